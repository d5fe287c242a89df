"""The FP64 3-D step on grids with many more columns than the transform needs:
column counts at the edges of the path's shapes and up to its limit, with and without the
toroidal channels; GPU = oracle to 1e-10 (response) and 1e-8 (memory) as in
test_gpu_parity.py. A grid past the limit is refused, and the handle is then as it was."""
import numpy as np
import pytest

from fastearth3d_b200 import lib as vlib
from fastearth3d_b200 import synth
from fastearth3d_b200.abi import VG_RHEOL_MAXWELL
from oracle import orc
from parity_util import TOL, TOL_STATE, rel

pytestmark = pytest.mark.gpu


def field(nlat, nphi):
    lat, lon = np.linspace(0.1, 3.0, nlat)[:, None], 2 * np.pi * np.arange(nphi)[None] / nphi
    rng = np.random.default_rng(nphi)
    return 0.3 * np.sin(2 * lon + 1.0) * np.sin(lat) + 0.05 * rng.standard_normal((nlat, nphi))


def pert(m):
    p, f = m.p, field(m.p.nlat, m.p.nphi)
    out = []
    for i in range(p.n_layer - 1, -1, -1):
        out += [f * (p.rheology[i] == VG_RHEOL_MAXWELL)] * p.ne_layer[i]
    return np.stack(out)


def pair(lmax, nlat, nphi, toroidal=0):
    ms = []
    for mk, cls in ((vlib, vlib.Model), (orc, orc.Oracle)):
        p = mk.default_params()
        p.lmax, p.nlat, p.nphi, p.toroidal = lmax, nlat, nphi, toroidal
        for i, c in enumerate([1, 2, 1, 1]):
            p.ne_layer[i] = c
        m = cls(p)
        m.set_dt(20.0 * synth.SEC_PER_YEAR)
        ms.append(m)
    return ms


def compare(g, o, toroidal=0, tol=TOL, tol_state=TOL_STATE):
    rng = np.random.default_rng(5)
    for _ in range(2):
        s = 1e4 * (rng.standard_normal(g.nlm) + 1j * rng.standard_normal(g.nlm))
        s[: g.p.lmax + 1] = s[: g.p.lmax + 1].real
        for m in (g, o):
            m.begin_step()
        for a, b in zip(g.apply(s), o.apply(s)):
            assert rel(a, b) < tol
        for m in (g, o):
            m.advance(s)
    for a, b in zip(g.state()[0], o.state()[0]):
        assert rel(a, b) < tol_state
    if toroidal:
        for a, b in zip(g.state_tor(), o.state_tor()):
            assert rel(a, b) < tol_state


# columns: a tile is eight base longitudes, nphi / 32 tiles; the shapes change at 24 tiles (770, 772)
@pytest.mark.parametrize("lmax,nlat,nphi,toroidal", [
    (20, 21, 578, 0), (20, 21, 580, 1), (20, 21, 770, 0), (20, 21, 770, 1), (20, 21, 772, 0), (20, 21, 772, 1),
    (20, 21, 774, 0), (20, 21, 1000, 1), (100, 101, 1024, 0), (20, 21, 1030, 0), (20, 21, 1298, 0), (2, 3, 1334, 0),
])
def test_wide_grids_match_oracle(lmax, nlat, nphi, toroidal):
    g, o = pair(lmax, nlat, nphi, toroidal)
    for m in (g, o):
        m.enable_visc3d(pert(m))
    compare(g, o, toroidal)


def test_gradient_on_a_wide_grid():
    """The transposed pass reads the grid that the forward one stores: central differences to 1e-6 of the gradient's
    scale, as in test_gpu_adjoint.py (the misfit is quadratic in the load)."""
    g, _ = pair(12, 13, 780)
    g.enable_visc3d(pert(g))
    rng = np.random.default_rng(3)
    sites = rng.choice(g.ng, size=9, replace=False)
    dt = 20.0 * synth.SEC_PER_YEAR

    def draw():
        s = 1e3 * (rng.standard_normal((3, g.nlm)) + 1j * rng.standard_normal((3, g.nlm)))
        s[:, :13] = s[:, :13].real
        return s

    sigma, obs = draw(), 0.01 * rng.standard_normal((3, 9))
    _, gr = g.misfit_grad(sigma, dt, sites, obs)
    for _ in range(2):
        d = draw()
        h = 1e-3
        fd = (g.misfit(sigma + h * d, dt, sites, obs) - g.misfit(sigma - h * d, dt, sites, obs)) / (2 * h)
        t = gr.real * d.real + gr.imag * d.imag
        assert abs(fd - t.sum()) <= 1e-6 * max(abs(fd), np.sqrt((t**2).sum()))

def test_refused_grid_leaves_the_handle_as_it_was():
    g, o = pair(8, 9, 1400)
    for _ in range(2):  # the second time for the same reason
        with pytest.raises(vlib.VilmaError, match="grid too large"):
            g.enable_visc3d(pert(g))
    assert g.info().ne3d == 0
    compare(g, o)  # the laterally uniform earth, as without the call
