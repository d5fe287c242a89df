"""The drift's band sweeps at the edges of their tiling: node counts with every
remainder of the four-node chunks (the smallest mesh has two chunks), degrees
with one, sixteen and seventeen slots, and the same factor through the rotation
channels; GPU = oracle to 1e-10 of the field maximum (test_gpu_parity.py's
tolerance of the response)."""
import numpy as np
import pytest

from fastearth3d_b200 import lib as vlib
from fastearth3d_b200 import synth
from oracle import orc
from parity_util import TOL, rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,counts", [(2, [1, 2, 2, 1]), (15, [1, 2, 3, 1]), (16, [2, 3, 2, 1]), (17, [2, 3, 3, 1]),
                                         (33, [3, 8, 9, 9])])
def test_drift_matches_oracle_at_chunk_edges(lmax, counts):
    ms = []
    for mk, model in ((vlib, vlib.Model), (orc, orc.Oracle)):
        p = mk.default_params()
        p.lmax, p.nlat, p.nphi = lmax, lmax + 1, 2 * lmax + 2
        for i, c in enumerate(counts):
            p.ne_layer[i] = c
        m = model(p)
        m.set_dt(100.0 * synth.SEC_PER_YEAR)
        ms.append(m)
    rng = np.random.default_rng(lmax)
    nlm = (lmax + 1) * (lmax + 2) // 2
    for _ in range(3):
        s = 1e4 * (rng.standard_normal(nlm) + 1j * rng.standard_normal(nlm))
        s[: lmax + 1] = s[: lmax + 1].real
        out = []
        for m in ms:
            m.begin_step()
            out.append(m.apply(s))
            m.advance(s)
        for a, b in zip(*out):
            assert rel(a, b) < TOL


@pytest.mark.parametrize("n_elem", [9, 10, 11, 12])
def test_rotation_channels_match_oracle_at_chunk_edges(n_elem):
    w = synth.Workload("edge", 8, n_elem, 200.0, 6, 2, "sawtooth", sle=True, visc3d=False, seed=3, rotation=True)
    g, o = vlib.Model(w.params(vlib.default_params)), orc.Oracle(w.params(orc.default_params))
    for m in (g, o):
        m.set_reference(*w.reference())
        for step in (100, 200, 300):
            m.update(w.ice_at(step), w.dt_yr)
    assert rel(g.fields()[0], o.fields()[0]) < TOL
    mg, mo = g.rotation()[0], o.rotation()[0]
    assert abs(mg - mo) <= TOL * abs(mo)


@pytest.mark.parametrize("lmax,counts,cm", [(2, [1, 2, 2, 1], 1), (15, [1, 2, 3, 1], 0), (16, [2, 3, 2, 1], 1),
                                            (17, [2, 3, 3, 1], 1)])
def test_transposed_sweeps_match_differences(lmax, counts, cm):
    """The gradient through the transposed solves: the misfit is quadratic in the load, so central differences are
    exact up to rounding; 1e-6 of the gradient's scale along the direction, as in test_gpu_adjoint_sle.py."""
    p = vlib.default_params()
    p.lmax, p.nlat, p.nphi, p.deg1_cm = lmax, lmax + 1, 2 * lmax + 2, cm
    for i, c in enumerate(counts):
        p.ne_layer[i] = c
    m = vlib.Model(p)
    rng = np.random.default_rng(lmax)
    sites = rng.choice(m.ng, size=9, replace=False)
    dt = 100.0 * synth.SEC_PER_YEAR

    def draw():
        s = 1e3 * (rng.standard_normal((5, m.nlm)) + 1j * rng.standard_normal((5, m.nlm)))
        s[:, : lmax + 1] = s[:, : lmax + 1].real
        return s

    sigma, obs = draw(), 0.01 * rng.standard_normal((5, 9))
    _, g = m.misfit_grad(sigma, dt, sites, obs, ckpt_every=2)
    for _ in range(3):
        d = draw()
        h = 1e-3
        fd = (m.misfit(sigma + h * d, dt, sites, obs) - m.misfit(sigma - h * d, dt, sites, obs)) / (2 * h)
        t = g.real * d.real + g.imag * d.imag
        assert abs(fd - t.sum()) <= 1e-6 * max(abs(fd), np.sqrt((t**2).sum()))
