"""The fused sea-level pass at the edges of its work split: grids with and
without an equator row, even, twice-odd and odd longitude counts, one order and
several a CTA (more orders than CTAs; three CTAs for everything), rows too long
for the square twiddle table, a work area larger than shared memory, a fixed coastline, the subgrid load, one inner
iteration, a solve with no ocean; GPU = oracle with test_gpu_parity.py's
tolerances, the same iteration counts, and the same result whatever the CTAs."""
import numpy as np
import pytest

from fastearth3d_b200 import lib as vlib
from fastearth3d_b200 import synth
from oracle import orc
from parity_util import check_models

pytestmark = pytest.mark.gpu


def fields(nlat, nphi, ocean):
    lat = np.linspace(0.0, np.pi, nlat + 2)[1:-1, None]
    lon = 2 * np.pi * np.arange(nphi)[None] / nphi
    topo = -900.0 + 2300.0 * np.sin(lon + 0.4) * np.sin(lat) ** 2 + 700.0 * np.cos(2 * lat)
    topo = topo + 350.0 * np.cos(2 * lon - 1.0) * np.sin(lat)
    if not ocean:
        topo = np.abs(topo) + 50.0
    ice = 2100.0 * np.exp(-((lat - 0.7) ** 2 + 0.4 * (1 - np.cos(lon - 1.1))) / 0.08)
    return topo.reshape(-1), ice.reshape(-1)


def run(lmax, nlat, nphi, opts, ctas=0, gpu=True, ocean=True):
    mk, model = (vlib, vlib.Model) if gpu else (orc, orc.Oracle)
    p = mk.default_params()
    p.lmax, p.nlat, p.nphi = lmax, nlat, nphi
    for i, c in enumerate([1, 2, 2, 1]):
        p.ne_layer[i] = c
    for k, v in opts.items():
        setattr(p, k, v)
    if gpu:
        p.sle_ctas = ctas
    m = model(p)
    topo, ice = fields(nlat, nphi, ocean)
    m.set_reference(topo, 0.25 * ice)
    for f in (0.5, 1.0, 0.6):
        m.update(f * ice, 150.0)
    return m


@pytest.mark.parametrize("lmax,nlat,nphi,opts", [
    (2, 3, 6, {}),
    (5, 6, 12, {"sle_subgrid": 1}),
    (7, 9, 15, {}),
    (16, 17, 34, {"sle_fixed_ocean": 1}),
    (21, 24, 46, {"sle_n_inner": 1}),
    (33, 40, 76, {"sle_n_outer": 1}),
    (150, 151, 302, {}),
    (16, 17, 800, {}),
    (4, 7000, 10, {}),
])
def test_pass_matches_oracle(lmax, nlat, nphi, opts):
    g, o = run(lmax, nlat, nphi, opts), run(lmax, nlat, nphi, opts, gpu=False)
    check_models(g, o)
    assert g.info().n_inner_last == o.info().n_inner_last


def test_no_ocean_matches_oracle():
    g, o = run(12, 13, 26, {}, ocean=False), run(12, 13, 26, {}, gpu=False, ocean=False)
    check_models(g, o)


def test_result_does_not_depend_on_the_ctas():
    a, b = run(33, 40, 76, {}), run(33, 40, 76, {}, ctas=3)
    for x, y in zip(a.fields(), b.fields()):
        assert np.array_equal(x, y)


def misfit(lmax, nlat, nphi, opts, ctas=0):
    m = run(lmax, nlat, nphi, opts, ctas)
    topo, ice = fields(nlat, nphi, True)
    rng = np.random.default_rng(lmax)
    sites = rng.choice(np.flatnonzero(topo > 100.0), 12).astype(np.int32)
    ices = np.stack([0.8 * ice, 0.7 * ice])
    return m, ices, sites, rng.standard_normal((2, 12))


@pytest.mark.parametrize("lmax,nlat,nphi,opts", [
    (7, 9, 15, {}),
    (21, 24, 46, {"sle_n_inner": 1}),
    (33, 40, 76, {"sle_fixed_ocean": 1}),
    (4, 7000, 10, {}),
])
def test_pass_adjoint_matches_differences(lmax, nlat, nphi, opts):
    """As test_gpu_adjoint_sle.py: quadratic in the ice, central differences to 1e-6 of the gradient's scale."""
    m, ices, sites, obs = misfit(lmax, nlat, nphi, opts)
    g = m.sle_misfit_grad(ices, 150.0, sites, obs)[1].reshape(2, -1)
    rng = np.random.default_rng(5)
    for _ in range(3):
        d = rng.standard_normal(ices.shape) * ices
        h = 1e-6
        fd = (m.sle_misfit(ices + h * d, 150.0, sites, obs) - m.sle_misfit(ices - h * d, 150.0, sites, obs)) / (2 * h)
        an = float(np.sum(g * d))
        scale = max(abs(an), abs(fd), float(np.sqrt(np.sum((g * d) ** 2))))
        assert abs(an - fd) <= 1e-6 * scale, (an, fd, scale)


def test_pass_adjoint_does_not_depend_on_the_ctas():
    out = []
    for ctas in (0, 3):
        m, ices, sites, obs = misfit(33, 40, 76, {}, ctas)
        out.append(m.sle_misfit_grad(ices, 150.0, sites, obs))
    assert out[0][0] == out[1][0]
    assert np.array_equal(out[0][1], out[1][1])
