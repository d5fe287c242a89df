"""The FP64 3-D stress products and the longitude pass at the edges of their tiles: row tiles of 40
northern latitudes (one, exactly full, one over), degree and latitude chunks
with remainders, grids with an equator row and without and with more rows and
columns than the transform needs, column counts below, at and past a
64-column tile, with and without the toroidal channels; GPU = oracle to
1e-10 (response) and 1e-8 (memory) as in test_gpu_parity.py."""
import numpy as np
import pytest

from fastearth3d_b200 import lib as vlib
from fastearth3d_b200 import synth
from fastearth3d_b200.abi import VG_RHEOL_MAXWELL
from oracle import orc
from parity_util import TOL, TOL_STATE, rel

pytestmark = pytest.mark.gpu


def models(lmax, nlat, nphi, counts, toroidal):
    out = []
    rng = np.random.default_rng(lmax + nphi)
    f = 0.3 * np.sin(2 * np.pi * np.arange(nphi) / nphi * 2 + 1)[None] * np.sin(np.linspace(0.1, 3.0, nlat))[:, None]
    f = f + 0.05 * rng.standard_normal((nlat, nphi))
    for mk, model in ((vlib, vlib.Model), (orc, orc.Oracle)):
        p = mk.default_params()
        p.lmax, p.nlat, p.nphi, p.toroidal = lmax, nlat, nphi, toroidal
        for i, c in enumerate(counts):
            p.ne_layer[i] = c
        pert = []
        for i in range(p.n_layer - 1, -1, -1):
            pert += [f * (p.rheology[i] == VG_RHEOL_MAXWELL)] * p.ne_layer[i]
        m = model(p)
        m.enable_visc3d(np.stack(pert))
        m.set_dt(20.0 * synth.SEC_PER_YEAR)
        out.append(m)
    return out


@pytest.mark.parametrize("lmax,nlat,nphi,counts,toroidal", [
    (2, 3, 6, [1, 1, 1, 1], 0),
    (7, 9, 16, [1, 5, 5, 1], 1),       # ncf 60
    (16, 17, 34, [1, 6, 5, 1], 0),     # ncf 66
    (31, 33, 66, [1, 1, 1, 2], 1),
    (39, 40, 82, [1, 2, 1, 1], 0),     # 20 northern rows, no equator
    (79, 80, 160, [1, 1, 1, 1], 0),    # 40 northern rows: a full row tile
    (80, 81, 162, [1, 1, 1, 1], 0),    # 41
    (81, 85, 170, [1, 1, 1, 1], 1),    # 43, more rows than the transform needs
    # longitude tiles: odd half period with most and with few of its orders, tables in shared memory and from L2
    (24, 25, 50, [1, 2, 1, 1], 0),
    (20, 21, 66, [1, 1, 1, 1], 1),
    (32, 33, 66, [1, 1, 1, 1], 1),
    (47, 48, 100, [1, 1, 1, 1], 0),
    (66, 67, 134, [1, 1, 1, 1], 0),
    (30, 31, 262, [1, 1, 1, 1], 1),
    (20, 21, 390, [1, 1, 1, 1], 0),
    (16, 17, 520, [1, 1, 1, 1], 0),
])
def test_products_match_oracle_at_tile_edges(lmax, nlat, nphi, counts, toroidal):
    g, o = models(lmax, nlat, nphi, counts, toroidal)
    assert g.info().ne3d == o.info().ne3d > 0
    rng = np.random.default_rng(5)
    nlm = (lmax + 1) * (lmax + 2) // 2
    for _ in range(2):
        s = 1e4 * (rng.standard_normal(nlm) + 1j * rng.standard_normal(nlm))
        s[: lmax + 1] = s[: lmax + 1].real
        g.begin_step()
        o.begin_step()
        for a, b in zip(g.apply(s), o.apply(s)):
            assert rel(a, b) < TOL
        g.advance(s)
        o.advance(s)
    for a, b in zip(g.state()[0], o.state()[0]):
        assert rel(a, b) < TOL_STATE
    if toroidal:
        for a, b in zip(g.state_tor(), o.state_tor()):
            assert rel(a, b) < TOL_STATE
