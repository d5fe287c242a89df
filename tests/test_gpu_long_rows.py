"""Rows of thousands of longitudes, at the edges of what the row transforms hold
in shared memory: the analysis with odd and even counts up to its limits (6144,
even counts as long as their tables fit), the closing load of a solve without an
ocean, and the refusal past the limits; GPU = oracle to 1e-12 (transforms) and with test_gpu_parity.py's
tolerances (solve)."""
import numpy as np
import pytest

from fastearth3d_b200 import lib as vlib
from oracle import orc
from parity_util import check_models, rel

pytestmark = pytest.mark.gpu


def model(mk, cls, lmax, nlat, nphi):
    p = mk.default_params()
    p.lmax, p.nlat, p.nphi = lmax, nlat, nphi
    for i, c in enumerate([1, 2, 2, 1]):
        p.ne_layer[i] = c
    return cls(p)


def pair(*size):
    return model(vlib, vlib.Model, *size), model(orc, orc.Oracle, *size)


@pytest.mark.parametrize("nphi", [5141, 5143, 5145, 6143, 6144, 6146, 6354])
def test_analysis_of_long_rows(nphi):
    g, o = pair(5, 6, nphi)
    f = np.random.default_rng(nphi).standard_normal(6 * nphi)
    assert rel(g.analysis(f), o.analysis(f)) < 1e-12


@pytest.mark.parametrize("nphi", [5143, 6143, 6346])
def test_solve_without_an_ocean_on_long_rows(nphi):
    ms = pair(4, 5, nphi)
    lat = np.linspace(0.2, 2.9, 5)[:, None]
    lon = 2 * np.pi * np.arange(nphi)[None] / nphi
    ice = (1500.0 * np.exp(-((lat - 0.8) ** 2 + 0.4 * (1 - np.cos(lon - 1.1))) / 0.3)).reshape(-1)
    for m in ms:
        m.set_reference(np.full(5 * nphi, 900.0), 0.25 * ice)
        for f in (0.5, 1.0):
            m.update(f * ice, 150.0)
    check_models(*ms)


@pytest.mark.parametrize("nphi", [6145, 6356, 9000])
def test_analysis_past_the_limit_is_refused(nphi):
    g = model(vlib, vlib.Model, 3, 4, nphi)
    with pytest.raises(vlib.VilmaError):
        g.analysis(np.zeros(4 * nphi))
