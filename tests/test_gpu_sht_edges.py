"""The scalar transforms at the edges of their tiles: degree chunks of 32 (one,
full, one over), latitude chunks of 32 and 256 northern rows, grids with and
without an equator row, even, twice-odd and odd longitude counts, more points
than the transform needs, and rows past what shared memory holds; GPU = oracle
to 1e-12 as in test_gpu_parity.py."""
import numpy as np
import pytest

from fastearth3d_b200 import lib as vlib
from oracle import orc
from parity_util import rel

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lmax,nlat,nphi", [
    (2, 3, 5), (5, 6, 12), (30, 31, 62), (31, 32, 66), (32, 63, 65), (33, 64, 70), (63, 65, 128),
    (40, 511, 84), (40, 513, 90), (4, 6, 3000), (3, 4, 9000),
])
def test_transforms_match_oracle(lmax, nlat, nphi):
    ms = []
    for mk, model in ((vlib, vlib.Model), (orc, orc.Oracle)):
        p = mk.default_params()
        p.lmax, p.nlat, p.nphi = lmax, nlat, nphi
        for i, c in enumerate([1, 2, 2, 1]):
            p.ne_layer[i] = c
        ms.append(model(p))
    g, o = ms
    rng = np.random.default_rng(lmax + nphi)
    q = rng.standard_normal((lmax + 1) * (lmax + 2) // 2) + 1j * rng.standard_normal((lmax + 1) * (lmax + 2) // 2)
    q[: lmax + 1] = q[: lmax + 1].real
    assert rel(g.synthesis(q), o.synthesis(q)) < 1e-12
    if nphi <= 6144:
        f = rng.standard_normal(nlat * nphi)
        assert rel(g.analysis(f), o.analysis(f)) < 1e-12


def test_noalloc_analysis_into_any_double():
    """The caller's device vectors may start at any double: shifted by one, the same spectrum to the bit."""
    import ctypes as C

    import torch

    p = vlib.default_params()
    p.lmax, p.nlat, p.nphi = 33, 34, 68
    m = vlib.Model(p)
    f = torch.from_numpy(np.random.default_rng(2).standard_normal(m.ng + 1)).cuda()
    out = []
    for shift in (0, 1):
        q = torch.zeros(2 * m.nlm + 1, dtype=torch.float64, device="cuda")
        g = torch.zeros(m.ng + 1, dtype=torch.float64, device="cuda")
        g[shift:shift + m.ng] = f[:m.ng]
        torch.cuda.synchronize()
        rc = vlib.lib().vg_sht_analysis_noalloc(m.h, C.c_void_p(g[shift:].data_ptr()), C.c_void_p(q[shift:].data_ptr()), 1)
        assert rc == 0
        torch.cuda.synchronize()
        out.append(q[shift:shift + 2 * m.nlm].cpu().numpy())
    assert np.array_equal(*out)
