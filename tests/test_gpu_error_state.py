"""A refused call leaves nothing behind: the next valid call, of the same or of
another handle, neither reports the earlier error nor computes anything else."""
import numpy as np
import pytest

from fastearth3d_b200 import lib as vlib
from oracle import orc
from parity_util import rel

pytestmark = pytest.mark.gpu


def test_valid_call_after_a_refused_one():
    ms = []
    for mk, cls in ((vlib, vlib.Model), (orc, orc.Oracle)):
        p = mk.default_params()
        p.lmax, p.nlat, p.nphi = 3, 4, 9000  # the analysis takes rows of up to 6144 longitudes, the synthesis any
        for i, c in enumerate([1, 2, 2, 1]):
            p.ne_layer[i] = c
        ms.append(cls(p))
    g, o = ms
    q = np.arange(1.0, g.nlm + 1) + 0j
    with pytest.raises(vlib.VilmaError):
        g.analysis(np.zeros(g.ng))
    assert rel(g.synthesis(q), o.synthesis(q)) < 1e-12
    p = vlib.default_params()
    p.lmax, p.nlat, p.nphi = 4000, 4001, 8002  # Legendre tables of 256 GB: more than the GPU has
    with pytest.raises(vlib.VilmaError, match="out of memory"):
        vlib.Model(p)
    assert rel(g.synthesis(q), o.synthesis(q)) < 1e-12
