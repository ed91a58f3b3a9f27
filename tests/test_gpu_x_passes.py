"""The x passes' row lengths: rows that share a warp, that fill it, and that
are cut into pieces of 512 voxels with sites near and across the cuts; every
reach from the least to the largest.  The closing commutes with the exchange
of x and z, which takes the same grid through rows of 32 voxels."""
import numpy as np
import pytest

from broxy_gb300 import _lib as L
from broxy_gb300 import api, synth

pytestmark = pytest.mark.gpu


def _grid(rx, seed):
    rng = np.random.default_rng(seed)
    n = 2 * rx
    occ = rng.random((32, 32, n)) < 0.0004
    for cut in range(512, n, 512):  # at the cuts: a pair of voxels, and one just inside each side
        occ[8, 8, cut - 1:cut + 1] = True
        occ[20, 9, cut] = occ[12, 25, cut - 1] = True
    occ[5, 6, 0] = occ[27, 16, n - 1] = True
    occ[16:20, 16:20, n // 3:n // 2] = True  # a bar: long runs of sites
    return occ


def _pack(occ):
    c = np.zeros(tuple(s // 2 for s in occ.shape), np.uint8)
    for k in range(8):
        c |= occ[k >> 2 & 1::2, k >> 1 & 1::2, k & 1::2].astype(np.uint8) << k
    return c


def _unpack(c):
    occ = np.zeros(tuple(2 * s for s in c.shape), bool)
    for k in range(8):
        occ[k >> 2 & 1::2, k >> 1 & 1::2, k & 1::2] = c >> k & 1
    return occ


@pytest.mark.parametrize("mode,se", [(L.GM_REF, L.GM_SE_SPHERE), (L.GM_EXACT, L.GM_SE_SPHERE), (L.GM_REF, L.GM_SE_CUBE)])
@pytest.mark.parametrize("rx", [32, 48, 128, 240, 256, 272, 512, 528])
@pytest.mark.parametrize("radius", [2, 9, 64, 127, -9, -127])
def test_rows_equal_exchanged_box(gm_ctx, rx, radius, mode, se):
    import torch
    occ = _grid(rx, 1000 + rx)
    R = None
    if radius < 0:  # a field with runs of one radius and single ones
        rng = np.random.default_rng(rx)
        R = np.repeat(rng.integers(2, -radius + 1, (32, 32, rx // 8)), 16, axis=2).astype(np.int8)
        one = rng.random(R.shape) < 0.2
        R[one] = rng.integers(2, -radius + 1, int(one.sum()))

    def run(o, r):
        z, y, x = (s // 2 for s in o.shape)
        t = None if r is None else torch.as_tensor(np.ascontiguousarray(r)).cuda()
        c = gm_ctx.close_box(api.make_box((x, y, z)), torch.as_tensor(_pack(o)).cuda(), t, max(radius, 2), mode, se)
        torch.cuda.synchronize()
        return _unpack(c.cpu().numpy().reshape(z, y, x))

    long = run(occ, R)
    short = run(np.ascontiguousarray(occ.transpose(2, 1, 0)), None if R is None else R.transpose(2, 1, 0))
    assert long.sum() > 0
    assert np.array_equal(long, short.transpose(2, 1, 0))
