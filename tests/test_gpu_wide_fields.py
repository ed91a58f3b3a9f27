"""Closings of boxes longer than 1024 cells along x with a radius field: the
map of the tiles' radius bounds takes their rows in several parts.  The
closing commutes with the exchange of x and z, which takes the same grid
through rows of 32 voxels."""
import numpy as np
import pytest

from broxy_gb300 import _lib as L
from broxy_gb300 import api

pytestmark = pytest.mark.gpu


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
@pytest.mark.parametrize("rx,rmax", [(1024, 9), (1040, 9), (1040, 127), (1536, 30), (2048, 9), (2048, 127)])
def test_field_on_long_rows(gm_ctx, rx, rmax, mode, se):
    import torch
    rng = np.random.default_rng(rx + rmax)
    occ = rng.random((32, 32, 2 * rx)) < 0.0006
    occ[14:18, 12:20, 2000:2100] = True  # across the first part's end
    R = np.repeat(rng.integers(2, 8, (32, 32, rx // 8)), 16, axis=2).astype(np.int8)
    R[15, 16, 40] = rmax                  # the largest radii near the row's ends and inside the last part
    R[9, 20, 2 * rx - 30] = R[20, 9, 2 * rx - 3] = rmax

    def run(o, r):
        z, y, x = (s // 2 for s in o.shape)
        X = torch.as_tensor(_pack(o)).cuda()
        out = torch.full_like(X, 0xA5)  # (random sites: no closing of them is all 0xa5)
        gm_ctx.close_box(api.make_box((x, y, z)), X, torch.as_tensor(np.ascontiguousarray(r)).cuda(), 0, mode, se, out=out)
        torch.cuda.synchronize()
        return _unpack(out.cpu().numpy().reshape(z, y, x))

    long = run(occ, R)
    short = run(np.ascontiguousarray(occ.transpose(2, 1, 0)), R.transpose(2, 1, 0))
    assert short.sum() > occ.sum()
    assert np.array_equal(long, short.transpose(2, 1, 0))
