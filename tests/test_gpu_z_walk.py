"""Contour, selection and tags on boxes whose rows take one, a few or all of a
warp's lanes and whose y and z extents end inside a block's rows and walk:
content away from the box's far sides closes as in a grid around it."""
import numpy as np
import pytest

from broxy_gb300 import _lib as L
from broxy_gb300 import api, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu

RES, RADIUS, MARGIN = 128, 3, 12  # voxels: dilation and erosion reach no further than 2 (RADIUS + 1) + 2


@pytest.mark.parametrize("dims", [(16, 112, 48), (32, 48, 80), (48, 80, 112), (80, 128, 16), (112, 16, 32)])
@pytest.mark.parametrize("mode", [L.GM_REF, L.GM_EXACT])
def test_box_equals_oracle(gm_ctx, dims, mode):
    import torch
    x, y, z = dims
    occ = np.zeros((2 * RES,) * 3, bool)
    inner = occ[MARGIN:2 * z - MARGIN, MARGIN:2 * y - MARGIN, MARGIN:2 * x - MARGIN]
    rng = np.random.default_rng(x)
    inner[:] = rng.random(inner.shape) < 0.004
    inner[inner.shape[0] // 2 - 1:inner.shape[0] // 2 + 1, :, inner.shape[2] // 3:] = True  # a slab
    X = synth.pack_dense(occ)
    box = np.ascontiguousarray(X.reshape(RES, RES, RES)[:z, :y, :x])
    C = gm_ctx.close_box(api.make_box(dims), torch.as_tensor(box).cuda(), None, RADIUS, mode, L.GM_SE_SPHERE)
    torch.cuda.synchronize()
    _, _, Co = O.close(X, RES, [RES] * 3, O.scale_grid(RES, uniform=RADIUS), mode)
    assert np.array_equal(C.cpu().numpy().reshape(z, y, x), Co.reshape(RES, RES, RES)[:z, :y, :x])
