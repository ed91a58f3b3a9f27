"""A batch with a captured graph, a larger one with radius fields (which is
not captured and moves the workspaces), and the first one again: each result
equals separate calls."""
import numpy as np
import pytest

from broxy_gb300 import _lib as L
from broxy_gb300 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mesh", [False, True])
@pytest.mark.parametrize("lanes", [2, 0, L.GM_BATCH_GROUPED])
def test_batch_again_after_a_larger_one(gm_ctx, lanes, mesh):
    import torch
    rng = np.random.default_rng(77)

    def batch(sizes, field):
        items, want = [], []
        for i, (res, edge) in enumerate(sizes):
            X = torch.zeros((res,) * 3, dtype=torch.uint8)
            X[2:edge, 2:edge, 2:edge] = torch.as_tensor(
                np.where(rng.random((edge - 2,) * 3) < 0.05, rng.integers(0, 256, (edge - 2,) * 3), 0).astype(np.uint8))
            X = X.view(-1).cuda()
            R = torch.as_tensor(rng.integers(2, 12, (2 * res) ** 3).astype(np.int8)).cuda() if field else None
            d = api.make_desc(res)
            C = gm_ctx.close(d, X, R, 3 + i)
            m = [t.clone() for t in gm_ctx.mesh(d, C, 3)] if mesh else []
            items.append((d, X, R, 3 + i, torch.empty_like(X)))
            want.append([C, *m])
        torch.cuda.synchronize()
        return items, want

    first, second = batch([(32, 20), (64, 20)], False), batch([(64, 60), (128, 100), (64, 30)], True)
    ctx = api.Context(0)
    try:
        for items, want in (first, first, second, first, first):
            for it in items:
                it[4].fill_(0x5A)
            got = ctx.batch_close_mesh(items, bilateral_iters=3, lanes=lanes, mesh=mesh)
            torch.cuda.synchronize()
            for i, it in enumerate(items):
                for a, b in zip([it[4], *(got[i] if mesh else [])], want[i]):
                    assert np.array_equal(a.cpu().numpy(), b.cpu().numpy(), equal_nan=a.is_floating_point())
    finally:
        ctx.close_ctx()
