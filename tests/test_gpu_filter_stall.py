"""The bounded wait of the small meshes' normal filter running out (injected:
its barrier waits for an arrival that never comes): NaN normals, the error
bit, an error from the calls that wait for the mesh, and a usable context."""
import numpy as np
import pytest

from broxy_gb300 import _lib as L
from broxy_gb300 import api, synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("res,iters", [(32, 2), (64, 20)])  # one block and many; the shortest filter that waits
def test_filter_barrier_runs_out(res, iters):
    import torch
    ctx = api.Context(0)
    try:
        desc = api.make_desc(res)
        C = torch.zeros((res,) * 3, dtype=torch.uint8, device="cuda")
        C[4:res - 4, 4:res // 2, 4:10] = 0xFF
        C = C.view(-1)
        want = [t.cpu().numpy() for t in ctx.mesh(desc, C, iters)]
        assert api.kernel_error_flags(clear=True) == 0 and np.isfinite(want[1]).all()
        assert ctx.lib.gm_mesh_inject_filter_stalls(ctx.ctx, 1) == L.GM_OK
        V, N, T = (t.cpu().numpy() for t in ctx.mesh(desc, C, iters))
        assert np.array_equal(V, want[0]) and np.array_equal(T, want[2]) and np.isnan(N).all()
        with pytest.raises(L.GMError) as e:
            ctx.mesh_download(len(V), len(T))
        assert e.value.status == L.GM_ERR_CUDA
        assert api.kernel_error_flags(clear=True) == 1
        got = [t.cpu().numpy() for t in ctx.mesh(desc, C, iters)]
        assert all(np.array_equal(a, b) for a, b in zip(got, want))
        assert all(np.array_equal(a, b) for a, b in zip(ctx.mesh_download(len(V), len(T)), want))
        assert api.kernel_error_flags() == 0
    finally:
        ctx.close_ctx()
        api.kernel_error_flags(clear=True)


def test_update_reports_it():
    ctx = api.Context(0)
    try:
        res, n = 32, 20000
        desc = api.make_desc(res)
        X = synth.random_grid(res, 5)
        hV, hN, hT = (np.zeros((k, 3), t) for k, t in ((n, np.float32), (n, np.float32), (2 * n, np.uint32)))
        args = (desc, X, None, 3 * desc.cell_size, hV, hN, hT)
        nv, _ = ctx.update_to_host(*args)
        want = hN.copy()
        assert nv > 0
        ctx.lib.gm_mesh_inject_filter_stalls(ctx.ctx, 1)
        with pytest.raises(L.GMError) as e:
            ctx.update_to_host(*args)
        assert e.value.status == L.GM_ERR_CUDA and np.isnan(hN[:nv]).all()
        assert ctx.update_to_host(*args)[0] == nv
        assert np.array_equal(hN, want, equal_nan=True)
    finally:
        ctx.close_ctx()
        api.kernel_error_flags(clear=True)
