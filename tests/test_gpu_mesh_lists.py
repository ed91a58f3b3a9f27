"""The mesh's vertex lists and triangle list where their pieces meet: vertex
counts around a chunk of 256 records, cells around a warp of four and a round
of 256, cells on brick and grid borders, fans of more than eight triangles and
surfaces that are no closed fan."""
import numpy as np
import pytest

from broxy_gb300 import api, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(ctx, occ, iters, filtered=True):
    import torch
    res = occ.shape[0] // 2
    C = synth.pack_dense(occ)
    desc = api.make_desc(res)
    V, N, T = ctx.mesh(desc, torch.as_tensor(C).cuda(), iters)
    torch.cuda.synchronize()
    Vo, To = O.mc(C, res, np.array(desc.bbox_min), desc.cell_size)
    assert V.shape == Vo.shape and np.array_equal(T.cpu().numpy(), To)
    np.testing.assert_allclose(V.cpu().numpy(), Vo, rtol=1e-6, atol=0)
    if filtered:
        np.testing.assert_allclose(N.cpu().numpy(), O.normals(Vo, To, iters), atol=2e-3, rtol=0, equal_nan=True)
    return len(Vo), To


@pytest.mark.parametrize("voxels", [1, 2, 42, 43, 85, 86, 128])
def test_isolated_voxels(gm_ctx, voxels):
    """Six vertices each: 252, 258, 510, 516, 768 around the chunks.  (A lone
    voxel's octahedron has no filtered normal: a vertex' four neighbours
    cancel exactly, and rounding decides between 0 / 0 and a direction.)"""
    occ = np.zeros((64, 64, 64), bool)
    at = np.stack(np.meshgrid(*[np.arange(4, 60, 4)] * 3, indexing="ij"), -1).reshape(-1, 3)[:voxels]
    occ[tuple(at.T)] = True
    assert _check(gm_ctx, occ, 0)[0] == 6 * voxels
    _check(gm_ctx, occ, 3, filtered=False)


@pytest.mark.parametrize("blocks", [10, 11, 21, 22, 32])
def test_small_blocks(gm_ctx, blocks):
    """Solid 2x2x2 blocks, 24 vertices each (240, 264, 504, 528, 768), filtered."""
    occ = np.zeros((64, 64, 64), bool)
    at = np.stack(np.meshgrid(*[np.arange(4, 58, 7)] * 3, indexing="ij"), -1).reshape(-1, 3)[:blocks]
    for z, y, x in at:
        occ[z:z + 2, y:y + 2, x:x + 2] = True
    assert _check(gm_ctx, occ, 3)[0] == 24 * blocks


@pytest.mark.parametrize("seed,density", [(1, 0.03), (2, 0.3), (3, 0.5)])
def test_noise(gm_ctx, seed, density):
    """Random voxels: every cube value, long lists, open fans, case 91 (the
    filtered normals of their lone voxels are undefined, as above)."""
    occ = np.random.default_rng(seed).random((64, 64, 64)) < density
    occ[:4] = occ[-4:] = occ[:, :4] = occ[:, -4:] = occ[:, :, :4] = occ[:, :, -4:] = False
    _check(gm_ctx, occ, 0)
    _check(gm_ctx, occ, 2, filtered=False)


@pytest.mark.parametrize("cut", [0, 1, 2, 3])
def test_border(gm_ctx, cut):
    """A ball cut by the grid's border: vertex 0 takes the missing edges'
    corners."""
    z, y, x = np.meshgrid(*[np.arange(32)] * 3, indexing="ij")
    occ = (x - (2.5 - 2 * cut)) ** 2 + (y - 16) ** 2 + (z - 16) ** 2 < 36
    _check(gm_ctx, occ, 4)


@pytest.mark.parametrize("blocks", [6475, 6490])
@pytest.mark.parametrize("iters", [1, 3])
def test_filter_around_one_vertex_a_thread(gm_ctx, blocks, iters):
    """Solid 2x2x2 blocks, 24 vertices each: 155400 and 155760 vertices, about
    as many as the chip holds threads of the resident filter (155648)."""
    occ = np.zeros((128, 128, 128), bool)
    at = np.stack(np.meshgrid(*[np.arange(4, 124, 5)] * 3, indexing="ij"), -1).reshape(-1, 3)[:blocks]
    for z, y, x in at:
        occ[z:z + 2, y:y + 2, x:x + 2] = True
    assert _check(gm_ctx, occ, iters)[0] == 24 * blocks
    assert api.kernel_error_flags() == 0
