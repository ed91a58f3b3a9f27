"""The voxelizer's forms against the oracle, bit for bit: triangles of less
than a voxel up to the whole grid, on voxel planes and corners (where single
precision decides nothing), skinny and degenerate ones, meshes that reach
beyond the grid or are far from it, and the smallest and the widest z-word
columns."""
import numpy as np
import pytest

from broxy_gb300 import api, synth
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _check(ctx, P, T, res, bbox_min, cell):
    import torch
    desc = api.make_desc(res, bbox_min=bbox_min, cell_size=cell)
    P = np.ascontiguousarray(P, np.float32)
    T = np.ascontiguousarray(T, np.uint32)
    g = ctx.voxelize(desc, torch.as_tensor(P).cuda(), torch.as_tensor(T.astype(np.int32)).cuda())
    torch.cuda.synchronize()
    ref = O.voxelize(P, T, res, np.array(desc.bbox_min), desc.cell_size)
    assert np.array_equal(g.cpu().numpy(), ref)
    return ref


def _soup(rng, n, size, lo=0.0, hi=1.0):
    """n triangles of about `size`, their centres in [lo, hi]^3."""
    c = rng.uniform(lo, hi, (n, 1, 3))
    P = (c + size * rng.normal(size=(n, 3, 3))).reshape(-1, 3)
    return P, np.arange(3 * n).reshape(-1, 3)


@pytest.mark.parametrize("res,level", [(16, 0), (16, 3), (32, 1), (64, 2), (64, 5), (256, 4)])
def test_closed_spheres(gm_ctx, res, level):
    V, F = synth.icosphere(level)
    P = np.concatenate([0.31 * V + 0.47, 0.11 * V + np.array([0.8, 0.75, 0.3])])
    ref = _check(gm_ctx, P, np.concatenate([F, F + len(V)]), res, (-0.013, 0.007, 0.0), 1.02 / res)
    assert ref.any()


@pytest.mark.parametrize("size", [1e-7, 1e-4, 3e-3, 0.02, 0.2, 1.5])
def test_triangle_sizes(gm_ctx, size):
    rng = np.random.default_rng(int(1 / size))
    P, T = _soup(rng, 400 if size < 0.1 else 60, size)
    _check(gm_ctx, P, T, 32, (0.1, 0.0, -0.05), 1.0 / 32)


def test_on_voxel_planes(gm_ctx):
    """Boxes, slopes and points on voxel faces, edges, corners and centres."""
    rng = np.random.default_rng(5)
    res = 32
    h = 0.5 / res
    P, T = [], []
    for k in range(300):
        step = (1.0, 0.5, 0.25)[k % 3]
        t = rng.integers(2, 60, (1, 3)) + step * rng.integers(-8, 9, (3, 3))
        if k % 4 == 0:
            t[:, rng.integers(3)] = t[0, rng.integers(3)]
        T.append(np.arange(3) + 3 * k)
        P.append(t)
    P = np.concatenate(P) * h
    _check(gm_ctx, P, np.stack(T), res, (0.0, 0.0, 0.0), 2 * h)


def test_skinny_and_degenerate(gm_ctx):
    rng = np.random.default_rng(6)
    tris = []
    for k in range(200):
        a, d = rng.uniform(0.2, 0.8, 3), rng.normal(size=3)
        d /= np.linalg.norm(d)
        u = np.cross(d, rng.normal(size=3))
        u /= np.linalg.norm(u)
        length = rng.uniform(0.05, 0.6)
        # an aspect ratio around the limit of 50, far past it, or none
        height = length / (49.9, 50.1, 50.0, 30.0, 500.0, 1e9)[k % 6]
        tris.append(np.stack([a, a + length * d, a + 0.4 * length * d + height * u]))
    tris += [np.full((3, 3), 0.4), np.array([[0.3] * 3, [0.3] * 3, [0.6] * 3])]
    P = np.concatenate(tris)
    _check(gm_ctx, P, np.arange(len(P)).reshape(-1, 3), 32, (0.0, 0.0, 0.0), 1.0 / 32)


@pytest.mark.parametrize("lo,hi,size", [(-0.5, 1.5, 0.3), (-40.0, 40.0, 30.0), (-300.0, 300.0, 200.0)])
def test_beyond_the_grid(gm_ctx, lo, hi, size):
    rng = np.random.default_rng(7)
    P, T = _soup(rng, 40, size, lo, hi)
    _check(gm_ctx, P, T, 16, (0.0, 0.0, 0.0), 1.0 / 16)


def test_widest_columns(gm_ctx):
    """64 z-words a column: the packing's parity goes over two warps' words."""
    import torch
    res = 1024
    V, F = synth.icosphere(2)
    desc = api.make_desc(res)
    P, T = (0.45 * V + 0.5).astype(np.float32), F.astype(np.uint32)
    g = gm_ctx.voxelize(desc, torch.as_tensor(P).cuda(), torch.as_tensor(T.astype(np.int32)).cuda())
    g = g.view(res, res, res)[:, res // 2, res // 2 - 8:res // 2 + 8].cpu().numpy()
    full = np.flatnonzero((g == 0xff).all(1))
    assert len(full) > 0.85 * res and np.array_equal(full, np.arange(full[0], full[-1] + 1))
    assert not g[:full[0] - 3].any() and not g[full[-1] + 4:].any()


@pytest.mark.parametrize("res", [16, 32, 64, 128])
@pytest.mark.parametrize("offset", [0, 1])
def test_zwords_to_packed(gm_ctx, res, offset):
    import torch
    rng = np.random.default_rng(res)
    occ = rng.random((2 * res,) * 3) < 0.3  # [z, y, x]
    bits = occ.transpose(1, 2, 0).reshape(2 * res, 2 * res, res // 16, 32).astype(np.uint64)
    zw = np.ascontiguousarray((bits << np.arange(32, dtype=np.uint64)).sum(-1).astype(np.uint32)).view(np.int32)
    buf = torch.zeros(res ** 3 + 16, dtype=torch.uint8, device="cuda")
    out = buf[offset:offset + res ** 3]
    gm_ctx.zwords_to_packed(res, torch.as_tensor(zw).cuda(), out)
    assert np.array_equal(out.cpu().numpy(), synth.pack_dense(occ))
    assert not buf[offset + res ** 3:].any() and not buf[:offset].any()
