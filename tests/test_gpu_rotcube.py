"""GPU parity of the frame-field closing (GMorpho::Update with use_frame_field:
DilateByRotCubeMipmap then ErodeBySphereMipmap, GMorpho/GMorpho.cu:3058-3230,
7785-7803) and of the frame field solver (FrameField::Generate with
BiHarmonicSystem, GMorpho/FrameFieldSparseBiharmonic.cu:449-647) against the
CPU oracle.

Grids: bit-exact (D, S, C), GM_REF and GM_EXACT, uniform and variable
radius, random quaternion fields of several lattice sizes, data_res below
res.  Frame field: the solver's quaternions within 1e-5 of the largest
component of the oracle's exact double-precision solution of the same
system (the GPU stops at a relative residual of 1e-10).
"""
import numpy as np
import pytest

from broxy_gb300 import _lib as L
from broxy_gb300 import api
from oracle import framefield as F
from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a)).cuda()


def _grid(res, seed, density=0.01, blocks=4):
    rng = np.random.default_rng(seed)
    X = np.where(rng.random((res, res, res)) < density, rng.integers(1, 256, (res, res, res)), 0).astype(np.uint8)
    for _ in range(blocks):
        lo = rng.integers(2, res - res // 4, 3)
        ext = rng.integers(2, res // 5, 3)
        X[lo[2]:lo[2] + ext[2], lo[1]:lo[1] + ext[1], lo[0]:lo[0] + ext[0]] = 0xFF
    X[:1] = 0
    X[-1:] = 0
    return X.reshape(-1)


def _field(qres, seed):
    rng = np.random.default_rng(seed)
    return rng.normal(size=(qres ** 3, 4)).astype(np.float32)


def _scale(res, seed, lo=2, hi=7):
    rng = np.random.default_rng(seed)
    return rng.integers(lo, hi, (2 * res) ** 3).astype(np.int8)


def _run(ctx, res, X, Q, qres, scale=None, uniform=3, mode=L.GM_REF, data_res=None):
    import torch
    desc = api.make_desc(res, data_res)
    Xd = _dev(X)
    Qd = _dev(Q)
    Rd = _dev(scale) if scale is not None else None
    D = torch.empty_like(Xd)
    S = torch.empty_like(Xd)
    Cg = ctx.close_rotcube(desc, Xd, Qd, qres, Rd, uniform, mode, D=D, S=S)
    torch.cuda.synchronize()
    return D.cpu().numpy(), S.cpu().numpy(), Cg.cpu().numpy()


def _oracle(res, X, Q, qres, scale, uniform, mode, data_res=None):
    sc = scale if scale is not None else O.scale_grid(res, uniform=uniform)
    return O.close_rotcube(X, res, data_res or [res] * 3, sc, Q, qres, mode)


@pytest.mark.parametrize("res,qres,uniform", [(32, 2, 3), (32, 4, 5), (64, 4, 4), (64, 3, 7)])
def test_rotcube_ref_uniform(gm_ctx, res, qres, uniform):
    X = _grid(res, 8000 + res + qres)
    Q = _field(qres, 8100 + qres)
    got = _run(gm_ctx, res, X, Q, qres, uniform=uniform)
    want = _oracle(res, X, Q, qres, None, uniform, 0)
    for g, w, name in zip(got, want, "DSC"):
        assert np.array_equal(g, w), name
    assert want[2].any()


@pytest.mark.parametrize("res,qres", [(32, 2), (64, 4)])
def test_rotcube_ref_variable_radius(gm_ctx, res, qres):
    X = _grid(res, 8200 + res)
    Q = _field(qres, 8300 + qres)
    sc = _scale(res, 8400 + res)
    got = _run(gm_ctx, res, X, Q, qres, scale=sc)
    want = _oracle(res, X, Q, qres, sc, 0, 0)
    for g, w, name in zip(got, want, "DSC"):
        assert np.array_equal(g, w), name


@pytest.mark.parametrize("uniform", [12, 24, None])
def test_rotcube_large_radius(gm_ctx, uniform):
    """Sparse voxels and one block with radii up to 24: the dilation covers
    most of the grid, so most queries are decided by the distance shortcuts
    and the rest by the warp search; D, S, C still equal the oracle's."""
    res, qres = 64, 4
    X = _grid(res, 9400 + (uniform or 0), density=0.0005, blocks=1)
    Q = _field(qres, 9500)
    sc = None if uniform else _scale(res, 9600, 2, 25)
    got = _run(gm_ctx, res, X, Q, qres, scale=sc, uniform=uniform or 0)
    want = _oracle(res, X, Q, qres, sc, uniform or 0, 0)
    for g, w, name in zip(got, want, "DSC"):
        assert np.array_equal(g, w), name
    assert 0.1 < (want[0] == 0xFF).mean() < 0.99


@pytest.mark.parametrize("angle", [0.0, 1e-4, 0.02, 0.049, 0.06, np.pi / 4])
@pytest.mark.parametrize("uniform", [2, 9, 30])
def test_rotcube_frames_near_the_axes(gm_ctx, angle, uniform):
    """Frames along the axes, turned by little and by 45 degrees, the smallest
    radius and radii whose cube meets the grid's border: the distance field's
    verdicts and the voxels it leaves to the predicate give the oracle's
    grids."""
    res, qres = 32, 3
    rng = np.random.default_rng(int(1000 * angle) + uniform)
    axis = rng.normal(size=(qres ** 3, 3)) if angle < 0.5 else np.tile([0.0, 0.0, 1.0], (qres ** 3, 1))
    axis /= np.linalg.norm(axis, axis=1, keepdims=True)
    Q = np.concatenate([np.sin(angle / 2) * axis, np.full((qres ** 3, 1), np.cos(angle / 2))], 1).astype(np.float32)
    X = _grid(res, 9900 + uniform, density=0.002 if uniform < 9 else 0.0002, blocks=1)
    for mode in (0, 1):
        got = _run(gm_ctx, res, X, Q, qres, uniform=uniform, mode=mode)
        want = _oracle(res, X, Q, qres, None, uniform, mode)
        for g, w, name in zip(got, want, "DSC"):
            assert np.array_equal(g, w), (name, mode)


@pytest.mark.parametrize("zero", ["some", "all"])
def test_rotcube_degenerate_frames(gm_ctx, zero):
    """Nodes with a zero quaternion have no frame (the reference's normalize
    divides zero by zero): those queries keep the tree search."""
    res, qres = 16, 4
    Q = _field(qres, 9950)
    Q[::5 if zero == "some" else 1] = 0
    X = _grid(res, 9960, density=0.003, blocks=1)
    got = _run(gm_ctx, res, X, Q, qres, uniform=3)
    want = _oracle(res, X, Q, qres, None, 3, 0)
    for g, w, name in zip(got, want, "DSC"):
        assert np.array_equal(g, w), name


@pytest.mark.parametrize("res,uniform", [(16, 3), (64, 75)])
def test_rotcube_smallest_grid_and_huge_radius(gm_ctx, res, uniform):
    """res 16 (four pyramid levels); and radius 75 around one corner block:
    the distance field saturates below the miss bound (3 x 76^2), so every
    query beyond the radius is searched."""
    qres = 2
    if uniform > 64:
        X = np.zeros((res, res, res), np.uint8)
        X[2:5, 3:6, 2:4] = 0xFF
        X = X.reshape(-1)
    else:
        X = _grid(res, 9700 + res, density=0.002, blocks=1)
    Q = _field(qres, 9800)
    got = _run(gm_ctx, res, X, Q, qres, uniform=uniform)
    want = _oracle(res, X, Q, qres, None, uniform, 0)
    for g, w, name in zip(got, want, "DSC"):
        assert np.array_equal(g, w), name
    assert 0 < (want[0] == 0xFF).mean() < 1


def test_rotcube_exact(gm_ctx):
    res, qres = 32, 3
    X = _grid(res, 8500)
    Q = _field(qres, 8600)
    sc = _scale(res, 8700, 2, 5)
    got = _run(gm_ctx, res, X, Q, qres, scale=sc, mode=L.GM_EXACT)
    want = _oracle(res, X, Q, qres, sc, 0, 1)
    for g, w, name in zip(got, want, "DSC"):
        assert np.array_equal(g, w), name


def test_rotcube_data_res(gm_ctx):
    res, qres = 32, 2
    X = _grid(res, 8800)
    Q = _field(qres, 8900)
    dr = [20, 27, 31]
    got = _run(gm_ctx, res, X, Q, qres, uniform=4, data_res=dr)
    want = _oracle(res, X, Q, qres, None, 4, 0, data_res=dr)
    for g, w, name in zip(got, want, "DSC"):
        assert np.array_equal(g, w), name


def test_rotcube_empty_and_zero_field(gm_ctx):
    res, qres = 32, 2
    X = np.zeros(res ** 3, np.uint8)
    Q = _field(qres, 9000)
    got = _run(gm_ctx, res, X, Q, qres)
    assert not got[0].any() and not got[2].any()
    # a zero quaternion normalises to NaN: every separating-axis test fails
    # to separate, as in the reference (oracle evaluates the same)
    X = _grid(res, 9100)
    Z = np.zeros((qres ** 3, 4), np.float32)
    got = _run(gm_ctx, res, X, Z, qres)
    want = _oracle(res, X, Z, qres, None, 3, 0)
    for g, w, name in zip(got, want, "DSC"):
        assert np.array_equal(g, w), name


def test_axis_aligned_field_equals_cube_closing_exact(gm_ctx):
    import torch
    res, qres = 32, 2
    X = _grid(res, 9200)
    Q = np.tile(np.array([0, 1, 0, 0], np.float32), (qres ** 3, 1))
    _, _, C = _run(gm_ctx, res, X, Q, qres, uniform=4, mode=L.GM_EXACT)
    Cc = gm_ctx.close(api.make_desc(res), _dev(X), None, 4, L.GM_EXACT, L.GM_SE_CUBE)
    torch.cuda.synchronize()
    assert np.array_equal(C, Cc.cpu().numpy())


def test_rotcube_rejects_bad_arguments(gm_ctx):
    import torch
    res = 32
    desc = api.make_desc(res)
    X = _dev(np.zeros(res ** 3, np.uint8))
    Q = _dev(np.zeros((8, 4), np.float32))
    out = torch.empty_like(X)
    for args in [(None, 2), (Q, 0), (Q, 2000)]:
        with pytest.raises(L.GMError):
            gm_ctx.close_rotcube(desc, X, args[0], args[1], None, 3, L.GM_REF, out=out)
    Qm = torch.zeros(8 * 4 + 1, dtype=torch.float32, device="cuda")[1:]  # 4-byte aligned only
    with pytest.raises(L.GMError):
        gm_ctx.close_rotcube(desc, X, Qm, 2, None, 3, L.GM_REF, out=out)
    torch.cuda.synchronize()


POINTS = [((0.30, 0.40, 0.50), (0.5, 0.2, 0.1)), ((0.80, 0.10, 0.60), (0.0, 0.0, 1.0)),
          ((0.15, 0.85, 0.25), (-0.7, 0.3, 0.2))]


@pytest.mark.parametrize("qres,npts", [(4, 1), (8, 2), (12, 3)])
def test_frame_field_matches_oracle(gm_ctx, qres, npts):
    import torch
    ff = api.FrameField(gm_ctx, (0, 0, 0), (1, 1, 1), qres)
    for pos, tw in POINTS[:npts]:
        ff.add_point(pos, tw)
    iters = ff.generate()
    got = ff.quats().cpu().numpy()
    torch.cuda.synchronize()
    want = F.generate(qres, (0, 0, 0), (1, 1, 1), POINTS[:npts])
    assert iters > 0
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    assert ff.num_points() == npts
    g, t = ff.point(0)
    assert list(g) == F.lattice_position(POINTS[0][0], (0, 0, 0), (1, 1, 1), qres)
    ff.destroy()


@pytest.mark.parametrize("qres,npts", [(2, 1), (2, 8), (3, 20), (5, 4), (7, 5), (16, 20), (17, 3), (18, 13)])
def test_frame_field_sizes(gm_ctx, qres, npts):
    """Odd and even lattices from the smallest on (the transforms fold a line
    in halves and run 16 lines a block), one constraint up to 20, points that
    share a node and a field solved again after a point changed."""
    import torch
    rng = np.random.default_rng(100 * qres + npts)
    pts = [(tuple(rng.uniform(0.01, 0.99, 3)), tuple(rng.normal(size=3))) for _ in range(npts)]
    ff = api.FrameField(gm_ctx, (0, 0, 0), (1, 1, 1), qres)
    for pos, tw in pts:
        ff.add_point(pos, tw)
    for again in range(2):
        ff.generate()
        got = ff.quats().cpu().numpy()
        torch.cuda.synchronize()
        want = F.generate(qres, (0, 0, 0), (1, 1, 1), pts)
        assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
        pts[0] = (pts[0][0], (0.4, -0.2, 0.9))
        ff.update_point(0, pts[0][1])
    ff.destroy()


def test_frame_field_by_lines(gm_ctx):
    """The first lattice past those transformed by planes; constraints in
    corners, on a face and inside."""
    import torch
    qres = 33
    pts = [((0.0, 0.0, 0.0), (0.3, 0.1, -0.2)), ((0.99, 0.99, 0.99), (-0.5, 0.2, 0.4)), ((0.4, 0.99, 0.7), (0.1, 0.9, 0.0)),
           ((0.52, 0.31, 0.63), (0.0, -0.4, 0.8))]
    ff = api.FrameField(gm_ctx, (0, 0, 0), (1, 1, 1), qres)
    for pos, tw in pts:
        ff.add_point(pos, tw)
    ff.generate()
    got = ff.quats().cpu().numpy()
    torch.cuda.synchronize()
    want = F.generate(qres, (0, 0, 0), (1, 1, 1), pts)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    ff.destroy()


def test_frame_field_same_node_last_wins(gm_ctx):
    """Two constraints on one lattice node: S is set once and b takes the
    later point's quaternion (FrameFieldSparseBiharmonic.cu:353-364,
    481-507), on a box that is not the unit cube."""
    import torch
    lo, hi, qres = (-2.0, 1.0, 0.5), (2.0, 3.0, 4.0), 10
    pts = [((0.1, 2.0, 2.0), (0.3, 0.0, 0.0)), ((1.5, 1.2, 3.5), (0.0, 0.8, 0.0)),
           ((0.15, 2.05, 2.02), (0.0, 0.0, -1.1))]
    g0 = F.lattice_position(pts[0][0], lo, hi, qres)
    assert g0 == F.lattice_position(pts[2][0], lo, hi, qres)
    ff = api.FrameField(gm_ctx, lo, hi, qres)
    for pos, tw in pts:
        ff.add_point(pos, tw)
    ff.generate()
    got = ff.quats().cpu().numpy()
    torch.cuda.synchronize()
    want = F.generate(qres, lo, hi, pts)
    assert np.abs(got - want).max() <= 1e-5 * np.abs(want).max()
    ff.destroy()


def test_frame_field_defaults_and_limits(gm_ctx):
    ff = api.FrameField(gm_ctx, (-1, -1, -1), (1, 1, 1), 6)
    with pytest.raises(L.GMError):
        ff.quats()  # before generate
    assert ff.generate() == 0
    q = ff.quats().cpu().numpy()
    assert np.array_equal(q, np.tile(np.array([0, 1, 0, 0], np.float32), (6 ** 3, 1)))
    with pytest.raises(L.GMError):
        ff.add_point((5, 0, 0), (0, 0, 1))  # outside the lattice
    for i in range(20):
        ff.add_point((-0.9 + 0.09 * i, 0, 0), (0, 0, 0.1 * i))
    with pytest.raises(L.GMError):
        ff.add_point((0, 0, 0), (0, 0, 1))  # a 21st point
    ff.update_point(3, (1, 0, 0))
    assert ff.point(3)[1] == (1.0, 0.0, 0.0)
    ff.destroy()


def test_generated_field_drives_the_closing(gm_ctx):
    """Generate on the GPU, close with the field, and compare with the
    oracle closing of the same (downloaded) quaternions."""
    import torch
    res, qres = 64, 4
    ff = api.FrameField(gm_ctx, (0, 0, 0), (1, 1, 1), qres)
    ff.add_point((0.2, 0.3, 0.4), (0.0, 0.0, 0.7))
    ff.add_point((0.7, 0.6, 0.5), (0.4, -0.4, 0.0))
    ff.generate()
    Qd = ff.quats()
    X = _grid(res, 9300)
    desc = api.make_desc(res)
    Xd = _dev(X)
    Cg = gm_ctx.close_rotcube(desc, Xd, Qd, qres, None, 5, L.GM_REF)
    torch.cuda.synchronize()
    Q = Qd.cpu().numpy()
    want = _oracle(res, X, Q, qres, None, 5, 0)[2]
    assert np.array_equal(Cg.cpu().numpy(), want)
    ff.destroy()
