// rotcube.cu — rotated-cube dilation under a frame field (reference:
// GMorpho::DilateByRotCubeMipmap, GMorpho/GMorpho.cu:3058-3230, with the
// kernels DilateByRotCubeByTexMipmapBase, GMorpho.cu:1712-1837, and
// DilateByRotCubeByTexMipmap, GMorpho.cu:2464-2602).
//
// The structuring element at a lattice point p is the cube of half size
// r(p) centred on p and rotated by the frame field's quaternion
// interpolated at p.  It is not separable, so this dilation keeps the
// reference's hierarchical search: an occupancy byte pyramid over the input
// grid (bit k of a node = child k holds any voxel) is descended while the
// children's boxes overlap the rotated cube (separating-axis test), and the
// point is dilated as soon as one occupied fine voxel is reached.
//
// * Shortcuts from the squared lattice distance field E of the input grid
//   (launch_edt): the cube of half size r contains the ball of radius r and
//   lies in the ball of radius r sqrt(3), so E(p) < r^2 is a hit and
//   E(p) >= 3 (r + 1)^2 a miss.  Both keep a margin of at least 1/(2r)
//   fine voxels to the float predicate's decision, far above its rounding
//   (about 1e-4 at these coordinates), so they never change a boolean.
//   Only the shell between them is searched.
// * The search halves the query's own cube and lets the field decide the
//   parts (k_rc_cover, below): it reads a voxel's byte only next to the
//   cube's boundary.  The descent of the occupancy pyramid, one warp per
//   query and 32 children tested at once (k_rc_search), remains for frames
//   that are no rotations (a zero or NaN quaternion has no cube to halve).
// * Base pass: cells inside data_res whose byte is not 0xff; frame at the
//   cell, centre 2c, radius of fine voxel 2c.  Contour: the cells whose byte
//   differs from a diagonal neighbour (ComputeContourBaseConservative,
//   GMorpho/Grid.cu:1464-1498, 2170-2230), listed with warp-aggregated
//   atomics; their eight fine voxels (frame on the 2 res lattice, own
//   radius) overwrite the byte.
//
// Every float expression is the reference's, evaluated left to right; this
// translation unit is compiled with -fmad=false so that no multiply-add is
// fused, and division and square root are IEEE round-to-nearest, as in the
// CPU oracle (compiled with -ffp-contract=off): both give the same booleans.
#include "gm_common.cuh"
#include "gm_internal.h"

namespace gm {

namespace {

constexpr int kRcThreads = 256;

// The occupancy pyramid: level 0 is the input grid (a node's bits are its
// fine voxels), levels 1..L ((res >> l)^3 node bytes) follow each other in
// `up`, level l at byte (8^L - 8^(L-l+1)) / 7.
struct RcLevels {
  const uint8_t* X;
  const uint8_t* up;
  int L;  // log2(res)
  __host__ __device__ __forceinline__ const uint8_t* level(int l) const {
    return l == 0 ? X : up + ((((int64_t)1 << (3 * L)) - ((int64_t)1 << (3 * (L - l + 1)))) / 7);
  }
  const uint8_t* level_host(int l) const { return level(l); }
};

// the structuring element of one lattice point
struct RcQuery {
  float c[3];             // centre, fine units
  float bx[3], by[3], bz[3];
  float se;               // half size
};

__device__ __forceinline__ float4 rc_node(const float4* __restrict__ Q, int64_t n, int64_t i) {
  // past the last node: clamped (the reference reads beyond its field there)
  return __ldg(Q + (i < n ? i : n - 1));
}

__device__ __forceinline__ float4 rc_lerp(float4 a, float4 b, float t) {
  const float s = 1.f - t;
  return make_float4(s * a.x + t * b.x, s * a.y + t * b.y, s * a.z + t * b.z, s * a.w + t * b.w);
}

// Hamilton product, terms in the reference's order (cuda_math.h:386-393)
__device__ __forceinline__ float4 rc_mul(float4 a, float4 b) {
  float4 r;
  r.w = a.w * b.w - a.x * b.x - a.y * b.y - a.z * b.z;
  r.x = a.w * b.x + a.x * b.w + a.y * b.z - a.z * b.y;
  r.y = a.w * b.y - a.x * b.z + a.y * b.w + a.z * b.x;
  r.z = a.w * b.z + a.x * b.y - a.y * b.x + a.z * b.w;
  return r;
}

// InterpolateQuaternionField (GMorpho.cu:1631-1710: trilinear, group size
// 0 = plain weighted sums), normalize (conj (quat)) and the rotated axes
// rotate (quat, e_k) (GMorpho.cu:1735-1745; cuda_math.h:396-401)
__device__ void rc_frame(const float4* __restrict__ Q, int qres, int ix, int iy, int iz, int res, RcQuery& q) {
  const float fres = (float)res, fq = (float)qres;
  const float fx = fq * ((float)ix / fres), fy = fq * ((float)iy / fres), fz = fq * ((float)iz / fres);
  const int jx = (int)fx, jy = (int)fy, jz = (int)fz;
  const int64_t sy = qres, sz = (int64_t)qres * qres, n = sz * qres;
  const int64_t b = jx + sy * jy + sz * jz;
  const float tx = fx - (float)jx, ty = fy - (float)jy, tz = fz - (float)jz;
  const float4 q00 = rc_lerp(rc_node(Q, n, b), rc_node(Q, n, b + 1), tx);
  const float4 q01 = rc_lerp(rc_node(Q, n, b + sz), rc_node(Q, n, b + 1 + sz), tx);
  const float4 q10 = rc_lerp(rc_node(Q, n, b + sy), rc_node(Q, n, b + 1 + sy), tx);
  const float4 q11 = rc_lerp(rc_node(Q, n, b + sy + sz), rc_node(Q, n, b + 1 + sy + sz), tx);
  float4 u = rc_lerp(rc_lerp(q00, q10, ty), rc_lerp(q01, q11, ty), tz);
  u.x = -u.x;
  u.y = -u.y;
  u.z = -u.z;
  const float len = sqrtf(u.x * u.x + u.y * u.y + u.z * u.z + u.w * u.w);
  u.x = u.x / len;
  u.y = u.y / len;
  u.z = u.z / len;
  u.w = u.w / len;
  const float4 uc = make_float4(-u.x, -u.y, -u.z, u.w);
  float4 r = rc_mul(uc, rc_mul(make_float4(1.f, 0.f, 0.f, 0.f), u));
  q.bx[0] = r.x, q.bx[1] = r.y, q.bx[2] = r.z;
  r = rc_mul(uc, rc_mul(make_float4(0.f, 1.f, 0.f, 0.f), u));
  q.by[0] = r.x, q.by[1] = r.y, q.by[2] = r.z;
  r = rc_mul(uc, rc_mul(make_float4(0.f, 0.f, 1.f, 0.f), u));
  q.bz[0] = r.x, q.bz[1] = r.y, q.bz[2] = r.z;
}

// HasRotCubeSEOverlap (GMorpho.cu:241-302, 334-349): the 15 separating
// axes of the rotated cube and the box (centre n, half size hs).  All 15
// comparisons are evaluated (no early exit) so that the lanes of a warp,
// each testing another box, stay together; the boolean is the same.
__device__ __forceinline__ bool rc_overlap(const RcQuery& q, float nx, float ny, float nz, float hs) {
  const float tx = q.c[0] - nx, ty = q.c[1] - ny, tz = q.c[2] - nz;
  const float* bx = q.bx;
  const float* by = q.by;
  const float* bz = q.bz;
  const float se = q.se;
  bool sep = fabsf(tx) > hs + se * (fabsf(bx[0]) + fabsf(by[0]) + fabsf(bz[0]));
  sep |= fabsf(ty) > hs + se * (fabsf(bx[1]) + fabsf(by[1]) + fabsf(bz[1]));
  sep |= fabsf(tz) > hs + se * (fabsf(bx[2]) + fabsf(by[2]) + fabsf(bz[2]));
  sep |= fabsf(tx * bx[0] + ty * bx[1] + tz * bx[2]) > hs * (fabsf(bx[0]) + fabsf(bx[1]) + fabsf(bx[2])) + se;
  sep |= fabsf(tx * by[0] + ty * by[1] + tz * by[2]) > hs * (fabsf(by[0]) + fabsf(by[1]) + fabsf(by[2])) + se;
  sep |= fabsf(tx * bz[0] + ty * bz[1] + tz * bz[2]) > hs * (fabsf(bz[0]) + fabsf(bz[1]) + fabsf(bz[2])) + se;
  sep |= fabsf(tz * bx[1] - ty * bx[2]) > hs * (fabsf(bx[2]) + fabsf(bx[1])) + se * (fabsf(bz[0]) + fabsf(by[0]));
  sep |= fabsf(tz * by[1] - ty * by[2]) > hs * (fabsf(by[2]) + fabsf(by[1])) + se * (fabsf(bz[0]) + fabsf(bx[0]));
  sep |= fabsf(tz * bz[1] - ty * bz[2]) > hs * (fabsf(bz[2]) + fabsf(bz[1])) + se * (fabsf(by[0]) + fabsf(bx[0]));
  sep |= fabsf(tx * bx[2] - tz * bx[0]) > hs * (fabsf(bx[2]) + fabsf(bx[0])) + se * (fabsf(bz[1]) + fabsf(by[1]));
  sep |= fabsf(tx * by[2] - tz * by[0]) > hs * (fabsf(by[2]) + fabsf(by[0])) + se * (fabsf(bz[1]) + fabsf(bx[1]));
  sep |= fabsf(tx * bz[2] - tz * bz[0]) > hs * (fabsf(bz[2]) + fabsf(bz[0])) + se * (fabsf(by[1]) + fabsf(bx[1]));
  sep |= fabsf(ty * bx[0] - tx * bx[1]) > hs * (fabsf(bx[1]) + fabsf(bx[0])) + se * (fabsf(bz[2]) + fabsf(by[2]));
  sep |= fabsf(ty * by[0] - tx * by[1]) > hs * (fabsf(by[1]) + fabsf(by[0])) + se * (fabsf(bz[2]) + fabsf(bx[2]));
  sep |= fabsf(ty * bz[0] - tx * bz[1]) > hs * (fabsf(bz[1]) + fabsf(bz[0])) + se * (fabsf(by[2]) + fabsf(bx[2]));
  return !sep;
}

__device__ __forceinline__ int rc_radius(const int8_t* __restrict__ R, int uniform_r, int fx, int fy, int fz, int n) {
  return clamp_radius(R ? (int)__ldg(R + fine_index(fx, fy, fz, n)) : uniform_r);
}

// Decision from the squared lattice distance e (saturated, a lower bound of
// the true one) of the query point to the nearest occupied fine voxel box:
// 1 = dilated, 0 = not dilated, -1 = search.
// * e < r^2: a voxel box reaches into the ball of radius r, which the cube
//   of half size r contains with a margin of at least 1/(2r) fine voxels
//   along every axis (also for each box containing that voxel box, i.e. the
//   voxel's pyramid ancestors), against float rounding of about 1e-4 here.
// * A voxel box passing the predicate passes its separating-axis tests 1-3
//   (box within se * A_i of the query along axis i, A_i = |b_x,i| + |b_y,i|
//   + |b_z,i|) and 4-6 (its centre within se + w_j / 2 of the query along
//   b_j, w_j = |b_j,x| + |b_j,y| + |b_j,z|), so it lies at squared distance
//   at most M1 = sum_i (se A_i)^2 and at most M2 = (sum_j (se + w_j / 2)^2
//   ^ 1/2 + 0.01)^2 (0.01 covers the tests' float rounding).  e > min(M1, M2)
//   leaves no voxel that could pass: not dilated, exactly.
__device__ __forceinline__ int rc_shortcut(const RcQuery& q, uint32_t e) {
  const float r = q.se;
  if ((float)e < r * r) return 1;
  const float* b[3] = {q.bx, q.by, q.bz};
  float m1 = 0.f, m2 = 0.f;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const float h = q.se * (fabsf(q.bx[i]) + fabsf(q.by[i]) + fabsf(q.bz[i]));
    m1 += h * h;
    const float g = q.se + 0.5f * (fabsf(b[i][0]) + fabsf(b[i][1]) + fabsf(b[i][2]));
    m2 += g * g;
  }
  m2 = sqrtf(m2) + 0.01f;
  m2 *= m2;
  // float rounding of these bounds: a few ulps, covered by 1e-5 relative
  const float m = (m1 < m2 ? m1 : m2) * 1.00001f + 1e-3f;
  if ((float)e > m) return 0;  // NaN axes: m is NaN, no decision
  return -1;
}

__device__ __forceinline__ uint64_t rc_pack(int x, int y, int z) {
  return (uint64_t)x | ((uint64_t)y << 21) | ((uint64_t)z << 42);
}

constexpr int kRcSearchWarps = kRcThreads / 32;

// One warp, one query.  Each round the warp takes up to NPL pending nodes
// of its level; lane l tests 8 / (32 / NPL) children of node l / (32 / NPL)
// (the lanes of a node start with the children away from the query, so that
// the compacted list ends with the nearest ones, which are taken first);
// the surviving children become the next level's pending list and the warp
// descends.  A level's list only receives children while it is empty (the
// warp climbs back only once a level is exhausted), so it never holds more
// than 8 NPL nodes.  True at the first surviving fine voxel.  Warp-uniform
// control flow; the per-level counts (<= 64) live in three registers.
template <int NPL>
__device__ bool rc_search(const RcLevels& P, const RcQuery& q, uint64_t (*lst)[8 * NPL], int lane) {
  constexpr int LPN = 32 / NPL;  // lanes per node
  constexpr int CPL = 8 / LPN;   // children per lane
  const int maxd = P.L + 1;
  uint32_t c0 = 1, c1 = 0, c2 = 0;  // 8-bit pending counts of levels 0..11
  auto getc = [&](int d) -> int {
    const uint32_t w = d < 4 ? c0 : (d < 8 ? c1 : c2);
    return (int)((w >> ((d & 3) * 8)) & 0xffu);
  };
  auto setc = [&](int d, int v) {
    const int sh = (d & 3) * 8;
    const uint32_t m = ~(0xffu << sh), x = (uint32_t)v << sh;
    if (d < 4) c0 = (c0 & m) | x;
    else if (d < 8) c1 = (c1 & m) | x;
    else c2 = (c2 & m) | x;
  };
  if (lane == 0) lst[0][0] = rc_pack(0, 0, 0);
  int d = 0;
  // each round consumes at least one pending node; the pending nodes are
  // finite (a tree), so the loop ends
  for (;;) {
    __syncwarp();
    const int cd = getc(d);
    if (cd == 0) {
      if (d == 0) return false;
      d--;
      continue;
    }
    const int m = cd < NPL ? cd : NPL;
    setc(d, cd - m);
    const int j = lane / LPN;
    bool ok[CPL];
    uint64_t child[CPL];
#pragma unroll
    for (int u = 0; u < CPL; u++) ok[u] = false, child[u] = 0;
    if (j < m) {
      const uint64_t nd = lst[d][cd - m + j];
      const int nx = (int)(nd & 0x1fffff), ny = (int)((nd >> 21) & 0x1fffff), nz = (int)(nd >> 42);
      const int level = P.L - d;
      const int64_t nl = (int64_t)1 << d;
      const uint32_t occ = __ldg(P.level(level) + nx + nl * ny + nl * nl * nz);
      const float ns = (float)(2 << level);
      const int near = (q.c[0] >= ns * ((float)nx + 0.5f)) | ((q.c[1] >= ns * ((float)ny + 0.5f)) << 1) |
                       ((q.c[2] >= ns * ((float)nz + 0.5f)) << 2);
      const float ncs = (float)(1 << level);  // child size: 2 res >> (d + 1)
#pragma unroll
      for (int u = 0; u < CPL; u++) {
        const int t = (lane % LPN) * CPL + u;  // 7 = the child on the query's side
        const int k = t ^ near ^ 7;
        if ((occ >> k) & 1) {
          const int cx = 2 * nx + (k & 1), cy = 2 * ny + ((k >> 1) & 1), cz = 2 * nz + (k >> 2);
          ok[u] = rc_overlap(q, ncs * ((float)cx + 0.5f), ncs * ((float)cy + 0.5f), ncs * ((float)cz + 0.5f),
                             0.5f * ncs);
          child[u] = rc_pack(cx, cy, cz);
        }
      }
    }
    uint32_t surv[CPL];
    int tot = 0;
#pragma unroll
    for (int u = 0; u < CPL; u++) {
      surv[u] = __ballot_sync(0xffffffffu, ok[u]);
      tot += __popc(surv[u]);
    }
    if (tot == 0) continue;
    if (d + 1 == maxd) return true;
    __syncwarp();
    int at = 0;
#pragma unroll
    for (int u = 0; u < CPL; u++) {
      if (ok[u]) lst[d + 1][at + __popc(surv[u] & ((1u << lane) - 1))] = child[u];
      at += __popc(surv[u]);
    }
    setc(d + 1, tot);
    d++;
  }
}

// ---- the search in the query's own cube
//
// A voxel passing the predicate passes its separating-axis tests 4-6, so its
// centre lies in the box B of half sizes H_j = r + w_j / 2 along the cube's
// axes.  B is halved along each axis level by level, and the distance field
// decides the parts:
//   * a part of centre s and half diagonal rho holds no occupied voxel's
//     centre when the field at the lattice point l next to s exceeds
//     rho + |s - l| - 1/2 (a voxel contains the ball of radius 1/2 around
//     its centre): dropped;
//   * when the field plus |s - l| is below the distance of s to the cube's
//     faces, some occupied voxel reaches into the cube: dilated.  Taken with
//     a margin of kRcInside against the float rounding of the predicate, and
//     only for frames whose edge-edge axes are long enough to keep it
//     (kRcAligned) or vanish;
//   * parts of half size <= 1 that remain are read: their occupied voxels
//     (at most 4^3 candidates) are put to the predicate itself, and on
//     success so are the voxel's ancestors, as the descent from the grid's
//     root would have: the same boolean.
// Depth first, a query at a time: a step halves one part and weighs its
// eight halves (eight field values in flight), the one nearest to an
// occupied voxel next; the halves still to do are a byte per level.
// k_rc_cover schedules the steps.
constexpr float kRcInside = 0.05f;
constexpr float kRcAligned = 0.99875f;

__device__ __forceinline__ float rc_sqrt(float x) {  // within 2^-22: the bounds have room for it
  float r;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}

// the frame is a rotation (not degenerate, not NaN)
__device__ __forceinline__ bool rc_is_rotation(const RcQuery& q) {
  bool ok = true;
  const float* b[3] = {q.bx, q.by, q.bz};
#pragma unroll
  for (int j = 0; j < 3; j++) ok = ok && fabsf(b[j][0] * b[j][0] + b[j][1] * b[j][1] + b[j][2] * b[j][2] - 1.f) < 1e-3f;
  return ok;
}

// Voxel (x, y, z) and its ancestors against the predicate.  The tests along
// the cube's axes come first: they refuse most voxels, and a centre inside
// the cube with a margin passes the others (rule, as above).  An ancestor
// contains the voxel, so its exact slack in every test is at least the
// voxel's; only when the voxel's smallest slack is within the rounding of
// the ancestors' tests (below 1e-3 up to 2048 voxels an axis) are they
// evaluated.
__device__ __forceinline__ bool rc_reached(const RcQuery& q, int x, int y, int z, int L, bool rule) {
  const float tx = q.c[0] - ((float)x + 0.5f), ty = q.c[1] - ((float)y + 0.5f), tz = q.c[2] - ((float)z + 0.5f);
  const float* bx = q.bx;
  const float* by = q.by;
  const float* bz = q.bz;
  const float se = q.se, hs = 0.5f;
  const float px = fabsf(tx * bx[0] + ty * bx[1] + tz * bx[2]), py = fabsf(tx * by[0] + ty * by[1] + tz * by[2]),
              pz = fabsf(tx * bz[0] + ty * bz[1] + tz * bz[2]);
  const float far = fmaxf(px, fmaxf(py, pz));
  if (rule && far < se - kRcInside) return true;
  float slack = hs * (fabsf(bx[0]) + fabsf(bx[1]) + fabsf(bx[2])) + se - px;
  slack = fminf(slack, hs * (fabsf(by[0]) + fabsf(by[1]) + fabsf(by[2])) + se - py);
  slack = fminf(slack, hs * (fabsf(bz[0]) + fabsf(bz[1]) + fabsf(bz[2])) + se - pz);
  if (slack < -4e-3f) return false;
  // the other twelve
  slack = fminf(slack, hs + se * (fabsf(bx[0]) + fabsf(by[0]) + fabsf(bz[0])) - fabsf(tx));
  slack = fminf(slack, hs + se * (fabsf(bx[1]) + fabsf(by[1]) + fabsf(bz[1])) - fabsf(ty));
  slack = fminf(slack, hs + se * (fabsf(bx[2]) + fabsf(by[2]) + fabsf(bz[2])) - fabsf(tz));
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const float* b = j == 0 ? bx : (j == 1 ? by : bz);
    const float* c = j == 0 ? bz : (j == 1 ? bz : by);
    const float* d = j == 0 ? by : bx;
    slack = fminf(slack, hs * (fabsf(b[2]) + fabsf(b[1])) + se * (fabsf(c[0]) + fabsf(d[0])) - fabsf(tz * b[1] - ty * b[2]));
    slack = fminf(slack, hs * (fabsf(b[2]) + fabsf(b[0])) + se * (fabsf(c[1]) + fabsf(d[1])) - fabsf(tx * b[2] - tz * b[0]));
    slack = fminf(slack, hs * (fabsf(b[1]) + fabsf(b[0])) + se * (fabsf(c[2]) + fabsf(d[2])) - fabsf(ty * b[0] - tx * b[1]));
  }
  if (slack > 4e-3f) return true;
  if (slack < -4e-3f) return false;
  // within rounding: the tests themselves
  for (int t = 0; t <= L; t++) {
    const float size = (float)(1 << t);
    if (!rc_overlap(q, size * ((float)(x >> t) + 0.5f), size * ((float)(y >> t) + 0.5f),
                    size * ((float)(z >> t) + 0.5f), 0.5f * size))
      return false;
  }
  return true;
}

// A lane's search: B, and the part to do next (its level and its index
// along the three axes, 8 bits each); pending: halves to do, a byte a level.
struct RcCover {
  float H[3], far;
  int depth;   // level of the parts that are read
  bool rule;   // the frame keeps the margin of the inside verdict
  int level;
  uint32_t at;
  uint64_t pending;
};

__device__ __forceinline__ void rc_begin(const RcQuery& q, RcCover& v) {
  const float* b[3] = {q.bx, q.by, q.bz};
  bool rule = true, square = true;
  float far2 = 0.f;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    v.H[j] = q.se + 0.5f * (fabsf(b[j][0]) + fabsf(b[j][1]) + fabsf(b[j][2])) + 2e-3f;
    far2 += v.H[j] * v.H[j];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const float t = fabsf(b[j][i]);
      rule = rule && t <= kRcAligned;
      square = square && (t == 0.f || t == 1.f);
    }
  }
  v.rule = rule || square;
  v.far = sqrtf(far2);
  const float big = fmaxf(v.H[0], fmaxf(v.H[1], v.H[2]));  // in (2, 128)
  v.depth = 32 - __clz((int)ceilf(big) - 1);                // big <= 2^depth
  v.level = 0;
  v.at = 0;
  v.pending = 0;
}

// the next pending half; false: none
__device__ __forceinline__ bool rc_next(RcCover& v) {
  if (v.pending == 0) return false;
  const int l = (63 - __clzll((long long)v.pending)) >> 3;
  const uint32_t byte = (uint32_t)(v.pending >> (8 * l)) & 0xffu;
  const int k = __ffs(byte) - 1;
  v.pending &= ~((uint64_t)1 << (8 * l + k));
  const int up = v.level - l;
  const uint32_t node = (v.at >> up) & ((0xffu >> up) * 0x010101u);
  v.at = (node << 1) | (uint32_t)(k & 1) | ((uint32_t)(k & 2) << 7) | ((uint32_t)(k & 4) << 14);
  v.level = l + 1;
  return true;
}

// Halves the part: 1 dilated, 0 no half left of it, -1 the next is set
__device__ __forceinline__ int rc_halve(const uint16_t* __restrict__ E, int N, const RcQuery& q, RcCover& v) {
  const float half = 1.f / (float)(2 << v.level);  // of the halves, in H
  float u[3], h[3], s[3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    h[j] = v.H[j] * half;
    u[j] = h[j] * (float)(4 * (int)((v.at >> (8 * j)) & 0xffu) + 2) - v.H[j];  // the part's centre
  }
  float dx[3], dy[3], dz[3], in_lo[3], in_hi[3];
#pragma unroll
  for (int i = 0; i < 3; i++) {
    s[i] = q.c[i] + (u[0] * q.bx[i] + u[1] * q.by[i] + u[2] * q.bz[i]);
    dx[i] = h[0] * q.bx[i], dy[i] = h[1] * q.by[i], dz[i] = h[2] * q.bz[i];
    in_lo[i] = fabsf(u[i] - h[i]), in_hi[i] = fabsf(u[i] + h[i]);
  }
  const float reach = half * v.far - 0.5f + 4e-3f;
  float off[8];
  uint32_t e[8];
#pragma unroll
  for (int k = 0; k < 8; k++) {
    float off2 = 0.f;
    int l[3];
#pragma unroll
    for (int i = 0; i < 3; i++) {
      const float p = s[i] + ((k & 1 ? dx[i] : -dx[i]) + (k & 2 ? dy[i] : -dy[i]) + (k & 4 ? dz[i] : -dz[i]));
      l[i] = min(max(__float2int_rn(p), 0), N - 1);
      const float o = p - (float)l[i];
      off2 += o * o;
    }
    off[k] = rc_sqrt(off2);
    e[k] = __ldg(E + fine_index(l[0], l[1], l[2], N));
  }
  uint32_t keep = 0, best = 0;
  float nearest = 1e30f;
  bool hit = false;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const float dist = rc_sqrt((float)e[k]);
    const float out = fmaxf(k & 1 ? in_hi[0] : in_lo[0], fmaxf(k & 2 ? in_hi[1] : in_lo[1], k & 4 ? in_hi[2] : in_lo[2]));
    hit = hit || dist + off[k] < q.se - out - kRcInside;
    if (dist <= reach + off[k]) {
      keep |= 1u << k;
      if (dist < nearest) nearest = dist, best = k;
    }
  }
  if (hit && v.rule) return 1;
  if (keep == 0) return 0;
  v.pending |= (uint64_t)(keep & ~(1u << best)) << (8 * v.level);
  v.at = (v.at << 1) | (best & 1u) | ((best & 2u) << 7) | ((best & 4u) << 14);
  v.level++;
  return -1;
}

// Reads a part of half size <= 1: true when one of its occupied voxels is
// reached.  Candidates: the voxels with their centre in the part's box
// along the grid's axes, 4 along each at most, i.e. 3 cells; the 27 bytes
// are loaded at once, the voxels outside the box masked off.
__device__ __forceinline__ bool rc_read(const uint8_t* __restrict__ X, int res, int L, const RcQuery& q,
                                        const RcCover& v) {
  const float half = 1.f / (float)(1 << v.level);
  float u[3], h[3];
#pragma unroll
  for (int j = 0; j < 3; j++) {
    h[j] = v.H[j] * half;
    u[j] = h[j] * (float)(2 * (int)((v.at >> (8 * j)) & 0xffu) + 1) - v.H[j];
  }
  int c0[3];
  uint32_t mask[3];  // per axis: the parities inside, two bits a cell (none outside the grid)
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const float s = q.c[i] + (u[0] * q.bx[i] + u[1] * q.by[i] + u[2] * q.bz[i]) - 0.5f;
    const float a = h[0] * fabsf(q.bx[i]) + h[1] * fabsf(q.by[i]) + h[2] * fabsf(q.bz[i]) + 2e-3f;
    const int lo = max(__float2int_ru(s - a), 0), hi = min(__float2int_rd(s + a), 2 * res - 1);
    c0[i] = min(lo >> 1, res - 1);  // (a box beyond the grid: no parity is inside)
    mask[i] = hi < lo ? 0u : ((2u << (hi - 2 * c0[i])) - 1u) & ~((1u << (lo - 2 * c0[i])) - 1u);
  }
  if (mask[0] == 0 || mask[1] == 0 || mask[2] == 0) return false;
  const uint8_t* base = X + cell_index(c0[0], c0[1], c0[2], res);
  uint32_t row[9];  // three cells along x a word
#pragma unroll
  for (int r = 0; r < 9; r++) {
    const int y = r % 3, z = r / 3;
    const uint32_t my = (mask[1] >> (2 * y)) & 3u, mz = (mask[2] >> (2 * z)) & 3u;
    // bits x + 2 y + 4 z of a byte, for every x
    const uint32_t m4 = (my & 1u ? 0x3u : 0u) | (my & 2u ? 0xcu : 0u);
    const uint32_t m8 = (mz & 1u ? m4 : 0u) | (mz & 2u ? m4 << 4 : 0u);
    uint32_t w = 0;
    if (m8) {
#pragma unroll
      for (int x = 0; x < 3; x++) {
        const uint32_t mx = (mask[0] >> (2 * x)) & 3u;
        if (mx) w |= ((uint32_t)__ldg(base + x + (int64_t)res * (y + (int64_t)res * z)) & m8 & (mx * 0x55u)) << (8 * x);
      }
    }
    row[r] = w;
  }
  uint32_t rows = 0;
#pragma unroll
  for (int r = 0; r < 9; r++) rows |= (row[r] ? 1u : 0u) << r;
  while (rows) {
    const int r = __ffs(rows) - 1;
    rows &= rows - 1;
    uint32_t w = 0;
#pragma unroll
    for (int i = 0; i < 9; i++) w = r == i ? row[i] : w;
    do {
      const int k = __ffs(w) - 1;
      w &= w - 1;
      if (rc_reached(q, 2 * (c0[0] + (k >> 3)) + (k & 1), 2 * (c0[1] + r % 3) + ((k >> 1) & 1),
                     2 * (c0[2] + r / 3) + ((k >> 2) & 1), L, v.rule))
        return true;
    } while (w);
  }
  return false;
}

// one node byte per thread: bit k = child k of the finer level non-empty
__global__ void k_rc_occ_up(const uint8_t* __restrict__ from, int nf, uint8_t* __restrict__ to) {
  const int nt = nf >> 1;
  const int64_t total = (int64_t)nt * nt * nt;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % nt), y = (int)((i / nt) % nt), z = (int)(i / ((int64_t)nt * nt));
    uint32_t b = 0;
#pragma unroll
    for (int k = 0; k < 8; k++)
      b |= (uint32_t)(from[cell_index(2 * x + (k & 1), 2 * y + ((k >> 1) & 1), 2 * z + (k >> 2), nf)] != 0) << k;
    to[i] = (uint8_t)b;
  }
}

// warp-aggregated append of (cell, voxel mask) entries
__device__ __forceinline__ void rc_append(bool want, uint64_t entry, uint64_t* __restrict__ list,
                                          uint32_t* __restrict__ count, int lane) {
  const uint32_t bal = __ballot_sync(0xffffffffu, want);
  if (bal == 0) return;
  uint32_t at = 0;
  if (lane == 0) at = atomicAdd(count, (uint32_t)__popc(bal));
  at = __shfl_sync(0xffffffffu, at, 0);
  if (want) list[at + __popc(bal & ((1u << lane) - 1))] = entry;
}

// DilateByRotCubeByTexMipmapBase, decided part: D[c] = X[c], or 0xff when
// the corner 2c is dilated by the distance shortcut; the undecided cells are
// listed for rc_search
__global__ void __launch_bounds__(kRcThreads) k_rc_base_cls(const uint8_t* __restrict__ X,
                                                            const uint16_t* __restrict__ E,
                                                            const int8_t* __restrict__ R, int uniform_r,
                                                            const float4* __restrict__ Q, int qres, int res, int dx,
                                                            int dy, int dz, uint8_t* __restrict__ D,
                                                            uint64_t* __restrict__ list, uint32_t* __restrict__ count) {
  const int lane = threadIdx.x & 31;
  const int64_t total = (int64_t)res * res * res, stride = (int64_t)gridDim.x * blockDim.x;
  const int N = 2 * res;
  for (int64_t base = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); base < total; base += stride) {
    const int64_t c = base + lane;
    bool search = false;
    if (c < total) {
      const int x = (int)(c % res), y = (int)((c / res) % res), z = (int)(c / ((int64_t)res * res));
      const uint8_t v = X[c];
      uint8_t out = v;
      if (v != 0xff && x < dx && y < dy && z < dz) {
        RcQuery q;
        rc_frame(Q, qres, x, y, z, res, q);
        q.c[0] = (float)(2 * x), q.c[1] = (float)(2 * y), q.c[2] = (float)(2 * z);
        q.se = (float)rc_radius(R, uniform_r, 2 * x, 2 * y, 2 * z, N);
        const int s = E ? rc_shortcut(q, __ldg(E + fine_index(2 * x, 2 * y, 2 * z, N))) : -1;
        if (s == 1) out = 0xff;
        search = s < 0;
      }
      D[c] = out;
    }
    rc_append(search, ((uint64_t)c << 8) | 1u, list, count, lane);
  }
}

// TagVoxelsContourBaseConservative on D, appended to tags
__global__ void __launch_bounds__(kRcThreads) k_rc_tag(const uint8_t* __restrict__ D, int res,
                                                       uint32_t* __restrict__ tags, uint32_t* __restrict__ count) {
  const int lane = threadIdx.x & 31;
  const int64_t total = (int64_t)res * res * res;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t s1 = res, s2 = (int64_t)res * res;
  for (int64_t base = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); base < total; base += stride) {
    const int64_t c = base + lane;
    bool tag = false;
    if (c < total) {
      const int x = (int)(c % res), y = (int)((c / res) % res), z = (int)(c / s2);
      if (x >= 1 && y >= 1 && z >= 1 && x <= res - 2 && y <= res - 2 && z <= res - 2) {
        const uint8_t v = D[c];
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const int64_t o = ((k & 1) ? 1 : -1) + s1 * (((k >> 1) & 1) ? 1 : -1) + s2 * ((k >> 2) ? 1 : -1);
          tag |= D[c + o] != v;
        }
      }
    }
    const uint32_t bal = __ballot_sync(0xffffffffu, tag);
    if (bal == 0) continue;
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(count, (uint32_t)__popc(bal));
    at = __shfl_sync(0xffffffffu, at, 0);
    if (tag) tags[at + __popc(bal & ((1u << lane) - 1))] = (uint32_t)c;
  }
}

// DilateByRotCubeByTexMipmap, decided part: one thread per cell (tags, or
// every cell when tags is null: GM_EXACT) writes the byte of its fine voxels
// decided by the distance shortcut and lists the others for rc_search
__global__ void __launch_bounds__(kRcThreads) k_rc_fine_cls(const uint16_t* __restrict__ E,
                                                            const int8_t* __restrict__ R, int uniform_r,
                                                            const float4* __restrict__ Q, int qres, int res,
                                                            const uint32_t* __restrict__ tags,
                                                            const uint32_t* __restrict__ ntags,
                                                            uint8_t* __restrict__ D, uint64_t* __restrict__ list,
                                                            uint32_t* __restrict__ count) {
  const int lane = threadIdx.x & 31;
  const int64_t total = tags ? (int64_t)*ntags : (int64_t)res * res * res;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int N = 2 * res;
  for (int64_t base = blockIdx.x * (int64_t)blockDim.x + (threadIdx.x & ~31); base < total; base += stride) {
    const int64_t i = base + lane;
    uint32_t undecided = 0;
    int64_t c = 0;
    if (i < total) {
      c = tags ? (int64_t)tags[i] : i;
      const int x = (int)(c % res), y = (int)((c / res) % res), z = (int)(c / ((int64_t)res * res));
      uint32_t hit = 0;
      for (int k = 0; k < 8; k++) {
        const int fx = 2 * x + (k & 1), fy = 2 * y + ((k >> 1) & 1), fz = 2 * z + (k >> 2);
        RcQuery q;
        rc_frame(Q, qres, fx, fy, fz, N, q);
        q.c[0] = (float)fx, q.c[1] = (float)fy, q.c[2] = (float)fz;
        q.se = (float)rc_radius(R, uniform_r, fx, fy, fz, N);
        const int s = E ? rc_shortcut(q, __ldg(E + fine_index(fx, fy, fz, N))) : -1;
        if (s == 1) hit |= 1u << k;
        if (s < 0) undecided |= 1u << k;
      }
      D[c] = (uint8_t)hit;
    }
    rc_append(undecided != 0, ((uint64_t)c << 8) | undecided, list, count, lane);
  }
}

constexpr int kRcRest = 48;  // an entry's voxels left to the tree search by k_rc_cover

// the query of a listed entry: cell (x, y, z), its corner (fine == 0) or
// fine voxel k
__device__ __forceinline__ void rc_query(RcQuery& q, const int8_t* __restrict__ R, int uniform_r,
                                         const float4* __restrict__ Q, int qres, int res, int x, int y, int z, int k,
                                         int fine) {
  const int N = 2 * res;
  const int fx = 2 * x + (fine ? k & 1 : 0), fy = 2 * y + (fine ? (k >> 1) & 1 : 0), fz = 2 * z + (fine ? k >> 2 : 0);
  if (fine) rc_frame(Q, qres, fx, fy, fz, N, q);
  else rc_frame(Q, qres, x, y, z, res, q);
  q.c[0] = (float)fx, q.c[1] = (float)fy, q.c[2] = (float)fz;
  q.se = (float)rc_radius(R, uniform_r, fx, fy, fz, N);
}

// The listed queries, one warp each (rc_search).  Base entries (fine == 0):
// corner 2c of the cell, frame on the res lattice, D[c] = 0xff on a hit.
// Fine entries: the voxels of the mask, frame on the 2 res lattice, hit
// bits or-ed into D[c] (one entry per cell: no other writer).
template <int NPL>
__global__ void __launch_bounds__(kRcThreads, 2) k_rc_search(RcLevels P, const int8_t* __restrict__ R, int uniform_r,
                                                          const float4* __restrict__ Q, int qres, int res,
                                                          const uint64_t* __restrict__ list,
                                                          const uint32_t* __restrict__ count,
                                                          uint32_t* __restrict__ next,
                                                          const uint32_t* __restrict__ left, int fine,
                                                          uint8_t* __restrict__ D) {
  __shared__ uint64_t lst[kRcSearchWarps][kRotCubeMaxLevels][8 * NPL];
  if (left != nullptr && *left == 0) return;  // (rc_cover took them all)
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t n = *count;
  // entries are taken one at a time from a shared counter: their costs
  // differ by orders of magnitude, a fixed split would leave warps idle
  for (;;) {
    uint32_t e = 0;
    if (lane == 0) e = atomicAdd(next, 1u);
    e = __shfl_sync(0xffffffffu, e, 0);
    if ((int64_t)e >= n) break;
    const uint64_t ent = list[e];
    const int64_t c = (int64_t)((ent & (((uint64_t)1 << kRcRest) - 1)) >> 8);
    uint32_t mask = (uint32_t)((left != nullptr ? ent >> kRcRest : ent) & 0xff);
    if (mask == 0) continue;
    const int x = (int)(c % res), y = (int)((c / res) % res), z = (int)(c / ((int64_t)res * res));
    uint32_t hits = 0;
    while (mask) {
      const int k = __ffs(mask) - 1;
      mask &= mask - 1;
      RcQuery q;
      rc_query(q, R, uniform_r, Q, qres, res, x, y, z, k, fine);
      if (rc_search<NPL>(P, q, lst[w], lane)) hits |= 1u << k;
    }
    if (lane == 0 && hits) D[c] = fine ? (uint8_t)(D[c] | hits) : (uint8_t)0xff;
  }
}

// The listed queries by halving, one voxel of an entry at a time (entries as
// for k_rc_search).  What it does not take (frames that are no rotations) is
// marked in its entry, from bit kRcRest on, and counted in left.
//
// Queries differ in what they want next (a new query, a part halved, a part
// read) and in how often.  A warp keeps kRcSlots queries in shared memory
// and each turn takes up to 32 that want the same, whatever most of them
// want, so that its lanes are busy and do the same.  8.25M queries at 512^3,
// radii up to 17: 3.6 ms, bound by instruction issue (six halvings and two
// parts read a query); 4.0 with six blocks an SM (spills), 6.7 with whole
// entries bound to a slot (a tail of long ones), 7.7 with a query bound to a
// lane (7 of 32 lanes active), 28.7 by the occupancy tree.
constexpr int kRcSlots = 64;
constexpr int kRcCoverWarps = 4;
enum {
  RC_AXES = 0, RC_C = 9, RC_SE = 12, RC_H = 13, RC_FAR = 16, RC_STATE = 17, RC_AT = 18, RC_PEND = 19, RC_CELL = 21,
  RC_VOXEL = 22, RC_WANT = 23, RC_WORDS = 24
};
enum { RC_NEW, RC_HALVE, RC_READ, RC_DONE };

__global__ void __launch_bounds__(32 * kRcCoverWarps, 5) k_rc_cover(const uint8_t* __restrict__ X,
                                                            const uint16_t* __restrict__ E, int L,
                                                            const int8_t* __restrict__ R, int uniform_r,
                                                            const float4* __restrict__ Q, int qres, int res,
                                                            uint64_t* __restrict__ list,
                                                            const uint32_t* __restrict__ count,
                                                            unsigned long long* __restrict__ next,
                                                            uint32_t* __restrict__ left,
                                                            int fine, uint8_t* __restrict__ D) {
  __shared__ uint32_t slots[kRcCoverWarps][RC_WORDS][kRcSlots];
  __shared__ uint8_t turn[kRcCoverWarps][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t(*S)[kRcSlots] = slots[wid];
  const uint32_t n = *count;
  const int N = 2 * res;
#pragma unroll
  for (int h = 0; h < kRcSlots; h += 32) {
    S[RC_WANT][lane + h] = RC_NEW;
  }
  // every turn takes a voxel, halves a part or reads one, for some query
  for (;;) {
    __syncwarp();
    const uint32_t w0 = S[RC_WANT][lane], w1 = S[RC_WANT][lane + 32];
    uint32_t b0[3], b1[3];
    int most = -1, phase = 0;
#pragma unroll
    for (int p = 0; p < 3; p++) {
      b0[p] = __ballot_sync(0xffffffffu, w0 == p);
      b1[p] = __ballot_sync(0xffffffffu, w1 == p);
      const int c = __popc(b0[p]) + __popc(b1[p]);
      if (c > most) most = c, phase = p;
    }
    if (most == 0) break;
    const uint32_t m0 = phase == 0 ? b0[0] : (phase == 1 ? b0[1] : b0[2]);
    const uint32_t m1 = phase == 0 ? b1[0] : (phase == 1 ? b1[1] : b1[2]);
    const uint32_t below = (1u << lane) - 1u;
    if ((m0 >> lane) & 1u) turn[wid][__popc(m0 & below)] = (uint8_t)lane;
    const int at1 = __popc(m0) + __popc(m1 & below);
    if (((m1 >> lane) & 1u) && at1 < 32) turn[wid][at1] = (uint8_t)(lane + 32);
    __syncwarp();
    if (lane >= most) continue;
    const int i = turn[wid][lane];
    const uint32_t on = most >= 32 ? 0xffffffffu : (1u << most) - 1u;
    RcQuery q;
    RcCover v;
    int verdict = -1;
    if (phase != RC_NEW) {
      float* axes[3] = {q.bx, q.by, q.bz};
#pragma unroll
      for (int j = 0; j < 9; j++) axes[j / 3][j % 3] = __uint_as_float(S[RC_AXES + j][i]);
#pragma unroll
      for (int j = 0; j < 3; j++) {
        q.c[j] = __uint_as_float(S[RC_C + j][i]);
        v.H[j] = __uint_as_float(S[RC_H + j][i]);
      }
      q.se = __uint_as_float(S[RC_SE][i]);
      v.far = __uint_as_float(S[RC_FAR][i]);
      const uint32_t st = S[RC_STATE][i];
      v.depth = st & 0xff;
      v.rule = (st >> 8) & 1;
      v.level = st >> 16;
      v.at = S[RC_AT][i];
      v.pending = S[RC_PEND][i] | ((uint64_t)S[RC_PEND + 1][i] << 32);
      int r;
      if (phase == RC_HALVE) r = rc_halve(E, N, q, v);
      else r = rc_read(X, res, L, q, v) ? 1 : 0;
      if (r == 1) verdict = 1;
      else if (r == 0 && !rc_next(v)) verdict = 0;
      if (verdict < 0) {
        S[RC_STATE][i] = (st & 0xffffu) | ((uint32_t)v.level << 16);
        S[RC_AT][i] = v.at;
        S[RC_PEND][i] = (uint32_t)v.pending;
        S[RC_PEND + 1][i] = (uint32_t)(v.pending >> 32);
        S[RC_WANT][i] = v.level == v.depth ? RC_READ : RC_HALVE;
      } else {
        if (verdict) {
          const uint32_t c = S[RC_CELL][i];
          if (fine) atomicOr(reinterpret_cast<uint32_t*>(D) + (c >> 2), 1u << (8 * (c & 3u) + S[RC_VOXEL][i]));
          else D[c] = 0xff;
        }
        S[RC_WANT][i] = RC_NEW;
      }
    } else {
      unsigned long long id = 0;  // voxel (fine) or entry
      if (lane == 0) id = atomicAdd(next, (unsigned long long)__popc(on));
      id = __shfl_sync(on, id, 0) + lane;
      const unsigned long long entry = fine ? id >> 3 : id;
      const int k = fine ? (int)(id & 7u) : 0;
      if (entry >= n) {
        S[RC_WANT][i] = RC_DONE;
        continue;
      }
      const uint64_t ent = list[entry];
      if ((ent >> k) & 1u) {
        const uint32_t c = (uint32_t)(ent >> 8);
        const int x = (int)(c % res), y = (int)((c / res) % res), z = (int)(c / ((uint32_t)res * res));
        rc_query(q, R, uniform_r, Q, qres, res, x, y, z, k, fine);
        if (rc_is_rotation(q)) {
          rc_begin(q, v);
          const float* axes[3] = {q.bx, q.by, q.bz};
#pragma unroll
          for (int j = 0; j < 9; j++) S[RC_AXES + j][i] = __float_as_uint(axes[j / 3][j % 3]);
#pragma unroll
          for (int j = 0; j < 3; j++) {
            S[RC_C + j][i] = __float_as_uint(q.c[j]);
            S[RC_H + j][i] = __float_as_uint(v.H[j]);
          }
          S[RC_SE][i] = __float_as_uint(q.se);
          S[RC_FAR][i] = __float_as_uint(v.far);
          S[RC_STATE][i] = (uint32_t)v.depth | (v.rule ? 0x100u : 0u);
          S[RC_AT][i] = 0;
          S[RC_PEND][i] = 0;
          S[RC_PEND + 1][i] = 0;
          S[RC_CELL][i] = c;
          S[RC_VOXEL][i] = (uint32_t)k;
          S[RC_WANT][i] = RC_HALVE;
        } else {
          atomicOr(reinterpret_cast<unsigned long long*>(list + entry), 1ull << (kRcRest + k));
          atomicAdd(left, 1u);
        }
      }
    }
  }
}

int ilog2_exact(int v) {
  int l = 0;
  while ((1 << l) < v) l++;
  return (1 << l) == v ? l : -1;
}

}  // namespace

// occupancy levels 1..L (contiguous), the tag list (u32 per cell) and the
// search list (u64 per cell), with their counters
size_t rotcube_scratch_bytes(int res) {
  const size_t cells = (size_t)res * res * res;
  const size_t up = (cells - 1) / 7;  // sum of (res >> l)^3, l = 1..L
  return ((up + 255) & ~(size_t)255) + 256 + ((4 * cells + 255) & ~(size_t)255) + 8 * cells;
}

cudaError_t launch_rotcube_dilation(const RotCubeArgs& a, cudaStream_t st, KernelCounter* kc) {
  const int res = a.res;
  const int L = ilog2_exact(res);
  if (L < 1 || L + 1 > kRotCubeMaxLevels || a.qres < 1 || !a.X || !a.Q || !a.D || !a.scratch)
    return cudaErrorInvalidValue;
  const size_t cells = (size_t)res * res * res;
  RcLevels P{};
  P.L = L;
  P.X = a.X;
  P.up = a.scratch;
  uint8_t* p = a.scratch + (((cells - 1) / 7 + 255) & ~(size_t)255);
  uint32_t* counts = reinterpret_cast<uint32_t*>(p);  // [0] tags, [1] search list, [2 .. 5] search
  p += 256;
  uint32_t* tags = reinterpret_cast<uint32_t*>(p);
  p += (4 * cells + 255) & ~(size_t)255;
  uint64_t* list = reinterpret_cast<uint64_t*>(p);
  // the distance field of the shortcuts first (launch_edt uses the
  // scratch region as its own temporaries): saturated at (re + 1)^2, with
  // re >= every radius (hits are decided below r^2) and, up to 127, beyond
  // the largest miss bound
  if (a.E) {
    // the largest miss bound M2 is (sqrt(3) (rmax + sqrt(3) / 2) + 0.01)^2
    int re = (int)(1.7321f * (float)a.rmax) + 3;
    if (re > 127) re = 127;
    if (re < a.rmax) return cudaErrorInvalidValue;
    cudaError_t e = launch_edt(a.X, res, re, a.edt_workspace, a.E, st, kc);
    if (e != cudaSuccess) return e;
  }
  for (int l = 1; l <= L; l++) {
    const int nf = res >> (l - 1);
    const int64_t nt = (int64_t)(nf / 2) * (nf / 2) * (nf / 2);
    int b = (int)((nt + 255) / 256);
    if (b > 152 * 16) b = 152 * 16;
    GM_LAUNCH(kc, "k_rc_occ_up", st,
              k_rc_occ_up<<<b, 256, 0, st>>>(P.level_host(l - 1), nf, const_cast<uint8_t*>(P.level_host(l))));
  }
  const float4* Q = reinterpret_cast<const float4*>(a.Q);
  const int sms = a.num_sms > 0 ? a.num_sms : 152;
  const int grid = sms * 8;
  // the listed queries: by the distance field, then by the occupancy tree
  // what that leaves (four nodes per round measured faster than one, two or
  // eight: breadth pays, up to the 32 lanes)
  auto search = [&](int fine) {
    uint32_t *left = counts + 4, *next = counts + 5;
    unsigned long long* next_voxel = reinterpret_cast<unsigned long long*>(counts + 2);
    cudaMemsetAsync(next_voxel, 0, 4 * sizeof(uint32_t), st);
    if (a.E)
      GM_LAUNCH(kc, "k_rc_cover", st,
                k_rc_cover<<<sms * 5, 32 * kRcCoverWarps, 0, st>>>(a.X, a.E, L, a.R, a.uniform_r, Q, a.qres, res, list,
                                                           counts + 1, next_voxel, left, fine, a.D));
    GM_LAUNCH(kc, "k_rc_search", st,
              k_rc_search<4><<<sms * 2, kRcThreads, 0, st>>>(P, a.R, a.uniform_r, Q, a.qres, res, list, counts + 1,
                                                             next, a.E ? left : nullptr, fine, a.D));
  };
  cudaMemsetAsync(counts, 0, 2 * sizeof(uint32_t), st);
  if (a.mode == 0) {
    GM_LAUNCH(kc, "k_rc_base_cls", st,
              k_rc_base_cls<<<grid, kRcThreads, 0, st>>>(a.X, a.E, a.R, a.uniform_r, Q, a.qres, res, a.data_res[0],
                                                         a.data_res[1], a.data_res[2], a.D, list, counts + 1));
    search(0);
    GM_LAUNCH(kc, "k_rc_tag", st, k_rc_tag<<<grid, kRcThreads, 0, st>>>(a.D, res, tags, counts));
    cudaMemsetAsync(counts + 1, 0, sizeof(uint32_t), st);
    GM_LAUNCH(kc, "k_rc_fine_cls", st,
              k_rc_fine_cls<<<grid, kRcThreads, 0, st>>>(a.E, a.R, a.uniform_r, Q, a.qres, res, tags, counts, a.D,
                                                         list, counts + 1));
  } else {
    GM_LAUNCH(kc, "k_rc_fine_cls", st,
              k_rc_fine_cls<<<grid, kRcThreads, 0, st>>>(a.E, a.R, a.uniform_r, Q, a.qres, res, nullptr, counts,
                                                         a.D, list, counts + 1));
  }
  search(1);
  return cudaGetLastError();
}

}  // namespace gm
