// voxelize.cu — conservative solid voxelization into the packed grid
// (reference row a2: Voxelizer::VoxelizeConservative, VoxelizeVolume,
// VoxelizeSurfaceConservative, ConvertBucketToPacketGrid;
// GMorpho/Voxelizer.cu:594-849 and the shaders vol_vox_bit.frag:35-51,
// surf_vox_conserv.geo:41-122, surf_vox_conserv_bit.frag:35-47).
//
// The reference rasterises with OpenGL (parity fill at pixel centres plus
// NVIDIA conservative rasterisation).  Here both passes are CUDA kernels
// with a precise definition (double precision, no contraction; computed in
// single precision where that decides the same):
//   (i)  volume: a triangle covers pixel (x, y) when the pixel centre is
//        inside its xy projection (top-left rule on edges); it flips every
//        voxel of that column at or below floor(z at the centre);
//   (ii) surface: every voxel whose closed box meets the triangle
//        (separating-axis test) is set; triangles with squared aspect ratio
//        >= 50^2 are skipped as the geometry shader does (Voxelizer.cu:680).
// Both passes work on z-word bit grids (32 consecutive z per uint32, the
// reference's GL bucket layout), which are then packed into 2x2x2 bytes.
#include "gm_common.cuh"
#include "gm_internal.h"

namespace gm {

constexpr int64_t kVoxChunk = 1 << 24;  // triangles per launch (bounds the list)

// the two z-word grids, the two list counts, the triangle list
size_t voxelize_scratch_bytes(int res, int64_t triangles) {
  const size_t N = 2 * (size_t)res;
  const int64_t n = triangles < 0 ? 0 : (triangles < kVoxChunk ? triangles : kVoxChunk);
  return 2 * (N * N * N / 8) + 512 + sizeof(uint32_t) * (size_t)n;
}

// What the kernels share: the grid (N fine voxels per axis, its corner, the
// voxel size and its two-float reciprocal) and the two z-word grids.
struct VoxParams {
  int N;
  float b[3];
  double h;
  float ih, il;
  uint32_t *mark, *surf;
};

__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }

__device__ __forceinline__ bool edge_covers(double ax, double ay, double bx, double by, double px, double py) {
  const double w = dsub(dmul(dsub(bx, ax), dsub(py, ay)), dmul(dsub(by, ay), dsub(px, ax)));
  if (w > 0) return true;
  if (w < 0) return false;
  const double ex = dsub(bx, ax), ey = dsub(by, ay);
  return (ey == 0 && ex < 0) || (ey < 0);
}

__device__ bool tri_box_overlap(const double c[3], double half, const double v0[3], const double v1[3],
                                const double v2[3]) {
  double a[3], b[3], d[3];
  for (int i = 0; i < 3; i++) {
    a[i] = dsub(v0[i], c[i]);
    b[i] = dsub(v1[i], c[i]);
    d[i] = dsub(v2[i], c[i]);
  }
  for (int ax = 0; ax < 3; ax++) {
    const double mn = fmin(a[ax], fmin(b[ax], d[ax])), mx = fmax(a[ax], fmax(b[ax], d[ax]));
    if (mn > half || mx < -half) return false;
  }
  double e[3][3];
  for (int i = 0; i < 3; i++) {
    e[0][i] = dsub(b[i], a[i]);
    e[1][i] = dsub(d[i], b[i]);
    e[2][i] = dsub(a[i], d[i]);
  }
  const double nrm[3] = {dsub(dmul(e[0][1], e[1][2]), dmul(e[0][2], e[1][1])),
                         dsub(dmul(e[0][2], e[1][0]), dmul(e[0][0], e[1][2])),
                         dsub(dmul(e[0][0], e[1][1]), dmul(e[0][1], e[1][0]))};
  const double dd = dadd(dadd(dmul(nrm[0], a[0]), dmul(nrm[1], a[1])), dmul(nrm[2], a[2]));
  const double rr = dmul(half, dadd(dadd(fabs(nrm[0]), fabs(nrm[1])), fabs(nrm[2])));
  if (dd > rr || dd < -rr) return false;
  const double* vv[3] = {a, b, d};
  for (int i = 0; i < 3; i++)
    for (int j = 0; j < 3; j++) {
      double ax[3] = {0, 0, 0};
      if (j == 0) { ax[1] = -e[i][2]; ax[2] = e[i][1]; }
      if (j == 1) { ax[0] = e[i][2]; ax[2] = -e[i][0]; }
      if (j == 2) { ax[0] = -e[i][1]; ax[1] = e[i][0]; }
      double p[3];
      for (int k = 0; k < 3; k++) p[k] = dadd(dadd(dmul(ax[0], vv[k][0]), dmul(ax[1], vv[k][1])), dmul(ax[2], vv[k][2]));
      const double mn = fmin(p[0], fmin(p[1], p[2])), mx = fmax(p[0], fmax(p[1], p[2]));
      const double r = dmul(half, dadd(dadd(fabs(ax[0]), fabs(ax[1])), fabs(ax[2])));
      if (mn > r || mx < -r) return false;
    }
  return true;
}

// The general form of both passes for one triangle in double precision, and
// what defines the result.  The column (x, y) of pixel tests and the voxel
// tests are separate calls: the float form below asks for them one at a
// time, the exact kernel runs over all of them.
struct TriD {
  double g[3][3];  // vertices in voxels
};

__device__ __forceinline__ void tri_load(const float* __restrict__ P, const uint32_t* __restrict__ T, uint32_t t,
                                         const VoxParams& vp, TriD& d) {
  for (int j = 0; j < 3; j++)
    for (int a = 0; a < 3; a++)
      d.g[j][a] = __ddiv_rn(dsub((double)P[3 * (size_t)T[3 * (size_t)t + j] + a], (double)vp.b[a]), vp.h);
}

// (i) volume parity: pixel (x, y) flips the voxel at floor(z) of its centre
__device__ void pixel_exact(const TriD& d, int x, int y, const VoxParams& vp) {
  const double(*g)[3] = d.g;
  double area = dsub(dmul(dsub(g[1][0], g[0][0]), dsub(g[2][1], g[0][1])),
                     dmul(dsub(g[1][1], g[0][1]), dsub(g[2][0], g[0][0])));
  if (!(area != 0)) return;
  int o1 = 1, o2 = 2;
  if (area < 0) { o1 = 2; o2 = 1; area = -area; }
  const double* A = g[0];
  const double* B = g[o1];
  const double* Cc = g[o2];
  const double px = x + 0.5, py = y + 0.5;
  if (!edge_covers(A[0], A[1], B[0], B[1], px, py)) return;
  if (!edge_covers(B[0], B[1], Cc[0], Cc[1], px, py)) return;
  if (!edge_covers(Cc[0], Cc[1], A[0], A[1], px, py)) return;
  const double wa = dsub(dmul(dsub(B[0], px), dsub(Cc[1], py)), dmul(dsub(B[1], py), dsub(Cc[0], px)));
  const double wb = dsub(dmul(dsub(Cc[0], px), dsub(A[1], py)), dmul(dsub(Cc[1], py), dsub(A[0], px)));
  const double wc = dsub(dsub(area, wa), wb);
  const double z = __ddiv_rn(dadd(dadd(dmul(wa, A[2]), dmul(wb, B[2])), dmul(wc, Cc[2])), area);
  int k = (int)floor(z);
  if (k < 0) return;
  if (k > vp.N - 1) k = vp.N - 1;
  atomicXor(vp.mark + ((int64_t)x + (int64_t)vp.N * y) * (vp.N >> 5) + (k >> 5), 1u << (k & 31));
}

// pixels that the volume pass looks at (a cover of the triangle's projection)
__device__ void pixel_range(const TriD& d, int N, int& x0, int& x1, int& y0, int& y1) {
  const double(*g)[3] = d.g;
  const double mnx = fmin(g[0][0], fmin(g[1][0], g[2][0])), mxx = fmax(g[0][0], fmax(g[1][0], g[2][0]));
  const double mny = fmin(g[0][1], fmin(g[1][1], g[2][1])), mxy = fmax(g[0][1], fmax(g[1][1], g[2][1]));
  x0 = max((int)floor(mnx - 0.5), 0), x1 = min((int)ceil(mxx - 0.5), N - 1);
  y0 = max((int)floor(mny - 0.5), 0), y1 = min((int)ceil(mxy - 0.5), N - 1);
}

// (ii) conservative surface: not for triangles of squared aspect ratio >= 50^2
__device__ bool surface_wanted(const TriD& d) {
  const double(*g)[3] = d.g;
  double d0[3], d1[3], d2[3];
  for (int a = 0; a < 3; a++) {
    d0[a] = dsub(g[0][a], g[1][a]);
    d1[a] = dsub(g[1][a], g[2][a]);
    d2[a] = dsub(g[2][a], g[0][a]);
  }
  const double l0 = dadd(dadd(dmul(d0[0], d0[0]), dmul(d0[1], d0[1])), dmul(d0[2], d0[2]));
  const double l1 = dadd(dadd(dmul(d1[0], d1[0]), dmul(d1[1], d1[1])), dmul(d1[2], d1[2]));
  const double l2 = dadd(dadd(dmul(d2[0], d2[0]), dmul(d2[1], d2[1])), dmul(d2[2], d2[2]));
  double maxl2 = l0 > l1 ? l0 : l1;
  if (l2 > maxl2) maxl2 = l2;
  const double cx = dsub(dmul(d0[1], d2[2]), dmul(d0[2], d2[1]));
  const double cy = dsub(dmul(d0[2], d2[0]), dmul(d0[0], d2[2]));
  const double cz = dsub(dmul(d0[0], d2[1]), dmul(d0[1], d2[0]));
  const double a2 = dadd(dadd(dmul(cx, cx), dmul(cy, cy)), dmul(cz, cz));
  return a2 > 0 && __ddiv_rn(dmul(maxl2, maxl2), a2) < 2500.0;
}

// voxels whose closed box [x, x + 1] meets [mn, mx] on every axis:
// ceil(mn) - 1 <= x <= floor(mx) (the box test of tri_box_overlap, so the
// voxels outside could not pass it)
__device__ void voxel_range(const TriD& d, int N, int lo[3], int hi[3]) {
  const double(*g)[3] = d.g;
  for (int a = 0; a < 3; a++) {
    const double mn = fmin(g[0][a], fmin(g[1][a], g[2][a])), mx = fmax(g[0][a], fmax(g[1][a], g[2][a]));
    lo[a] = max((int)ceil(mn) - 1, 0);
    hi[a] = min((int)floor(mx), N - 1);
  }
}

__device__ __forceinline__ bool voxel_exact(const TriD& d, int x, int y, int z) {
  const double c[3] = {x + 0.5, y + 0.5, z + 0.5};
  return tri_box_overlap(c, 0.5, d.g[0], d.g[1], d.g[2]);
}

__device__ __forceinline__ uint32_t* zword(uint32_t* g, int N, int x, int y) {
  return g + ((int64_t)x + (int64_t)N * y) * (N >> 5);
}

// What the float form cannot decide (rare: out of line)
__device__ __noinline__ void ask_pixel(const float* __restrict__ P, const uint32_t* __restrict__ T, uint32_t t, int x,
                                       int y, const VoxParams& vp) {
  TriD d;
  tri_load(P, T, t, vp, d);
  int x0, x1, y0, y1;
  pixel_range(d, vp.N, x0, x1, y0, y1);
  if (x >= x0 && x <= x1 && y >= y0 && y <= y1) pixel_exact(d, x, y, vp);
}

__device__ __noinline__ void ask_voxels(const float* __restrict__ P, const uint32_t* __restrict__ T, uint32_t t, int x,
                                        int y, int z0, int z1, const VoxParams& vp) {
  TriD d;
  tri_load(P, T, t, vp, d);
  int lo[3], hi[3];
  voxel_range(d, vp.N, lo, hi);
  if (x < lo[0] || x > hi[0] || y < lo[1] || y > hi[1]) return;
  for (int z = max(z0, lo[2]); z <= min(z1, hi[2]); z++)
    if (voxel_exact(d, x, y, z)) atomicOr(zword(vp.surf, vp.N, x, y) + (z >> 5), 1u << (z & 31));
}

// Such tests of a warp's walks, kept for the end, where its lanes make them
// together: a test takes microseconds at the rate of FP64 here, and the warp
// waited for each of them: 42 -> 34 us for 82k triangles into 128^3, and
// 84 where one warp had many.
constexpr uint32_t kAsks = 32;
constexpr int kVoxThreads = 64;
struct Asks {
  uint32_t n;
  uint4 q[kAsks];  // triangle, x | y << 16, first and last z; first z -1: the column's pixel
};
__device__ __forceinline__ void make_ask(const float* __restrict__ P, const uint32_t* __restrict__ T, uint4 a,
                                         const VoxParams& vp) {
  const int x = (int)(a.y & 0xffffu), y = (int)(a.y >> 16);
  if ((int)a.z < 0) ask_pixel(P, T, a.x, x, y, vp);
  else ask_voxels(P, T, a.x, x, y, (int)a.z, (int)a.w, vp);
}
__device__ __forceinline__ Asks& warp_asks() {
  __shared__ Asks asks[kVoxThreads / 32];
  return asks[threadIdx.x >> 5];
}
// (KEEP false: at once)
template <bool KEEP>
__device__ __forceinline__ void ask(const float* __restrict__ P, const uint32_t* __restrict__ T, uint32_t t, int x,
                                    int y, int z0, int z1, const VoxParams& vp) {
  const uint4 a = make_uint4(t, (uint32_t)x | ((uint32_t)y << 16), (uint32_t)z0, (uint32_t)z1);
  const uint32_t i = KEEP ? atomicAdd(&warp_asks().n, 1u) : kAsks;
  if (i < kAsks) warp_asks().q[i] = a;
  else make_ask(P, T, a, vp);
}

__device__ __noinline__ bool ask_surface(const float* __restrict__ P, const uint32_t* __restrict__ T, uint32_t t,
                                         const VoxParams& vp) {
  TriD d;
  tri_load(P, T, t, vp, d);
  return surface_wanted(d);
}

// ---- the float form
//
// Each separating-axis test of a voxel (centre c) reads L <= axis . c <= H:
// a slab.  In single precision, with coordinates relative to the triangle's
// own corner and a bound eps on everything that was rounded, a slab says in,
// out or undecided; and along a column of voxels (x, y fixed) each slab is
// an interval of z.  So a column costs ten slabs whatever its length: the
// three xy slabs decide it, the intersection of the other seven intervals is
// set as whole words, and only the voxels between the shrunk and the grown
// interval (about one column in 10^5) are asked in double precision.  The
// vertices' coordinates are computed as a pair of floats (46 bits), so no
// double arithmetic is left on the common path: FP64 issues at 1/64 of the
// FP32 rate here and was what bounded the voxelizer (115 ms for 4.0M
// triangles into 1024^3, 1.94 ms for 82k into 128^3; k_vox_tris: 0.84 and
// 0.034 ms).
struct Slab {
  // z interval at the column coordinate u: [lo - k u, hi - k u], rounding
  // within w; a slab that hardly depends on z (flat) is a test of k u
  // against [lo, hi] instead
  float lo, hi, k, w;
};

struct ZRange {
  float dlo, dhi, plo, phi;  // decided inside / possibly inside (centres)
};

struct TriF {
  int o[3];              // origin (voxels)
  int lo[3], hi[3];      // possible voxels, clamped to the grid
  int dlo[2], dhi[2];    // columns that are decided to be inside the box in x, y
  int zdlo, zdhi;
  float ax[3], ay[3], L[3], H[3], W[3], exy;  // xy slabs; W: the edge's own value; eps
  Slab yz[3], xz[3], pl;
  float pky;             // the plane's y coefficient (pl.k: x)
  float pz0, pzw;        // z of the plane at the origin column and its rounding
  uint32_t flat;         // bit i: yz, 3 + i: xz, 6: plane
  bool surf, steep;      // steep: no usable z of the plane
};

__device__ __forceinline__ float min3(float a, float b, float c) { return fminf(a, fminf(b, c)); }
__device__ __forceinline__ float max3(float a, float b, float c) { return fmaxf(a, fmaxf(b, c)); }

// slab of axis . c = cu u + cz z in [L, H] with rounding eps; zext: extent
// of z over the triangle
__device__ __forceinline__ bool make_slab(float L, float H, float cu, float cz, float eps, float zext, Slab& s) {
  if (fabsf(cz) < 64.f * eps) {  // flat
    s = Slab{L, H, cu, eps + fabsf(cz) * zext};
    return true;
  }
  const float inv = 1.f / cz;
  const float a = L * inv, b = H * inv;
  s = Slab{fminf(a, b), fmaxf(a, b), cu * inv, eps * fabsf(inv)};
  return false;
}

// false: out
__device__ __forceinline__ bool cut(ZRange& r, const Slab& s, float ku, bool flat) {
  if (flat) {
    if (ku < s.lo - s.w || ku > s.hi + s.w) return false;
    if (ku < s.lo + s.w || ku > s.hi - s.w) r.dhi = -1e30f;  // undecided
    return true;
  }
  const float a = s.lo - ku, b = s.hi - ku;
  r.dlo = fmaxf(r.dlo, a + s.w);
  r.dhi = fminf(r.dhi, b - s.w);
  r.plo = fmaxf(r.plo, a - s.w);
  r.phi = fminf(r.phi, b + s.w);
  return r.plo <= r.phi;
}

enum TriClass { TRI_FLOAT = 0, TRI_EXACT = 1 };

// The float form of a triangle.  TRI_EXACT: outside its range (coordinates
// of 4096 voxels or more or not finite, a degenerate size).
__device__ __forceinline__ TriClass tri_setup(const float* __restrict__ P, const uint32_t* __restrict__ T, uint32_t t,
                                              const VoxParams& vp, TriF& f) {
  float p[3][3], q[3][3], v[3][3], e[3][3];
  bool ok = true;
#pragma unroll
  for (int j = 0; j < 3; j++) {
    const float* src = P + 3 * (size_t)T[3 * (size_t)t + j];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      // (P - b) / h as a pair of floats: an exact two-float difference times
      // the two-float reciprocal of h
      const float x = src[a], b = vp.b[a];
      const float s = __fsub_rn(x, b), bb = __fsub_rn(s, x);
      const float r = __fadd_rn(__fsub_rn(x, __fsub_rn(s, bb)), -__fadd_rn(b, bb));
      const float m = __fmul_rn(s, vp.ih);
      p[j][a] = m;
      q[j][a] = fmaf(s, vp.ih, -m) + fmaf(s, vp.il, r * vp.ih);
      ok = ok && fabsf(m) < 4096.f;
    }
  }
  if (!ok) return TRI_EXACT;
  float mn[3], mx[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const float o = floorf(min3(p[0][a], p[1][a], p[2][a]));
    f.o[a] = (int)o;
#pragma unroll
    for (int j = 0; j < 3; j++) {
      v[j][a] = (p[j][a] - o) + q[j][a];
      const int k = j == 2 ? 0 : j + 1;
      e[j][a] = (p[k][a] - p[j][a]) + (q[k][a] - q[j][a]);
    }
    mn[a] = min3(v[0][a], v[1][a], v[2][a]);
    mx[a] = max3(v[0][a], v[1][a], v[2][a]);
  }
  const float S = max3(mx[0] - mn[0], mx[1] - mn[1], mx[2] - mn[2]) + 2.f;  // bounds every local coordinate
  const float ec = S * 1.2e-7f + 1e-9f;
  const int N = vp.N;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    f.lo[a] = max(f.o[a] + (int)ceilf(mn[a] - ec) - 1, 0);
    f.hi[a] = min(f.o[a] + (int)floorf(mx[a] + ec), N - 1);
    const int dl = f.o[a] + (int)ceilf(mn[a] + ec) - 1, dh = f.o[a] + (int)floorf(mx[a] - ec);
    if (a < 2) f.dlo[a] = dl, f.dhi[a] = dh;
    else f.zdlo = dl, f.zdhi = dh;
  }
  float l2 = 0.f;
#pragma unroll
  for (int i = 0; i < 3; i++) l2 = fmaxf(l2, e[i][0] * e[i][0] + e[i][1] * e[i][1] + e[i][2] * e[i][2]);
  if (l2 < 1e-8f) return TRI_EXACT;
  const float n[3] = {e[0][1] * e[1][2] - e[0][2] * e[1][1], e[0][2] * e[1][0] - e[0][0] * e[1][2],
                      e[0][0] * e[1][1] - e[0][1] * e[1][0]};
  const float n2 = n[0] * n[0] + n[1] * n[1] + n[2] * n[2];
  f.surf = l2 * l2 < 2500.f * n2;
  if (l2 * l2 > 2475.f * n2 && l2 * l2 < 2525.f * n2) f.surf = ask_surface(P, T, t, vp);  // at the limit
  const float zext = S;
  const float ep = S * (l2 * 2e-6f + 2e-10f);  // plane
  f.flat = 0;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    // axes e x unit: (0, -e2, e1), (e2, 0, -e0), (-e1, e0, 0); an axis that
    // vanishes (an edge along the unit) separates nothing
    const float e0 = e[i][0], e1 = e[i][1], e2 = e[i][2];
    const float a0 = fabsf(e0), a1 = fabsf(e1), a2 = fabsf(e2);
    {
      const float q0 = e1 * v[0][2] - e2 * v[0][1], q1 = e1 * v[1][2] - e2 * v[1][1], q2 = e1 * v[2][2] - e2 * v[2][1];
      const float r = a1 + a2 > 0.f ? 0.5f * (a1 + a2) : 1e30f, eps = S * ((a1 + a2) * 1e-6f + 2e-10f);
      if (make_slab(min3(q0, q1, q2) - r, max3(q0, q1, q2) + r, -e2, e1, eps, zext, f.yz[i])) f.flat |= 1u << i;
    }
    {
      const float q0 = e2 * v[0][0] - e0 * v[0][2], q1 = e2 * v[1][0] - e0 * v[1][2], q2 = e2 * v[2][0] - e0 * v[2][2];
      const float r = a0 + a2 > 0.f ? 0.5f * (a0 + a2) : 1e30f, eps = S * ((a0 + a2) * 1e-6f + 2e-10f);
      if (make_slab(min3(q0, q1, q2) - r, max3(q0, q1, q2) + r, e2, -e0, eps, zext, f.xz[i])) f.flat |= 8u << i;
    }
    {
      const float q0 = e0 * v[0][1] - e1 * v[0][0], q1 = e0 * v[1][1] - e1 * v[1][0], q2 = e0 * v[2][1] - e1 * v[2][0];
      const float r = a0 + a1 > 0.f ? 0.5f * (a0 + a1) : 1e30f;
      f.ax[i] = -e1, f.ay[i] = e0;
      f.L[i] = min3(q0, q1, q2) - r, f.H[i] = max3(q0, q1, q2) + r;
      f.W[i] = i == 0 ? q0 : (i == 1 ? q1 : q2);
    }
  }
  f.exy = S * ((max3(fabsf(e[0][0]), fabsf(e[1][0]), fabsf(e[2][0])) +
                max3(fabsf(e[0][1]), fabsf(e[1][1]), fabsf(e[2][1]))) * 1e-6f + 2e-10f);
  const float D = n[0] * v[0][0] + n[1] * v[0][1] + n[2] * v[0][2];
  const float r = 0.5f * (fabsf(n[0]) + fabsf(n[1]) + fabsf(n[2]));
  f.pky = n[1];
  if (make_slab(D - r, D + r, n[0], n[2], ep, zext, f.pl)) {
    f.flat |= 64u;
    f.steep = true;
    f.pz0 = f.pzw = 0.f;
  } else {
    const float inv = 1.f / n[2];
    f.pky *= inv;
    f.pz0 = D * inv;
    // beside this form's rounding, that of the double form's interpolation
    f.pzw = (ep + 1e-9f * S * S) * fabsf(inv);
    f.steep = false;
  }
  return TRI_FLOAT;
}

// One column of a triangle: parity pixel and surface voxels
template <bool KEEP>
__device__ __forceinline__ void tri_column(const float* __restrict__ P, const uint32_t* __restrict__ T, uint32_t t,
                                           const VoxParams& vp, const TriF& f, int x, int y, ZRange zr, bool zy_in) {
  const int N = vp.N;
  const float X = (float)(x - f.o[0]) + 0.5f, Y = (float)(y - f.o[1]) + 0.5f;
  bool in = zy_in && x >= f.dlo[0] && x <= f.dhi[0] && y >= f.dlo[1] && y <= f.dhi[1], out = !f.surf;
  float wmin = 1e30f, wmax = -1e30f;
#pragma unroll
  for (int i = 0; i < 3; i++) {
    const float s = fmaf(f.ax[i], X, f.ay[i] * Y);
    out |= s < f.L[i] - f.exy || s > f.H[i] + f.exy;
    in = in && s > f.L[i] + f.exy && s < f.H[i] - f.exy;
    const float w = s - f.W[i];  // the pixel centre's side of edge i
    wmin = fminf(wmin, w);
    wmax = fmaxf(wmax, w);
  }
  // (i) parity.  Sides of both signs: outside; one sign: inside
  if (!(wmin < -f.exy && wmax > f.exy)) {
    bool sure = wmin > f.exy || wmax < -f.exy;
    int k = 0;
    if (sure && !f.steep) {
      const float z = f.pz0 - fmaf(f.pl.k, X, f.pky * Y);
      const float k0 = floorf(z - f.pzw), k1 = floorf(z + f.pzw);
      sure = k0 == k1;
      k = f.o[2] + (int)k0;
    } else {
      sure = false;
    }
    if (sure) {
      if (k >= 0) {
        k = min(k, N - 1);
        atomicXor(zword(vp.mark, N, x, y) + (k >> 5), 1u << (k & 31));
      }
    } else {
      ask<KEEP>(P, T, t, x, y, -1, -1, vp);
    }
  }
  // (ii) surface
  if (out || zr.plo > zr.phi) return;
#pragma unroll
  for (int i = 0; i < 3; i++)
    if (!cut(zr, f.xz[i], f.xz[i].k * X, (f.flat >> (3 + i)) & 1u)) return;
  if (!cut(zr, f.pl, fmaf(f.pl.k, X, f.pky * Y), (f.flat >> 6) & 1u)) return;
  const int p0 = max(f.o[2] + (int)ceilf(fminf(fmaxf(zr.plo, -1.f), 8192.f) - 0.5f), f.lo[2]);
  const int p1 = min(f.o[2] + (int)floorf(fmaxf(fminf(zr.phi, 8192.f), -2.f) - 0.5f), f.hi[2]);
  if (p0 > p1) return;
  int d0 = p1 + 1, d1 = p1;  // decided voxels
  if (in && zr.dlo <= zr.dhi) {
    d0 = max(max(f.o[2] + (int)ceilf(fminf(fmaxf(zr.dlo, -1.f), 8192.f) - 0.5f), f.zdlo), p0);
    d1 = min(min(f.o[2] + (int)floorf(fmaxf(fminf(zr.dhi, 8192.f), -2.f) - 0.5f), f.zdhi), p1);
    if (d0 > d1) d0 = p1 + 1, d1 = p1;
  }
  uint32_t* col = zword(vp.surf, N, x, y);
  for (int z = d0; z <= d1;) {
    const int w = z >> 5, last = min(d1, 32 * w + 31);
    atomicOr(col + w, (0xffffffffu >> (31 - (last - z))) << (z & 31));
    z = last + 1;
  }
  if (d0 > p0) ask<KEEP>(P, T, t, x, y, p0, min(d0 - 1, p1), vp);
  if (d0 <= d1 && d1 < p1) ask<KEEP>(P, T, t, x, y, d1 + 1, p1, vp);
}

// z interval of the yz slabs of a row of columns; false: no voxel passes
// them (the row's pixels are still to be tested)
__device__ __forceinline__ bool tri_row(const TriF& f, int y, ZRange& zr) {
  const float Y = (float)(y - f.o[1]) + 0.5f;
  zr = ZRange{-1e30f, 1e30f, -1e30f, 1e30f};
#pragma unroll
  for (int i = 0; i < 3; i++)
    if (!cut(zr, f.yz[i], f.yz[i].k * Y, (f.flat >> i) & 1u)) return false;
  return true;
}

// One thread per triangle of at most kVoxCols columns; larger ones are
// listed from the front, those outside the float form's range from the back
// (counts: [0] large, [1] exact).  Bound by the latency of a warp's longest
// walk (a triangle of a 4.0M-triangle surface in 1024^3 has five columns on
// average, up to a dozen): six blocks of 64 an SM (168 registers, no spills
// to speak of) take 0.84 ms, a third fewer warps 1.00, a third more (128
// registers) 0.95; blocks of 128 were 3 % slower, seven of 64 32 %.
constexpr int kVoxCols = 64;
__global__ void __launch_bounds__(kVoxThreads, 6) k_vox_tris(const float* __restrict__ P, const uint32_t* __restrict__ T,
                                                  uint32_t nf, const __grid_constant__ VoxParams vp,
                                                  uint32_t* __restrict__ list, uint32_t* __restrict__ counts) {
  if ((threadIdx.x & 31) == 0) warp_asks().n = 0;
  __syncwarp();
  const uint32_t t = blockIdx.x * kVoxThreads + threadIdx.x;  // (at most kVoxChunk)
  if (t < nf) {
    TriF f;
    if (tri_setup(P, T, t, vp, f) == TRI_EXACT) {
      list[nf - 1 - atomicAdd(counts + 1, 1u)] = t;
    } else {
      const int nx = f.hi[0] - f.lo[0] + 1, ny = f.hi[1] - f.lo[1] + 1;
      if (nx > 0 && ny > 0 && (nx > kVoxCols || ny > kVoxCols || nx * ny > kVoxCols)) {
        list[atomicAdd(counts, 1u)] = t;
      } else if (nx > 0) {
        for (int y = f.lo[1]; y <= f.hi[1]; y++) {
          ZRange zr;
          const bool zy = tri_row(f, y, zr);
          if (!zy) zr.phi = -1e30f, zr.plo = 1e30f;  // pixels only
          for (int x = f.lo[0]; x <= f.hi[0]; x++) tri_column<true>(P, T, t, vp, f, x, y, zr, zy);
        }
      }
    }
  }
  __syncwarp();
  const uint32_t lane = threadIdx.x & 31;
  if (lane < min(warp_asks().n, kAsks)) make_ask(P, T, warp_asks().q[lane], vp);
}

// One block per listed triangle, its threads over the columns of a large
// one, or over the voxels of one that the float form does not take
__global__ void __launch_bounds__(128) k_vox_listed(const float* __restrict__ P, const uint32_t* __restrict__ T,
                                                    int64_t nf, const __grid_constant__ VoxParams vp,
                                                    const uint32_t* __restrict__ list,
                                                    const uint32_t* __restrict__ counts) {
  const uint32_t n = counts[0], m = counts[1];
  for (uint32_t i = blockIdx.x; i < n; i += gridDim.x) {
    const uint32_t t = list[i];
    TriF f;
    tri_setup(P, T, t, vp, f);
    const int nx = f.hi[0] - f.lo[0] + 1, ny = f.hi[1] - f.lo[1] + 1;
    for (int c = threadIdx.x; c < nx * ny; c += blockDim.x) {
      const int x = f.lo[0] + c % nx, y = f.lo[1] + c / nx;
      ZRange zr;
      const bool zy = tri_row(f, y, zr);
      if (!zy) zr.phi = -1e30f, zr.plo = 1e30f;
      tri_column<false>(P, T, t, vp, f, x, y, zr, zy);
    }
  }
  for (uint32_t i = blockIdx.x; i < m; i += gridDim.x) {
    TriD d;
    tri_load(P, T, list[nf - 1 - i], vp, d);
    int x0, x1, y0, y1;
    pixel_range(d, vp.N, x0, x1, y0, y1);
    const int64_t npix = x1 >= x0 && y1 >= y0 ? (int64_t)(x1 - x0 + 1) * (y1 - y0 + 1) : 0;
    for (int64_t c = threadIdx.x; c < npix; c += blockDim.x)
      pixel_exact(d, x0 + (int)(c % (x1 - x0 + 1)), y0 + (int)(c / (x1 - x0 + 1)), vp);
    if (!surface_wanted(d)) continue;
    int lo[3], hi[3];
    voxel_range(d, vp.N, lo, hi);
    if (lo[0] > hi[0] || lo[1] > hi[1] || lo[2] > hi[2]) continue;
    const int nx = hi[0] - lo[0] + 1, ny = hi[1] - lo[1] + 1;
    const int64_t nvox = (int64_t)nx * ny * (hi[2] - lo[2] + 1);
    for (int64_t c = threadIdx.x; c < nvox; c += blockDim.x) {
      const int x = lo[0] + (int)(c % nx), y = lo[1] + (int)((c / nx) % ny), z = lo[2] + (int)(c / ((int64_t)nx * ny));
      if (voxel_exact(d, x, y, z)) atomicOr(zword(vp.surf, vp.N, x, y) + (z >> 5), 1u << (z & 31));
    }
  }
}

// z-words to packed bytes, 64 columns (32 cells) of two rows y a block.
// With SOLID the words are the volume pass's marks: voxel z of a column is
// set when an odd number of marks sit at or above it, or when its surface
// bit is (an xor scan down the column: within a word by shifts, across the
// words of a column by a ballot of their parities).  The columns' words go
// through shared memory so that both sides are coalesced: words of a column
// in, cells along x out, four cells and 32 z a thread as sixteen 4-byte
// stores; the bits of the four columns of a cell are interleaved two, four
// and eight at a time (34 operations for 16 bytes).  Bound by HBM: at
// 1024^3 it moves 256 MB of words and 128 MB of cells in 0.133 ms, 2.9 TB/s
// (0.167 without the fourfold unrolling that keeps loads in flight); one
// thread per byte, reading eight strided words, took 5.6 ms and the parity
// pass that this includes 0.43 ms.
constexpr int kPackCols = 64;
template <bool SOLID>
__global__ void __launch_bounds__(256) k_pack_columns(const uint32_t* __restrict__ zw,
                                                      const uint32_t* __restrict__ surf, uint8_t* __restrict__ grid,
                                                      int res, int aligned) {
  extern __shared__ uint32_t words[];  // [2][kPackCols][W + 1]
  const int N = 2 * res, W = N >> 5;   // W: a power of two
  const int x0 = blockIdx.x * kPackCols, cy = blockIdx.y;
  const int cols = min(kPackCols, N - x0);
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if (W <= 32) {
    const int total = cols * W;  // words of one row, contiguous; cols >= 32, so a multiple of 32
#pragma unroll 4
    for (int i = wid * 32 + lane; i < 2 * total; i += 256) {
      const int r = i >= total ? 1 : 0, k = i - r * total;
      const int64_t at = ((int64_t)x0 + (int64_t)N * (2 * cy + r)) * W + k;
      uint32_t m = zw[at];
      if (SOLID) {
        m ^= m >> 1;
        m ^= m >> 2;
        m ^= m >> 4;
        m ^= m >> 8;
        m ^= m >> 16;  // bit 0: the word's parity
        const uint32_t par = __ballot_sync(0xffffffffu, m & 1u);
        // the words above this one in its column: lanes up to the end of its group of W
        const uint32_t group = W == 32 ? 0xffffffffu : ((1u << W) - 1u) << (lane & ~(W - 1));
        const uint32_t above = group & ~(0xffffffffu >> (31 - lane));
        m = ((__popc(par & above) & 1) ? ~m : m) | surf[at];
      }
      words[(r * kPackCols + k / W) * (W + 1) + (k & (W - 1))] = m;
    }
  } else {
    for (int c = wid; c < 2 * cols; c += 8) {  // a warp per column, from its top word down
      const int r = c >= cols ? 1 : 0, x = c - r * cols;
      const int64_t at = ((int64_t)(x0 + x) + (int64_t)N * (2 * cy + r)) * W;
      uint32_t carry = 0;  // parity of the marks above
      for (int w = W - 32 + lane; w >= 0; w -= 32) {
        uint32_t m = zw[at + w];
        if (SOLID) {
          m ^= m >> 1;
          m ^= m >> 2;
          m ^= m >> 4;
          m ^= m >> 8;
          m ^= m >> 16;
          const uint32_t par = __ballot_sync(0xffffffffu, m & 1u);
          const uint32_t above = ~(0xffffffffu >> (31 - lane));
          m = (((__popc(par & above) & 1) ^ carry) ? ~m : m) | surf[at + w];
          carry ^= __popc(par) & 1;
        }
        words[(r * kPackCols + x) * (W + 1) + w] = m;
      }
    }
  }
  __syncthreads();
  const int quads = cols >> 3;  // groups of four cells
  for (int i = threadIdx.x; i < quads * W; i += 256) {
    const int g = i % quads, w = i / quads;
    uint32_t out[4][4];  // [k mod 4][cell]: bytes of z pairs k, k + 4, k + 8, k + 12
#pragma unroll
    for (int c = 0; c < 4; c++) {
      const uint32_t* s = words + (8 * g + 2 * c) * (W + 1) + w;
      const uint32_t a = s[0], b = s[W + 1], d = s[kPackCols * (W + 1)], e = s[(kPackCols + 1) * (W + 1)];
      const uint32_t m5 = 0x55555555u, m3 = 0x33333333u, mf = 0x0f0f0f0fu;
      const uint32_t u0 = (a & m5) | ((b & m5) << 1), u1 = ((a >> 1) & m5) | (b & ~m5);  // y even, z even / odd
      const uint32_t v0 = (d & m5) | ((e & m5) << 1), v1 = ((d >> 1) & m5) | (e & ~m5);  // y odd
      const uint32_t e0 = (u0 & m3) | ((v0 & m3) << 2), e1 = (u1 & m3) | ((v1 & m3) << 2);      // even k
      const uint32_t f0 = ((u0 >> 2) & m3) | (v0 & ~m3), f1 = ((u1 >> 2) & m3) | (v1 & ~m3);    // odd k
      out[0][c] = (e0 & mf) | ((e1 & mf) << 4);
      out[2][c] = ((e0 >> 4) & mf) | (e1 & ~mf);
      out[1][c] = (f0 & mf) | ((f1 & mf) << 4);
      out[3][c] = ((f0 >> 4) & mf) | (f1 & ~mf);
    }
    uint8_t* dst = grid + cell_index((x0 >> 1) + 4 * g, cy, 16 * w, res);
#pragma unroll
    for (int q = 0; q < 4; q++) {
      const uint32_t t0 = __byte_perm(out[q][0], out[q][1], 0x5140), t1 = __byte_perm(out[q][0], out[q][1], 0x7362);
      const uint32_t s0 = __byte_perm(out[q][2], out[q][3], 0x5140), s1 = __byte_perm(out[q][2], out[q][3], 0x7362);
      const uint32_t o[4] = {__byte_perm(t0, s0, 0x5410), __byte_perm(t0, s0, 0x7632), __byte_perm(t1, s1, 0x5410),
                             __byte_perm(t1, s1, 0x7632)};
#pragma unroll
      for (int j = 0; j < 4; j++) {
        uint8_t* to = dst + (int64_t)res * res * (q + 4 * j);
        if (aligned) {
          *reinterpret_cast<uint32_t*>(to) = o[j];
        } else {
#pragma unroll
          for (int k = 0; k < 4; k++) to[k] = (uint8_t)(o[j] >> (8 * k));
        }
      }
    }
  }
}

__global__ void k_packed_to_zwords(const uint8_t* __restrict__ grid, uint32_t* __restrict__ zw, int res) {
  const int N = 2 * res, W = N >> 5;
  const int64_t total = (int64_t)N * N * W;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const int kz = (int)(i % W);
    const int64_t col = i / W;
    const int fx = (int)(col % N), fy = (int)(col / N);
    uint32_t w = 0;
    for (int j = 0; j < 32; j++) {
      const int fz = 32 * kz + j;
      const uint8_t b = grid[cell_index(fx >> 1, fy >> 1, fz >> 1, res)];
      w |= (uint32_t)((b >> child_bit(fx, fy, fz)) & 1u) << j;
    }
    zw[i] = w;
  }
}

static int blocks_for(int64_t n) {
  int64_t b = (n + 255) / 256;
  if (b > 152 * 32) b = 152 * 32;
  return (int)(b < 1 ? 1 : b);
}

template <bool SOLID>
static cudaError_t launch_pack(const uint32_t* zw, const uint32_t* surf, uint8_t* grid, int res, cudaStream_t st,
                               KernelCounter* kc) {
  const int N = 2 * res, W = N >> 5;
  const size_t smem = sizeof(uint32_t) * 2 * kPackCols * (W + 1);
  const dim3 g((N + kPackCols - 1) / kPackCols, res);
  GM_LAUNCH(kc, "k_pack_columns", st,
            k_pack_columns<SOLID><<<g, 256, smem, st>>>(zw, surf, grid, res,
                                                        (reinterpret_cast<uintptr_t>(grid) & 3) == 0 ? 1 : 0));
  return cudaGetLastError();
}

cudaError_t launch_voxelize(const float* P, int64_t nv, const uint32_t* T, int64_t nf, int res,
                            const float* bbox_min, float cell_size, uint8_t* grid, uint8_t* scratch,
                            cudaStream_t st, KernelCounter* kc) {
  (void)nv;
  const int N = 2 * res;
  const size_t words = (size_t)N * N * N / 32;
  VoxParams vp;
  vp.N = N;
  for (int a = 0; a < 3; a++) vp.b[a] = bbox_min[a];
  vp.h = 0.5 * (double)cell_size;
  vp.ih = (float)(1.0 / vp.h);
  vp.il = (float)(1.0 / vp.h - (double)vp.ih);
  vp.mark = reinterpret_cast<uint32_t*>(scratch);
  vp.surf = vp.mark + words;
  uint32_t* counts = vp.surf + words;  // [2], then the list
  uint32_t* list = counts + 64;
  cudaMemsetAsync(vp.mark, 0, (2 * words + 2) * sizeof(uint32_t), st);
  for (int64_t t0 = 0; t0 < nf; t0 += kVoxChunk) {
    const int64_t n = nf - t0 < kVoxChunk ? nf - t0 : kVoxChunk;
    const uint32_t* Tc = T + 3 * t0;
    if (t0 > 0) cudaMemsetAsync(counts, 0, 2 * sizeof(uint32_t), st);
    GM_LAUNCH(kc, "k_vox_tris", st,
              k_vox_tris<<<(unsigned)((n + kVoxThreads - 1) / kVoxThreads), kVoxThreads, 0, st>>>(P, Tc, (uint32_t)n, vp, list, counts));
    const unsigned b = (unsigned)(n < 152 * 16 ? n : 152 * 16);
    GM_LAUNCH(kc, "k_vox_listed", st, k_vox_listed<<<b, 128, 0, st>>>(P, Tc, n, vp, list, counts));
  }
  return launch_pack<true>(vp.mark, vp.surf, grid, res, st, kc);
}

cudaError_t launch_layout(int res, const uint32_t* zw, uint8_t* grid, int dir, cudaStream_t st, KernelCounter* kc) {
  if (dir == 0) return launch_pack<false>(zw, nullptr, grid, res, st, kc);
  const int N = 2 * res;
  GM_LAUNCH(kc, "k_packed_to_zwords", st, k_packed_to_zwords<<<blocks_for((int64_t)N * N * (N / 32)), 256, 0, st>>>(grid, const_cast<uint32_t*>(zw), res));
  return cudaGetLastError();
}

}  // namespace gm
