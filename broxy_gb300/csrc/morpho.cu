// morpho.cu — variable-radius ball/cube closing on GB300 (reference rows
// a5..a11: GMorpho::DilateBySphereMipmap / DilateByCubeMipmap /
// ErodeBySphereMipmap, GMorpho/GMorpho.cu:3231-3314, 3538-3596, 6627-6702).
//
// The reference answers every dilation/erosion predicate by a per-thread
// stack traversal of a texture pyramid.  Here the same predicates are
// computed as separable min-plus distance transforms over fine-voxel
// fields, one axis per pass, each pass a tiled, coalesced, HBM-streaming
// kernel:
//
//   dilation (query radius r(p), GMorpho.cu:2858-2867):
//       D(p) = min_q sum_a d_a(q - p)^2 < (r(p) + 1)^2   (sphere)
//       D(p) = max_a-combined L-inf lattice distance <= r(p)   (cube)
//     with d(delta) the distance from lattice point p to the box of voxel q.
//   erosion (source radius r(q), GMorpho.cu:4403-4411, 5283-5349):
//       E(s) = min_q [K - 4 (r(q)-1)^2 + sum_a e_a^2] < K,  q in contour S,
//     in half-voxel units (e = box distance from point s to voxel q),
//     K = 4 (rmax - 1)^2, at voxel centres (fine pass) and at the lattice
//     points 2c+1 (base pass).
//
// The two-level structure of the reference (base pass on whole cells,
// refinement of contour cells only) is then applied exactly by the select
// kernels, which reproduces the reference grids bit for bit (GM_REF), or
// skipped (GM_EXACT).
#include <string.h>

#include <algorithm>
#include <vector>

#include "gm_common.cuh"
#include "gm_internal.h"

namespace gm {

// Error bits that kernels with a bounded wait record instead of trapping
// (bit 0: the grid barrier of the resident normal filter gave up); read and
// cleared by kernel_error_flags().
__device__ unsigned int g_kernel_errors = 0;

// A radius field read in place: element (x, y, z) at p[x + y sy + z sz]
// (a whole field, or a crop of a larger one without copying it).
struct RField {
  const int8_t* p;
  int64_t sy, sz;
};
__device__ __forceinline__ int rget(const RField& f, int x, int y, int z) {
  return f.p[(int64_t)x + (int64_t)y * f.sy + (int64_t)z * f.sz];
}

// A box of cells [lo, hi) where a pass's outputs are needed (the whole grid
// unless the caller needs the closing on part of it only).
struct CBox {
  int lo[3], hi[3];
};
__host__ __device__ __forceinline__ bool cbox_meets(const CBox& b, int x0, int x1, int y0, int y1, int z0, int z1) {
  return x1 >= b.lo[0] && x0 < b.hi[0] && y1 >= b.lo[1] && y0 < b.hi[1] && z1 >= b.lo[2] && z0 < b.hi[2];
}

// The two x-bits of fine row r (y parity r & 1, z parity r >> 1) of four
// packed bytes, gathered into 8 bits (byte b -> bits 2b, 2b+1).
__device__ __forceinline__ uint32_t row_bits8(uint32_t w, int r) {
  uint32_t x = (w >> (2 * r)) & 0x03030303u;
  x = (x | (x >> 6)) & 0x000f000fu;
  return (x | (x >> 12)) & 0xffu;
}

// ---------------------------------------------------------------------
// x passes: distances along the fine rows of the packed byte grid.
//
// A lane holds a strip of 16 voxels of four fine rows (8 bytes of the grid)
// and computes the four rows side by side, two to a register in 16-bit
// halves: from right to left the distance to the next site, from left to
// right the nearer of that and of the position before plus one.  What a lane
// needs of the strips beside it is one number a row and side, from a scan
// over the warp (min-plus: 16 per strip).  A warp takes 32 strips of one
// byte row, or several whole rows where they are shorter; longer rows are
// cut and the warp looks 16 strips past each end (no distance above 129 is
// asked for).
// ---------------------------------------------------------------------
constexpr int kStrip = 16;        // voxels
constexpr uint32_t kFar2 = 0x20002000u;  // no site (16-bit halves)

// Four packed bytes to 8 voxels of each fine row, row r = 2 z + y in byte r:
// a transposition of 4 x 4 pairs of bits.
__device__ __forceinline__ uint32_t rows_of_word(uint32_t x) {
  uint32_t t = (x ^ (x >> 12)) & 0x0000f0f0u;
  x ^= t ^ (t << 12);
  t = (x ^ (x >> 6)) & 0x00cc00ccu;
  return x ^ t ^ (t << 6);
}
// halves: 0xffff where byte LO (low half) and byte LO + 1 (high half) have their top bit set
template <int LO>
__device__ __forceinline__ uint32_t spread_tops(uint32_t x) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %1, %2;" : "=r"(r) : "r"(x), "n"(LO == 0 ? 0x9988 : 0xbbaa));
  return r;
}
// per half, the distance from the strip's last position back to its last
// site (last), or from its first on to its first; rows LO and LO + 1
template <int LO>
__device__ __forceinline__ uint32_t strip_end(const uint32_t u[2], bool last) {
  uint32_t w = __byte_perm(u[0], u[1], LO == 0 ? 0x5140 : 0x7362);
  uint32_t lo = w & 0xffffu, hi = w >> 16;
  if (!last) lo = __brev(lo) >> 16, hi = __brev(hi) >> 16;
  const uint32_t a = lo ? (uint32_t)__clz((int)lo) - 16u : kFar2 & 0xffffu;
  const uint32_t b = hi ? (uint32_t)__clz((int)hi) - 16u : kFar2 & 0xffffu;
  return a | (b << 16);
}

// The strips of a warp: bits of the lane's own strip and, where the row is
// cut, of one strip beside the warp's (lanes 0-15 those before, 16-31 those
// after it).
struct Strips {
  uint32_t u[2], h[2];
  int cy, cz, x0;  // byte row, first voxel of the lane's strip
  int seg;         // lanes per row (a power of 2)
  bool mine;       // the strip is in the grid
};

template <bool HALO>
__device__ __forceinline__ bool strips_load(const uint8_t* __restrict__ G, int rx, int ry, CBox rows, int64_t row0,
                                            int64_t row_end, int seg, int cuts, Strips& s) {
  const int lane = threadIdx.x & 31, sub = lane & (seg - 1), n = rx >> 3;  // strips of a row
  const int64_t unit = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  const int64_t row = row0 + (HALO ? unit / cuts : unit * (32 / seg) + lane / seg);
  const int cut = HALO ? (int)(unit % cuts) : 0, strip = 32 * cut + sub;
  s.seg = seg;
  s.cy = (int)(row % ry), s.cz = (int)(row / ry), s.x0 = kStrip * strip;
  const bool asked = row < row_end && s.cy >= rows.lo[1] && s.cy < rows.hi[1] && s.cz >= rows.lo[2] &&
                     s.cz < rows.hi[2];  // (else a row that nobody reads)
  s.mine = asked && strip < n;
  s.u[0] = s.u[1] = s.h[0] = s.h[1] = 0u;
  const uint8_t* g = G + (int64_t)rx * row;
  if (s.mine) {
    const uint2 q = *reinterpret_cast<const uint2*>(g + 8 * strip);
    s.u[0] = rows_of_word(q.x), s.u[1] = rows_of_word(q.y);
  }
  if (HALO && asked) {
    const int beside = lane < 16 ? 32 * cut - 16 + lane : 32 * cut + 16 + lane;
    if (beside >= 0 && beside < n) {
      const uint2 q = *reinterpret_cast<const uint2*>(g + 8 * beside);
      s.h[0] = rows_of_word(q.x), s.h[1] = rows_of_word(q.y);
    }
  }
  return __any_sync(0xffffffffu, s.mine);
}

// Per half (rows LO and LO + 1), the distances at the position before the
// lane's strip (to the last site up to there) and at the one after it (to
// the next site from there on).
template <bool HALO, int LO>
__device__ __forceinline__ void strip_carries(const Strips& s, uint32_t& before, uint32_t& after) {
  const int lane = threadIdx.x & 31, sub = lane & (s.seg - 1);
  uint32_t f = strip_end<LO>(s.u, true), b = strip_end<LO>(s.u, false), left = kFar2, right = kFar2;
  if (HALO) {
    uint32_t e = strip_end<LO>(s.h, lane < 16) + 0x100010u * (uint32_t)(lane < 16 ? 15 - lane : lane - 16);
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) e = __vminu2(e, __shfl_xor_sync(0xffffffffu, e, o));
    left = __shfl_sync(0xffffffffu, e, 0);
    right = __shfl_sync(0xffffffffu, e, 16);
    if (lane == 0) f = __viaddmin_u16x2(left, 0x100010u, f);
    if (lane == 31) b = __viaddmin_u16x2(right, 0x100010u, b);
  }
  for (int o = 1; o < s.seg; o <<= 1) {  // (a lane with no such neighbour gets its own value)
    const uint32_t d = 0x100010u * (uint32_t)o;
    f = __viaddmin_u16x2(__shfl_up_sync(0xffffffffu, f, o, s.seg), d, f);
    b = __viaddmin_u16x2(__shfl_down_sync(0xffffffffu, b, o, s.seg), d, b);
  }
  before = __shfl_up_sync(0xffffffffu, f, 1, s.seg);
  after = __shfl_down_sync(0xffffffffu, b, 1, s.seg);
  if (sub == 0) before = left;
  if (sub == s.seg - 1) after = right;
}

// Launch shape of the x passes: rows shorter than a warp share one.
struct StripGrid {
  int seg, cuts;
  unsigned blocks;
};
static StripGrid strip_grid(int rx, int64_t rows) {
  StripGrid g;
  const int n = rx / 8;  // strips of a row
  g.seg = 2;
  while (g.seg < n && g.seg < 32) g.seg *= 2;
  g.cuts = (n + 31) / 32;
  const int64_t warps = g.cuts > 1 ? rows * g.cuts : (rows + 32 / g.seg - 1) / (32 / g.seg);
  g.blocks = (unsigned)((warps + 7) / 8);
  return g;
}

// Pass X of the dilation: the lattice distance (at the lattice points that
// bound an occupied voxel: 0) to the nearest occupied voxel along each fine
// row, up to dcap, in bytes.  Bound by its instructions (4 a voxel, a third of
// them the scan and the halo).  Against a bit search per voxel in lanes of 32
// voxels, which left most lanes of short rows idle: 0.450 -> 0.326 ms at
// 1024^3 (1.07 GB written), 0.108 -> 0.038 at 512^3, 16.8 -> 7.2 us at 128^3.
template <bool HALO>
__global__ void __launch_bounds__(256) k_dil_pass_x(const uint8_t* __restrict__ X, uint8_t* __restrict__ A, int rx,
                                                    int ry, int dcap, CBox rows, int64_t row0, int64_t row_end,
                                                    int seg, int cuts) {
  Strips s;
  if (!strips_load<HALO>(X, rx, ry, rows, row0, row_end, seg, cuts, s)) return;
  const int N = 2 * rx, Ny = 2 * ry;
  const uint32_t own = s.u[0] | s.u[1], beside = s.h[0] | s.h[1];
  const bool none = !__any_sync(0xffffffffu, own | beside);
  if (none || __all_sync(0xffffffffu, !s.mine || (s.u[0] & s.u[1]) == 0xffffffffu)) {
    // nothing within reach, or every corner a site
    const uint32_t v = none ? (uint32_t)dcap * 0x01010101u : 0u;
    if (s.mine) {
#pragma unroll
      for (int r = 0; r < 4; r++)
        *reinterpret_cast<uint4*>(A + idx3(s.x0, 2 * s.cy + (r & 1), 2 * s.cz + (r >> 1), N, Ny)) =
            make_uint4(v, v, v, v);
    }
    return;
  }
  // corner sets: lattice point p bounds voxels p - 1 and p
  {
    const int lane = threadIdx.x & 31;
    uint32_t prev = __shfl_up_sync(0xffffffffu, s.u[1], 1, seg);
    if (HALO) {
      uint32_t hprev = __shfl_up_sync(0xffffffffu, s.h[1], 1, 16);
      if ((lane & 15) == 0) hprev = 0u;  // (out of reach; of no effect past the warp's end)
      const uint32_t first = __shfl_sync(0xffffffffu, s.h[1], 15);
      s.h[1] |= ((s.h[1] << 1) & 0xfefefefeu) | ((s.h[0] >> 7) & 0x01010101u);
      s.h[0] |= ((s.h[0] << 1) & 0xfefefefeu) | ((hprev >> 7) & 0x01010101u);
      if (lane == 0) prev = first;
    } else if ((lane & (seg - 1)) == 0) {
      prev = 0u;
    }
    s.u[1] |= ((s.u[1] << 1) & 0xfefefefeu) | ((s.u[0] >> 7) & 0x01010101u);
    s.u[0] |= ((s.u[0] << 1) & 0xfefefefeu) | ((prev >> 7) & 0x01010101u);
  }
  uint32_t d0, d1, r0, r1;
  strip_carries<HALO, 0>(s, d0, r0);
  strip_carries<HALO, 2>(s, d1, r1);
  uint32_t t0[16], t1[16];
#pragma unroll
  for (int p = 15; p >= 0; p--) {
    const uint32_t w = ~s.u[p >> 3] << (7 - (p & 7));
    t0[p] = r0 = __viaddmin_u16x2(r0, 0x10001u, spread_tops<0>(w));
    t1[p] = r1 = __viaddmin_u16x2(r1, 0x10001u, spread_tops<2>(w));
  }
  const uint32_t cap2 = (uint32_t)dcap * 0x10001u;
  uint32_t out[4][4];
#pragma unroll
  for (int q = 0; q < 4; q++) {
    uint32_t m0[4], m1[4];
#pragma unroll
    for (int j = 0; j < 4; j++) {
      d0 = __viaddmin_u16x2(d0, 0x10001u, t0[4 * q + j]);
      d1 = __viaddmin_u16x2(d1, 0x10001u, t1[4 * q + j]);
      m0[j] = __vminu2(d0, cap2);
      m1[j] = __vminu2(d1, cap2);
    }
    const uint32_t a = __byte_perm(m0[0], m0[1], 0x6240), b = __byte_perm(m0[2], m0[3], 0x6240);
    const uint32_t c = __byte_perm(m1[0], m1[1], 0x6240), d = __byte_perm(m1[2], m1[3], 0x6240);
    out[0][q] = __byte_perm(a, b, 0x5410);
    out[1][q] = __byte_perm(a, b, 0x7632);
    out[2][q] = __byte_perm(c, d, 0x5410);
    out[3][q] = __byte_perm(c, d, 0x7632);
  }
  if (!s.mine) return;
#pragma unroll
  for (int r = 0; r < 4; r++)
    *reinterpret_cast<uint4*>(A + idx3(s.x0, 2 * s.cy + (r & 1), 2 * s.cz + (r >> 1), N, Ny)) =
        make_uint4(out[r][0], out[r][1], out[r][2], out[r][3]);
}

// launch of the dilation's x pass over the rows of `rows`
static cudaError_t launch_dil_pass_x(const uint8_t* X, uint8_t* A, int rx, int ry, int rz, int dcap, CBox rows,
                                     cudaStream_t st, KernelCounter* kc) {
  // the rows of the box's z range only (row id = y + ry z)
  const int64_t row0 = (int64_t)ry * (rows.lo[2] > 0 ? rows.lo[2] : 0);
  const int64_t row_end = (int64_t)ry * (rows.hi[2] < rz ? rows.hi[2] : rz);
  if (row_end <= row0) return cudaSuccess;
  const StripGrid sg = strip_grid(rx, row_end - row0);
  if (sg.cuts > 1)
    GM_LAUNCH(kc, "k_dil_pass_x", st,
              k_dil_pass_x<true><<<sg.blocks, 256, 0, st>>>(X, A, rx, ry, dcap, rows, row0, row_end, sg.seg, sg.cuts));
  else
    GM_LAUNCH(kc, "k_dil_pass_x", st,
              k_dil_pass_x<false><<<sg.blocks, 256, 0, st>>>(X, A, rx, ry, dcap, rows, row0, row_end, sg.seg, 1));
  return cudaGetLastError();
}

// ---------------------------------------------------------------------
// pass X of the erosion: sites are the contour voxels of one fine row;
// outputs the half-voxel-unit partial sums K - 4 (r - 1)^2 + e^2, at most K,
// at every voxel centre (HC) and at the odd lattice points x = 2c+1 (HL).
// ---------------------------------------------------------------------

// With one radius the sums follow from the distance to the nearest site.
// With d twice the distance in voxels (the recurrences' steps are 2), the
// centres' box distance is max(d - 1, 0), and that of the lattice point
// before voxel p the least of voxel p's towards the right and voxel p - 1's.
// Bound by the bytes it writes (3 a voxel: 57 us of 76 at 512^3, where
// splatting the sites took 152; 22.8 -> 8.6 us at 128^3).
template <bool HALO>
__global__ void __launch_bounds__(256, 3) k_ero_pass_x_one(const uint8_t* __restrict__ S, int r, int rx, int ry,
                                                        uint32_t K, uint16_t* __restrict__ HC,
                                                        uint16_t* __restrict__ HL, CBox rows, int64_t row0,
                                                        int64_t row_end, int seg, int cuts) {
  Strips s;
  if (!strips_load<HALO>(S, rx, ry, rows, row0, row_end, seg, cuts, s)) return;
  const int N = 2 * rx, Ny = 2 * ry;
  if (!__any_sync(0xffffffffu, s.u[0] | s.u[1] | s.h[0] | s.h[1])) {
    // no site within reach: every output keeps the saturation value K
    if (s.mine) {
      const uint32_t k2 = K | (K << 16);
      const uint4 v = make_uint4(k2, k2, k2, k2);
#pragma unroll
      for (int i = 0; i < 4; i++) {
        const int fy = 2 * s.cy + (i & 1), fz = 2 * s.cz + (i >> 1);
        uint4* c = reinterpret_cast<uint4*>(HC + idx3(s.x0, fy, fz, N, Ny));
        c[0] = c[1] = v;
        *reinterpret_cast<uint4*>(HL + idx3(s.x0 >> 1, fy, fz, rx, Ny)) = v;
      }
    }
    return;
  }
  const uint32_t cap = 2u * (uint32_t)(r - 1), cap2 = cap | (cap << 16);
  const uint32_t u = K - cap * cap, u2 = u | (u << 16);
  // values of two positions of a row: u + e^2 per half
  auto squares = [&](uint32_t e) {
    const uint32_t a = e & 0xffffu, b = e >> 16;
    return b * (e & 0xffff0000u) + (a * a + u2);
  };
#pragma unroll
  for (int half = 0; half < 2; half++) {  // rows 0, 1, then 2, 3
    uint32_t d, q;
    if (half == 0) strip_carries<HALO, 0>(s, d, q);
    else strip_carries<HALO, 2>(s, d, q);
    d = __vminu2(d, cap2) << 1, q = __vminu2(q, cap2) << 1;
    uint32_t t[16];
#pragma unroll
    for (int p = 15; p >= 0; p--) {
      const uint32_t w = ~s.u[p >> 3] << (7 - (p & 7));
      t[p] = q = __viaddmin_u16x2(q, 0x20002u, half == 0 ? spread_tops<0>(w) : spread_tops<2>(w));
    }
    uint32_t c0[8], c1[8], l0[4], l1[4];
#pragma unroll
    for (int p4 = 0; p4 < 4; p4++) {
      uint32_t c[4], l[2];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int p = 4 * p4 + j;
        if (j & 1) l[j >> 1] = __vimin3_u16x2(d, t[p], cap2);
        d = __viaddmin_u16x2(d, 0x20002u, t[p]);
        c[j] = __viaddmin_s16x2_relu(d, 0xffffffffu, cap2);
      }
      c0[2 * p4] = squares(__byte_perm(c[0], c[1], 0x5410)), c0[2 * p4 + 1] = squares(__byte_perm(c[2], c[3], 0x5410));
      c1[2 * p4] = squares(__byte_perm(c[0], c[1], 0x7632)), c1[2 * p4 + 1] = squares(__byte_perm(c[2], c[3], 0x7632));
      l0[p4] = squares(__byte_perm(l[0], l[1], 0x5410));
      l1[p4] = squares(__byte_perm(l[0], l[1], 0x7632));
    }
    if (s.mine) {
      const int fy = 2 * s.cy, fz = 2 * s.cz + half;
      uint4* c = reinterpret_cast<uint4*>(HC + idx3(s.x0, fy, fz, N, Ny));
      c[0] = make_uint4(c0[0], c0[1], c0[2], c0[3]), c[1] = make_uint4(c0[4], c0[5], c0[6], c0[7]);
      c = reinterpret_cast<uint4*>(HC + idx3(s.x0, fy + 1, fz, N, Ny));
      c[0] = make_uint4(c1[0], c1[1], c1[2], c1[3]), c[1] = make_uint4(c1[4], c1[5], c1[6], c1[7]);
      *reinterpret_cast<uint4*>(HL + idx3(s.x0 >> 1, fy, fz, rx, Ny)) = make_uint4(l0[0], l0[1], l0[2], l0[3]);
      *reinterpret_cast<uint4*>(HL + idx3(s.x0 >> 1, fy + 1, fz, rx, Ny)) = make_uint4(l1[0], l1[1], l1[2], l1[3]);
    }
  }
}

// With a radius field: one warp per fine row and no block barrier.  The
// warp's slice of shared memory holds the row's outputs; sites are sparse
// (the contour shell), so they splat their sums: 32 voxels of the row at a
// time, a lane reading its voxel's radius (the next word's radii on their
// way meanwhile), one run of adjacent sites of one radius after the other,
// lanes over the run's taps, so that the lanes of a splat touch distinct
// outputs and need no atomics.  Rows without sites are written straight away.
// Bound by instructions (a row's sites, 70 % of the issue slots), then by the
// 3 bytes a voxel it writes: 0.754 ms at 1024^3 (0.850 with four rows a warp
// one after the other, whose radii came one dependent load a site; the bytes
// alone take 0.48).
constexpr int kEroXWarps = 8;
constexpr int kEroPad = 128;  // voxels past each end of a row that a splat may reach (at most 126)

__host__ __device__ inline size_t ero_x_warp_bytes(int rx) {
  return 6 * ((size_t)rx + 2 * kEroPad / 2);  // outputs at centres and at lattice points
}

__global__ void __launch_bounds__(256, 6) k_ero_pass_x(const uint8_t* __restrict__ S, RField R, int rx, int ry, int halo,
                                                    uint32_t K, uint16_t* __restrict__ HC, uint16_t* __restrict__ HL,
                                                    CBox rows, int64_t row0, int64_t row_end) {
  extern __shared__ uint4 sm_ero[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int N = 2 * rx, Ny = 2 * ry, W = N >> 5;
  const int64_t row_id = row0 + ((int64_t)blockIdx.x * kEroXWarps + wid) / 4;
  const int r = wid & 3;
  if (row_id >= row_end) return;
  const int cy = (int)(row_id % ry), cz = (int)(row_id / ry);
  if (cy < rows.lo[1] || cy >= rows.hi[1] || cz < rows.lo[2] || cz >= rows.hi[2]) return;  // rows nobody reads
  uint8_t* slice = reinterpret_cast<uint8_t*>(sm_ero) + (size_t)wid * ero_x_warp_bytes(rx);
  uint16_t* hc = reinterpret_cast<uint16_t*>(slice) + kEroPad;
  uint16_t* hl = hc + N + kEroPad + kEroPad / 2;
  const int fy = 2 * cy + (r & 1), fz = 2 * cz + (r >> 1);
  const uint8_t* srow = S + idx3(0, cy, cz, rx, ry);
  const int8_t* rrow = R.p + (int64_t)fy * R.sy + (int64_t)fz * R.sz;
  uint4* hcrow = reinterpret_cast<uint4*>(HC + idx3(0, fy, fz, N, Ny));
  uint4* hlrow = reinterpret_cast<uint4*>(HL + idx3(0, fy, fz, rx, Ny));
  const uint32_t k2 = K | (K << 16);
  const uint4 K4 = make_uint4(k2, k2, k2, k2);
  bool filled = false;
  for (int w0 = 0; w0 < W; w0 += 32) {
    // the row's bits, a word per lane
    uint32_t bits = 0u;
    const int w = w0 + lane;
    if (w < W) {
      const uint4 q = *reinterpret_cast<const uint4*>(srow + 16 * (size_t)w);
      bits = row_bits8(q.x, r) | (row_bits8(q.y, r) << 8) | (row_bits8(q.z, r) << 16) | (row_bits8(q.w, r) << 24);
    }
    uint32_t left = __ballot_sync(0xffffffffu, bits != 0u);  // words with sites
    if (!left) continue;
    if (!filled) {
      for (int i = lane; i < N >> 3; i += 32) reinterpret_cast<uint4*>(hc)[i] = K4;
      for (int i = lane; i < rx >> 3; i += 32) reinterpret_cast<uint4*>(hl)[i] = K4;
      __syncwarp();
      filled = true;
    }
    int src = __ffs(left) - 1;
    uint32_t m = __shfl_sync(0xffffffffu, bits, src);
    int rq = (m >> lane) & 1u ? rrow[32 * (w0 + src) + lane] : 0;
    while (left) {
      const int x0 = 32 * (w0 + src);
      const bool site = (m >> lane) & 1u;
      const int rm1 = clamp_radius(rq) - 1;
      // the next word's radii
      left &= left - 1;
      src = __ffs(left) - 1;
      m = __shfl_sync(0xffffffffu, bits, src & 31);
      rq = left && ((m >> lane) & 1u) ? rrow[32 * (w0 + src) + lane] : 0;
      // Runs of adjacent sites with the same radius splat as one: every
      // output inside the run has a site at distance 0 (value u), and one
      // outside it is nearest to the run's end on its side (both kernels grow
      // with the distance), so the run's taps are [q0 - reach, qe + reach]
      // with the nearest site of each, instead of 2 reach + 1 per site.
      const int before = __shfl_up_sync(0xffffffffu, site ? rm1 : -1, 1);
      const uint32_t cont = __ballot_sync(0xffffffffu, site && lane > 0 && before == rm1);
      uint32_t starts = __ballot_sync(0xffffffffu, site) & ~cont;
      while (starts) {
        const int b = __ffs(starts) - 1;
        starts &= starts - 1;
        const uint32_t more = ~((cont >> b) >> 1);
        const int len = more ? __ffs(more) : 32, q0 = x0 + b;
        const int rr = __shfl_sync(0xffffffffu, rm1, b);
        // (a point at |q - p| >= r(q) is never eroded by q: e >= 2 (r(q) - 1))
        const int reach = rr < halo ? rr : halo;
        const uint32_t u = K - 4u * (uint32_t)(rr * rr);
        for (int o = lane - reach; o < len + reach; o += 32) {
          const int p = q0 + o;  // output position (the row is padded)
          // center_dist2 and twice lattice_dist to the nearest site of the run
          const int ec = max(2 * max(-o, o - len + 1) - 1, 0), el = 2 * max(max(-o, o - len), 0);
          const uint32_t vc = u + (uint32_t)(ec * ec), vl = u + (uint32_t)(el * el);
          if (vc < hc[p]) hc[p] = (uint16_t)vc;
          if ((p & 1) && vl < hl[p >> 1]) hl[p >> 1] = (uint16_t)vl;
        }
        __syncwarp();
      }
    }
  }
  if (!filled) {
    for (int i = lane; i < N >> 3; i += 32) hcrow[i] = K4;
    for (int i = lane; i < rx >> 3; i += 32) hlrow[i] = K4;
    return;
  }
  for (int i = lane; i < N >> 3; i += 32) hcrow[i] = reinterpret_cast<const uint4*>(hc)[i];
  for (int i = lane; i < rx >> 3; i += 32) hlrow[i] = reinterpret_cast<const uint4*>(hl)[i];
}

// launch of the erosion's x pass over the rows of `rows`
static cudaError_t launch_ero_pass_x(const uint8_t* S, RField R, int uniform_r, int rx, int ry, int rz, int halo,
                                     uint32_t K, uint16_t* HC, uint16_t* HL, CBox rows, cudaStream_t st,
                                     KernelCounter* kc) {
  const int64_t row0 = (int64_t)ry * (rows.lo[2] > 0 ? rows.lo[2] : 0);
  const int64_t row_end = (int64_t)ry * (rows.hi[2] < rz ? rows.hi[2] : rz);
  if (row_end <= row0) return cudaSuccess;
  if (R.p != nullptr) {
    const size_t smem = kEroXWarps * ero_x_warp_bytes(rx);
    ensure_dynamic_smem(reinterpret_cast<const void*>(k_ero_pass_x), smem);
    const unsigned blocks = (unsigned)((4 * (row_end - row0) + kEroXWarps - 1) / kEroXWarps);
    GM_LAUNCH(kc, "k_ero_pass_x", st,
              k_ero_pass_x<<<blocks, 32 * kEroXWarps, smem, st>>>(S, R, rx, ry, halo, K, HC, HL, rows, row0, row_end));
    return cudaGetLastError();
  }
  const int r = clamp_radius(uniform_r);
  const StripGrid sg = strip_grid(rx, row_end - row0);
  if (sg.cuts > 1)
    GM_LAUNCH(kc, "k_ero_pass_x", st,
              k_ero_pass_x_one<true><<<sg.blocks, 256, 0, st>>>(S, r, rx, ry, K, HC, HL, rows, row0, row_end, sg.seg,
                                                                sg.cuts));
  else
    GM_LAUNCH(kc, "k_ero_pass_x", st,
              k_ero_pass_x_one<false><<<sg.blocks, 256, 0, st>>>(S, r, rx, ry, K, HC, HL, rows, row0, row_end, sg.seg,
                                                                 1));
  return cudaGetLastError();
}

// ---------------------------------------------------------------------
// generic axis pass (y or z): out(o) = min over delta of
//     in(pos(o) + delta) (+) g(delta)
// ---------------------------------------------------------------------

enum Kern { KERN_LAT = 0, KERN_LAT2 = 1, KERN_CEN2 = 2, KERN_CUBE = 3 };

template <int G>
__device__ __forceinline__ uint32_t kern_g(int delta) {
  if (G == KERN_LAT) { const int d = lattice_dist(delta); return (uint32_t)(d * d); }
  if (G == KERN_LAT2) { const int d = 2 * lattice_dist(delta); return (uint32_t)(d * d); }
  if (G == KERN_CEN2) { const int d = center_dist2(delta); return (uint32_t)(d * d); }
  return (uint32_t)lattice_dist(delta);  // KERN_CUBE
}

template <int G>
__device__ __forceinline__ uint32_t combine(uint32_t v, uint32_t g) {
  if (G == KERN_CUBE) return v > g ? v : g;
  return v + g;
}

// Minimum over a window of the tile column `col` (stride 32 between
// consecutive positions) around index sp, scanning outward and stopping as
// soon as the kernel alone reaches the best value (inputs are >= 0).
template <int G>
__device__ __forceinline__ uint32_t column_min(const uint16_t* col, int sp, int span, int halo) {
  uint32_t best = combine<G>(col[sp * 32], kern_g<G>(0));
  for (int k = 1; k <= halo; k++) {
    const uint32_t gp = kern_g<G>(k), gm_ = kern_g<G>(-k);
    if ((gp < gm_ ? gp : gm_) >= best) break;
    if (sp + k < span) { const uint32_t v = combine<G>(col[(sp + k) * 32], gp); best = v < best ? v : best; }
    if (sp - k >= 0) { const uint32_t v = combine<G>(col[(sp - k) * 32], gm_); best = v < best ? v : best; }
  }
  return best;
}

constexpr int kTileOut = 64;  // outputs per block along the pass axis
constexpr int kRows = 8;      // blockDim.y

// Input element conversion: u8 fields hold 1-D distances d (pass X of the
// dilation) and enter the sphere kernel squared.
template <int G, typename TIn>
__device__ __forceinline__ uint16_t load_in(const TIn* p, uint32_t cap) {
  const uint32_t v = (uint32_t)*p;
  if (sizeof(TIn) == 1 && G != KERN_CUBE) { const uint32_t s = v * v; return (uint16_t)(s < cap ? s : cap); }
  return (uint16_t)(v < cap ? v : cap);
}

// in/out fields are x-fastest with dims (nx, ny, nz).  axis = 1 (y) or 2
// (z).  sub: output only the odd input positions 2o+1 along the axis.
template <int G, typename TIn>
__global__ void __launch_bounds__(256) k_axis_pass(const TIn* __restrict__ in, uint16_t* __restrict__ out,
                                                   int nx, int ny, int nz, int axis, int sub, int halo,
                                                   uint32_t cap) {
  extern __shared__ uint16_t tile[];  // [span][32]
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int x = blockIdx.x * 32 + tx;
  const int na = axis == 1 ? ny : nz;
  const int nout = sub ? na / 2 : na;
  const int third = blockIdx.z;  // z for axis y, y for axis z
  const int64_t sa = axis == 1 ? (int64_t)nx : (int64_t)nx * ny;
  const int64_t s3 = axis == 1 ? (int64_t)nx * ny : (int64_t)nx;
  const int o0 = blockIdx.y * kTileOut;
  const int p_first = sub ? 2 * o0 + 1 : o0;
  const int o_last = min(o0 + kTileOut, nout) - 1;
  const int p_last = sub ? 2 * o_last + 1 : o_last;
  const int lo = p_first - halo;
  const int span = p_last + halo - lo + 1;
  for (int s = ty; s < span; s += kRows) {
    const int a = lo + s;
    uint16_t v = (uint16_t)cap;
    if (x < nx && a >= 0 && a < na) v = load_in<G, TIn>(in + x + sa * a + s3 * third, cap);
    tile[s * 32 + tx] = v;
  }
  __syncthreads();
  if (x >= nx) return;
  // output dims: same as input except the pass axis (nout)
  const int64_t osa = sa;
  const int64_t os3 = axis == 1 ? (int64_t)nx * nout : (int64_t)nx;
  for (int o = o0 + ty; o <= o_last; o += kRows) {
    const int p = sub ? 2 * o + 1 : o;
    const uint32_t best = column_min<G>(tile + tx, p - lo, span, halo);
    out[x + osa * o + os3 * third] = (uint16_t)(best < cap ? best : cap);
  }
}

// ---------------------------------------------------------------------
// final z pass at full resolution, fused with the per-voxel threshold and
// the packing of 2x2x2 bits into reference bytes.
//   FIN_DIL: bit = sum < (r(p)+1)^2 (sphere) / sum <= r(p) (cube)
//   FIN_ERO: bit = sum < K (eroded)
// block (32, 8): tx = x, ty & 1 = y parity, ty >> 1 = group of 16 z.
// ---------------------------------------------------------------------

enum Fin { FIN_DIL = 0, FIN_ERO = 1 };

template <int G, int F>
__global__ void __launch_bounds__(256) k_final_z(const uint16_t* __restrict__ in, uint8_t* __restrict__ out_cells,
                                                 RField R, int uniform_r, int rx, int ry, int rz,
                                                 int halo, uint32_t cap) {
  extern __shared__ uint16_t tile2[];  // [2][span][32]
  const int Nx = 2 * rx, Ny = 2 * ry, N = 2 * rz;  // N: fine extent along the pass axis z
  const int tx = threadIdx.x, yp = threadIdx.y & 1, zg = threadIdx.y >> 1;
  const int x = blockIdx.x * 32 + tx;
  const int y = 2 * blockIdx.z + yp;
  const int z0 = blockIdx.y * kTileOut;
  const int z_last = min(z0 + kTileOut, N) - 1;
  const int lo = z0 - halo;
  const int span = z_last + halo - lo + 1;
  uint16_t* tile = tile2 + yp * span * 32;
  for (int s = zg; s < span; s += 4) {
    const int a = lo + s;
    uint16_t v = (uint16_t)cap;
    if (x < Nx && a >= 0 && a < N) {
      const uint32_t t = in[idx3(x, y, a, Nx, Ny)];
      v = (uint16_t)(t < cap ? t : cap);
    }
    tile[s * 32 + tx] = v;
  }
  __syncthreads();
  // each thread: 16 consecutive z = z0 + 16 zg + j
  uint32_t bits = 0;
  const int ru = clamp_radius(uniform_r);
  if (x < Nx) {
#pragma unroll 1
    for (int j = 0; j < 16; j++) {
      const int z = z0 + 16 * zg + j;
      if (z > z_last) break;
      const uint32_t v = column_min<G>(tile + tx, z - lo, span, halo);
      bool b;
      if (F == FIN_DIL) {
        const int r = R.p != nullptr ? clamp_radius(rget(R, x, y, z)) : ru;
        if (G == KERN_CUBE) b = v <= (uint32_t)r;
        else b = v < (uint32_t)((r + 1) * (r + 1));
      } else {
        b = v < cap;
      }
      bits |= (uint32_t)b << j;
    }
  }
  // pack: for z pair q (0..7), this voxel contributes bit (xb + 2 yb) for the
  // lower z and (xb + 2 yb + 4) for the upper z.
  const int xb = x & 1;
  uint32_t packed = 0;  // byte q in bits 8q..8q+7, q = 0..3 (first 8 z) / second word
  uint32_t packed_hi = 0;
#pragma unroll
  for (int q = 0; q < 8; q++) {
    const uint32_t lo_b = (bits >> (2 * q)) & 1u, hi_b = (bits >> (2 * q + 1)) & 1u;
    const uint32_t byte = (lo_b << (xb + 2 * yp)) | (hi_b << (xb + 2 * yp + 4));
    if (q < 4) packed |= byte << (8 * q);
    else packed_hi |= byte << (8 * (q - 4));
  }
  packed |= __shfl_xor_sync(0xffffffffu, packed, 1);
  packed_hi |= __shfl_xor_sync(0xffffffffu, packed_hi, 1);
  __shared__ uint32_t ex[2][4][32][2];
  ex[yp][zg][tx][0] = packed;
  ex[yp][zg][tx][1] = packed_hi;
  __syncthreads();
  if (yp == 0 && (tx & 1) == 0 && x < Nx) {
    const uint32_t w0 = packed | ex[1][zg][tx][0];
    const uint32_t w1 = packed_hi | ex[1][zg][tx][1];
    const int cx = x >> 1, cyy = y >> 1;
#pragma unroll
    for (int q = 0; q < 8; q++) {
      const int zc = (z0 + 16 * zg) / 2 + q;
      if (2 * zc > z_last) break;
      const uint32_t byte = q < 4 ? (w0 >> (8 * q)) & 0xffu : (w1 >> (8 * (q - 4))) & 0xffu;
      out_cells[idx3(cx, cyy, zc, rx, ry)] = (uint8_t)byte;
    }
  }
}

// final z pass of the base erosion: lattice points 2c+1 only; one flag byte
// per base cell (1 = the cell centre is eroded).
__global__ void __launch_bounds__(256) k_final_z_base(const uint16_t* __restrict__ in, uint8_t* __restrict__ flags,
                                                      int rx, int ry, int rz, int halo, uint32_t cap) {
  extern __shared__ uint16_t tile[];
  const int N = 2 * rz;
  const int tx = threadIdx.x, ty = threadIdx.y;
  const int x = blockIdx.x * 32 + tx;  // cx
  const int cyy = blockIdx.z;
  const int o0 = blockIdx.y * kTileOut;
  const int o_last = min(o0 + kTileOut, rz) - 1;
  const int lo = 2 * o0 + 1 - halo;
  const int span = 2 * o_last + 1 + halo - lo + 1;
  for (int s = ty; s < span; s += kRows) {
    const int a = lo + s;
    uint16_t v = (uint16_t)cap;
    if (x < rx && a >= 0 && a < N) {
      const uint32_t t = in[idx3(x, cyy, a, rx, ry)];
      v = (uint16_t)(t < cap ? t : cap);
    }
    tile[s * 32 + tx] = v;
  }
  __syncthreads();
  if (x >= rx) return;
  for (int o = o0 + ty; o <= o_last; o += kRows) {
    const uint32_t v = column_min<KERN_LAT2>(tile + tx, 2 * o + 1 - lo, span, halo);
    flags[idx3(x, cyy, o, rx, ry)] = v < cap ? 1 : 0;
  }
}

// ---------------------------------------------------------------------
// packed 16-bit min-plus pass (y or z) with DPX add-min
//
// Each thread owns two adjacent x columns (one u32 = two u16 lanes) and 16
// consecutive outputs along the pass axis, so one __viaddmin_u16x2 updates
// two outputs per tap.  A block is 64 columns x 64 outputs x 2 "third"
// coordinates (256 threads); the input tile with its halo sits in shared
// memory.  Taps are visited outward (|delta| = 0, 1, 2, ...); a warp stops
// as soon as the kernel alone exceeds every output it holds.  A tile with
// no finite input is written directly.  Requires cap <= 32767 so that
// value + kernel never wraps in 16 bits.
//   FIN 0: write the u16 field;  FIN 1: dilation threshold + packed bytes;
//   FIN 2: erosion threshold (centres) + packed bytes;
//   FIN 3: erosion threshold at lattice points 2c+1, one flag per cell;
//   FIN 4: FIN 2's bytes e applied to the closing (out8): a cell tagged 0xff
//          in the tags, handed over in R.p, becomes ~e, the others stay (a
//          kernel of its own for it took 14.6 us at 512^3, 47 at 1024^3).
// ---------------------------------------------------------------------

constexpr int kDpxCols = 64;   // x columns per block
constexpr int kDpxOut = 64;    // outputs per block along the axis (4 warps x 16)
constexpr int kDpxPer = 16;    // outputs per thread

template <int G>
__device__ __forceinline__ uint32_t gpair(int delta, uint32_t cap) {
  uint32_t g = kern_g<G>(delta);
  g = g < cap ? g : cap;
  return g | (g << 16);
}

// kernel value at delta = k >= 1 (the +side), without the general
// lattice_dist; the -side of LAT and CUBE at -k equals the +side at k - 1,
// and CEN2 is symmetric
template <int G>
__device__ __forceinline__ uint32_t kern_pos(int k) {
  if (G == KERN_LAT) return (uint32_t)(k * k);
  if (G == KERN_LAT2) return (uint32_t)(4 * k * k);
  if (G == KERN_CEN2) return (uint32_t)((2 * k - 1) * (2 * k - 1));
  return (uint32_t)k;  // KERN_CUBE
}

__device__ __forceinline__ uint32_t pack_cap(uint32_t g, uint32_t cap) {
  g = g < cap ? g : cap;
  return g | (g << 16);
}

template <int G>
__device__ __forceinline__ uint32_t step_min(uint32_t row, uint32_t g, uint32_t best) {
  if (G == KERN_CUBE) return __vminu2(__vmaxu2(row, g), best);
  return __viaddmin_u16x2(row, g, best);
}

// Four packed words (8 columns) of a u16 field.
__device__ __forceinline__ uint4 clamp4(uint4 v, uint32_t capp) {
  return make_uint4(__vminu2(v.x, capp), __vminu2(v.y, capp), __vminu2(v.z, capp), __vminu2(v.w, capp));
}
__device__ __forceinline__ uint32_t min4(uint4 v, uint32_t m) {
  return __vimin3_u16x2(__vimin3_u16x2(v.x, v.y, m), v.z, v.w);
}
// Two u8 distances (the low bytes of a word's halves) as packed u16: squared
// for the ball, themselves for the cube.
template <int G>
__device__ __forceinline__ uint32_t widen_pair(uint32_t w, uint32_t sel) {
  const uint32_t p = __byte_perm(w, 0u, sel);  // the two bytes, zero-extended
  if (G == KERN_CUBE) return p;
  const uint32_t hi = p >> 16;
  return (p & 0xffffu) * (p & 0xffffu) + (p & 0xffff0000u) * hi;
}

size_t dpx_smem_bytes(int sub, int halo) {
  const int span = (sub ? 2 * kDpxOut - 1 : kDpxOut) + 2 * halo;
  return (size_t)2 * span * 32 * sizeof(uint32_t);
}

// Where a pass's outputs are needed: tiles whose cells, grown by (gx, ga,
// gt) cells along (x, pass axis, third axis), hold no non-empty cell of the
// 8^3-cell occupancy map of the dilation are skipped.  The x coordinate and
// the third coordinate are fine voxels (shift 1) or cells (shift 0); the
// outputs along the pass axis are fine voxels (sub = 0) or cells (sub = 1).
struct NeedMap {
  const uint8_t* dmap;  // nullptr: no occupancy test
  int mdx, mdy, mdz;
  int x_shift, t_shift;
  int gx, ga, gt;
  CBox roi;             // tiles whose own cells miss it are skipped as well
  // launch over third-axis block rows third0 .. third0 + third_n - 1 and
  // output tiles out0 .. out0 + out_n - 1 only (0: all); a skipped tile
  // writes saturation values, so a part of a pass that must leave the rest
  // of its output alone is launched this way
  int third0 = 0, third_n = 0, out0 = 0, out_n = 0;
};

__device__ bool tile_needed(const NeedMap& nm, int axis, int sub, int o0, int nout, int bx, int bz) {
  const int x0 = bx * kDpxCols;
  const int cx0 = x0 >> nm.x_shift, cx1 = (x0 + kDpxCols - 1) >> nm.x_shift;
  const int oa = o0, ob = min(o0 + kDpxOut, nout) - 1;
  const int ca0 = sub ? oa : oa >> 1, ca1 = sub ? ob : ob >> 1;
  const int ct0 = (2 * bz) >> nm.t_shift, ct1 = (2 * bz + 1) >> nm.t_shift;
  // (a, t) are (y, z) for the y pass and (z, y) for the z pass
  {
    const int ya = axis == 1 ? ca0 : ct0, yb = axis == 1 ? ca1 : ct1;
    const int za = axis == 1 ? ct0 : ca0, zb = axis == 1 ? ct1 : ca1;
    if (!cbox_meets(nm.roi, cx0, cx1, ya, yb, za, zb)) return false;  // block-uniform
  }
  if (nm.dmap == nullptr) return true;
  const int lo[3] = {cx0 - nm.gx, (axis == 1 ? ca0 - nm.ga : ct0 - nm.gt), (axis == 1 ? ct0 - nm.gt : ca0 - nm.ga)};
  const int hi[3] = {cx1 + nm.gx, (axis == 1 ? ca1 + nm.ga : ct1 + nm.gt), (axis == 1 ? ct1 + nm.gt : ca1 + nm.ga)};
  const int md[3] = {nm.mdx, nm.mdy, nm.mdz};
  int a[3], b[3];
  for (int k = 0; k < 3; k++) {
    a[k] = max(lo[k], 0) >> 3;
    b[k] = min(hi[k] >> 3, md[k] - 1);
  }
  // eight blocks along x, four along y a step of the warp
  const int lane = threadIdx.x & 31;
  for (int z = a[2]; z <= b[2]; z++)
    for (int y = a[1] + (lane >> 3); y - (lane >> 3) <= b[1]; y += 4)
      for (int x = a[0] + (lane & 7); x - (lane & 7) <= b[0]; x += 8) {
        const bool any = x <= b[0] && y <= b[1] && nm.dmap[idx3(x, y, z, nm.mdx, nm.mdy)] != 0;
        if (__any_sync(0xffffffffu, any)) return true;
      }
  return false;
}

// Radius bound of one tile of a dilation pass, from the map of the largest
// raw radius per 16^3 fine voxels: over the tile's x columns and outputs,
// and its two third-axis coordinates widened by `rext` (the y pass feeds z
// outputs up to a halo away).  Every warp finds it for itself (4 x 4 map
// cells across the tile and two along the third axis a step): no barrier.
__device__ int tile_radius(const uint8_t* __restrict__ rmap, int mbx, int mby, int nx, int n3, int axis, int nout,
                           int o0, int rext, int bx, int bz) {
  const int lane = threadIdx.x & 31;
  const int ix = ((bx * kDpxCols) >> 4) + (lane & 3), ia = (o0 >> 4) + ((lane >> 2) & 3);
  const int ta = max(2 * bz - rext, 0) >> 4, tb = min(2 * bz + 1 + rext, n3 - 1) >> 4;
  int m = 0;
  if (16 * ix < nx && 16 * ia < nout)
    for (int it = ta + (lane >> 4); it <= tb; it += 2) {
      const int v = rmap[idx3(ix, axis == 1 ? ia : it, axis == 1 ? it : ia, mbx, mby)];
      m = v > m ? v : m;
    }
  return clamp_radius(__reduce_max_sync(0xffffffffu, m));
}

// First tap k at which the kernel alone reaches d (the -side of LAT lags by
// one tap and ends with it).
template <int G>
__device__ __forceinline__ int last_tap(uint32_t d) {
  if (G == KERN_CUBE) return (int)d;
  const float s = __fsqrt_rn((float)d);
  if (G == KERN_LAT) return (int)ceilf(s);
  if (G == KERN_CEN2) return (int)ceilf(0.5f * (s + 1.f));
  return (int)ceilf(0.5f * s) + 1;  // KERN_LAT2
}

// One tile of a min-plus pass: 64 columns x 64 outputs x 2 third-axis
// slices, at tile coordinates (bx, by, bz) along (x, outputs, slice pairs),
// the need map's out0 / third0 offsets included.  The whole block works on
// it.  The taps are at most a third of what a tile costs, so the rest is
// kept short: 16-byte loads (a thread: 8 or 16 columns of a row, every 16th
// or 32nd row of its slice), window ends by a square root, the radius bound
// and the need test per warp without barriers, thresholds as packed adds
// whose sign bits collect in one word.  Warps whose 16 outputs lie past the
// field skip the taps (extents are multiples of 16).  Against row-wise
// 4-byte loads or a TMA box re-read for its minimum, a search loop for the
// window's end, two walks over the maps with divisions and barriers, and a
// packing of its own per output: dilation z at 512^3, radius 12, 2017 -> 851
// instructions a warp's 16 rows (the taps are 448) and 0.287 -> 0.152 ms;
// the six passes at 1024^3 with a radius field 9.6 -> 6.4 ms.  Bound by the
// ALU pipe (70-74% busy) and, at the start of a tile, by its loads; sums on
// the FMA pipe with three-input minima instead of add-mins, three blocks an
// SM instead of four and an exit test every fourth tap were no faster.
template <int G, typename TIn, int FIN>
__device__ __forceinline__ void dpx_tile(const TIn* __restrict__ in, uint16_t* __restrict__ out16,
                                         uint8_t* __restrict__ out8, int nx, int ny, int nz, int axis, int sub,
                                         int halo, uint32_t cap, RField R, int uniform_r, int rx, int ry,
                                         const uint8_t* __restrict__ rmap, int rext, const NeedMap& need, int bx,
                                         int by, int bz) {
  extern __shared__ uint4 tile_raw[];
  uint32_t* tileu = reinterpret_cast<uint32_t*>(tile_raw);
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int tpar = w >> 2, grp = w & 3;
  const int x = bx * kDpxCols + 2 * lane;
  const int na = axis == 1 ? ny : nz;
  const int n3 = axis == 1 ? nz : ny;
  const int nout = sub ? na / 2 : na;
  const int third = 2 * bz + tpar;
  const int64_t sa = axis == 1 ? (int64_t)nx : (int64_t)nx * ny;
  const int64_t s3 = axis == 1 ? (int64_t)nx * ny : (int64_t)nx;
  const int o0 = by * kDpxOut;
  const int lo = (sub ? 2 * o0 + 1 : o0) - halo;
  const int span = (sub ? 2 * kDpxOut - 1 : kDpxOut) + 2 * halo;
  // Dilation passes with a radius field use the tile's own radius bound:
  // a smaller window (halo_e) and saturation value (cap_e).  Every output
  // that reads this tile has r(p) <= rt, so terms >= (rt+1)^2 never decide.
  int halo_e = halo;
  if (rmap != nullptr && !sub) {
    const int rt = tile_radius(rmap, nx >> 4, ny >> 4, nx, n3, axis, nout, o0, rext, bx, bz);
    const uint32_t ct = G == KERN_CUBE ? (uint32_t)(rt + 1) : (uint32_t)((rt + 1) * (rt + 1));
    cap = ct < cap ? ct : cap;
    halo_e = rt + 2 < halo ? rt + 2 : halo;
  }
  // Erosion outputs matter only where the dilation has voxels (and the
  // passes feeding them within their window): a tile outside writes its
  // saturation value ("not eroded") without work.
  const bool needed = tile_needed(need, axis, sub, o0, nout, bx, bz);
  if (FIN == 4 && !needed) return;  // (block-uniform; no tagged cell)
  const int skip = needed ? halo - halo_e : span;  // tile rows never read
  const uint32_t capp = cap | (cap << 16);
  uint32_t* tile = tileu + tpar * span * 32;
  const bool colok = x < nx && third < n3;
  __shared__ uint32_t warp_min[8];
  {
    uint32_t vmin = capp;  // smallest loaded value (both lanes)
    const bool slice = third < n3;
    if (sizeof(TIn) == 1) {
      const int c = threadIdx.x & 3, x0 = bx * kDpxCols + 16 * c;
      const TIn* src = in + x0 + s3 * third;
      const bool ok = slice && x0 < nx;
#pragma unroll 2
      for (int s = skip + ((threadIdx.x & 127) >> 2); s < span - skip; s += 32) {
        const int p = lo + s;
        uint4 v0 = make_uint4(capp, capp, capp, capp), v1 = v0;
        if (ok && p >= 0 && p < na) {
          const uint4 q = *reinterpret_cast<const uint4*>(src + sa * p);
          v0 = clamp4(make_uint4(widen_pair<G>(q.x, 0x4140u), widen_pair<G>(q.x, 0x4342u), widen_pair<G>(q.y, 0x4140u),
                                 widen_pair<G>(q.y, 0x4342u)), capp);
          v1 = clamp4(make_uint4(widen_pair<G>(q.z, 0x4140u), widen_pair<G>(q.z, 0x4342u), widen_pair<G>(q.w, 0x4140u),
                                 widen_pair<G>(q.w, 0x4342u)), capp);
        }
        uint4* dst = reinterpret_cast<uint4*>(tile + s * 32 + 8 * c);
        dst[0] = v0;
        dst[1] = v1;
        vmin = min4(v1, min4(v0, vmin));
      }
    } else {
      const int c = threadIdx.x & 7, x0 = bx * kDpxCols + 8 * c;
      const TIn* src = in + x0 + s3 * third;
      const bool ok = slice && x0 < nx;
#pragma unroll 4
      for (int s = skip + ((threadIdx.x & 127) >> 3); s < span - skip; s += 16) {
        const int p = lo + s;
        uint4 v = make_uint4(capp, capp, capp, capp);
        if (ok && p >= 0 && p < na) v = clamp4(*reinterpret_cast<const uint4*>(src + sa * p), capp);
        *reinterpret_cast<uint4*>(tile + s * 32 + 4 * c) = v;
        vmin = min4(v, vmin);
      }
    }
    const uint32_t mw = __reduce_min_sync(0xffffffffu, min(vmin & 0xffffu, vmin >> 16));
    if (lane == 0) warp_min[w] = mw;
  }
  __syncthreads();
  // Every tile value is >= tmin, so a tap whose kernel value reaches
  // cap - tmin cannot bring an output below the saturation value cap: the
  // window of this tile ends at the last tap below it (kernels grow with
  // |delta|).  Erosion passes: their inputs carry the per-site offset
  // K - 4 (r - 1)^2, so tiles whose sites all have small radii need short
  // windows; dilation passes: tiles whose inputs are all far from the input
  // stop early.
  uint32_t tmin = warp_min[0];
#pragma unroll
  for (int i = 1; i < 8; i++) tmin = min(tmin, warp_min[i]);
  const int obase = o0 + grp * kDpxPer;
  const bool finite = needed && tmin < cap && obase < nout;  // else every output keeps cap
  // (the cube combines by the larger of value and kernel: its window ends
  // with the kernel alone)
  if (G == KERN_CUBE) tmin = 0;
  const int halo_t = min(halo_e, max(last_tap<G>(cap - tmin), 1));
  const int sp0 = (sub ? 2 * obase + 1 : obase) - lo;
  uint32_t best[kDpxPer];
  // The lattice-point erosion (KERN_LAT2) is the only pass with outputs at
  // every other position (sub, step 2) and the only one that has them:
  // each instantiation compiles one of the two tap loops.
  constexpr bool kSub = G == KERN_LAT2;
  if (finite && !kSub) {
    // Register sliding windows: wp[(j + k) % 16] holds tile row sp0 + j + k
    // and wm[(j - k) mod 16] holds row sp0 + j - k, so that after tap k only
    // one new row per side is loaded (into the slot its leaving row frees).
    // Rows read: sp0 - halo_t .. sp0 + 15 + halo_t (halo_t <= halo_e, and
    // at least the rows sp0 - 1 and sp0 + 16 of the first window), inside
    // [skip, span - skip).
    const uint32_t* tcol = tile + lane;
    uint32_t wp[kDpxPer], wm[kDpxPer];
#pragma unroll
    for (int j = 0; j < kDpxPer; j++) {
      wp[j] = tcol[(sp0 + j + (j < 1 ? kDpxPer : 0)) * 32];
      wm[j] = tcol[(sp0 + (j < kDpxPer - 1 ? j : -1)) * 32];
    }
    const uint32_t g0 = gpair<G>(0, cap);
#pragma unroll
    for (int j = 0; j < kDpxPer; j++) best[j] = step_min<G>(tcol[(sp0 + j) * 32], g0, capp);
    uint32_t gprev = g0;  // +side kernel of the previous tap (the -side of this one for LAT, CUBE)
    for (int kb = 0; kb <= halo_t; kb += kDpxPer) {
#pragma unroll
      for (int u = 0; u < kDpxPer; u++) {
        const int k = kb + u;
        if (k == 0) continue;
        if (k > halo_t) goto dpx_done;
        const uint32_t graw = kern_pos<G>(k);
        const uint32_t gp = pack_cap(graw, cap);
        const uint32_t gm_ = G == KERN_CEN2 ? gp : gprev;
        gprev = gp;
#pragma unroll
        for (int j = 0; j < kDpxPer; j++) {
          best[j] = step_min<G>(wp[(j + u) % kDpxPer], gp, best[j]);
          best[j] = step_min<G>(wm[(j - u + kDpxPer) % kDpxPer], gm_, best[j]);
        }
        if (k == halo_t) goto dpx_done;  // no further tap: load nothing past the window
        // rows sp0 + k + 16 and sp0 - k - 1 enter; the slots of rows
        // sp0 + k and sp0 + 15 - k are free now (k < halo_e keeps both in the window)
        wp[u] = tcol[(sp0 + k + kDpxPer) * 32];
        wm[(kDpxPer - 1 - u) % kDpxPer] = tcol[(sp0 - k - 1) * 32];
        if ((u & 7) == 3) {  // every eighth tap: leave once no output can improve
          uint32_t m = best[0];
#pragma unroll
          for (int j = 1; j + 1 < kDpxPer; j += 2) m = __vimax3_u16x2(m, best[j], best[j + 1]);
          m = __vmaxu2(m, best[kDpxPer - 1]);
          const uint32_t mx = (m & 0xffffu) > (m >> 16) ? (m & 0xffffu) : (m >> 16);
          // smallest kernel value of the taps to come (k + 1 on either side)
          const uint32_t nxt = G == KERN_CEN2 ? kern_pos<G>(k + 1) : graw;
          if (__all_sync(0xffffffffu, nxt + tmin >= mx)) goto dpx_done;
        }
      }
    }
  dpx_done:;
  } else if (finite && kSub) {
    // Outputs at every other position (sub): output j sits on tile row
    // sp0 + 2j and reads rows sp0 + 2j + delta.  The taps split by the
    // parity of delta into two stride-1 sequences over the rows of one
    // parity, R(h) = row b + 2h (b = sp0: delta = 2d; b = sp0 - 1:
    // delta = 2d - 1; h = j + d), each run with the register sliding window
    // of the full-resolution path: one new row per side and tap instead of
    // one load per output and tap.
#pragma unroll
    for (int j = 0; j < kDpxPer; j++) best[j] = capp;
    const uint32_t* tcol = tile + lane;
#pragma unroll 1
    for (int par = 0; par < 2; par++) {
      const int e0 = -par;                   // delta of the group's centre tap (d = 0)
      const uint32_t* tb = tcol + (sp0 - par) * 32;  // R(h) = tb[64 h]
      const int kp = (halo_t - e0) >> 1;     // plus taps d = k: delta = 2k + e0 <= halo_t
      const int km = (halo_t + e0) >> 1;     // minus taps d = -k: delta = -2k + e0 >= -halo_t
      const int kmax = kp > km ? kp : km;
      uint32_t wp[kDpxPer], wm[kDpxPer];
#pragma unroll
      for (int j = 0; j < kDpxPer; j++) {
        wp[j] = tb[(j < 1 ? kDpxPer : j) * 64];
        wm[j] = tb[(j < kDpxPer - 1 ? j : -1) * 64];
      }
      const uint32_t gc = pack_cap(kern_g<G>(e0), cap);
#pragma unroll
      for (int j = 0; j < kDpxPer; j++) best[j] = step_min<G>(tb[j * 64], gc, best[j]);
      for (int kb = 0; kb <= kmax; kb += kDpxPer) {
#pragma unroll
        for (int u = 0; u < kDpxPer; u++) {
          const int k = kb + u;
          if (k == 0) continue;
          if (k > kmax) goto sub_done;
          if (k <= kp) {
            const uint32_t gp = pack_cap(kern_g<G>(2 * k + e0), cap);
#pragma unroll
            for (int j = 0; j < kDpxPer; j++) best[j] = step_min<G>(wp[(j + u) % kDpxPer], gp, best[j]);
          }
          if (k <= km) {
            const uint32_t gm_ = pack_cap(kern_g<G>(-2 * k + e0), cap);
#pragma unroll
            for (int j = 0; j < kDpxPer; j++)
              best[j] = step_min<G>(wm[(j - u + kDpxPer) % kDpxPer], gm_, best[j]);
          }
          if (k == kmax) goto sub_done;
          // R(k + 16) and R(-k - 1) enter for the next tap, in the slots
          // that R(k) and R(15 - k) leave
          if (k < kp) wp[u] = tb[(k + kDpxPer) * 64];
          if (k < km) wm[(kDpxPer - 1 - u) % kDpxPer] = tb[(-k - 1) * 64];
          if ((u & 7) == 3) {  // every eighth tap: leave once no output can improve
            uint32_t m = best[0];
#pragma unroll
            for (int j = 1; j + 1 < kDpxPer; j += 2) m = __vimax3_u16x2(m, best[j], best[j + 1]);
            m = __vmaxu2(m, best[kDpxPer - 1]);
            const uint32_t mx = (m & 0xffffu) > (m >> 16) ? (m & 0xffffu) : (m >> 16);
            const uint32_t np = k + 1 <= kp ? kern_g<G>(2 * (k + 1) + e0) : 0xffffu;
            const uint32_t nm = k + 1 <= km ? kern_g<G>(-2 * (k + 1) + e0) : 0xffffu;
            const uint32_t nxt = np < nm ? np : nm;
            if (__all_sync(0xffffffffu, nxt + tmin >= mx)) goto sub_done;
          }
        }
      }
    sub_done:;
    }
  } else {
#pragma unroll
    for (int j = 0; j < kDpxPer; j++) best[j] = capp;
  }
  if (FIN == 0) {
    if (!colok || obase >= nout) return;
    const int64_t osa = axis == 1 ? (int64_t)nx : (int64_t)nx * ny;
    const int64_t os3 = axis == 1 ? (int64_t)nx * nout : (int64_t)nx;
    uint16_t* dst = out16 + x + osa * obase + os3 * third;
#pragma unroll
    for (int j = 0; j < kDpxPer; j++) *reinterpret_cast<uint32_t*>(dst + osa * j) = best[j];
  } else if (FIN == 3) {
    if (!colok || obase >= nout) return;
    // x is a cell index here; outputs are cells (x, third, o)
    uint8_t* dst = out8 + idx3(x, third, obase, rx, ry);
    const uint32_t t1 = 0x80008000u - capp;
#pragma unroll
    for (int j = 0; j < kDpxPer; j++) {
      const uint32_t f = ~(best[j] + t1);  // bit 15 of a half: value < cap
      *reinterpret_cast<uint16_t*>(dst + (int64_t)rx * ry * j) = (uint16_t)(((f >> 15) & 1u) | ((f >> 23) & 0x100u));
    }
  } else {
    // threshold then pack 2 (x) x 2 (y = third pair) x 2 (z) bits per byte.
    // value < T exactly when bit 15 of value + 0x8000 - T is clear (both at
    // most 0x7fff); the 16 outputs' bits collect in one word, the lower
    // column's in its lower half.
    __shared__ uint32_t xch[4][32][2];
    uint32_t acc = 0xffffffffu;  // bit j of a half: output j is not below its threshold
    if (colok && obase < nout) {
      const bool field = FIN == 1 && R.p != nullptr;
      const int8_t* rp = nullptr;
      uint32_t t1;
      if (FIN == 1) {
        const uint32_t r1 = (uint32_t)clamp_radius(uniform_r) + 1u, t = G == KERN_CUBE ? r1 : r1 * r1;
        t1 = 0x80008000u - (t | (t << 16));
        if (field) rp = R.p + (int64_t)x + third * R.sy + obase * R.sz;
      } else {
        t1 = 0x80008000u - capp;
      }
      if (field) {
#pragma unroll
        for (int j = 0; j < kDpxPer; j++) {
          // x even and even strides: a 2-byte aligned pair of radii,
          // sign-extended to the halves, at least 2 (at most 127 as bytes)
          const uint32_t rr = *reinterpret_cast<const uint16_t*>(rp + j * R.sz);
          uint32_t r2;
          asm("prmt.b32 %0, %1, 0, 0x9180;" : "=r"(r2) : "r"(rr));
          const uint32_t r1 = __vmaxs2(r2, 0x00020002u) + 0x00010001u;  // r + 1 (<= 128)
          uint32_t e = best[j] + 0x80008000u;
          if (G == KERN_CUBE) {
            e -= r1;  // value <= r
          } else {
            const uint32_t a = r1 & 0xffffu, b = r1 >> 16;
            e = e - a * a - (r1 & 0xffff0000u) * b;  // value < (r + 1)^2
          }
          acc = ((acc >> 1) & 0x7fff7fffu) | (e & 0x80008000u);
        }
      } else {
#pragma unroll
        for (int j = 0; j < kDpxPer; j++) acc = ((acc >> 1) & 0x7fff7fffu) | ((best[j] + t1) & 0x80008000u);
      }
    }
    // bits of z pair q to byte q: z even to bits 0, 1, z odd to bits 4, 5
    uint32_t bytes[2];
    {
      const uint32_t f = ~acc, u = f & 0xffffu, v = f >> 16;  // the two columns
      const uint32_t e = (u & 0x5555u) | ((v & 0x5555u) << 1), o = ((u >> 1) & 0x5555u) | (v & 0xaaaau);
#pragma unroll
      for (int h = 0; h < 2; h++) {
        uint32_t p = ((e >> (8 * h)) & 0xffu) | (((o >> (8 * h)) & 0xffu) << 16);  // four 2-bit fields of each
        p = (p | (p << 4)) & 0x0f0f0f0fu;
        p = (p | (p << 2)) & 0x33333333u;  // nibble per field
        // e fields in the lower half, o fields in the upper: byte q = e_q | o_q << 4
        const uint32_t lo16 = p & 0xffffu, hi16 = p >> 16;
        uint32_t be = (lo16 | (lo16 << 8)) & 0x00ff00ffu, bo = (hi16 | (hi16 << 8)) & 0x00ff00ffu;
        be = (be | (be << 4)) & 0x0f0f0f0fu;
        bo = (bo | (bo << 4)) & 0x0f0f0f0fu;
        bytes[h] = (be | (bo << 4)) << (2 * tpar);
      }
    }
    if (tpar == 1) {
      xch[grp][lane][0] = bytes[0];
      xch[grp][lane][1] = bytes[1];
    }
    __syncthreads();
    if (tpar == 0 && colok && obase < nout) {
      bytes[0] |= xch[grp][lane][0];
      bytes[1] |= xch[grp][lane][1];
      const int64_t o = idx3(x >> 1, third >> 1, obase / 2, rx, ry);
      uint8_t* dst = out8 + o;
#pragma unroll
      for (int q = 0; q < kDpxPer / 2; q++) {
        const uint32_t e = (bytes[q >> 2] >> (8 * (q & 3))) & 0xffu;
        if (FIN == 4) {
          // (tags exist in groups of 16 cells along x that meet the region)
          const int cx = x >> 1, cy = third >> 1, cz = obase / 2 + q;
          if (cbox_meets(need.roi, cx & ~15, cx | 15, cy, cy, cz, cz) && R.p[o + (int64_t)rx * ry * q] != 0)
            dst[(int64_t)rx * ry * q] = (uint8_t)~e;
        } else {
          dst[(int64_t)rx * ry * q] = (uint8_t)e;
        }
      }
    }
  }
}

template <int G, typename TIn, int FIN>
__global__ void __launch_bounds__(256, 4) k_pass_dpx(const TIn* __restrict__ in, uint16_t* __restrict__ out16,
                                                  uint8_t* __restrict__ out8, int nx, int ny, int nz, int axis,
                                                  int sub, int halo, uint32_t cap, RField R,
                                                  int uniform_r, int rx, int ry, const uint8_t* __restrict__ rmap,
                                                  int rext, const __grid_constant__ NeedMap need) {
  dpx_tile<G, TIn, FIN>(in, out16, out8, nx, ny, nz, axis, sub, halo, cap, R, uniform_r, rx, ry, rmap, rext, need,
                        (int)blockIdx.x, (int)blockIdx.y + need.out0, (int)blockIdx.z + need.third0);
}

template <int G, typename TIn, int FIN>
static void launch_dpx(const TIn* in, uint16_t* out16, uint8_t* out8, int nx, int ny, int nz, int axis, int sub,
                       int halo, uint32_t cap, RField R, int uniform_r, int rx, int ry, cudaStream_t st,
                       KernelCounter* kc, const char* name, const uint8_t* rmap = nullptr, int rext = 0,
                       NeedMap need = NeedMap{nullptr, 0, 0, 0, 0, 0, 0, 0, 0, CBox{{0, 0, 0}, {1 << 30, 1 << 30, 1 << 30}}}) {
  if ((G == KERN_LAT2) != (sub != 0)) return;  // (every call site pairs them; see k_pass_dpx)
  const size_t smem = dpx_smem_bytes(sub, halo);
  ensure_dynamic_smem(reinterpret_cast<const void*>(k_pass_dpx<G, TIn, FIN>), smem);
  const int na = axis == 1 ? ny : nz;
  const int n3 = axis == 1 ? nz : ny;
  const int nout = sub ? na / 2 : na;
  dim3 g((nx + kDpxCols - 1) / kDpxCols, need.out_n > 0 ? need.out_n : (nout + kDpxOut - 1) / kDpxOut,
         need.third_n > 0 ? need.third_n : (n3 + 1) / 2);
  GM_LAUNCH(kc, name, st,
            k_pass_dpx<G, TIn, FIN><<<g, 256, smem, st>>>(in, out16, out8, nx, ny, nz, axis, sub, halo, cap, R,
                                                          uniform_r, rx, ry, rmap, rext, need));
}

// ---- grouped min-plus passes (many grids, one persistent launch) ----
//
// One pass of the closing of many grids (the same pass of each: same
// kernel shape, own sizes, radius bounds, buffers and need maps), recorded
// by launch_close in phase mode and run as one launch: a grid of resident
// blocks pulls tiles of all the grids from one work counter, so that small
// grids fill the GPU together and the cost differences between tiles
// (window lengths vary with the local radius and the early exits) balance
// across blocks.  The tiles and their results are those of the per-grid
// launches (the same tile function on the same tile coordinates).
struct DpxJob {
  const void* in;
  uint16_t* out16;
  uint8_t* out8;
  int nx, ny, nz, axis, sub, halo;
  uint32_t cap;
  RField R;
  int uniform_r, rx, ry;
  const uint8_t* rmap;
  int rext;
  NeedMap need;
  int gx, gy, gz;  // tiles of this grid's pass
  int first;       // its first work item (tiles of the jobs before it)
};

// Instantiations a grouped launch may hold: the passes of launch_close.
enum DpxKind {
  DPXK_LAT_U8_0 = 0,   // sphere dilation y
  DPXK_LAT_U16_1,      // sphere dilation z (threshold + packing)
  DPXK_CUBE_U8_0,      // cube dilation y
  DPXK_CUBE_U16_1,     // cube dilation z
  DPXK_CEN2_U16_0,     // centre erosion y
  DPXK_CEN2_U16_2,     // centre erosion z
  DPXK_CEN2_U16_4,     // the same, applied to the closing (GM_REF)
  DPXK_LAT2_U16_0,     // lattice-point erosion y
  DPXK_LAT2_U16_3,     // lattice-point erosion z
  DPXK_COUNT
};
template <int G, typename TIn, int FIN>
constexpr int dpx_kind() {
  return G == KERN_LAT && sizeof(TIn) == 1 && FIN == 0    ? DPXK_LAT_U8_0
         : G == KERN_LAT && sizeof(TIn) == 2 && FIN == 1  ? DPXK_LAT_U16_1
         : G == KERN_CUBE && sizeof(TIn) == 1 && FIN == 0 ? DPXK_CUBE_U8_0
         : G == KERN_CUBE && sizeof(TIn) == 2 && FIN == 1 ? DPXK_CUBE_U16_1
         : G == KERN_CEN2 && sizeof(TIn) == 2 && FIN == 0 ? DPXK_CEN2_U16_0
         : G == KERN_CEN2 && sizeof(TIn) == 2 && FIN == 2 ? DPXK_CEN2_U16_2
         : G == KERN_CEN2 && sizeof(TIn) == 2 && FIN == 4 ? DPXK_CEN2_U16_4
         : G == KERN_LAT2 && sizeof(TIn) == 2 && FIN == 0 ? DPXK_LAT2_U16_0
         : G == KERN_LAT2 && sizeof(TIn) == 2 && FIN == 3 ? DPXK_LAT2_U16_3
                                                          : -1;
}

template <int G, typename TIn, int FIN>
__global__ void __launch_bounds__(256, 4) k_pass_dpx_group(const DpxJob* __restrict__ jobs, int njobs, int total,
                                                        unsigned int* __restrict__ counter) {
  __shared__ int item_s;     // the block's current work item
  __shared__ int job_end_s;  // first item past the job held in job_s
  // the job of the current item (kept while the block's items stay in it)
  __shared__ __align__(16) unsigned char job_raw[sizeof(DpxJob)];
  DpxJob& job_s = *reinterpret_cast<DpxJob*>(job_raw);
  if (threadIdx.x == 0) {
    item_s = (int)atomicAdd(counter, 1u);
    job_end_s = -1;
  }
  __syncthreads();
  for (;;) {
    const int item = item_s;
    if (item >= total) return;  // block-uniform
    const bool other_job = item >= job_end_s || item < job_s.first;  // (job_end_s = -1 at first)
    // every thread has read job_s / job_end_s before warp 0 may rewrite
    // them, so that the branch below (and its barrier) is block-uniform
    __syncthreads();
    if (other_job) {
      if (threadIdx.x < 32) {
        // the job holding the item: the last one whose first item is <= it
        int lo = 0, hi = njobs - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if (jobs[mid].first <= item) lo = mid; else hi = mid - 1;
        }
        const uint32_t* src = reinterpret_cast<const uint32_t*>(jobs + lo);
        uint32_t* dst = reinterpret_cast<uint32_t*>(&job_s);
        for (int k = threadIdx.x; k < (int)(sizeof(DpxJob) / 4); k += 32) dst[k] = src[k];
        if (threadIdx.x == 0) job_end_s = jobs[lo].first + jobs[lo].gx * jobs[lo].gy * jobs[lo].gz;
      }
      __syncthreads();
    }
    // the next item, fetched while this tile runs (consumed after it)
    int next = 0;
    if (threadIdx.x == 0) next = (int)atomicAdd(counter, 1u);
    const DpxJob& b = job_s;
    const int t = item - b.first;
    const int bx = t % b.gx, by = (t / b.gx) % b.gy, bz = t / (b.gx * b.gy);
    dpx_tile<G, TIn, FIN>(static_cast<const TIn*>(b.in), b.out16, b.out8, b.nx, b.ny, b.nz, b.axis, b.sub, b.halo,
                          b.cap, b.R, b.uniform_r, b.rx, b.ry, b.rmap, b.rext, b.need, bx, by + b.need.out0, bz + b.need.third0);
    __syncthreads();  // every thread is done with this tile (its shared memory, job_s, item_s)
    if (threadIdx.x == 0) item_s = next;
    __syncthreads();
  }
}

struct DpxGroup {
  int kind = -1;
  size_t smem = 0;
  std::vector<DpxJob> jobs;
  int total = 0;
  DpxJob* h_jobs = nullptr;  // pinned copy read by the upload (also at graph replays)
  DpxJob* d_jobs = nullptr;
  unsigned int* d_counter = nullptr;
  int cap = 0;
  cudaEvent_t uploaded = nullptr;  // after the last upload outside a capture (h_jobs free again)
};

DpxGroup* dpx_group_new() { return new DpxGroup(); }

void dpx_group_free(DpxGroup* g) {
  if (!g) return;
  if (g->uploaded) {
    cudaEventSynchronize(g->uploaded);
    cudaEventDestroy(g->uploaded);
  }
  if (g->h_jobs) cudaFreeHost(g->h_jobs);
  cudaFree(g->d_jobs);
  cudaFree(g->d_counter);
  delete g;
}

void dpx_group_clear(DpxGroup* g) {
  g->kind = -1;
  g->smem = 0;
  g->jobs.clear();
  g->total = 0;
}

int dpx_group_size(const DpxGroup* g) { return (int)g->jobs.size(); }

int dpx_group_room(const DpxGroup* g) { return g->cap; }

cudaError_t dpx_group_reserve(DpxGroup* g, int njobs) {
  if (njobs <= g->cap) return cudaSuccess;
  cudaError_t e;
  if (g->uploaded && (e = cudaEventSynchronize(g->uploaded)) != cudaSuccess) return e;
  if (!g->uploaded && (e = cudaEventCreateWithFlags(&g->uploaded, cudaEventDisableTiming)) != cudaSuccess) return e;
  if (g->h_jobs) cudaFreeHost(g->h_jobs);
  cudaFree(g->d_jobs);
  g->h_jobs = nullptr;
  g->d_jobs = nullptr;
  g->cap = 0;
  if ((e = cudaMallocHost(&g->h_jobs, sizeof(DpxJob) * njobs)) != cudaSuccess) return e;
  if ((e = cudaMalloc(&g->d_jobs, sizeof(DpxJob) * njobs)) != cudaSuccess) return e;
  if (!g->d_counter && (e = cudaMalloc(&g->d_counter, sizeof(unsigned int))) != cudaSuccess) return e;
  g->cap = njobs;
  return cudaSuccess;
}

// Records one grid's pass (the arguments of launch_dpx) into the group.
template <int G, typename TIn, int FIN>
static bool dpx_record(DpxGroup* grp, const TIn* in, uint16_t* out16, uint8_t* out8, int nx, int ny, int nz, int axis,
                       int sub, int halo, uint32_t cap, RField R, int uniform_r, int rx, int ry,
                       const uint8_t* rmap, int rext, NeedMap need) {
  constexpr int kind = dpx_kind<G, TIn, FIN>();
  if (kind < 0 || (grp->kind >= 0 && grp->kind != kind) || (G == KERN_LAT2) != (sub != 0)) return false;
  grp->kind = kind;
  grp->smem = std::max(grp->smem, dpx_smem_bytes(sub, halo));
  const int na = axis == 1 ? ny : nz;
  const int n3 = axis == 1 ? nz : ny;
  const int nout = sub ? na / 2 : na;
  DpxJob j;
  j.in = in;
  j.out16 = out16;
  j.out8 = out8;
  j.nx = nx;
  j.ny = ny;
  j.nz = nz;
  j.axis = axis;
  j.sub = sub;
  j.halo = halo;
  j.cap = cap;
  j.R = R;
  j.uniform_r = uniform_r;
  j.rx = rx;
  j.ry = ry;
  j.rmap = rmap;
  j.rext = rext;
  j.need = need;
  j.gx = (nx + kDpxCols - 1) / kDpxCols;
  j.gy = need.out_n > 0 ? need.out_n : (nout + kDpxOut - 1) / kDpxOut;
  j.gz = need.third_n > 0 ? need.third_n : (n3 + 1) / 2;
  j.first = grp->total;
  const long long tiles = (long long)j.gx * j.gy * j.gz;
  if (tiles <= 0) return true;
  if (grp->total + tiles > 0x7fffffffLL) return false;
  grp->total += (int)tiles;
  grp->jobs.push_back(j);
  return true;
}

static const char* const kDpxGroupNames[DPXK_COUNT] = {
    "k_pass_dil_y_group", "k_pass_dil_z_group",  "k_pass_dil_y_group",  "k_pass_dil_z_group",
    "k_pass_ero_y_group", "k_pass_ero_z_group", "k_pass_ero_z_group", "k_pass_erob_y_group", "k_pass_erob_z_group"};

template <int G, typename TIn, int FIN>
static cudaError_t dpx_group_go(DpxGroup* g, int sms, cudaStream_t st, KernelCounter* kc) {
  const void* k = reinterpret_cast<const void*>(k_pass_dpx_group<G, TIn, FIN>);
  cudaError_t e = ensure_dynamic_smem(k, g->smem);
  if (e != cudaSuccess) return e;
  int per_sm = 0;
  if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_pass_dpx_group<G, TIn, FIN>, 256, g->smem)) !=
      cudaSuccess)
    return e;
  const int blocks = std::max(1, std::min(g->total, std::max(1, sms) * std::max(1, per_sm)));
  GM_LAUNCH(kc, kDpxGroupNames[g->kind], st,
            k_pass_dpx_group<G, TIn, FIN><<<blocks, 256, g->smem, st>>>(g->d_jobs, (int)g->jobs.size(), g->total,
                                                                        g->d_counter));
  return cudaGetLastError();
}

cudaError_t dpx_group_launch(DpxGroup* g, int sms, cudaStream_t st, KernelCounter* kc) {
  if (g->jobs.empty()) return cudaSuccess;
  const int n = (int)g->jobs.size();
  if (n > g->cap) return cudaErrorInvalidValue;  // dpx_group_reserve first (not while capturing)
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaError_t e = cudaStreamIsCapturing(st, &cs);
  if (e != cudaSuccess) return e;
  const bool capturing = cs == cudaStreamCaptureStatusActive;
  // the previous upload has read the pinned table (in a capture the caller
  // guarantees that no replay of an earlier graph over it is in flight)
  if (!capturing && (e = cudaEventSynchronize(g->uploaded)) != cudaSuccess) return e;
  memcpy(g->h_jobs, g->jobs.data(), sizeof(DpxJob) * n);
  if ((e = cudaMemcpyAsync(g->d_jobs, g->h_jobs, sizeof(DpxJob) * n, cudaMemcpyHostToDevice, st)) != cudaSuccess)
    return e;
  if (!capturing && (e = cudaEventRecord(g->uploaded, st)) != cudaSuccess) return e;
  if ((e = cudaMemsetAsync(g->d_counter, 0, sizeof(unsigned int), st)) != cudaSuccess) return e;
  switch (g->kind) {
    case DPXK_LAT_U8_0: return dpx_group_go<KERN_LAT, uint8_t, 0>(g, sms, st, kc);
    case DPXK_LAT_U16_1: return dpx_group_go<KERN_LAT, uint16_t, 1>(g, sms, st, kc);
    case DPXK_CUBE_U8_0: return dpx_group_go<KERN_CUBE, uint8_t, 0>(g, sms, st, kc);
    case DPXK_CUBE_U16_1: return dpx_group_go<KERN_CUBE, uint16_t, 1>(g, sms, st, kc);
    case DPXK_CEN2_U16_0: return dpx_group_go<KERN_CEN2, uint16_t, 0>(g, sms, st, kc);
    case DPXK_CEN2_U16_2: return dpx_group_go<KERN_CEN2, uint16_t, 2>(g, sms, st, kc);
    case DPXK_CEN2_U16_4: return dpx_group_go<KERN_CEN2, uint16_t, 4>(g, sms, st, kc);
    case DPXK_LAT2_U16_0: return dpx_group_go<KERN_LAT2, uint16_t, 0>(g, sms, st, kc);
    case DPXK_LAT2_U16_3: return dpx_group_go<KERN_LAT2, uint16_t, 3>(g, sms, st, kc);
    default: return cudaErrorInvalidValue;
  }
}

// A pass of launch_close: launched (a.phase < 0), recorded into a.group
// when it is the pass of the phase asked for, or skipped.  `at` counts the
// passes met so far.
template <int G, typename TIn, int FIN>
static bool dpx_step(const CloseArgs& a, int& at, const TIn* in, uint16_t* out16, uint8_t* out8, int nx, int ny,
                     int nz, int axis, int sub, int halo, uint32_t cap, RField R, int uniform_r, int rx, int ry,
                     cudaStream_t st, KernelCounter* kc, const char* name, const uint8_t* rmap = nullptr,
                     int rext = 0,
                     NeedMap need = NeedMap{nullptr, 0, 0, 0, 0, 0, 0, 0, 0,
                                            CBox{{0, 0, 0}, {1 << 30, 1 << 30, 1 << 30}}}) {
  bool ok = true;
  if (a.phase < 0)
    launch_dpx<G, TIn, FIN>(in, out16, out8, nx, ny, nz, axis, sub, halo, cap, R, uniform_r, rx, ry, st, kc, name,
                            rmap, rext, need);
  else if (a.phase == at)
    ok = a.group != nullptr && dpx_record<G, TIn, FIN>(a.group, in, out16, out8, nx, ny, nz, axis, sub, halo, cap, R,
                                                        uniform_r, rx, ry, rmap, rext, need);
  at++;
  return ok;
}

unsigned int* kernel_error_word() {
  void* p = nullptr;
  return cudaGetSymbolAddress(&p, g_kernel_errors) == cudaSuccess ? static_cast<unsigned int*>(p) : nullptr;
}

cudaError_t kernel_error_flags(unsigned int* flags, bool clear) {
  cudaError_t e = cudaMemcpyFromSymbol(flags, g_kernel_errors, sizeof(unsigned int));
  if (e == cudaSuccess && clear && *flags != 0) {
    const unsigned int zero = 0;
    e = cudaMemcpyToSymbol(g_kernel_errors, &zero, sizeof(unsigned int));
  }
  return e;
}

// Largest raw radius (>= 0) of each 16^3 block of fine voxels of a radius
// field (nx, ny, nz multiples of 16).  One block per (map y, map z) row of
// map cells (per 32 * CELLS of them where the rows are longer, blockIdx.z); a
// warp reads whole fine rows (lane l owns the 16-byte segments of map cells
// l, l + 32, ...), the 8 warps take every 8th of the 256 rows, so the block
// streams its 16 x 16 rows of the field front to back, eight 16-byte loads a
// lane in flight.  With d_rmax, the largest clamped radius is folded into
// *d_rmax as well.  Bound by the bytes it reads: 0.150 ms for 1024^3 (7.2
// TB/s; 0.172 with two rows in flight and bytewise maxima), and 23 instead of
// 32 us for 64 x 512 x 512.
constexpr int kRmapCells = 4;  // map cells per lane along x, at most (registers and shared memory)

// maxima of signed bytes, in 16-bit halves whose upper byte counts (the one
// below it decides between equals only): the odd bytes, and the even ones
// shifted up
struct ByteMax {
  uint32_t odd, even;
};
__device__ __forceinline__ void max_bytes(ByteMax& m, uint4 v) {
  m.odd = __vimax3_s16x2(__vimax3_s16x2(m.odd, v.x, v.y), v.z, v.w);
  m.even = __vimax3_s16x2(__vimax3_s16x2(m.even, v.x << 8, v.y << 8), v.z << 8, v.w << 8);
}

template <int CELLS>
__global__ void __launch_bounds__(256) k_radius_map(RField R, int mbx, int mby, int aligned,
                                                     uint8_t* __restrict__ out, int* __restrict__ d_rmax) {
  const int my = blockIdx.x, mz = blockIdx.y;
  const int wid = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int c0 = 32 * CELLS * (int)blockIdx.z, n = min(mbx - c0, 32 * CELLS);  // the block's map cells
  R.p += 16 * c0;
  __shared__ int part[8][32 * CELLS];
  int m[CELLS];
#pragma unroll
  for (int c = 0; c < CELLS; c++) m[c] = 0;
  if (aligned) {
    ByteMax b[CELLS];
#pragma unroll
    for (int c = 0; c < CELLS; c++) b[c].odd = b[c].even = 0u;  // (negative radii count as none)
    constexpr int kAhead = 8 / CELLS;  // rows in flight: eight loads a lane
    for (int r0 = wid; r0 < 256; r0 += 8 * kAhead) {
      uint4 v[kAhead][CELLS];
#pragma unroll
      for (int k = 0; k < kAhead; k++) {
        const int r = r0 + 8 * k;
        const int8_t* row = R.p + (int64_t)(16 * my + (r & 15)) * R.sy + (int64_t)(16 * mz + (r >> 4)) * R.sz;
#pragma unroll
        for (int c = 0; c < CELLS; c++) {
          const int cx = lane + 32 * c;
          v[k][c] = cx < n ? __ldcs(reinterpret_cast<const uint4*>(row + 16 * cx)) : make_uint4(0u, 0u, 0u, 0u);
        }
      }
#pragma unroll
      for (int k = 0; k < kAhead; k++)
#pragma unroll
        for (int c = 0; c < CELLS; c++) max_bytes(b[c], v[k][c]);
    }
#pragma unroll
    for (int c = 0; c < CELLS; c++) {
      const uint32_t t = __vmaxs2(b[c].odd, b[c].even);
      m[c] = (int)max((t >> 8) & 0xffu, t >> 24);
    }
  } else {
    for (int r = wid; r < 256; r += 8) {
      const int8_t* row = R.p + (int64_t)(16 * my + (r & 15)) * R.sy + (int64_t)(16 * mz + (r >> 4)) * R.sz;
#pragma unroll
      for (int c = 0; c < CELLS; c++) {
        const int cx = lane + 32 * c;
        if (cx < n)
#pragma unroll
          for (int j = 0; j < 16; j++) m[c] = max(m[c], (int)row[16 * cx + j]);
      }
    }
  }
#pragma unroll
  for (int c = 0; c < CELLS; c++) part[wid][lane + 32 * c] = m[c];
  __syncthreads();
  int gmax = 0;
  for (int cx = threadIdx.x; cx < n; cx += blockDim.x) {
    int t = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) t = max(t, part[k][cx]);
    out[c0 + cx + (int64_t)mbx * (my + (int64_t)mby * mz)] = (uint8_t)t;
    gmax = max(gmax, t);
  }
  if (d_rmax != nullptr && wid * 32 < n) {
    for (int o = 16; o > 0; o >>= 1) gmax = max(gmax, __shfl_xor_sync(0xffffffffu, gmax, o));
    if (lane == 0) atomicMax(d_rmax, clamp_radius(gmax));
  }
}

cudaError_t launch_radius_map(RField R, int nx, int ny, int nz, uint8_t* out, int* d_rmax, cudaStream_t st,
                              KernelCounter* kc) {
  const int mbx = nx / 16, mby = ny / 16, mbz = nz / 16;
  const int aligned = ((uintptr_t)R.p % 16 == 0 && R.sy % 16 == 0 && R.sz % 16 == 0) ? 1 : 0;
  if (d_rmax) cudaMemsetAsync(d_rmax, 0, sizeof(int), st);
  auto* kernel = mbx <= 32 ? k_radius_map<1> : (mbx <= 64 ? k_radius_map<2> : k_radius_map<kRmapCells>);
  const int parts = (mbx + 32 * kRmapCells - 1) / (32 * kRmapCells);
  GM_LAUNCH(kc, "k_radius_map", st, kernel<<<dim3(mby, mbz, parts), 256, 0, st>>>(R, mbx, mby, aligned, out, d_rmax));
  return cudaGetLastError();
}

cudaError_t launch_radius_map_dense(const int8_t* R, int nx, int ny, int nz, uint8_t* out, int* d_rmax,
                                    cudaStream_t st, KernelCounter* kc) {
  return launch_radius_map(RField{R, (int64_t)nx, (int64_t)nx * ny}, nx, ny, nz, out, d_rmax, st, kc);
}

// 1 for each 8^3 block of cells of a cell grid (rx, ry, rz multiples of
// 16) holding a non-zero byte: one warp per block, two 8-byte rows a lane.
__global__ void __launch_bounds__(256) k_occ_map8(const uint8_t* __restrict__ G, int rx, int ry, int mdx, int mdy,
                                                  int nblocks, uint8_t* __restrict__ out) {
  const int b = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (b >= nblocks) return;
  const int bx = b % mdx, by = (b / mdx) % mdy, bz = b / (mdx * mdy);
  uint64_t acc = 0;
#pragma unroll
  for (int k = 0; k < 2; k++) {
    const int r = lane + 32 * k;  // row r of the block: y = r & 7, z = r >> 3
    acc |= *reinterpret_cast<const uint64_t*>(G + idx3(8 * bx, 8 * by + (r & 7), 8 * bz + (r >> 3), rx, ry));
  }
  const int any = __any_sync(0xffffffffu, acc != 0);
  if (lane == 0) out[b] = any ? 1 : 0;
}

// ---------------------------------------------------------------------
// cell-level kernels; cell grids of this section are boxes of rx * ry * rz
// cells (Dims), z = blockIdx.z
// ---------------------------------------------------------------------

struct DataRes { int v[3]; };

struct Dims { int x, y, z; };
__device__ __forceinline__ int64_t cidx(int x, int y, int z, Dims d) { return idx3(x, y, z, d.x, d.y); }

// Dilation flags from a resident squared lattice distance field E of the
// input grid (u16 per fine voxel: the value the dilation's z pass computes,
// saturated at (rmax + 1)^2 for a bound rmax of every radius asked for).
// The flag of fine voxel p is E(p) < (r(p) + 1)^2, the z pass's own test, so
// the bytes equal the passes' output.  Four cells per thread, bit
// x + 2y + 4z of the 2x2x2 fine voxels of a cell.
__global__ void __launch_bounds__(256) k_dil_threshold(const uint16_t* __restrict__ E, int64_t esy, int64_t esz,
                                                       RField R, int uniform_r, Dims g, uint8_t* __restrict__ out,
                                                       CBox roi) {
  const int x4 = 4 * (blockIdx.x * 64 + threadIdx.x);
  const int y = blockIdx.y * 4 + threadIdx.y, z = blockIdx.z;
  if (x4 >= g.x || y >= g.y || !cbox_meets(roi, x4, x4 + 3, y, y, z, z)) return;
  const int ru = clamp_radius(uniform_r);
  uint32_t out4 = 0;
#pragma unroll
  for (int r = 0; r < 4; r++) {  // fine row: y parity r & 1, z parity r >> 1
    const int fy = 2 * y + (r & 1), fz = 2 * z + (r >> 1);
    const uint16_t* er = E + fy * esy + fz * esz + 2 * x4;
    const int8_t* rr = R.p != nullptr ? R.p + fy * R.sy + fz * R.sz + 2 * x4 : nullptr;
#pragma unroll
    for (int i = 0; i < 4; i++) {  // fine x 2(x4 + i) and 2(x4 + i) + 1
      const uint32_t e2 = *reinterpret_cast<const uint32_t*>(er + 2 * i);
      int r0 = ru, r1 = ru;
      if (rr != nullptr) {
        const uint32_t w = *reinterpret_cast<const uint16_t*>(rr + 2 * i);
        r0 = clamp_radius((int)(int8_t)(w & 0xffu));
        r1 = clamp_radius((int)(int8_t)(w >> 8));
      }
      const uint32_t b0 = (e2 & 0xffffu) < (uint32_t)((r0 + 1) * (r0 + 1)) ? 1u : 0u;
      const uint32_t b1 = (e2 >> 16) < (uint32_t)((r1 + 1) * (r1 + 1)) ? 2u : 0u;
      out4 |= (b0 | b1) << (2 * r + 8 * i);
    }
  }
  *reinterpret_cast<uint32_t*>(out + cidx(x4, y, z, g)) = out4;
}


__device__ __forceinline__ uint32_t c0_of(uint32_t x, uint32_t d, uint32_t eb, bool inside) {
  return (inside && d != 0u && x != 0xffu && eb) ? 0u : d;
}


static dim3 quad_grid(Dims g) { return dim3((g.x / 4 + 63) / 64, (g.y + 3) / 4, g.z); }

// ---------------------------------------------------------------------
// The same cell-level kernels on 16 consecutive cells per thread (one
// 16-byte load per row), four cells per 32-bit word at a time: the
// per-byte rules become byte masks (__vcmp*4) and shifts that stay within
// bytes.  Block (32, 8): x along threadIdx.x, y along threadIdx.y.
// ---------------------------------------------------------------------

__device__ __forceinline__ uint4 ld16(const uint8_t* g, int x16, int y, int z, Dims d) {
  return *reinterpret_cast<const uint4*>(g + cidx(x16, y, z, d));
}
__device__ __forceinline__ uint32_t w_of(const uint4& q, int j) {
  return j == 0 ? q.x : (j == 1 ? q.y : (j == 2 ? q.z : q.w));
}
// 0xff in byte i where cell x0 + i satisfies lo <= x < hi
__device__ __forceinline__ uint32_t xrange_mask(int x0, int lo, int hi) {
  uint32_t m = 0;
#pragma unroll
  for (int i = 0; i < 4; i++) m |= (x0 + i >= lo && x0 + i < hi) ? (0xffu << (8 * i)) : 0u;
  return m;
}
// the word of cells x0 + 1 .. x0 + 4 (x0 - 1 .. x0 + 2) from the word of
// x0 .. x0 + 3 and the byte after (before) it
__device__ __forceinline__ uint32_t next_cells(uint32_t w, uint32_t after) { return (w >> 8) | (after << 24); }
__device__ __forceinline__ uint32_t prev_cells(uint32_t w, uint32_t before) { return (w << 8) | before; }

// Blocks of the kernels that walk along z over threads of 16 cells: as many
// threads along x as the rows have (a power of 2, at most 32), the others
// along y, `halo` rows of them beside the outputs.  Walks of 16 cells re-read
// least; shorter ones, down to 2, where the grid gives fewer than 512 blocks
// (each step waits for its loads).  Tags, selection and contour with 32
// threads along x and 16 cells against this: 22, 19 and 14 -> 8, 8 and 7 us
// at 128^3 (walks of 2; 10, 8 and 8 with 4), 53, 49 and 29 -> 35, 25 and 21
// at 512^3 (walks of 4; 37, 29 and 21 with 2), and at 1024^3 (walks of 16)
// 166, 137 and 92 (246, 192 and 115 with 2).
constexpr int kWalkThreads = 320, kWalkBlocks = 512;
__device__ __forceinline__ bool walk_meets(const CBox& roi, int bx, int out, int z0, int z1) {
  const int x0 = 16 * (int)blockIdx.x * bx, y0 = (int)blockIdx.y * out;
  return cbox_meets(roi, x0, x0 + 16 * bx - 1, y0, y0 + out - 1, z0, z1 - 1);
}
struct ZWalk {
  dim3 blocks, threads;
  int zs;
};
static ZWalk z_walk(Dims g, int halo) {
  int bx = 1;
  while (16 * bx < g.x && bx < 32) bx *= 2;
  const int by = kWalkThreads / bx, out = by - halo;
  ZWalk w;
  w.threads = dim3(bx, by);
  const int plane = ((g.x / 16 + bx - 1) / bx) * ((g.y + out - 1) / out);
  for (w.zs = 16; w.zs > 2 && plane * ((g.z + w.zs - 1) / w.zs) < kWalkBlocks; w.zs /= 2) {}
  w.blocks = dim3((g.x / 16 + bx - 1) / bx, (g.y + out - 1) / out, (g.z + w.zs - 1) / w.zs);
  return w;
}

// Contour of the dilation: fine voxels outside D that are 6-adjacent to D.
// GM_REF: only for cells in [1, res-2]^3 whose byte is not 0xff
// (TagVoxelsContourByErosion, Grid.cu:1230-1327); GM_EXACT: whole grid.
// A block walks along z (z_walk), each thread keeping its row of D at z - 1,
// z, z + 1 in registers; the rows y - 1 and y + 1 come from the block's
// other threads through shared memory (its first and last rows are halo
// only) and the bytes before and after a thread's 16 cells from its
// neighbouring lanes, so each row of D is read once.
__global__ void __launch_bounds__(kWalkThreads) k_contour_z(const uint8_t* __restrict__ D, uint8_t* __restrict__ S,
                                                            Dims g, int zs, int exact, CBox roi) {
  __shared__ uint4 rows_s[kWalkThreads];
  const int bx = blockDim.x, tx = threadIdx.x, ty = threadIdx.y, me = ty * bx + tx;
  const int x16 = 16 * (blockIdx.x * bx + tx);
  const int y = (int)blockIdx.y * (blockDim.y - 2) - 1 + ty;
  const int z0 = (int)blockIdx.z * zs, z1 = min(z0 + zs, g.z);
  if (!walk_meets(roi, bx, (int)blockDim.y - 2, z0, z1)) return;
  const bool xok = x16 < g.x, yok = y >= 0 && y < g.y;
  const uint4 z4 = make_uint4(0u, 0u, 0u, 0u);
  auto row = [&](int zz) { return xok && yok && zz >= 0 && zz < g.z ? ld16(D, x16, y, zz, g) : z4; };
  uint4 zm = row(z0 - 1), v = row(z0);
  for (int z = z0; z < z1; z++) {
    const uint4 zp = row(z + 1);
    rows_s[me] = v;
    __syncthreads();
    uint32_t before = __shfl_up_sync(0xffffffffu, v.w >> 24, 1, bx);
    uint32_t after = __shfl_down_sync(0xffffffffu, v.x & 0xffu, 1, bx);
    if (ty >= 1 && ty < (int)blockDim.y - 1 && xok && yok && cbox_meets(roi, x16, x16 + 15, y, y, z, z)) {
      if (tx == 0) before = x16 > 0 ? D[cidx(x16 - 1, y, z, g)] : 0u;
      if (tx == bx - 1 || x16 + 16 >= g.x) after = x16 + 16 < g.x ? D[cidx(x16 + 16, y, z, g)] : 0u;
      const uint4 ym = rows_s[me - bx], yp = rows_s[me + bx];
      const bool yz_in = y >= 1 && z >= 1 && y <= g.y - 2 && z <= g.z - 2;
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint32_t vw = w_of(v, j);
        const uint32_t l = prev_cells(vw, j > 0 ? w_of(v, j - 1) >> 24 : before);
        const uint32_t r = next_cells(vw, j < 3 ? w_of(v, j + 1) & 0xffu : after);
        // 6-neighbours of each fine voxel (bit x + 2y + 4z of a byte)
        uint32_t t = ((vw & 0xAAAAAAAAu) >> 1) | ((r & 0x55555555u) << 1);
        t |= ((vw & 0x55555555u) << 1) | ((l & 0xAAAAAAAAu) >> 1);
        t |= ((vw & 0xCCCCCCCCu) >> 2) | ((w_of(yp, j) & 0x33333333u) << 2);
        t |= ((vw & 0x33333333u) << 2) | ((w_of(ym, j) & 0xCCCCCCCCu) >> 2);
        t |= ((vw & 0xF0F0F0F0u) >> 4) | ((w_of(zp, j) & 0x0F0F0F0Fu) << 4);
        t |= ((vw & 0x0F0F0F0Fu) << 4) | ((w_of(zm, j) & 0xF0F0F0F0u) >> 4);
        uint32_t m = 0xffffffffu;
        if (!exact) m = yz_in ? (__vcmpne4(vw, 0xffffffffu) & xrange_mask(x16 + 4 * j, 1, g.x - 1)) : 0u;
        o[j] = t & ~vw & m;
      }
      *reinterpret_cast<uint4*>(S + cidx(x16, y, z, g)) = make_uint4(o[0], o[1], o[2], o[3]);
    }
    __syncthreads();  // rows_s is rewritten for the next z
    zm = v;
    v = zp;
  }
}

// GM_REF dilation select: base pass (cells inside data_res that are not
// full take 0xff when their child-0 corner is dilated, GMorpho.cu:2848-2927)
// then the tight contour (forward 2x2x2 block mixes full and non-full,
// Grid.cu:1589-1607) takes the fine per-voxel byte (GMorpho.cu:2930-3056).
//
// base-pass bytes of the dilation (GM_REF) of one row of 16 cells and the
// full flags (0xff per full byte) of the cells x16 + 1 .. x16 + 16
__device__ __forceinline__ void base_dil_row(const uint8_t* X, const uint8_t* Df, int x16, int yy, int zz, Dims g,
                                             const DataRes& dr, uint32_t d0[4], uint32_t f[4], uint32_t fr[4],
                                             uint32_t dfw[4]) {
  if (yy >= g.y || zz >= g.z) {
#pragma unroll
    for (int j = 0; j < 4; j++) { d0[j] = 0u; f[j] = 0u; fr[j] = 0u; dfw[j] = 0u; }
    return;
  }
  const bool iyz = yy < dr.v[1] && zz < dr.v[2];
  const uint4 xq = ld16(X, x16, yy, zz, g), dq = ld16(Df, x16, yy, zz, g);
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint32_t xw = w_of(xq, j), dw = w_of(dq, j);
    const uint32_t in = iyz ? xrange_mask(x16 + 4 * j, 0, dr.v[0]) : 0u;
    const uint32_t cond = in & __vcmpne4(xw, 0xffffffffu) & ((dw & 0x01010101u) * 0xffu);
    d0[j] = xw | cond;
    f[j] = __vcmpeq4(d0[j], 0xffffffffu);
    dfw[j] = dw;
  }
  // full flag of cell x16 + 16
  uint32_t fa = 0u;
  if (x16 + 16 < g.x) {
    const int64_t c = cidx(x16 + 16, yy, zz, g);
    const uint32_t xb = X[c], db = Df[c];
    const bool inside = iyz && x16 + 16 < dr.v[0];
    const uint32_t d = (inside && xb != 0xffu && (db & 1u)) ? 0xffu : xb;
    fa = d == 0xffu ? 0xffu : 0u;
  }
#pragma unroll
  for (int j = 0; j < 4; j++) fr[j] = next_cells(f[j], j < 3 ? f[j + 1] & 0xffu : fa);
}

// The select kernel computes each base-pass row once: a block walks along z,
// each thread keeping its row's flags at z and z + 1 in registers; the row
// y + 1 comes from the block's next row of threads through shared memory (its
// last row is that halo only).  It marks the 8^3-cell blocks of D that hold a
// non-zero byte in dmap (zeroed by the caller; reading D again for them took
// 12.5 us at 512^3, 63 at 1024^3).
__global__ void __launch_bounds__(kWalkThreads) k_dil_select_z(const uint8_t* __restrict__ X,
                                                               const uint8_t* __restrict__ Df, uint8_t* __restrict__ D,
                                                               Dims g, int zs, DataRes dr, CBox roi,
                                                               uint8_t* __restrict__ dmap, int mdx, int mdy) {
  __shared__ uint4 flags_s[4][kWalkThreads];  // per thread: f, fr at z; f, fr at z + 1
  const int bx = blockDim.x, ty = threadIdx.y, me = ty * bx + threadIdx.x;
  const int x16 = 16 * (blockIdx.x * bx + threadIdx.x);
  const int y = (int)blockIdx.y * (blockDim.y - 1) + ty;
  const int z0 = (int)blockIdx.z * zs, z1 = min(z0 + zs, g.z);
  if (!walk_meets(roi, bx, (int)blockDim.y - 1, z0, z1)) return;
  const bool xok = x16 < g.x;
  auto row = [&](int zz, uint32_t d0[4], uint32_t f[4], uint32_t fr[4], uint32_t dfw[4]) {
    if (xok) {
      base_dil_row(X, Df, x16, y, zz, g, dr, d0, f, fr, dfw);  // zeros outside the grid
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++) d0[j] = f[j] = fr[j] = dfw[j] = 0u;
    }
  };
  uint32_t d0c[4], fc[4], frc[4], dfc[4];
  uint32_t seen0 = 0, seen1 = 0;  // of the two 8-cell blocks along x, since the last mark
  row(z0, d0c, fc, frc, dfc);
  for (int z = z0; z < z1; z++) {
    uint32_t d0n[4], fn[4], frn[4], dfn[4];
    row(z + 1, d0n, fn, frn, dfn);
    flags_s[0][me] = make_uint4(fc[0], fc[1], fc[2], fc[3]);
    flags_s[1][me] = make_uint4(frc[0], frc[1], frc[2], frc[3]);
    flags_s[2][me] = make_uint4(fn[0], fn[1], fn[2], fn[3]);
    flags_s[3][me] = make_uint4(frn[0], frn[1], frn[2], frn[3]);
    __syncthreads();
    if (ty < (int)blockDim.y - 1 && xok && y < g.y && cbox_meets(roi, x16, x16 + 15, y, y, z, z)) {
      const uint4 f1 = flags_s[0][me + bx], fr1 = flags_s[1][me + bx];
      const uint4 f2 = flags_s[2][me + bx], fr2 = flags_s[3][me + bx];
      // the forward 2x2x2 block mixes full and non-full bytes (cells <= dims - 2)
      const bool yz_ok = y <= g.y - 2 && z <= g.z - 2;
      uint32_t o[4];
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const uint32_t any = fc[j] | frc[j] | fn[j] | frn[j] | w_of(f1, j) | w_of(fr1, j) | w_of(f2, j) | w_of(fr2, j);
        const uint32_t all = fc[j] & frc[j] & fn[j] & frn[j] & w_of(f1, j) & w_of(fr1, j) & w_of(f2, j) & w_of(fr2, j);
        const uint32_t tag = yz_ok ? (any & ~all & xrange_mask(x16 + 4 * j, 0, g.x - 1)) : 0u;
        o[j] = (tag & dfc[j]) | (~tag & d0c[j]);
      }
      *reinterpret_cast<uint4*>(D + cidx(x16, y, z, g)) = make_uint4(o[0], o[1], o[2], o[3]);
      seen0 |= o[0] | o[1];
      seen1 |= o[2] | o[3];
    }
    if ((z & 7) == 7 || z == z1 - 1) {
      uint8_t* m = dmap + idx3(x16 >> 3, y >> 3, z >> 3, mdx, mdy);
      if (seen0) m[0] = 1;
      if (seen1) m[1] = 1;
      seen0 = seen1 = 0;
    }
    __syncthreads();  // flags_s is rewritten for the next z
#pragma unroll
    for (int j = 0; j < 4; j++) {
      d0c[j] = d0n[j];
      fc[j] = fn[j];
      frc[j] = frn[j];
      dfc[j] = dfn[j];
    }
  }
}

// GM_REF erosion select: base pass (cells inside data_res with D != 0 and
// X != 0xff are cleared when the centre 2c+1 is eroded, GMorpho.cu:4360-4370,
// 4644-4646), then cells whose byte differs from a 6-neighbour
// (Grid.cu:1499-1570) take 0xff & ~eroded (GMorpho.cu:5353-5360).
//
// C0 = base erosion of 16 cells of one row: 0 where the cell is inside the
// data, D != 0, X != 0xff and its lattice point 2c+1 is eroded; D otherwise
__device__ __forceinline__ void base_ero_row(const uint8_t* X, const uint8_t* D, const uint8_t* Eb, int x16, int yy,
                                             int zz, Dims g, const DataRes& dr, uint32_t c0[4]) {
  const bool iyz = yy < dr.v[1] && zz < dr.v[2];
  const uint4 xq = ld16(X, x16, yy, zz, g), dq = ld16(D, x16, yy, zz, g), eq = ld16(Eb, x16, yy, zz, g);
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint32_t dw = w_of(dq, j);
    const uint32_t in = iyz ? xrange_mask(x16 + 4 * j, 0, dr.v[0]) : 0u;
    const uint32_t cond = in & __vcmpne4(dw, 0u) & __vcmpne4(w_of(xq, j), 0xffffffffu) & __vcmpne4(w_of(eq, j), 0u);
    c0[j] = dw & ~cond;
  }
}

__global__ void __launch_bounds__(256) k_ero_select16(const uint8_t* __restrict__ X, const uint8_t* __restrict__ D,
                                                      const uint8_t* __restrict__ Eb, const uint8_t* __restrict__ Ef,
                                                      uint8_t* __restrict__ C, Dims g, DataRes dr, int exact,
                                                      CBox roi) {
  const int x16 = 16 * (blockIdx.x * 32 + threadIdx.x);
  const int y = blockIdx.y * 8 + threadIdx.y, z = blockIdx.z;
  if (x16 >= g.x || y >= g.y || !cbox_meets(roi, x16, x16 + 15, y, y, z, z)) return;
  const uint4 ef = ld16(Ef, x16, y, z, g);
  if (exact) {
    const uint4 d = ld16(D, x16, y, z, g);
    *reinterpret_cast<uint4*>(C + cidx(x16, y, z, g)) =
        make_uint4(d.x & ~ef.x, d.y & ~ef.y, d.z & ~ef.z, d.w & ~ef.w);
    return;
  }
  uint32_t c0[4];
  base_ero_row(X, D, Eb, x16, y, z, g, dr, c0);
  // C0 of the cells x16 - 1 and x16 + 16
  const bool iyz = y < dr.v[1] && z < dr.v[2];
  uint32_t before = 0u, after = 0u;
  if (x16 > 0) {
    const int64_t c = cidx(x16 - 1, y, z, g);
    before = c0_of(X[c], D[c], Eb[c], iyz && x16 - 1 < dr.v[0]);
  }
  if (x16 + 16 < g.x) {
    const int64_t c = cidx(x16 + 16, y, z, g);
    after = c0_of(X[c], D[c], Eb[c], iyz && x16 + 16 < dr.v[0]);
  }
  const bool interior_yz = y >= 1 && z >= 1 && y <= g.y - 2 && z <= g.z - 2;
  uint32_t diff[4] = {0u, 0u, 0u, 0u};
  if (interior_yz) {
    const int ny[4] = {y - 1, y + 1, y, y};
    const int nz[4] = {z, z, z - 1, z + 1};
#pragma unroll
    for (int n = 0; n < 4; n++) {
      uint32_t cn[4];
      base_ero_row(X, D, Eb, x16, ny[n], nz[n], g, dr, cn);
#pragma unroll
      for (int j = 0; j < 4; j++) diff[j] |= __vcmpne4(c0[j], cn[j]);
    }
  }
  uint32_t o[4];
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint32_t l = prev_cells(c0[j], j > 0 ? c0[j - 1] >> 24 : before);
    const uint32_t r = next_cells(c0[j], j < 3 ? c0[j + 1] & 0xffu : after);
    const uint32_t tag = interior_yz ? ((diff[j] | __vcmpne4(c0[j], l) | __vcmpne4(c0[j], r)) &
                                        xrange_mask(x16 + 4 * j, 1, g.x - 1))
                                     : 0u;
    o[j] = (tag & ~w_of(ef, j)) | (~tag & c0[j]);
  }
  *reinterpret_cast<uint4*>(C + cidx(x16, y, z, g)) = make_uint4(o[0], o[1], o[2], o[3]);
}

static dim3 grid16(Dims g) { return dim3((g.x / 16 + 31) / 32, (g.y + 7) / 8, g.z); }

// GM_REF erosion select in two steps, so that the centre erosion is computed
// only where it is read.  k_ero_tag_z writes the base erosion C0 into C (final
// for untagged cells), the refinement tags (0xff per tagged cell) into T and
// marks the 8^3-cell blocks holding a tagged cell in tmap (zeroed by the
// caller); the centre erosion's z pass then runs on those blocks and writes
// 0xff & ~e on the tagged cells.  The bytes equal k_ero_select16's.
// The tag kernel computes each base-erosion row once: a block walks along z,
// each thread keeping its row's C0 at z - 1, z, z + 1 in registers; the rows
// y - 1 and y + 1 at z come from the block's other threads through shared
// memory (its first and last rows are halo only), and the bytes before and
// after a thread's 16 cells from its neighbouring lanes.
__global__ void __launch_bounds__(kWalkThreads) k_ero_tag_z(const uint8_t* __restrict__ X,
                                                            const uint8_t* __restrict__ D,
                                                            const uint8_t* __restrict__ Eb, uint8_t* __restrict__ C,
                                                            uint8_t* __restrict__ T, uint8_t* __restrict__ tmap,
                                                            int mdx, int mdy, Dims g, int zs, DataRes dr, CBox roi) {
  __shared__ uint4 rows_s[kWalkThreads];
  const int bx = blockDim.x, tx = threadIdx.x, ty = threadIdx.y, me = ty * bx + tx;
  const int x16 = 16 * (blockIdx.x * bx + tx);
  const int y = (int)blockIdx.y * (blockDim.y - 2) - 1 + ty;
  const int z0 = (int)blockIdx.z * zs, z1 = min(z0 + zs, g.z);
  if (!walk_meets(roi, bx, (int)blockDim.y - 2, z0, z1)) return;
  const bool xok = x16 < g.x, yok = y >= 0 && y < g.y;
  auto row = [&](int zz, uint32_t c[4]) {
    if (xok && yok && zz >= 0 && zz < g.z) {
      base_ero_row(X, D, Eb, x16, y, zz, g, dr, c);
    } else {
#pragma unroll
      for (int j = 0; j < 4; j++) c[j] = 0u;
    }
  };
  uint32_t cp[4], cc[4], cn[4];
  row(z0 - 1, cp);
  row(z0, cc);
  for (int z = z0; z < z1; z++) {
    row(z + 1, cn);
    rows_s[me] = make_uint4(cc[0], cc[1], cc[2], cc[3]);
    __syncthreads();
    // C0 of the cells x16 - 1 and x16 + 16 (the neighbouring lanes' rows;
    // at the block's x edges, from the grid)
    uint32_t before = __shfl_up_sync(0xffffffffu, cc[3] >> 24, 1, bx);
    uint32_t after = __shfl_down_sync(0xffffffffu, cc[0] & 0xffu, 1, bx);
    const bool out = ty >= 1 && ty < (int)blockDim.y - 1 && xok && yok && cbox_meets(roi, x16, x16 + 15, y, y, z, z);
    if (out) {
      const bool iyz = y < dr.v[1] && z < dr.v[2];
      if (tx == 0)
        before = 0u;
      if (tx == 0 && x16 > 0) {
        const int64_t c = cidx(x16 - 1, y, z, g);
        before = c0_of(X[c], D[c], Eb[c], iyz && x16 - 1 < dr.v[0]);
      }
      if (tx == bx - 1 || x16 + 16 >= g.x) after = 0u;
      if (tx == bx - 1 && x16 + 16 < g.x) {
        const int64_t c = cidx(x16 + 16, y, z, g);
        after = c0_of(X[c], D[c], Eb[c], iyz && x16 + 16 < dr.v[0]);
      }
      const bool interior_yz = y >= 1 && z >= 1 && y <= g.y - 2 && z <= g.z - 2;
      uint32_t tag[4] = {0u, 0u, 0u, 0u};
      if (interior_yz) {
        const uint4 ym = rows_s[me - bx], yp = rows_s[me + bx];
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const uint32_t diff = __vcmpne4(cc[j], w_of(ym, j)) | __vcmpne4(cc[j], w_of(yp, j)) |
                                __vcmpne4(cc[j], cp[j]) | __vcmpne4(cc[j], cn[j]);
          const uint32_t l = prev_cells(cc[j], j > 0 ? cc[j - 1] >> 24 : before);
          const uint32_t r = next_cells(cc[j], j < 3 ? cc[j + 1] & 0xffu : after);
          tag[j] = (diff | __vcmpne4(cc[j], l) | __vcmpne4(cc[j], r)) & xrange_mask(x16 + 4 * j, 1, g.x - 1);
        }
      }
      const int64_t o = cidx(x16, y, z, g);
      *reinterpret_cast<uint4*>(C + o) = make_uint4(cc[0], cc[1], cc[2], cc[3]);
      *reinterpret_cast<uint4*>(T + o) = make_uint4(tag[0], tag[1], tag[2], tag[3]);
      const int64_t mb = idx3(x16 >> 3, y >> 3, z >> 3, mdx, mdy);
      if (tag[0] | tag[1]) tmap[mb] = 1;
      if (tag[2] | tag[3]) tmap[mb + 1] = 1;
    }
    __syncthreads();  // rows_s is rewritten for the next z
#pragma unroll
    for (int j = 0; j < 4; j++) {
      cp[j] = cc[j];
      cc[j] = cn[j];
    }
  }
}

// max clamped radius over the fine radius grid
__global__ void k_rmax(const int8_t* __restrict__ R, int64_t n, int* __restrict__ out) {
  int m = 2;
  for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) * 16; i < n;
       i += (int64_t)gridDim.x * blockDim.x * 16) {
    const uint4 v = *reinterpret_cast<const uint4*>(R + i);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int j = 0; j < 16; j++) {
      const int s = (int)(int8_t)((w[j >> 2] >> (8 * (j & 3))) & 0xff);
      const int r = clamp_radius(s);
      m = r > m ? r : m;
    }
  }
  for (int o = 16; o > 0; o >>= 1) { const int t = __shfl_xor_sync(0xffffffffu, m, o); m = t > m ? t : m; }
  if ((threadIdx.x & 31) == 0) atomicMax(out, m);
}

// ---------------------------------------------------------------------
// host orchestration
// ---------------------------------------------------------------------

static inline int cdiv(int a, int b) { return (a + b - 1) / b; }

static int grid_stride_blocks(int64_t n, int threads, int sms) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)sms * 32;
  return (int)(b < cap ? b : cap);
}

// tile-need test by output box only (x and third coordinates in fine voxels
// or cells by the shifts)
static NeedMap roi_only(const CBox& b, int x_shift, int t_shift) {
  return NeedMap{nullptr, 0, 0, 0, x_shift, t_shift, 0, 0, 0, b};
}

// box grown by g cells along each axis flagged in `axes` (bit a), clamped
static CBox cbox_grow(const CBox& b, int g, int axes, const int dims[3]) {
  CBox r = b;
  for (int a = 0; a < 3; a++) {
    if ((axes >> a) & 1) {
      r.lo[a] = b.lo[a] - g;
      r.hi[a] = b.hi[a] + g;
    }
    r.lo[a] = r.lo[a] < 0 ? 0 : r.lo[a];
    r.hi[a] = r.hi[a] > dims[a] ? dims[a] : r.hi[a];
  }
  return r;
}

size_t close_workspace_bytes_box(int rx, int ry, int rz) {
  const size_t Nx = 2 * (size_t)rx, Ny = 2 * (size_t)ry, Nz = 2 * (size_t)rz, V = Nx * Ny * Nz;
  const size_t cells = (size_t)rx * ry * rz;
  // buf16 x2, buf8, HL1, HL2, Df, Eb, Ef, S, D, radius map, D and tag block maps + alignment slack
  return 2 * V * 2 + V + (size_t)rx * Ny * Nz * 2 + (size_t)rx * ry * Nz * 2 + 5 * cells + V / 4096 + 2 * (cells / 512) +
         17 * 256;
}

size_t close_workspace_bytes(int res) { return close_workspace_bytes_box(res, res, res); }

static inline uint8_t* carve(uint8_t*& p, size_t bytes) {
  uint8_t* r = p;
  p += (bytes + 255) & ~(size_t)255;
  return r;
}

// The closing's workspace, carved the same way by every entry point that
// works in it (launch_close and the parts that run before it).
struct CloseWs {
  uint16_t *buf16a, *buf16b, *HL1, *HL2;
  uint8_t *buf8, *Df, *Eb, *Ef, *S, *D, *rmap, *dmap, *tmap;
};

static CloseWs close_ws(const CloseArgs& a, int rx, int ry, int rz) {
  const size_t Nx = 2 * (size_t)rx, Ny = 2 * (size_t)ry, Nz = 2 * (size_t)rz, V = Nx * Ny * Nz;
  const size_t cells = (size_t)rx * ry * rz, blocks8 = cells / 512;
  uint8_t* p = a.workspace;
  CloseWs w;
  w.buf16a = reinterpret_cast<uint16_t*>(carve(p, V * 2));
  w.buf16b = reinterpret_cast<uint16_t*>(carve(p, V * 2));
  w.buf8 = carve(p, V);
  w.HL1 = reinterpret_cast<uint16_t*>(carve(p, (size_t)rx * Ny * Nz * 2));
  w.HL2 = reinterpret_cast<uint16_t*>(carve(p, (size_t)rx * ry * Nz * 2));
  w.Df = carve(p, cells);
  w.Eb = carve(p, cells);
  w.Ef = carve(p, cells);
  w.S = carve(p, cells);
  w.D = a.D_out != nullptr ? a.D_out : carve(p, cells);
  w.rmap = carve(p, V / 4096);
  w.dmap = carve(p, blocks8);
  w.tmap = carve(p, blocks8);
  return w;
}

uint8_t* close_ws_dilation(const CloseArgs& a) {
  const int rx = a.dims[0] > 0 ? a.dims[0] : a.res;
  const int ry = a.dims[0] > 0 ? a.dims[1] : a.res;
  const int rz = a.dims[0] > 0 ? a.dims[2] : a.res;
  return close_ws(a, rx, ry, rz).D;
}

// buf16a: first written by the dilation's passes or, when the dilation is
// done, by the erosion's x pass
uint8_t* close_ws_scratch(const CloseArgs& a, size_t* bytes) {
  const int rx = a.dims[0] > 0 ? a.dims[0] : a.res;
  const int ry = a.dims[0] > 0 ? a.dims[1] : a.res;
  const int rz = a.dims[0] > 0 ? a.dims[2] : a.res;
  const CloseWs w = close_ws(a, rx, ry, rz);
  if (bytes) *bytes = (size_t)(reinterpret_cast<uint8_t*>(w.buf16b) - reinterpret_cast<uint8_t*>(w.buf16a));
  return reinterpret_cast<uint8_t*>(w.buf16a);
}

uint16_t* close_ws_field(const CloseArgs& a) {
  const int rx = a.dims[0] > 0 ? a.dims[0] : a.res;
  const int ry = a.dims[0] > 0 ? a.dims[1] : a.res;
  const int rz = a.dims[0] > 0 ? a.dims[2] : a.res;
  return close_ws(a, rx, ry, rz).buf16b;
}

cudaError_t launch_close(const CloseArgs& a, cudaStream_t st, KernelCounter* kc) {
  const int rx = a.dims[0] > 0 ? a.dims[0] : a.res;
  const int ry = a.dims[0] > 0 ? a.dims[1] : a.res;
  const int rz = a.dims[0] > 0 ? a.dims[2] : a.res;
  if (rx % 16 != 0 || ry % 16 != 0 || rz % 16 != 0 || rx <= 0 || ry <= 0 || rz <= 0) return cudaErrorInvalidValue;
  const Dims g{rx, ry, rz};
  const int Nx = 2 * rx, Ny = 2 * ry, Nz = 2 * rz;
  const size_t cells = (size_t)rx * ry * rz;
  const CloseWs w = close_ws(a, rx, ry, rz);
  uint16_t* buf16a = w.buf16a;
  uint16_t* buf16b = w.buf16b;
  uint8_t* buf8 = w.buf8;
  uint16_t* HL1 = w.HL1;
  uint16_t* HL2 = w.HL2;
  uint8_t* Df = w.Df;
  uint8_t* Eb = w.Eb;
  uint8_t* Ef = w.Ef;
  uint8_t* S = w.S;
  uint8_t* D = w.D;
  uint8_t* rmap = w.rmap;
  const int mdx = rx / 8, mdy = ry / 8, mdz = rz / 8;
  uint8_t* dmap = w.dmap;
  uint8_t* tmap = w.tmap;  // 8^3-cell blocks holding refinement-tagged cells
  const int rmax = a.rmax;
  DataRes dr{{a.data_res[0], a.data_res[1], a.data_res[2]}};
  const bool exact = a.mode == 1;
  const RField RF{a.R, a.r_sy > 0 ? a.r_sy : (int64_t)Nx, a.r_sz > 0 ? a.r_sz : (int64_t)Nx * Ny};
  const RField RNONE{nullptr, 0, 0};
  // Output boxes of the passes (cells).  F: where the caller needs the
  // closing.  Working backwards: the erosion flags on F (centres) and F + 1
  // (lattice points, read by the neighbour test), the contour within the
  // erosion reach of those, the dilation one cell further (contour
  // neighbours) and its fine flags one more (forward 2x2x2 block); each
  // y (z) pass also within the window of the following pass.
  const int dims[3] = {rx, ry, rz};
  CBox F{{0, 0, 0}, {rx, ry, rz}};
  if (a.roi_hi[0] > 0)
    for (int k = 0; k < 3; k++) {
      F.lo[k] = a.roi_lo[k] < 0 ? 0 : a.roi_lo[k];
      F.hi[k] = a.roi_hi[k] > dims[k] ? dims[k] : a.roi_hi[k];
    }
  const int win = (rmax + 3) / 2 + 2;  // cells covering a pass window (rmax + 2 fine voxels) with rounding
  const CBox R_Ef = F, R_Eb = cbox_grow(F, 1, 7, dims);
  const CBox R_S = cbox_grow(F, win + 2, 7, dims), R_D = cbox_grow(R_S, 1, 7, dims), R_Df = cbox_grow(R_D, 1, 7, dims);
  const CBox B_dil_y = cbox_grow(R_Df, win, 4, dims), B_dil_x = cbox_grow(R_Df, win, 6, dims);
  const CBox B_ero_y = cbox_grow(R_Ef, win, 4, dims), B_erob_y = cbox_grow(R_Eb, win, 4, dims);
  const CBox B_ero_x = cbox_grow(R_Eb, win, 6, dims);
  // phase mode: the steps of phase a.phase only (see CloseArgs::phase)
  if (a.phase >= 0 && (a.edt != nullptr || !close_phase_ok(rmax, a.se) || a.group == nullptr))
    return cudaErrorInvalidValue;
  cudaError_t e;  // (the launchers of a pass report and clear the errors so far)
  int at = 0;  // min-plus passes met so far
  auto here = [&]() { return a.phase < 0 || a.phase == at; };

  // ---- dilation ---- (skipped when the caller has put it in D already)
  if (!a.dilation_done) {
    const int dil_r = rmax + 1;  // "Safety Measure" radius + 1 (GMorpho.cu:2864)
    const int dcap = (a.se == 1 ? rmax + 2 : dil_r + 1) < 255 ? (a.se == 1 ? rmax + 2 : dil_r + 1) : 255;
    const uint32_t dil_cap = a.se == 1 ? (uint32_t)(rmax + 1) : (uint32_t)(dil_r * dil_r);
    const int dil_halo = dil_r + 1;
    const uint8_t* tile_map = nullptr;  // per-tile radius bounds of the dilation passes
    if (a.edt != nullptr) {
      // resident distance field: the dilation is its per-voxel threshold
      if (a.se != 0) return cudaErrorInvalidValue;
    } else if (a.R != nullptr && a.rmap_in != nullptr) {
      tile_map = a.rmap_in;  // built by the caller together with the radius bound
    } else if (a.R != nullptr) {
      if (here() && (e = launch_radius_map(RF, Nx, Ny, Nz, rmap, nullptr, st, kc)) != cudaSuccess) return e;
      tile_map = rmap;
    }
    if (a.edt != nullptr) {
      GM_LAUNCH(kc, "k_dil_threshold", st,
                k_dil_threshold<<<quad_grid(g), dim3(64, 4), 0, st>>>(a.edt, a.e_sy, a.e_sz, RF, a.uniform_r, g,
                                                                      exact ? D : Df, R_Df));
    } else {
      if (!a.xpass_done && here() &&
          (e = launch_dil_pass_x(a.X, buf8, rx, ry, rz, dcap, B_dil_x, st, kc)) != cudaSuccess)
        return e;
      uint8_t* dst = exact ? D : Df;
      if ((a.ypass_done || a.zpass_done) && a.se != 0) return cudaErrorInvalidValue;
      if (dil_cap <= 32767) {
        bool ok = true;
        if (a.se == 1) {
          ok &= dpx_step<KERN_CUBE, uint8_t, 0>(a, at, buf8, buf16a, nullptr, Nx, Ny, Nz, 1, 0, dil_halo, dil_cap, RNONE,
                                                0, rx, ry, st, kc, "k_pass_dil_y", tile_map, dil_halo,
                                                roi_only(B_dil_y, 1, 1));
          ok &= dpx_step<KERN_CUBE, uint16_t, 1>(a, at, buf16a, nullptr, dst, Nx, Ny, Nz, 2, 0, dil_halo, dil_cap, RF,
                                                 a.uniform_r, rx, ry, st, kc, "k_pass_dil_z", tile_map, 0,
                                                 roi_only(R_Df, 1, 1));
        } else {
          if (!a.ypass_done)
            ok &= dpx_step<KERN_LAT, uint8_t, 0>(a, at, buf8, buf16a, nullptr, Nx, Ny, Nz, 1, 0, dil_halo, dil_cap,
                                                 RNONE, 0, rx, ry, st, kc, "k_pass_dil_y", tile_map, dil_halo,
                                                 roi_only(B_dil_y, 1, 1));
          else
            at++;
          if (!a.zpass_done)
            ok &= dpx_step<KERN_LAT, uint16_t, 1>(a, at, buf16a, nullptr, dst, Nx, Ny, Nz, 2, 0, dil_halo, dil_cap, RF,
                                                  a.uniform_r, rx, ry, st, kc, "k_pass_dil_z", tile_map, 0,
                                                  roi_only(R_Df, 1, 1));
          else
            at++;
        }
        if (!ok) return cudaErrorInvalidValue;
      } else {
        const int span = kTileOut + 2 * dil_halo;
        dim3 gy(cdiv(Nx, 32), cdiv(Ny, kTileOut), Nz);
        if (a.se == 1)
          GM_LAUNCH(kc, "k_axis_pass", st, k_axis_pass<KERN_CUBE, uint8_t><<<gy, dim3(32, kRows), span * 32 * 2, st>>>(
                                               buf8, buf16a, Nx, Ny, Nz, 1, 0, dil_halo, dil_cap));
        else
          GM_LAUNCH(kc, "k_axis_pass", st, k_axis_pass<KERN_LAT, uint8_t><<<gy, dim3(32, kRows), span * 32 * 2, st>>>(
                                               buf8, buf16a, Nx, Ny, Nz, 1, 0, dil_halo, dil_cap));
        dim3 gz(cdiv(Nx, 32), cdiv(Nz, kTileOut), Ny / 2);
        if (a.se == 1)
          GM_LAUNCH(kc, "k_final_z", st, k_final_z<KERN_CUBE, FIN_DIL><<<gz, dim3(32, 8), 2 * span * 32 * 2, st>>>(
                                             buf16a, dst, RF, a.uniform_r, rx, ry, rz, dil_halo, dil_cap));
        else
          GM_LAUNCH(kc, "k_final_z", st, k_final_z<KERN_LAT, FIN_DIL><<<gz, dim3(32, 8), 2 * span * 32 * 2, st>>>(
                                             buf16a, dst, RF, a.uniform_r, rx, ry, rz, dil_halo, dil_cap));
      }
    }
    if (!exact && here()) {
      const ZWalk w = z_walk(g, 1);
      cudaMemsetAsync(dmap, 0, (size_t)(tmap - dmap) + (size_t)mdx * mdy * mdz, st);  // both block maps
      GM_LAUNCH(kc, "k_dil_select", st,
                k_dil_select_z<<<w.blocks, w.threads, 0, st>>>(a.X, Df, D, g, w.zs, dr, R_D, dmap, mdx, mdy));
    }
  } else {
    at += 2;  // the dilation's two passes
  }
  // ---- occupancy map of D (erosion outputs are needed on D only) ----
  // (k_dil_select has marked it already)
  const bool mapped = !exact && !a.dilation_done;
  if (!mapped && here()) {
    const int nb = mdx * mdy * mdz;
    GM_LAUNCH(kc, "k_occ_map8", st, k_occ_map8<<<(nb + 7) / 8, 256, 0, st>>>(D, rx, ry, mdx, mdy, nb, dmap));
  }
  // ---- contour ----
  if (here()) {
    const ZWalk w = z_walk(g, 2);
    GM_LAUNCH(kc, "k_contour", st,
              k_contour_z<<<w.blocks, w.threads, 0, st>>>(D, S, g, w.zs, exact ? 1 : 0, R_S));
    // (S holds the refinement tags after the erosion's x pass in GM_REF)
    if (a.S_out) cudaMemcpyAsync(a.S_out, S, cells, cudaMemcpyDeviceToDevice, st);
  }
  // ---- erosion ----
  {
    const uint32_t K = 4u * (uint32_t)((rmax - 1) * (rmax - 1));
    const int ehalo = rmax + 1;
    if (here() &&
        (e = launch_ero_pass_x(S, RF, a.uniform_r, rx, ry, rz, ehalo, K, buf16a, HL1, B_ero_x, st, kc)) != cudaSuccess)
      return e;
    if (K <= 32767) {
      const int gz = (ehalo + 1) / 2 + 1;  // cells covering the z window (ehalo fine voxels) of a z pass
      bool ok = true;
      if (exact) {
        // ero z needs its outputs on D grown by one cell, ero y its outputs
        // there and within the z window of it
        ok &= dpx_step<KERN_CEN2, uint16_t, 0>(a, at, buf16a, buf16b, nullptr, Nx, Ny, Nz, 1, 0, ehalo, K, RNONE, 0, rx,
                                               ry, st, kc, "k_pass_ero_y", nullptr, 0,
                                               NeedMap{dmap, mdx, mdy, mdz, 1, 1, 1, 1, 1 + gz, B_ero_y});
        ok &= dpx_step<KERN_CEN2, uint16_t, 2>(a, at, buf16b, nullptr, Ef, Nx, Ny, Nz, 2, 0, ehalo, K, RNONE, 0, rx, ry,
                                               st, kc, "k_pass_ero_z", nullptr, 0,
                                               NeedMap{dmap, mdx, mdy, mdz, 1, 1, 1, 1, 1, R_Ef});
      } else {
        // erob z needs its flags on D only, erob y within its z window
        ok &= dpx_step<KERN_LAT2, uint16_t, 0>(a, at, HL1, HL2, nullptr, rx, Ny, Nz, 1, 1, ehalo, K, RNONE, 0, rx, ry,
                                               st, kc, "k_pass_erob_y", nullptr, 0,
                                               NeedMap{dmap, mdx, mdy, mdz, 0, 1, 0, 0, gz, B_erob_y});
        ok &= dpx_step<KERN_LAT2, uint16_t, 3>(a, at, HL2, nullptr, Eb, rx, ry, Nz, 2, 1, ehalo, K, RNONE, 0, rx, ry,
                                               st, kc, "k_pass_erob_z", nullptr, 0,
                                               NeedMap{dmap, mdx, mdy, mdz, 0, 0, 0, 0, 0, R_Eb});
        // base erosion and refinement tags (the contour S is read by nobody
        // any more: it holds the tags), then the centre erosion only on the
        // blocks of tagged cells (ero y within the z window of them)
        if (here()) {
          if (!mapped) cudaMemsetAsync(tmap, 0, (size_t)mdx * mdy * mdz, st);
          const ZWalk w = z_walk(g, 2);
          GM_LAUNCH(kc, "k_ero_tag", st,
                    k_ero_tag_z<<<w.blocks, w.threads, 0, st>>>(a.X, D, Eb, a.C_out, S, tmap, mdx, mdy, g, w.zs, dr, F));
        }
        ok &= dpx_step<KERN_CEN2, uint16_t, 0>(a, at, buf16a, buf16b, nullptr, Nx, Ny, Nz, 1, 0, ehalo, K, RNONE, 0, rx,
                                               ry, st, kc, "k_pass_ero_y", nullptr, 0,
                                               NeedMap{tmap, mdx, mdy, mdz, 1, 1, 0, 0, gz, B_ero_y});
        ok &= dpx_step<KERN_CEN2, uint16_t, 4>(a, at, buf16b, nullptr, a.C_out, Nx, Ny, Nz, 2, 0, ehalo, K,
                                               RField{reinterpret_cast<const int8_t*>(S), 0, 0}, 0, rx, ry, st, kc,
                                               "k_pass_ero_z", nullptr, 0,
                                               NeedMap{tmap, mdx, mdy, mdz, 1, 1, 0, 0, 0, R_Ef});
      }
      if (!ok) return cudaErrorInvalidValue;
    } else {
      const int span = kTileOut + 2 * ehalo;
      dim3 gy(cdiv(Nx, 32), cdiv(Ny, kTileOut), Nz);
      GM_LAUNCH(kc, "k_axis_pass", st, k_axis_pass<KERN_CEN2, uint16_t><<<gy, dim3(32, kRows), span * 32 * 2, st>>>(
                                           buf16a, buf16b, Nx, Ny, Nz, 1, 0, ehalo, K));
      dim3 gz(cdiv(Nx, 32), cdiv(Nz, kTileOut), Ny / 2);
      GM_LAUNCH(kc, "k_final_z", st, k_final_z<KERN_CEN2, FIN_ERO><<<gz, dim3(32, 8), 2 * span * 32 * 2, st>>>(
                                         buf16b, Ef, RNONE, 0, rx, ry, rz, ehalo, K));
      if (!exact) {
        const int span_s = 2 * kTileOut + 2 * ehalo;
        dim3 gyb(cdiv(rx, 32), cdiv(ry, kTileOut), Nz);
        GM_LAUNCH(kc, "k_axis_pass", st, k_axis_pass<KERN_LAT2, uint16_t><<<gyb, dim3(32, kRows), span_s * 32 * 2, st>>>(
                                             HL1, HL2, rx, Ny, Nz, 1, 1, ehalo, K));
        dim3 gzb(cdiv(rx, 32), cdiv(rz, kTileOut), ry);
        GM_LAUNCH(kc, "k_final_z_base", st, k_final_z_base<<<gzb, dim3(32, kRows), span_s * 32 * 2, st>>>(
                                                HL2, Eb, rx, ry, rz, ehalo, K));
      }
    }
    if ((exact || K > 32767) && here())
      GM_LAUNCH(kc, "k_ero_select", st,
                k_ero_select16<<<grid16(g), dim3(32, 8), 0, st>>>(a.X, D, Eb, Ef, a.C_out, g, dr, exact ? 1 : 0, F));
  }
  return cudaGetLastError();
}

int close_phases(int mode) { return mode == 1 ? 5 : 7; }

bool close_phase_ok(int rmax, int se) {
  // the min-plus passes' saturation values fit 15 bits: the dilation's
  // (rmax + 1)^2 (sphere) or rmax + 1 (cube), the erosion's 4 (rmax - 1)^2
  const int r = clamp_radius(rmax);
  return (se == 1 || (r + 1) * (r + 1) <= 32767) && 4 * (r - 1) * (r - 1) <= 32767;
}

cudaError_t launch_edt(const uint8_t* X, int res, int rmax, uint8_t* workspace, uint16_t* E, cudaStream_t st,
                       KernelCounter* kc) {
  if (res % 16 != 0 || res <= 0 || rmax < 2 || rmax > 127) return cudaErrorInvalidValue;
  const int N = 2 * res;
  const size_t V = (size_t)N * N * N;
  uint8_t* p = workspace;
  uint16_t* buf16a = reinterpret_cast<uint16_t*>(carve(p, V * 2));
  carve(p, V * 2);
  uint8_t* buf8 = carve(p, V);
  // the sphere dilation's passes with the saturation of the largest radius
  // and no per-tile radius bound (every radius up to rmax may be asked)
  const int dil_r = rmax + 1, dil_halo = dil_r + 1, dcap = dil_r + 1;
  const uint32_t dil_cap = (uint32_t)(dil_r * dil_r);
  const RField RNONE{nullptr, 0, 0};
  const cudaError_t e = launch_dil_pass_x(X, buf8, res, res, res, dcap, CBox{{0, 0, 0}, {res, res, res}}, st, kc);
  if (e != cudaSuccess) return e;
  launch_dpx<KERN_LAT, uint8_t, 0>(buf8, buf16a, nullptr, N, N, N, 1, 0, dil_halo, dil_cap, RNONE, 0, res, res, st,
                                   kc, "k_pass_dil_y");
  launch_dpx<KERN_LAT, uint16_t, 0>(buf16a, E, nullptr, N, N, N, 2, 0, dil_halo, dil_cap, RNONE, 0, res, res, st,
                                    kc, "k_pass_edt_z");
  return cudaGetLastError();
}

cudaError_t launch_close_xpass(const CloseArgs& a, cudaStream_t st, KernelCounter* kc) {
  const int rx = a.dims[0] > 0 ? a.dims[0] : a.res;
  const int ry = a.dims[0] > 0 ? a.dims[1] : a.res;
  const int rz = a.dims[0] > 0 ? a.dims[2] : a.res;
  if (rx % 16 != 0 || ry % 16 != 0 || rz % 16 != 0 || rx <= 0 || ry <= 0 || rz <= 0) return cudaErrorInvalidValue;
  uint8_t* buf8 = close_ws(a, rx, ry, rz).buf8;
  // saturation of the largest clamped radius (127): exact distances up to
  // 129, so any radius bound found later is covered
  return launch_dil_pass_x(a.X, buf8, rx, ry, rz, 129, CBox{{0, 0, 0}, {rx, ry, rz}}, st, kc);
}

cudaError_t launch_close_ypass(const CloseArgs& a, int z0, int z1, int r_bound, cudaStream_t st, KernelCounter* kc) {
  const int rx = a.dims[0] > 0 ? a.dims[0] : a.res;
  const int ry = a.dims[0] > 0 ? a.dims[1] : a.res;
  const int rz = a.dims[0] > 0 ? a.dims[2] : a.res;
  if (rx % 16 != 0 || ry % 16 != 0 || rz % 16 != 0 || rx <= 0 || ry <= 0 || rz <= 0 || a.se != 0 ||
      a.rmap_in == nullptr || z0 < 0 || z1 > rz || z0 >= z1)
    return cudaErrorInvalidValue;
  const int Nx = 2 * rx, Ny = 2 * ry, Nz = 2 * rz;
  const CloseWs w = close_ws(a, rx, ry, rz);
  uint16_t* buf16a = w.buf16a;
  uint8_t* buf8 = w.buf8;
  const int rb = clamp_radius(r_bound);
  const int dil_r = rb + 1, dil_halo = dil_r + 1;
  const uint32_t dil_cap = (uint32_t)(dil_r * dil_r);
  const RField RNONE{nullptr, 0, 0};
  launch_dpx<KERN_LAT, uint8_t, 0>(buf8, buf16a, nullptr, Nx, Ny, Nz, 1, 0, dil_halo, dil_cap, RNONE, 0, rx, ry, st,
                                   kc, "k_pass_dil_y", a.rmap_in, dil_halo,
                                   NeedMap{nullptr, 0, 0, 0, 1, 1, 0, 0, 0,
                                           CBox{{0, 0, 0}, {1 << 30, 1 << 30, 1 << 30}}, z0, z1 - z0});
  return cudaGetLastError();
}

cudaError_t launch_close_zpass(const CloseArgs& a, int z0, int z1, int r_bound, cudaStream_t st, KernelCounter* kc) {
  const int rx = a.dims[0] > 0 ? a.dims[0] : a.res;
  const int ry = a.dims[0] > 0 ? a.dims[1] : a.res;
  const int rz = a.dims[0] > 0 ? a.dims[2] : a.res;
  // whole output tiles (32 cells along z) only
  if (rx % 16 != 0 || ry % 16 != 0 || rz % 16 != 0 || rx <= 0 || ry <= 0 || rz <= 0 || a.se != 0 ||
      a.rmap_in == nullptr || a.R == nullptr || z0 < 0 || z1 > rz || z0 >= z1 || z0 % 32 != 0 || z1 % 32 != 0)
    return cudaErrorInvalidValue;
  const int Nx = 2 * rx, Ny = 2 * ry, Nz = 2 * rz;
  const CloseWs w = close_ws(a, rx, ry, rz);
  uint8_t* dst = a.mode == 1 ? w.D : w.Df;
  const int rb = clamp_radius(r_bound);
  const int dil_r = rb + 1, dil_halo = dil_r + 1;
  const uint32_t dil_cap = (uint32_t)(dil_r * dil_r);
  const RField RF{a.R, a.r_sy > 0 ? a.r_sy : (int64_t)Nx, a.r_sz > 0 ? a.r_sz : (int64_t)Nx * Ny};
  launch_dpx<KERN_LAT, uint16_t, 1>(w.buf16a, nullptr, dst, Nx, Ny, Nz, 2, 0, dil_halo, dil_cap, RF, a.uniform_r, rx,
                                    ry, st, kc, "k_pass_dil_z", a.rmap_in, 0,
                                    NeedMap{nullptr, 0, 0, 0, 1, 1, 0, 0, 0,
                                            CBox{{0, 0, 0}, {1 << 30, 1 << 30, 1 << 30}}, 0, 0, z0 / 32,
                                            (z1 - z0) / 32});
  return cudaGetLastError();
}

cudaError_t launch_contour(const uint8_t* D, uint8_t* S, int res, int exact, cudaStream_t st, KernelCounter* kc) {
  const Dims g{res, res, res};
  const ZWalk w = z_walk(g, 2);
  GM_LAUNCH(kc, "k_contour", st,
            k_contour_z<<<w.blocks, w.threads, 0, st>>>(D, S, g, w.zs, exact, CBox{{0, 0, 0}, {res, res, res}}));
  return cudaGetLastError();
}

cudaError_t launch_rmax(const int8_t* R, int64_t n, int* d_out, int sms, cudaStream_t st, KernelCounter* kc) {
  cudaMemsetAsync(d_out, 0, sizeof(int), st);
  const int64_t vec = n / 16;
  int blocks = grid_stride_blocks(vec, 256, sms);
  if (blocks < 1) blocks = 1;
  GM_LAUNCH(kc, "k_rmax", st, k_rmax<<<blocks, 256, 0, st>>>(R, n, d_out));
  return cudaGetLastError();
}

}  // namespace gm
