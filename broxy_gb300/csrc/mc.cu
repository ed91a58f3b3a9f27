// mc.cu — contour marching cubes and mesh normals (reference rows a12..a16:
// Grid::ComputeContourMCM, ComputeMCMData/CompactMCMData, SplatIndices/
// BuildNeighbors, MarchingCubesMesher::createMesh3D, ComputeMeshNormals,
// BilateralMeshFiltering; GMorpho/Grid.cu:1329-1462, 1873-1973,
// GMorpho/GMorpho.cu:6109-6496, 6498-6620, 6814-7001,
// GMorpho/MarchingCubesMesher.cu:1297-1618).
//
// Emission order equals the reference's: base cells in Morton order (the
// reference sorts its contour list by 30-bit Morton code), eight sub-cubes
// per cell in child order, non-empty cubes compacted, owned edges 0, 3, 8
// numbered in that order.  Instead of a sort, cells are visited directly in
// Morton order: a 16^3 brick of cells is one contiguous 4096-code Morton
// range, so one block per brick with an in-block scan and a scan of the
// brick totals gives every cell its output offsets.  Instead of the 4V-byte
// splat map, a neighbour cube's vertex offset is its cell's offset (one u32
// per cell) plus an in-cell prefix recomputed from the grid.
#include "gm_common.cuh"
#include "gm_internal.h"
#include "mc_tables.inc"

namespace gm {

// (global, not constant memory: the lanes of a warp read different entries)
__device__ const uint64_t d_tri_packed[256] = GM_MC_TRI_PACKED_INIT;
__device__ const uint8_t d_tri_count[256] = GM_MC_TRI_COUNT_INIT;
__device__ const uint8_t d_tri_len[256] = GM_MC_TRI_LEN_INIT;

// A cell's corner block: the occupancy of the 3^3 fine voxels at 2c + (i, j,
// k), bit i + 3 j + 9 k, from which everything about its eight sub-cubes
// follows by shifts: cube k (child order) has its corner at one of the eight
// positions kCubes, corner bits at +0, 1, 4, 3, 9, 10, 13, 12
// (ComputeMCMData, GMorpho.cu:6146-6232), and crossed edges 0, 3, 8 where
// the bits at +1, +3, +9 differ.
constexpr uint32_t kCubes = 0x361bu;  // positions 0, 1, 3, 4, 9, 10, 12, 13

__device__ __forceinline__ uint32_t mixed_cubes(uint32_t b) {
  uint32_t o = b | (b >> 1), a = b & (b >> 1);
  o |= o >> 3, a &= a >> 3;
  o |= o >> 9, a &= a >> 9;
  return o & ~a & kCubes;
}
// crossed owned edges by cube position (a cube with one is mixed)
__device__ __forceinline__ uint32_t edges0(uint32_t b) { return (b ^ (b >> 1)) & kCubes; }
__device__ __forceinline__ uint32_t edges3(uint32_t b) { return (b ^ (b >> 3)) & kCubes; }
__device__ __forceinline__ uint32_t edges8(uint32_t b) { return (b ^ (b >> 9)) & kCubes; }
__device__ __forceinline__ int owned_vertices(uint32_t b) {
  return __popc(edges0(b)) + __popc(edges3(b)) + __popc(edges8(b));
}
// the MC value of the cube at position p
__device__ __forceinline__ uint32_t cube_value(uint32_t b, int p) {
  const uint32_t x = b >> p;
  return (x & 3u) | ((x >> 2) & 4u) | (x & 8u) | ((x >> 5) & 0x30u) | ((x >> 7) & 0x40u) | ((x >> 5) & 0x80u);
}
// position of the cube at (x, y, z) of its cell, each 0 or 1
__device__ __forceinline__ int cube_pos(int x, int y, int z) { return x + 3 * y + 9 * z; }

constexpr int kBrick = 16;               // cells per brick edge
constexpr int kTileE = kBrick + 2;       // tile edge (halo 2 for neighbour cells)
constexpr int kTileP = 32;               // tile row pitch (bytes): rows are one 16-byte and one 2-byte store
constexpr int kTileCells = kTileP * kTileE * kTileE;
__device__ __forceinline__ int tix(int x, int y, int z) { return x + kTileP * (y + kTileE * z); }
constexpr int kCellsPerBrick = kBrick * kBrick * kBrick;
constexpr int kMcThreads = 256;
constexpr int kCellsPerThread = kCellsPerBrick / kMcThreads;

__device__ __forceinline__ void brick_origin(int b, int& ox, int& oy, int& oz) {
  ox = (int)gather_bits3((uint32_t)b) * kBrick;
  oy = (int)gather_bits3((uint32_t)b >> 1) * kBrick;
  oz = (int)gather_bits3((uint32_t)b >> 2) * kBrick;
}

// grid dimensions in cells (x, y, z); x-fastest
struct GDims { int x, y, z; };
__device__ __forceinline__ int64_t gidx(int x, int y, int z, GDims d) { return idx3(x, y, z, d.x, d.y); }

// Loads the tile (cells o .. o + 17 per axis, zero outside the grid) and
// tells (block-uniformly) whether it can hold a mixed cube: a tile whose
// bytes are all 0x00 or all 0xff has none.  One row (18 cells along x) is
// a 16-byte and a 2-byte load: bricks start at multiples of 16 cells and
// grid edges are multiples of 16, so a row is either inside the grid up to
// cell o + 15 or outside, and so are cells o + 16, o + 17.
__device__ bool load_tile_mixed(const uint8_t* __restrict__ C, GDims d, int ox, int oy, int oz, uint8_t* tile) {
  int seen0 = 0, seen1 = 0, part = 0;
  for (int row = threadIdx.x; row < kTileE * kTileE; row += blockDim.x) {
    const int ly = row % kTileE, lz = row / kTileE;
    const int y = oy + ly, z = oz + lz;
    uint4 q = make_uint4(0u, 0u, 0u, 0u);
    uint32_t h = 0u;
    if (y < d.y && z < d.z && ox < d.x) {
      q = *reinterpret_cast<const uint4*>(C + gidx(ox, y, z, d));
      if (ox + kBrick < d.x) h = *reinterpret_cast<const uint16_t*>(C + gidx(ox + kBrick, y, z, d));
    }
    uint8_t* trow = tile + kTileP * row;
    *reinterpret_cast<uint4*>(trow) = q;
    *reinterpret_cast<uint16_t*>(trow + kBrick) = (uint16_t)h;
    // the two halo bytes, repeated to fill a word (repeats change no test)
    const uint32_t w[5] = {q.x, q.y, q.z, q.w, h | (h << 16)};
#pragma unroll
    for (int k = 0; k < 5; k++) {
      const uint32_t z4 = __vcmpeq4(w[k], 0u), f4 = __vcmpeq4(w[k], 0xffffffffu);
      seen0 |= z4 != 0u;
      seen1 |= f4 != 0u;
      part |= (~(z4 | f4)) != 0u;
    }
  }
  const int mixed = __syncthreads_or(part | (seen0 & seen1));
  if (mixed) return true;
  // a block may have seen only zeros while another saw only full bytes
  return __syncthreads_or(seen0) && __syncthreads_or(seen1);
}

// The corner block of tile cell (lx, ly, lz).
__device__ __forceinline__ uint32_t corner_block(const uint8_t* tile, int lx, int ly, int lz) {
  uint32_t c = tile[tix(lx, ly, lz)];
  uint32_t b = (c & 3u) | ((c & 0xcu) << 1) | ((c & 0x30u) << 5) | ((c & 0xc0u) << 6);
  c = tile[tix(lx + 1, ly, lz)];
  b |= ((c & 1u) << 2) | ((c & 4u) << 3) | ((c & 0x10u) << 7) | ((c & 0x40u) << 8);
  c = tile[tix(lx, ly + 1, lz)];
  b |= ((c & 3u) << 6) | ((c & 0x30u) << 11);
  c = tile[tix(lx + 1, ly + 1, lz)];
  b |= ((c & 1u) << 8) | ((c & 0x10u) << 13);
  c = tile[tix(lx, ly, lz + 1)];
  b |= ((c & 3u) << 18) | ((c & 0xcu) << 19);
  c = tile[tix(lx + 1, ly, lz + 1)];
  b |= ((c & 1u) << 20) | ((c & 4u) << 21);
  c = tile[tix(lx, ly + 1, lz + 1)];
  b |= (c & 3u) << 24;
  c = tile[tix(lx + 1, ly + 1, lz + 1)];
  return b | ((c & 1u) << 26);
}

// Tagging / emission window of one meshing run.  A whole grid is its own
// window: off = 0, gdim = its size, tag and emit boxes = the whole grid.  The edit
// server meshes the dirty box of a crop: the crop's cells sit at global
// cells off + local, the border rule uses the global resolution, cubes are
// tagged (own vertices) in the dirty box plus one cell on the + side (the
// neighbour cubes whose edges the box's triangles use), and triangles come
// from the dirty box only.
struct McWin {
  int off[3];
  int gdim[3];         // global grid (cells): cubes of cells outside [1, gdim-2] are never tagged
  int tlo[3], thi[3];  // local cells whose cubes may be tagged, [lo, hi)
  int elo[3], ehi[3];  // local cells whose cubes emit triangles, [lo, hi)
};

// cells outside [1, gres-2]^3 are never tagged (TagVoxelsContourMCM,
// Grid.cu:1334-1340)
__device__ __forceinline__ bool win_tag(const McWin& w, int x, int y, int z) {
  const int gx = x + w.off[0], gy = y + w.off[1], gz = z + w.off[2];
  return gx >= 1 && gy >= 1 && gz >= 1 && gx <= w.gdim[0] - 2 && gy <= w.gdim[1] - 2 && gz <= w.gdim[2] - 2 &&
         x >= w.tlo[0] && y >= w.tlo[1] && z >= w.tlo[2] && x < w.thi[0] && y < w.thi[1] && z < w.thi[2];
}
__device__ __forceinline__ bool win_emit(const McWin& w, int x, int y, int z) {
  return x >= w.elo[0] && y >= w.elo[1] && z >= w.elo[2] && x < w.ehi[0] && y < w.ehi[1] && z < w.ehi[2];
}
// block-uniform: does the 16^3 brick at (ox, oy, oz) meet the tag box?
__device__ __forceinline__ bool brick_live(const McWin& w, int ox, int oy, int oz) {
  return ox < w.thi[0] && oy < w.thi[1] && oz < w.thi[2] && ox + kBrick > w.tlo[0] && oy + kBrick > w.tlo[1] &&
         oz + kBrick > w.tlo[2];
}

__device__ __forceinline__ void local_coords(int l, int& lx, int& ly, int& lz) {
  lx = (int)gather_bits3((uint32_t)l);
  ly = (int)gather_bits3((uint32_t)l >> 1);
  lz = (int)gather_bits3((uint32_t)l >> 2);
}

// block-wide exclusive scan of one counter (256 threads); total in `total`
__device__ __forceinline__ uint32_t block_scan1(uint32_t v, uint32_t& total) {
  __shared__ uint32_t wt[kMcThreads / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  uint32_t x = v;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t t = __shfl_up_sync(0xffffffffu, x, o);
    if (lane >= o) x += t;
  }
  if (lane == 31) wt[wid] = x;
  __syncthreads();
  uint32_t pre = 0, tot = 0;
#pragma unroll
  for (int k = 0; k < kMcThreads / 32; k++) {
    pre += k < wid ? wt[k] : 0u;
    tot += wt[k];
  }
  __syncthreads();
  total = tot;
  return pre + x - v;
}

// Cells of one row of a tile that may hold a tagged mixed cube (bit x): those
// whose 2x2x2 block of cells is neither all empty nor all full, four at a
// time as bytes of a word, inside the tag window.
__device__ __forceinline__ uint32_t row_candidates(const uint8_t* tile, const McWin& w, int ox, int oy, int oz, int ly,
                                                   int lz) {
  const int gy = oy + ly + w.off[1], gz = oz + lz + w.off[2];
  if (gy < 1 || gz < 1 || gy > w.gdim[1] - 2 || gz > w.gdim[2] - 2 || oy + ly < w.tlo[1] || oz + lz < w.tlo[2] ||
      oy + ly >= w.thi[1] || oz + lz >= w.thi[2])
    return 0u;
  uint32_t o[5] = {0u, 0u, 0u, 0u, 0u}, a[5] = {~0u, ~0u, ~0u, ~0u, ~0u};
#pragma unroll
  for (int r = 0; r < 4; r++) {
    const uint8_t* row = tile + tix(0, ly + (r & 1), lz + (r >> 1));
    const uint4 q = *reinterpret_cast<const uint4*>(row);
    const uint32_t h = *reinterpret_cast<const uint16_t*>(row + kBrick);
    const uint32_t v[5] = {q.x, q.y, q.z, q.w, h};
#pragma unroll
    for (int j = 0; j < 5; j++) o[j] |= v[j], a[j] &= v[j];
  }
  uint32_t cand = 0;
#pragma unroll
  for (int j = 0; j < 4; j++) {
    const uint32_t on = o[j] | (o[j] >> 8) | (o[j + 1] << 24), an = a[j] & ((a[j] >> 8) | (a[j + 1] << 24));
    const uint32_t uniform = __vcmpeq4(on, 0u) | __vcmpeq4(an, 0xffffffffu);
    cand |= (((~uniform & 0x08040201u) * 0x01010101u) >> 24) << (4 * j);
  }
  const int lo = max(max(1 - w.off[0], w.tlo[0]) - ox, 0), hi = min(min(w.gdim[0] - 1 - w.off[0], w.thi[0]) - ox, kBrick);
  return hi <= lo ? 0u : cand & ((1u << hi) - (1u << lo));
}

// Counting pass, a block per brick: the mixed cells' corner blocks go to
// cells[].x (where their cell lies: later passes and neighbours find them
// there) and the brick's mask of them, in Morton order, to brick_mask, so
// that the tile is read once per mesh; totals of mixed cells, vertices,
// triangles and case-91 cubes to brick_tot.  At 1024^3 (4.4M vertices) 0.145
// ms, bound by its tile loads and barriers; 0.264 when every cell was tested
// byte by byte and its cubes built corner by corner.
constexpr int kMaskWords = kCellsPerBrick / 32;
__global__ void __launch_bounds__(kMcThreads, 6) k_mc_count(const uint8_t* __restrict__ C, GDims gd, McWin w,
                                                          uint32_t* __restrict__ brick_tot,
                                                          uint32_t* __restrict__ brick_mask, uint2* __restrict__ cells) {
  __shared__ __align__(16) uint8_t tile[kTileCells];
  __shared__ uint16_t list[kCellsPerBrick];
  __shared__ uint32_t mask[kMaskWords], tot[4];
  __shared__ uint8_t tab[256];  // triangles of a value, bit 7: one more than its slots (case 91)
  int ox, oy, oz;
  brick_origin(blockIdx.x, ox, oy, oz);
  if (threadIdx.x < 4) tot[threadIdx.x] = 0u;
  if (threadIdx.x < kMaskWords) mask[threadIdx.x] = 0u;
  if (!brick_live(w, ox, oy, oz) || !load_tile_mixed(C, gd, ox, oy, oz, tile)) {
    if (threadIdx.x < 4) brick_tot[4 * (size_t)blockIdx.x + threadIdx.x] = 0;
    return;
  }
  {
    const uint32_t n = d_tri_count[threadIdx.x];
    tab[threadIdx.x] = (uint8_t)(n | (d_tri_len[threadIdx.x] > n ? 0x80u : 0u));
  }
  const int ly = threadIdx.x & 15, lz = threadIdx.x >> 4;
  uint32_t cand = row_candidates(tile, w, ox, oy, oz, ly, lz), nc;
  uint32_t k = block_scan1(__popc(cand), nc);
  while (cand) {
    list[k++] = (uint16_t)((__ffs(cand) - 1) | (ly << 4) | (lz << 8));
    cand &= cand - 1;
  }
  __syncthreads();
  uint32_t n_cells = 0, n_verts = 0, n_tris = 0, n91 = 0;
  for (uint32_t j = threadIdx.x; j < nc; j += kMcThreads) {
    const int e = list[j], x = e & 15, y = (e >> 4) & 15, z = e >> 8;
    const uint32_t b = corner_block(tile, x, y, z);
    uint32_t m = mixed_cubes(b);
    if (!m) continue;
    cells[gidx(ox + x, oy + y, oz + z, gd)].x = b;
    const uint32_t l = morton3((uint32_t)x, (uint32_t)y, (uint32_t)z);
    atomicOr(mask + (l >> 5), 1u << (l & 31u));
    n_cells++;
    n_verts += owned_vertices(b);
    if (!win_emit(w, ox + x, oy + y, oz + z)) continue;
    while (m) {
      const uint32_t t = tab[cube_value(b, __ffs(m) - 1)];
      m &= m - 1;
      n_tris += t & 7u;
      n91 += t >> 7;
    }
  }
  n_cells = __reduce_add_sync(0xffffffffu, n_cells);
  n_verts = __reduce_add_sync(0xffffffffu, n_verts);
  n_tris = __reduce_add_sync(0xffffffffu, n_tris);
  n91 = __reduce_add_sync(0xffffffffu, n91);
  if ((threadIdx.x & 31) == 0 && n_cells) {
    atomicAdd(tot + 0, n_cells);
    atomicAdd(tot + 1, n_verts);
    atomicAdd(tot + 2, n_tris);
    atomicAdd(tot + 3, n91);
  }
  __syncthreads();
  if (threadIdx.x < 4) brick_tot[4 * (size_t)blockIdx.x + threadIdx.x] = tot[threadIdx.x];
  if (tot[0] && threadIdx.x < kMaskWords) brick_mask[(size_t)blockIdx.x * kMaskWords + threadIdx.x] = mask[threadIdx.x];
}

// Exclusive scan of the four brick counters, in place, totals at index nb:
// chunks of 1024 bricks, one block each.  k_brick_sums leaves each chunk's
// sums after the counters (index nb + 1 + chunk); k_scan_bricks adds the
// sums of the chunks before its own and scans its chunk (16-byte loads).
constexpr int kBrickChunk = 1024;

__device__ __forceinline__ uint4 add4(uint4 a, uint4 b) { return make_uint4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }
__device__ __forceinline__ uint4 shfl_up4(uint4 v, int o) {
  return make_uint4(__shfl_up_sync(0xffffffffu, v.x, o), __shfl_up_sync(0xffffffffu, v.y, o),
                    __shfl_up_sync(0xffffffffu, v.z, o), __shfl_up_sync(0xffffffffu, v.w, o));
}
__device__ __forceinline__ uint4 shfl4(uint4 v, int src) {
  return make_uint4(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src),
                    __shfl_sync(0xffffffffu, v.z, src), __shfl_sync(0xffffffffu, v.w, src));
}
// inclusive scan over the block (1024 threads); *total = the block's sum
__device__ __forceinline__ uint4 block_incl_scan4(uint4 v, uint4* total) {
  __shared__ uint4 warp_tot[32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint4 t = shfl_up4(v, o);
    if (lane >= o) v = add4(v, t);
  }
  if (lane == 31) warp_tot[wid] = v;
  __syncthreads();
  if (wid == 0) {
    uint4 w = warp_tot[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const uint4 t = shfl_up4(w, o);
      if (lane >= o) w = add4(w, t);
    }
    warp_tot[lane] = w;
  }
  __syncthreads();
  if (wid > 0) v = add4(v, warp_tot[wid - 1]);
  *total = warp_tot[31];
  return v;
}

__global__ void __launch_bounds__(kBrickChunk) k_brick_sums(uint32_t* __restrict__ bt, int nb) {
  const int b = blockIdx.x * kBrickChunk + threadIdx.x;
  const uint4 v = b < nb ? reinterpret_cast<const uint4*>(bt)[b] : make_uint4(0u, 0u, 0u, 0u);
  uint4 tot;
  block_incl_scan4(v, &tot);
  if (threadIdx.x == 0) reinterpret_cast<uint4*>(bt)[nb + 1 + blockIdx.x] = tot;
}

__global__ void __launch_bounds__(kBrickChunk) k_scan_bricks(uint32_t* __restrict__ bt, int nb) {
  // sums of the chunks before this one (at most kBrickChunk chunks)
  const int t = threadIdx.x;
  uint4 prev = t < (int)blockIdx.x ? reinterpret_cast<const uint4*>(bt)[nb + 1 + t] : make_uint4(0u, 0u, 0u, 0u);
  uint4 off;
  block_incl_scan4(prev, &off);
  __syncthreads();  // the scan's shared totals are reused below
  const int b = blockIdx.x * kBrickChunk + t;
  const uint4 v = b < nb ? reinterpret_cast<const uint4*>(bt)[b] : make_uint4(0u, 0u, 0u, 0u);
  uint4 tot;
  const uint4 incl = block_incl_scan4(v, &tot);
  const uint4 excl = make_uint4(incl.x - v.x, incl.y - v.y, incl.z - v.z, incl.w - v.w);
  if (b < nb) reinterpret_cast<uint4*>(bt)[b] = add4(off, excl);
  if (t == 0 && blockIdx.x == gridDim.x - 1) reinterpret_cast<uint4*>(bt)[nb] = add4(off, tot);
}

// Float expressions of findIntersection (MarchingCubesMesher.cu:98-100) with
// the corner point minC + idx * cellSize (MarchingCubesMesher.cu:1329-1331),
// evaluated with explicit rounding so that host and device agree bit for bit.
// The corner values are 0 or 1 and differ along an edge, so v2 - v1 is +1 or
// -1 and the IEEE quotient is the numerator or its negation, exactly
// (signed zeros included): no division is issued.
__device__ __forceinline__ float lerp_coord(float p1, float p2, float v1, float v2, float iso) {
  const float t = __fsub_rn(iso, v1);
  const float num = __fmul_rn(t, __fsub_rn(p2, p1));
  return __fadd_rn(p1, __fsub_rn(v2, v1) > 0.f ? num : -num);
}

// A mixed cell in Morton order: its brick and place (33 bits: the upper one
// above the corner block's 27 bits), first vertex and first triangle.
__device__ __forceinline__ uint4 pack_entry(uint32_t brick, uint32_t l, uint32_t b, uint32_t v, uint32_t t) {
  return make_uint4((brick << 12) | l, b | ((brick >> 20) << 27), v, t);
}

// The mixed cells of a brick listed in Morton order (entries), each with its
// first vertex and triangle from one scan per round of 256, and their
// vertices.  A block per brick, from the counting pass's mask: no tile
// (0.304 -> 0.090 ms at 1024^3).
__global__ void __launch_bounds__(kMcThreads, 6) k_mc_vertices(GDims gd, McWin w,
                                                          const uint32_t* __restrict__ brick_off,
                                                          const uint32_t* __restrict__ brick_mask,
                                                          uint2* __restrict__ cells, uint4* __restrict__ entries,
                                                          float* __restrict__ V, float bx, float by, float bz,
                                                          float cs, float iso) {
  __shared__ uint16_t list[kCellsPerBrick];
  __shared__ uint8_t tab[256];
  const uint4 off = reinterpret_cast<const uint4*>(brick_off)[blockIdx.x];
  const int nc = (int)(reinterpret_cast<const uint4*>(brick_off)[blockIdx.x + 1].x - off.x);
  if (nc == 0) return;
  int ox, oy, oz;
  brick_origin(blockIdx.x, ox, oy, oz);
  tab[threadIdx.x] = d_tri_count[threadIdx.x];
  {
    // 16 cells a thread
    uint32_t m = reinterpret_cast<const uint16_t*>(brick_mask + (size_t)blockIdx.x * kMaskWords)[threadIdx.x], n;
    uint32_t k = block_scan1(__popc(m), n);
    while (m) {
      list[k++] = (uint16_t)(threadIdx.x * kCellsPerThread + __ffs(m) - 1);
      m &= m - 1;
    }
  }
  __syncthreads();
  uint32_t run = 0;  // vertices and triangles of the rounds before (16 bits each a round, 32 in all)
  uint32_t run_t = 0;
  for (int j0 = 0; j0 < nc; j0 += kMcThreads) {
    const int j = j0 + (int)threadIdx.x;
    uint32_t l = 0, b = 0, nv = 0, nt = 0;
    int gx = 0, gy = 0, gz = 0;
    int64_t g = 0;
    if (j < nc) {
      l = list[j];
      int lx, ly, lz;
      local_coords((int)l, lx, ly, lz);
      gx = ox + lx, gy = oy + ly, gz = oz + lz;
      g = gidx(gx, gy, gz, gd);
      b = cells[g].x;
      nv = owned_vertices(b);
      if (win_emit(w, gx, gy, gz))
        for (uint32_t m = mixed_cubes(b); m; m &= m - 1) nt += tab[cube_value(b, __ffs(m) - 1)];
    }
    uint32_t total;
    const uint32_t pre = block_scan1(nv | (nt << 16), total);  // (at most 24 and 40 a cell)
    uint32_t vo = off.y + run + (pre & 0xffffu);
    const uint32_t to = off.z + run_t + (pre >> 16);
    run += total & 0xffffu;
    run_t += total >> 16;
    if (j >= nc) continue;
    entries[off.x + j] = pack_entry(blockIdx.x, l, b, vo, to);
    cells[g].y = vo;
    for (uint32_t own = edges0(b) | edges3(b) | edges8(b); own; own &= own - 1) {
      const int p = __ffs(own) - 1, sz = p >= 9 ? 1 : 0, sy = p - 9 * sz >= 3 ? 1 : 0, sx = p - 9 * sz - 3 * sy;
      const uint32_t c = b >> p;
      // corner point from GLOBAL fine coordinates, so that a crop's vertices
      // are bit-identical to the whole grid's
      const float px = __fmaf_rn((float)(2 * (gx + w.off[0]) + sx), cs, bx);
      const float py = __fmaf_rn((float)(2 * (gy + w.off[1]) + sy), cs, by);
      const float pz = __fmaf_rn((float)(2 * (gz + w.off[2]) + sz), cs, bz);
      const float v0 = (c & 1u) ? 1.f : 0.f, v1 = (c & 2u) ? 1.f : 0.f, v3 = (c & 8u) ? 1.f : 0.f,
                  v4 = (c & 512u) ? 1.f : 0.f;
      if (v0 != v1) {  // edge 0: point -> point + (cs,0,0)
        float* o = V + 3 * (size_t)vo++;
        o[0] = lerp_coord(px, __fadd_rn(px, cs), v0, v1, iso);
        o[1] = lerp_coord(py, py, v0, v1, iso);
        o[2] = lerp_coord(pz, pz, v0, v1, iso);
      }
      if (v0 != v3) {  // edge 3: point + (0,cs,0) -> point
        const float p1y = __fadd_rn(py, cs);
        float* o = V + 3 * (size_t)vo++;
        o[0] = lerp_coord(px, px, v3, v0, iso);
        o[1] = lerp_coord(p1y, py, v3, v0, iso);
        o[2] = lerp_coord(pz, pz, v3, v0, iso);
      }
      if (v0 != v4) {  // edge 8: point -> point + (0,0,cs)
        float* o = V + 3 * (size_t)vo++;
        o[0] = lerp_coord(px, px, v0, v4, iso);
        o[1] = lerp_coord(py, py, v0, v4, iso);
        o[2] = lerp_coord(pz, __fadd_rn(pz, cs), v0, v4, iso);
      }
    }
  }
}

// Triangles: eight lanes per listed cell, one per sub-cube, over the whole
// list (a small grid's bricks spread over all SMs).  Lane k also holds the
// neighbour cell at offset k (corner block and first vertex): the cubes whose
// edges a cube's triangles use lie in those eight cells, so their vertices
// come by shuffles.  A neighbour outside the tag window has no vertices (its
// edges take index 0); inside it, a crossed edge's owner is mixed, so its
// words are this mesh's.  0.626 -> 0.214 ms at 1024^3, and 84 -> 11 us at
// 128^3, where a block per brick (tile, summaries of 17^3 cells, rounds with
// three barriers each) left most SMs idle.
__global__ void __launch_bounds__(kMcThreads) k_mc_triangles(GDims gd, McWin w, const uint2* __restrict__ cells,
                                                            const uint4* __restrict__ entries, uint32_t ncells,
                                                            uint32_t* __restrict__ T, uint32_t nt_total,
                                                            uint32_t* __restrict__ fix, int fix_cap) {
  __shared__ uint64_t tab[256];             // edges of a value's triangles, its count in the upper bits
  __shared__ uint32_t vert[12][kMcThreads];  // edge vertices of each thread's cube
  {
    const uint32_t n = d_tri_count[threadIdx.x];
    tab[threadIdx.x] = d_tri_packed[threadIdx.x] | ((uint64_t)(n | (d_tri_len[threadIdx.x] > n ? 8u : 0u)) << 60);
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, k = lane & 7, kx = k & 1, ky = (k >> 1) & 1, kz = k >> 2;
  // (the grid covers whole warps: all lanes of a warp run as many rounds)
  const uint32_t stride = gridDim.x * (kMcThreads / 8);
  for (uint32_t i0 = (blockIdx.x * kMcThreads + (threadIdx.x & ~31u)) / 8; i0 < ncells; i0 += stride) {
    const uint32_t i = i0 + (lane >> 3);
    uint4 e = make_uint4(0u, 0u, 0u, 0u);
    int gx = 0, gy = 0, gz = 0;
    uint32_t b = 0, nb = 0, nvo = 0;  // own block; the neighbour's block and first vertex
    bool tagged = false, emit = false;
    if (i < ncells) {
      e = entries[i];
      b = e.y & 0x7ffffffu;
      const uint32_t brick = (e.x >> 12) | ((e.y >> 27) << 20);
      int ox, oy, oz, lx, ly, lz;
      brick_origin((int)brick, ox, oy, oz);
      local_coords((int)(e.x & 0xfffu), lx, ly, lz);
      gx = ox + lx, gy = oy + ly, gz = oz + lz;
      emit = win_emit(w, gx, gy, gz);
      const int x = gx + kx, y = gy + ky, z = gz + kz;
      tagged = x < gd.x && y < gd.y && z < gd.z && win_tag(w, x, y, z);
      if (k == 0) {
        nb = b, nvo = e.z;
      } else if (tagged && emit) {
        const uint2 c = cells[gidx(x, y, z, gd)];
        nb = c.x, nvo = c.y;
      }
    }
    const uint32_t tags = __ballot_sync(0xffffffffu, tagged) >> (lane & 24);
    const int p = cube_pos(kx, ky, kz);
    const bool cube = emit && ((mixed_cubes(b) >> p) & 1u);
    const uint32_t val = cube_value(b, p);
    const uint64_t tl = tab[val];
    const uint32_t cnt = cube ? (uint32_t)(tl >> 60) & 7u : 0u;
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
      const uint32_t t = __shfl_up_sync(0xffffffffu, incl, o, 8);
      if (k >= o) incl += t;
    }
    const uint32_t to = e.w + incl - cnt;
    // crossed edges: 0 (0,1) 1 (1,2) 2 (2,3) 3 (3,0) 4 (4,5) 5 (5,6) 6 (6,7)
    // 7 (7,4) 8 (0,4) 9 (1,5) 10 (2,6) 11 (3,7); their owner cubes are this
    // one and those at +x, +x+y, +y, +z, +x+z, +y+z, their own edges 0, 3, 8
    // (BuildNeighbors order, GMorpho.cu:6480-6487;
    // MarchingCubesMesher.cu:1392-1456)
    auto owner = [&](int dx, int dy, int dz, uint32_t& first, uint32_t& e0, uint32_t& e3) -> bool {
      const int fx = kx + dx, fy = ky + dy, fz = kz + dz;
      const int cell = (fx >> 1) | ((fy >> 1) << 1) | ((fz >> 1) << 2);
      const uint32_t ob = __shfl_sync(0xffffffffu, nb, cell, 8), ov = __shfl_sync(0xffffffffu, nvo, cell, 8);
      const int q = cube_pos(fx & 1, fy & 1, fz & 1);
      const uint32_t below = (1u << q) - 1u, m0 = edges0(ob), m3 = edges3(ob), m8 = edges8(ob);
      first = ov + __popc(m0 & below) + __popc(m3 & below) + __popc(m8 & below);
      e0 = (m0 >> q) & 1u;
      e3 = (m3 >> q) & 1u;
      return (tags >> cell) & 1u;
    };
    uint32_t f, e0, e3;
    uint32_t(*my)[kMcThreads] = reinterpret_cast<uint32_t(*)[kMcThreads]>(&vert[0][threadIdx.x]);
    bool ok = owner(0, 0, 0, f, e0, e3);
    my[0][0] = f, my[3][0] = f + e0, my[8][0] = f + e0 + e3;
    ok = owner(1, 0, 0, f, e0, e3);
    my[1][0] = ok ? f + e0 : 0u, my[9][0] = ok ? f + e0 + e3 : 0u;
    ok = owner(1, 1, 0, f, e0, e3);
    my[10][0] = ok ? f + e0 + e3 : 0u;
    ok = owner(0, 1, 0, f, e0, e3);
    my[2][0] = ok ? f : 0u, my[11][0] = ok ? f + e0 + e3 : 0u;
    ok = owner(0, 0, 1, f, e0, e3);
    my[4][0] = ok ? f : 0u, my[7][0] = ok ? f + e0 : 0u;
    ok = owner(1, 0, 1, f, e0, e3);
    my[5][0] = ok ? f + e0 : 0u;
    ok = owner(0, 1, 1, f, e0, e3);
    my[6][0] = ok ? f : 0u;
    // reversed winding (MarchingCubesMesher.cu:1487-1497)
    for (uint32_t t = 0; t < cnt; t++) {
      uint32_t* o = T + 3 * (size_t)(to + t);
      o[0] = my[(tl >> (4 * (3 * t + 2))) & 0xf][0];
      o[1] = my[(tl >> (4 * (3 * t + 1))) & 0xf][0];
      o[2] = my[(tl >> (4 * (3 * t))) & 0xf][0];
    }
    if (cube && (tl >> 63)) {
      // Case 91: the reference writes one more triangle than its slot
      // count; it lands on the next slot (the next cube's first triangle)
      // and, written later, wins; past the end it is dropped.
      const uint32_t slot = to + cnt;
      if (slot < nt_total) {
        const int idx = (int)atomicAdd(fix, 1u);
        if (idx < fix_cap) {
          uint32_t* o = fix + 1 + 4 * idx;
          o[0] = slot;
          o[1] = my[(tl >> (4 * (3 * cnt + 2))) & 0xf][0];
          o[2] = my[(tl >> (4 * (3 * cnt + 1))) & 0xf][0];
          o[3] = my[(tl >> (4 * (3 * cnt))) & 0xf][0];
        }
      }
    }
  }
}

__global__ void k_mc_fix91(const uint32_t* __restrict__ fix, int fix_cap, uint32_t* __restrict__ T) {
  const int n = min((int)fix[0], fix_cap);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const uint32_t* f = fix + 1 + 4 * i;
    uint32_t* o = T + 3 * (size_t)f[0];
    o[0] = f[1]; o[1] = f[2]; o[2] = f[3];
  }
}

// ------------------------------------------------------------------ normals

// Vertex -> corner lists.  A vertex sits on an edge shared by four cubes of
// at most five triangles, so it has at most kAdjMax corners and its list is
// a row of fixed size: one pass of atomics fills it, in any order, and
// k_adj_finish sorts it (no counting pass, no scan).  The first kAdjRow
// slots (32 bytes, enough for nearly every vertex) and the others are
// separate arrays.  Vertex 0 is special: the reference's triangles take
// index 0 for an edge whose owning cube is not tagged (cubes of border
// cells), so on grids whose surface reaches the border vertex 0 collects an
// unbounded number of corners; past kAdjMax they are collected apart.
constexpr int kAdjMax = 20;
constexpr int kAdjRow = 8;

// counters after the vertices' in `cursor`: records placed, blocks that
// finished an iteration
enum { kCntRecords = 0, kCntArrived = 1, kCntWords = 4 };

__global__ void k_adj_slots(const uint32_t* __restrict__ T, int64_t nt, uint32_t* __restrict__ cursor,
                            uint32_t* __restrict__ adj, uint32_t* __restrict__ adj_more,
                            uint32_t* __restrict__ row0) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < 3 * nt; i += (int64_t)gridDim.x * blockDim.x) {
    const uint32_t v = T[i];
    const uint32_t slot = atomicAdd(cursor + v, 1u);
    if (slot < kAdjRow) adj[(size_t)kAdjRow * v + slot] = (uint32_t)i;  // corner id = 3 t + role
    else if (slot < kAdjMax) adj_more[(size_t)(kAdjMax - kAdjRow) * v + slot - kAdjRow] = (uint32_t)i;
    if (v == 0u) row0[slot] = (uint32_t)i;
  }
}

__device__ __forceinline__ float3 ld3(const float* p, uint32_t i) {
  return make_float3(p[3 * (size_t)i], p[3 * (size_t)i + 1], p[3 * (size_t)i + 2]);
}

__device__ __forceinline__ float3 normalize3(float3 n) {
  const float l = __fsqrt_rn(__fadd_rn(__fadd_rn(__fmul_rn(n.x, n.x), __fmul_rn(n.y, n.y)), __fmul_rn(n.z, n.z)));
  return make_float3(__fdiv_rn(n.x, l), __fdiv_rn(n.y, l), __fdiv_rn(n.z, l));
}


__device__ __forceinline__ float dist2(float3 a, float3 b) {
  const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y), dz = __fsub_rn(a.z, b.z);
  return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}


__device__ __forceinline__ float dist2n(float4 a, float4 b) {
  const float dx = __fsub_rn(a.x, b.x), dy = __fsub_rn(a.y, b.y), dz = __fsub_rn(a.z, b.z);
  return __fadd_rn(__fadd_rn(__fmul_rn(dx, dx), __fmul_rn(dy, dy)), __fmul_rn(dz, dz));
}

// Compare-exchange networks over M values in registers.
template <int M>
__device__ __forceinline__ void bitonic_sort(uint32_t (&k)[M]) {
#pragma unroll
  for (int s = 2; s <= M; s <<= 1)
#pragma unroll
    for (int j = s >> 1; j > 0; j >>= 1)
#pragma unroll
      for (int i = 0; i < M; i++) {
        const int l = i ^ j;
        if (l > i) {
          const uint32_t a = k[i], b = k[l];
          const bool up = (i & s) == 0;
          k[i] = up ? min(a, b) : max(a, b);
          k[l] = up ? max(a, b) : min(a, b);
        }
      }
}

// one incident corner: its triangle's other vertices, the one after it and
// the one before it in the triangle's orientation, and its normal term
// (ComputeMeshNormals, GMorpho.cu:6498-6524)
__device__ __forceinline__ void adj_corner(const float* __restrict__ V, const uint32_t* __restrict__ T,
                                           uint32_t corner, float3& n, uint32_t& next, uint32_t& prev) {
  const uint32_t t = corner / 3, role = corner - 3 * t;
  const uint32_t i0 = T[3 * (size_t)t], i1 = T[3 * (size_t)t + 1], i2 = T[3 * (size_t)t + 2];
  const float3 p0 = ld3(V, i0), p1 = ld3(V, i1), p2 = ld3(V, i2);
  const float3 a = make_float3(__fsub_rn(p1.x, p0.x), __fsub_rn(p1.y, p0.y), __fsub_rn(p1.z, p0.z));
  const float3 b = make_float3(__fsub_rn(p2.x, p0.x), __fsub_rn(p2.y, p0.y), __fsub_rn(p2.z, p0.z));
  n.x = __fsub_rn(__fmul_rn(a.y, b.z), __fmul_rn(a.z, b.y));
  n.y = __fsub_rn(__fmul_rn(a.z, b.x), __fmul_rn(a.x, b.z));
  n.z = __fsub_rn(__fmul_rn(a.x, b.y), __fmul_rn(a.y, b.x));
  next = role == 0 ? i1 : (role == 1 ? i2 : i0);
  prev = role == 0 ? i2 : (role == 1 ? i0 : i1);
}

__device__ __forceinline__ float3 add3(float3 a, float3 b) {
  return make_float3(__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z));
}

// Filter records of a vertex: (neighbour, position term bits |pa - pb|^2),
// one per neighbour or per two occurrences of it among the incident
// triangles (an edge shared by two of them), the sign bit marking a double;
// in (neighbour, term) order.  sigma_p is 1 (GMorpho.cu:6959-6969), so the
// term of GMorpho.cu:6561-6569 is the squared distance itself.
//
// The records of kRecChunk consecutive vertices are packed, the chunks in
// any order (each takes its place from a counter: no scan over the mesh);
// a chunk has its own row of offsets, one more than its vertices, after
// vertex 0's own start and end (its records may lie apart).  (The
// iterations are bound by the records' bytes and the gathers' latency: rows
// of eight slots a vertex, or slots of 32 vertices interleaved, were 18%
// slower.)
constexpr int kRecChunk = 256;
constexpr int kPool = 4;  // general vertices that a warp takes together (more go one a lane)
__device__ __forceinline__ uint32_t roff_at(uint32_t v) { return v == 0u ? 0u : v + v / kRecChunk + 2u; }

// pairs (neighbour << 32 | term bits) sorted; merged in place into records
// (they never overtake the pairs still to be read); returns how many
__device__ uint32_t merge_pairs(uint64_t* kv, uint32_t m) {
  uint32_t w = 0, prev = 0;
  int run = 0;
  for (uint32_t i = 0; i < m; i++) {
    const uint64_t x = kv[i];
    const uint32_t id = (uint32_t)(x >> 32);
    run = (i > 0 && id == prev) ? run + 1 : 0;
    prev = id;
    if (run & 1) continue;
    const bool dbl = i + 1 < m && (uint32_t)(kv[i + 1] >> 32) == id;
    kv[w++] = ((uint64_t)id << 32) | (uint32_t)x | (dbl ? 0x80000000u : 0u);
  }
  return w;
}
__device__ __forceinline__ uint2 as_record(uint64_t kv) { return make_uint2((uint32_t)(kv >> 32), (uint32_t)kv); }

// A vertex in general: more than kAdjRow corners, or a surface around it
// that is not a closed fan.  Returns its normal sum; its records to kv.
__device__ __noinline__ float3 finish_general(const float* __restrict__ V, const uint32_t* __restrict__ T, int64_t v,
                                              uint32_t n, const uint32_t* __restrict__ adj,
                                              const uint32_t* __restrict__ adj_more, float3 pa, uint64_t* kv,
                                              uint32_t* records) {
  uint32_t key[kAdjMax];
  for (uint32_t i = 0; i < n; i++) {
    const uint32_t c = i < kAdjRow ? adj[(size_t)kAdjRow * v + i]
                                   : adj_more[(size_t)(kAdjMax - kAdjRow) * v + i - kAdjRow];
    uint32_t j = i;
    while (j > 0 && key[j - 1] > c) { key[j] = key[j - 1]; j--; }
    key[j] = c;
  }
  float3 acc = make_float3(0.f, 0.f, 0.f);
  uint32_t m = 0;
  for (uint32_t i = 0; i < n; i++) {
    float3 nn;
    uint32_t id[2];
    adj_corner(V, T, key[i], nn, id[0], id[1]);
    acc = add3(acc, nn);
    for (int h = 0; h < 2; h++) {
      const uint64_t x = ((uint64_t)id[h] << 32) | __float_as_uint(dist2(pa, ld3(V, id[h])));
      uint32_t j = m++;
      while (j > 0 && kv[j - 1] > x) { kv[j] = kv[j - 1]; j--; }
      kv[j] = x;
    }
  }
  *records = merge_pairs(kv, m);
  return acc;
}

// The same by a warp whose lanes hold the corners (all lanes call it; n at
// most kAdjMax): ranks instead of sorts, so that a vertex costs its three
// dependent loads and a few hundred instructions, not a chain of them: nearly
// every chunk has one (0.3 % of a solid's vertices have more than eight
// corners) and waited for it, 27 -> 18.5 us at 97k vertices, 0.471 -> 0.416 ms
// at 5.7M.
__device__ __noinline__ float3 finish_by_warp(const float* __restrict__ V, const uint32_t* __restrict__ T, uint32_t v,
                                              uint32_t n, const uint32_t* __restrict__ adj,
                                              const uint32_t* __restrict__ adj_more, bool records_wanted, uint64_t* kv,
                                              uint32_t* records) {
  const uint32_t lane = threadIdx.x & 31;
  const bool has = lane < n;
  uint32_t key = 0xffffffffu, id[2] = {0xffffffffu, 0xffffffffu}, rank = 0;
  float3 nn = make_float3(0.f, 0.f, 0.f), acc = nn;
  if (has) {
    key = lane < kAdjRow ? adj[(size_t)kAdjRow * v + lane]
                         : adj_more[(size_t)(kAdjMax - kAdjRow) * v + lane - kAdjRow];
    adj_corner(V, T, key, nn, id[0], id[1]);
  }
  for (uint32_t j = 0; j < n; j++) rank += __shfl_sync(0xffffffffu, key, j) < key;
  for (uint32_t j = 0; j < n; j++) {
    const int src = __ffs(__ballot_sync(0xffffffffu, has && rank == j)) - 1;
    acc = add3(acc, make_float3(__shfl_sync(0xffffffffu, nn.x, src), __shfl_sync(0xffffffffu, nn.y, src),
                                __shfl_sync(0xffffffffu, nn.z, src)));
  }
  *records = 0;
  if (!records_wanted) return acc;
  // a neighbour's occurrences have one term, so they differ by their place
  // (2 lane + h) only: every second one is kept, as a double if it has a next
  uint32_t less[2] = {0, 0}, run[2] = {0, 0}, all[2] = {0, 0};
  for (uint32_t j = 0; j < n; j++) {
    const uint32_t a = __shfl_sync(0xffffffffu, id[0], j), b = __shfl_sync(0xffffffffu, id[1], j);
#pragma unroll
    for (int h = 0; h < 2; h++) {
      less[h] += (a < id[h]) + (b < id[h]);
      all[h] += (a == id[h]) + (b == id[h]);
      run[h] += (a == id[h] && (h == 0 ? j < lane : j <= lane)) + (b == id[h] && j < lane);
    }
  }
  uint32_t lo = 0, hi = 0;
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const uint32_t at = less[h] + run[h];  // its place in (neighbour, occurrence) order
    if (has && !(run[h] & 1)) (at < 32 ? lo : hi) |= 1u << (at & 31);
  }
  lo = __reduce_or_sync(0xffffffffu, lo);
  hi = __reduce_or_sync(0xffffffffu, hi);
  const float3 pa = ld3(V, v);
#pragma unroll
  for (int h = 0; h < 2; h++) {
    const uint32_t at = less[h] + run[h];
    if (has && !(run[h] & 1)) {
      const uint32_t place = __popc(lo & (at < 32 ? (1u << at) - 1u : 0xffffffffu)) +
                             (at < 32 ? 0 : __popc(hi & ((1u << (at - 32)) - 1u)));
      kv[place] = ((uint64_t)id[h] << 32) | __float_as_uint(dist2(pa, ld3(V, id[h]))) |
                  (run[h] + 1 < all[h] ? 0x80000000u : 0u);
    }
  }
  *records = __popc(lo) + __popc(hi);
  __syncwarp();
  return acc;
}

// The per-vertex steps after the corner rows are filled, in one kernel: the
// row sorted into triangle order; the area-weighted normal summed in that
// order and normalised (GMorpho.cu:6498-6537); and, when the normals are
// filtered (rec), the filter records.
//
// Around a vertex whose triangles form closed fans, every neighbour follows
// it in one incident triangle and precedes it in another: the sorted lists
// of both are equal, and each entry is a neighbour shared by two triangles.
// Two networks over eight 32-bit values and a comparison thus replace the
// sort of sixteen 64-bit pairs, and the records go straight to their packed
// place: with the corner rows' single pass, 4.4M vertices' lists and records
// went from 1.27 ms (count, scan, fill, finish, scan, pack) to 0.6.
__global__ void __launch_bounds__(kRecChunk, 4) k_adj_finish(const float* __restrict__ V, const uint32_t* __restrict__ T,
                             const uint32_t* __restrict__ cursor, const uint32_t* __restrict__ adj,
                             const uint32_t* __restrict__ adj_more, int64_t nv,
                             int zero_isolated, float4* __restrict__ N4, float* __restrict__ N3,
                             uint2* __restrict__ rec, uint32_t* __restrict__ roff, uint32_t* __restrict__ counters) {
  __shared__ uint32_t base_s;
  __shared__ uint64_t pool[kRecChunk / 32][kPool][2 * kAdjMax];  // records of a warp's general vertices
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int64_t v = blockIdx.x * (int64_t)kRecChunk + threadIdx.x;
  const uint32_t n = v < nv ? cursor[v] : 0u;
  const bool isolated = n == 0 && (zero_isolated || v >= nv);
  const bool here = !isolated && n <= kAdjMax;  // (more: vertex 0, k_row0_finish)
  float3 acc = make_float3(0.f, 0.f, 0.f);
  uint32_t p[8], t[8], records = 0;
  uint64_t kv[2 * kAdjMax];
  bool fan = here && n <= kAdjRow;
  if (fan) {
    uint32_t key[8], q[8];
    const uint4* row = reinterpret_cast<const uint4*>(adj + (size_t)kAdjRow * v);
    const uint4 r0 = row[0], r1 = row[1];
    key[0] = r0.x, key[1] = r0.y, key[2] = r0.z, key[3] = r0.w;
    key[4] = r1.x, key[5] = r1.y, key[6] = r1.z, key[7] = r1.w;
#pragma unroll
    for (int k = 0; k < 8; k++) key[k] = (uint32_t)k < n ? key[k] : 0xffffffffu;
    bitonic_sort<8>(key);
#pragma unroll
    for (int k = 0; k < 8; k++) {
      p[k] = q[k] = 0xffffffffu;
      if ((uint32_t)k < n) {
        float3 nn;
        adj_corner(V, T, key[k], nn, p[k], q[k]);
        acc = add3(acc, nn);
      }
    }
    if (rec) {
      bitonic_sort<8>(p);
      bitonic_sort<8>(q);
#pragma unroll
      for (int k = 0; k < 8; k++) fan = fan && p[k] == q[k];
      if (fan) {
        const float3 pa = ld3(V, (uint32_t)v);
        records = n;
#pragma unroll
        for (int k = 0; k < 8; k++)
          if ((uint32_t)k < n) t[k] = __float_as_uint(dist2(pa, ld3(V, p[k]))) | 0x80000000u;
      }
    }
  }
  int slot = -1, used = 0;
  for (uint32_t todo = __ballot_sync(0xffffffffu, here && !fan); todo && used < kPool; used++) {
    const int src = __ffs(todo) - 1;
    todo &= todo - 1;
    uint32_t count;
    const float3 sum = finish_by_warp(V, T, (uint32_t)(v - lane + src), __shfl_sync(0xffffffffu, n, src), adj, adj_more,
                                      rec != nullptr, pool[wid][used], &count);
    if (lane == src) acc = sum, records = count, slot = used;
  }
  if (here && !fan && slot < 0) acc = finish_general(V, T, v, n, adj, adj_more, ld3(V, (uint32_t)v), kv, &records);
  if (rec) {
    uint32_t total;
    const uint32_t pre = block_scan1(records, total);
    if (threadIdx.x == 0) base_s = atomicAdd(counters + kCntRecords, total);
    __syncthreads();
    const uint32_t at = base_s + pre;
    if (v < nv && n <= kAdjMax) {
      roff[roff_at((uint32_t)v)] = at;
      if (v == 0 || threadIdx.x == kRecChunk - 1 || v == nv - 1) roff[roff_at((uint32_t)v) + 1] = at + records;
    }
    if (fan) {
#pragma unroll
      for (int k = 0; k < 8; k++)
        if ((uint32_t)k < records) rec[at + k] = make_uint2(p[k], t[k]);
    } else if (slot < 0) {
      for (uint32_t i = 0; i < records; i++) rec[at + i] = as_record(kv[i]);
    }
    for (int u = 0; u < used; u++) {
      const int src = __ffs(__ballot_sync(0xffffffffu, slot == u)) - 1;
      const uint32_t to = __shfl_sync(0xffffffffu, at, src), count = __shfl_sync(0xffffffffu, records, src);
      for (uint32_t i = lane; i < count; i += 32) rec[to + i] = as_record(pool[wid][u][i]);
    }
  }
  if (v >= nv || !(here || isolated)) return;
  float3 nn = make_float3(0.f, 0.f, 0.f);
  if (here) nn = normalize3(acc);
  N4[v] = make_float4(nn.x, nn.y, nn.z, 0.f);
  if (N3) { N3[3 * v] = nn.x; N3[3 * v + 1] = nn.y; N3[3 * v + 2] = nn.z; }
}

// Ascending sort of n values in global memory by one block (a bitonic
// network whose exchanges all put the smaller value first, so that the
// places past n need no padding).
template <typename K>
__device__ void block_sort(K* k, uint32_t n) {
  for (uint32_t s = 2; s / 2 < n; s <<= 1) {
    for (uint32_t j = s >> 1; j > 0; j >>= 1) {
      for (uint32_t t = threadIdx.x; t < n; t += blockDim.x) {
        // the first step of a merge mirrors the second half
        const uint32_t l = j == s >> 1 ? (t & ~(s - 1)) + (s - 1 - (t & (s - 1))) : t ^ j;
        if (l > t && l < n) {
          const K a = k[t], b = k[l];
          if (b < a) k[t] = b, k[l] = a;
        }
      }
      __syncthreads();
    }
  }
}

// Vertex 0 with more than kAdjMax corners (else nothing to do): the steps of
// k_adj_finish by one block, the terms in parallel and their sum in corner
// order by one thread.  Its pairs and then its records lie at the end of the
// records' buffer (the other vertices' fill it from the front; together they
// are at most two a corner).
__global__ void __launch_bounds__(1024) k_row0_finish(const float* __restrict__ V, const uint32_t* __restrict__ T,
                                                      const uint32_t* __restrict__ cursor, uint32_t* __restrict__ row0,
                                                      int64_t nt, float4* __restrict__ N4, float* __restrict__ N3,
                                                      uint2* __restrict__ rec, uint32_t* __restrict__ roff) {
  const uint32_t n = cursor[0];
  if (n <= kAdjMax) return;
  __shared__ float3 term[1024];
  block_sort(row0, n);
  const uint32_t start = (uint32_t)(6 * nt - 2 * (int64_t)n);
  uint64_t* kv = reinterpret_cast<uint64_t*>(rec + start);  // (8 bytes a record, 8 bytes a pair)
  const float3 pa = ld3(V, 0u);
  float3 acc = make_float3(0.f, 0.f, 0.f);
  for (uint32_t c0 = 0; c0 < n; c0 += blockDim.x) {
    const uint32_t c = c0 + threadIdx.x;
    if (c < n) {
      uint32_t id[2];
      adj_corner(V, T, row0[c], term[threadIdx.x], id[0], id[1]);
      if (rec)
        for (int h = 0; h < 2; h++)
          kv[2 * (size_t)c + h] = ((uint64_t)id[h] << 32) | __float_as_uint(dist2(pa, ld3(V, id[h])));
    }
    __syncthreads();
    if (threadIdx.x == 0)
      for (uint32_t i = 0; i < blockDim.x && c0 + i < n; i++) acc = add3(acc, term[i]);
    __syncthreads();
  }
  if (rec) block_sort(kv, 2 * n);
  if (threadIdx.x != 0) return;
  if (rec) {
    const uint32_t w = merge_pairs(kv, 2 * n);
    for (uint32_t i = 0; i < w; i++) kv[i] = (kv[i] << 32) | (kv[i] >> 32);  // a record's word order
    roff[0] = start;
    roff[1] = start + w;
  }
  const float3 nn = normalize3(acc);
  N4[0] = make_float4(nn.x, nn.y, nn.z, 0.f);
  if (N3) { N3[0] = nn.x; N3[1] = nn.y; N3[2] = nn.z; }
}

// One bilateral normal iteration (BilateralMeshFiltering{,Normalize},
// GMorpho.cu:6539-6620): each incident triangle adds w1 n_b + w2 n_c.  A
// neighbour shared by two incident triangles appears twice in that sum with
// the same weight and is read once.  The sum runs over the neighbours in
// vertex order (deterministic).
// one neighbour's term, added to acc
__device__ __forceinline__ void bilateral_add(float3& acc, uint2 e, float4 nb, float4 na, float sn2) {
  // the reference library is built with -use_fast_math (GMorpho/cuda.prf:47),
  // so its exp and division here are the fast forms.  Where neighbours nearly
  // cancel, one rounding decides a normal's third digit: the sums are not
  // fused and the division is not a product.
  float w = __expf(-__fadd_rn(__uint_as_float(e.y & 0x7fffffffu), __fdividef(dist2n(na, nb), sn2)));
  if (e.y >> 31) w = __fadd_rn(w, w);
  acc.x = __fadd_rn(acc.x, __fmul_rn(w, nb.x));
  acc.y = __fadd_rn(acc.y, __fmul_rn(w, nb.y));
  acc.z = __fadd_rn(acc.z, __fmul_rn(w, nb.z));
}

// The records two at a time, the next two loaded one step ahead, so that
// two neighbour-normal gathers are in flight per thread; the terms are
// added in record order (the same sum, bit for bit, as one at a time).
__device__ __forceinline__ float3 bilateral_sum(const float4* __restrict__ Nin, const uint2* __restrict__ rec,
                                                uint32_t n, float4 na, float sn2) {
  float3 acc = make_float3(0.f, 0.f, 0.f);
  const uint2 z2 = make_uint2(0u, 0u);
  uint2 f0 = n > 0 ? rec[0] : z2, f1 = n > 1 ? rec[1] : z2;  // the next pair
  uint32_t i = 0;
  for (; i + 1 < n; i += 2) {
    const uint2 e0 = f0, e1 = f1;
    if (i + 2 < n) f0 = rec[i + 2];
    if (i + 3 < n) f1 = rec[i + 3];
    const float4 nb0 = Nin[e0.x], nb1 = Nin[e1.x];
    bilateral_add(acc, e0, nb0, na, sn2);
    bilateral_add(acc, e1, nb1, na, sn2);
  }
  if (i < n) bilateral_add(acc, f0, Nin[f0.x], na, sn2);
  return acc;
}

// one vertex of an iteration
__device__ __forceinline__ void bilateral_vertex(const float4* __restrict__ Nin, const uint2* __restrict__ rec,
                                                 const uint32_t* __restrict__ roff, uint32_t v, float sn2,
                                                 int zero_isolated, float4* __restrict__ Nout,
                                                 float* __restrict__ N3) {
  const uint32_t at = roff_at(v), r0 = roff[at], n = roff[at + 1] - r0;
  float3 nn = make_float3(0.f, 0.f, 0.f);
  if (!(zero_isolated && n == 0)) nn = normalize3(bilateral_sum(Nin, rec + r0, n, Nin[v], sn2));
  Nout[v] = make_float4(nn.x, nn.y, nn.z, 0.f);
  if (N3) {
    float* o = N3 + 3 * (size_t)v;
    o[0] = nn.x; o[1] = nn.y; o[2] = nn.z;
  }
}

// (the 32 registers that keep eight blocks on an SM decide the time: 99 us for
// 4.4M vertices; 115 to 118 at 44, spilled or not)
__global__ void k_bilateral(const float4* __restrict__ Nin, const uint2* __restrict__ rec,
                            const uint32_t* __restrict__ roff, uint32_t nv,
                            float sn2, int zero_isolated, float4* __restrict__ Nout, float* __restrict__ N3) {
  for (uint32_t v = blockIdx.x * blockDim.x + threadIdx.x; v < nv; v += gridDim.x * blockDim.x)
    bilateral_vertex(Nin, rec, roff, v, sn2, zero_isolated, Nout, N3);
}

// All iterations in one cooperative launch, for meshes whose vertices all fit
// on the chip as threads: a thread keeps its vertex' first kResGathers records
// in shared memory, and an iteration is one round of gathers (97 % of the
// vertices have no more), the same sum in the same order, a store and a
// barrier over the grid.  A launch per iteration took 7.5 us at 97k vertices,
// most of it launch, ramp and dependent loads; this takes 4.4, half of it the
// barrier's round trips (as much with 379 blocks in place of one an SM, and
// with gathers past L1).
//
// The barrier counts arrivals and never resets within a launch (the caller
// zeroes the counter before it).  The acquire of the count and the block
// barrier after it order the other blocks' normals before the plain loads of
// the next iteration.  The blocks are resident together, so the wait ends, and
// it gives up after `polls` polls all the same: an error bit, a word that the
// host reads after it has waited for the kernel (gave_up), and NaN normals for
// the block's vertices.  (missing: arrivals that never come, for tests.)
constexpr int kResGathers = 8;
constexpr int kResThreads = 1024;  // at most; one block per SM, so that few arrive
constexpr uint32_t kResPolls = 1u << 24, kResPollsStalled = 1u << 12;

__global__ void __launch_bounds__(kResThreads) k_bilateral_resident(float4* Na, float4* Nb,
                                                                    const uint2* __restrict__ rec,
                                                                    const uint32_t* __restrict__ roff, uint32_t nv,
                                                                    int iters, int zero_isolated, uint32_t* arrived,
                                                                    uint32_t missing, uint32_t polls,
                                                                    float* __restrict__ N3, unsigned int* errors,
                                                                    uint32_t* gave_up) {
  extern __shared__ uint32_t mine_s[];  // [2 kResGathers][threads]: the first records' neighbours, then terms
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x, pitch = blockDim.x;
  uint32_t* mine = mine_s + threadIdx.x;
  uint32_t n = 0, r0 = 0;
  float4 na = make_float4(0.f, 0.f, 0.f, 0.f);
  if (v < nv) {
    const uint32_t at = roff_at(v);
    r0 = roff[at], n = roff[at + 1] - r0;
    na = Na[v];
    for (uint32_t k = 0; k < kResGathers && k < n; k++) {
      const uint2 e = rec[r0 + k];
      mine[k * pitch] = e.x;
      mine[(kResGathers + k) * pitch] = e.y;
    }
  }
  for (int it = 0; it < iters; it++) {
    const float sn = it < 2 ? 1e10f : 0.2f, sn2 = sn * sn;  // GMorpho.cu:6959-6969
    const float4* Nin = (it & 1) ? Nb : Na;
    float4* Nout = (it & 1) ? Na : Nb;
    if (v < nv) {
      float3 nn = make_float3(0.f, 0.f, 0.f);
      if (!(zero_isolated && n == 0)) {
        float3 acc = make_float3(0.f, 0.f, 0.f);
        float4 nb[kResGathers];
#pragma unroll
        for (int k = 0; k < kResGathers; k++)
          if (k < n) nb[k] = Nin[mine[k * pitch]];
#pragma unroll
        for (int k = 0; k < kResGathers; k++)
          if (k < n) bilateral_add(acc, make_uint2(0u, mine[(kResGathers + k) * pitch]), nb[k], na, sn2);
        for (uint32_t i = kResGathers; i < n; i++) {
          const uint2 e = rec[r0 + i];
          bilateral_add(acc, e, Nin[e.x], na, sn2);
        }
        nn = normalize3(acc);
      }
      na = make_float4(nn.x, nn.y, nn.z, 0.f);
      if (it == iters - 1) {
        float* o = N3 + 3 * (size_t)v;
        o[0] = nn.x; o[1] = nn.y; o[2] = nn.z;
      } else {
        __stcg(Nout + v, na);
      }
    }
    if (it == iters - 1) return;
    __syncthreads();
    int ok = 1;
    if (threadIdx.x == 0) {
      const uint32_t want = (uint32_t)(it + 1) * gridDim.x + missing;
      __threadfence();  // the block's normals before its arrival
      atomicAdd(arrived, 1u);
      uint32_t seen, left = polls;
      do {
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(arrived) : "memory");
      } while (seen < want && --left);
      if (seen < want) {
        ok = 0;
        atomicOr(errors, 1u);
        if (gave_up) *reinterpret_cast<volatile uint32_t*>(gave_up) = 1u;
      }
    }
    if (!__syncthreads_and(ok)) {
      if (v < nv) {
        float* o = N3 + 3 * (size_t)v;
        o[0] = o[1] = o[2] = __int_as_float(0x7fffffff);
      }
      return;
    }
  }
}

// The same iteration over the vertices of several meshes at once (one
// launch per iteration for a batch): a block takes 256 vertices of one mesh,
// chunk g of the concatenation belonging to the mesh m with start[m] <= g <
// start[m + 1], so that a mesh's pointers are the block's and 32 registers
// suffice (48 with a search per vertex; 72 -> 66 us for 16 meshes of 32^3 to
// 256^3 cells).
struct BilMesh {
  const float4* Na;       // normals of even iterations' inputs (N4a)
  float4* Nb;             // and odd (N4b)
  const uint2* rec;
  const uint32_t* roff;
  float* N3;              // final normals (last iteration)
  uint32_t nv;
  int zero_isolated;
};

__global__ void __launch_bounds__(256, 8) k_bilateral_group(const BilMesh* __restrict__ meshes,
                                                            const int64_t* __restrict__ start, int n, int odd,
                                                            int last, float sn2) {
  const int64_t chunks = start[n];
  for (int64_t g = blockIdx.x; g < chunks; g += gridDim.x) {
    int lo = 0, hi = n - 1;  // last m with start[m] <= g
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (start[mid] <= g) lo = mid; else hi = mid - 1;
    }
    const BilMesh& M = meshes[lo];
    const uint32_t v = (uint32_t)(g - start[lo]) * 256u + threadIdx.x;
    const float4* Nin = odd ? M.Nb : M.Na;
    float4* Nout = odd ? const_cast<float4*>(M.Na) : M.Nb;
    if (v < M.nv) bilateral_vertex(Nin, M.rec, M.roff, v, sn2, M.zero_isolated, Nout, last ? M.N3 : nullptr);
  }
}

// ------------------------------------------------------------------ host

static int gs_blocks(int64_t n, int threads, int sms) {
  int64_t b = (n + threads - 1) / threads;
  const int64_t cap = (int64_t)(sms > 0 ? sms : 152) * 16;
  if (b > cap) b = cap;
  return (int)(b < 1 ? 1 : b);
}

// Grid of a grid-stride kernel as one wave of resident blocks (SMs x the
// blocks of 256 threads one SM holds at once), at most one block per 256
// items: the filter iterations measured 8% faster so than with two waves.
static int wave_blocks(const void* kernel, int64_t n, int sms) {
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, 256, 0) != cudaSuccess || per_sm < 1) {
    cudaGetLastError();
    per_sm = 1;
  }
  int64_t b = (int64_t)(sms > 0 ? sms : 152) * per_sm;
  const int64_t need = (n + 255) / 256;
  if (b > need) b = need;
  return (int)(b < 1 ? 1 : b);
}

void MeshBuffers::release() {
  cudaFree(V); cudaFree(N); cudaFree(N4a); cudaFree(N4b); cudaFree(T); cudaFree(adj); cudaFree(row0);
  cudaFree(rec); cudaFree(roff); cudaFree(cursor); cudaFree(cells); cudaFree(brick_tot);
  cudaFree(brick_mask); cudaFree(entries);
  cudaFree(fix);
  *this = MeshBuffers();
}

// Bricks are visited in Morton order over the smallest power-of-two cube of
// bricks covering the grid; bricks outside the grid or the tag box return
// at once.
static int brick_count(const int d[3]) {
  const int m = d[0] > d[1] ? (d[0] > d[2] ? d[0] : d[2]) : (d[1] > d[2] ? d[1] : d[2]);
  int p = kBrick;
  while (p < m) p *= 2;
  const int e = p / kBrick;
  return e * e * e;
}

static void grid_dims(const MeshArgs& a, int d[3]) {
  for (int k = 0; k < 3; k++) d[k] = a.dims[0] > 0 ? a.dims[k] : a.res;
}

static McWin window_of(const MeshArgs& a) {
  McWin w;
  int d[3];
  grid_dims(a, d);
  const bool crop = a.gres > 0;
  for (int k = 0; k < 3; k++) {
    w.gdim[k] = crop ? a.gres : d[k];
    w.off[k] = crop ? a.off[k] : 0;
    w.tlo[k] = crop ? a.tag_lo[k] : 0;
    w.thi[k] = crop ? a.tag_hi[k] : d[k];
    w.elo[k] = crop ? a.emit_lo[k] : 0;
    w.ehi[k] = crop ? a.emit_hi[k] : d[k];
  }
  return w;
}

// capacity helpers: buffers grow (never shrink) to the sizes asked for
static cudaError_t ensure_grid_buffers(MeshBuffers& b, int64_t cells, int nb) {
  cudaError_t e;
  if (nb + 1 > b.bricks_cap || cells > b.cells_cap) b.grid_moves++;
  if (nb + 1 > b.bricks_cap) {
    cudaFree(b.brick_tot);
    cudaFree(b.brick_mask);
    b.brick_tot = b.brick_mask = nullptr;
    b.bricks_cap = 0;
    if ((e = cudaMalloc(&b.brick_mask, sizeof(uint32_t) * kMaskWords * (size_t)nb)) != cudaSuccess) return e;
    // counters and totals (nb + 1), then the chunk sums of the scan
    e = cudaMalloc(&b.brick_tot, sizeof(uint32_t) * 4 * ((size_t)nb + 1 + (nb + kBrickChunk - 1) / kBrickChunk));
    if (e != cudaSuccess) return e;
    b.bricks_cap = nb + 1;
  }
  if (cells > b.cells_cap) {
    cudaFree(b.cells);
    b.cells = nullptr;
    b.cells_cap = 0;
    e = cudaMalloc(&b.cells, sizeof(uint2) * (size_t)cells);
    if (e != cudaSuccess) return e;
    b.cells_cap = cells;
  }
  return cudaSuccess;
}

static cudaError_t ensure_vertex_buffers(MeshBuffers& b, int64_t nv) {
  cudaError_t e;
  if (b.v_cap < nv || b.V == nullptr) {
    cudaFree(b.V); cudaFree(b.N); cudaFree(b.N4a); cudaFree(b.N4b); cudaFree(b.cursor);
    cudaFree(b.adj); cudaFree(b.roff);
    b.V = b.N = nullptr;
    b.N4a = b.N4b = nullptr;
    b.cursor = b.adj = b.roff = nullptr;
    b.v_cap = 0;
    const int64_t c = nv + nv / 4 + 1024;
    if ((e = cudaMalloc(&b.V, sizeof(float) * 3 * (size_t)c)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&b.N, sizeof(float) * 3 * (size_t)c)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&b.N4a, sizeof(float4) * (size_t)c)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&b.N4b, sizeof(float4) * (size_t)c)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&b.cursor, sizeof(uint32_t) * ((size_t)c + kCntWords))) != cudaSuccess) return e;
    if ((e = cudaMalloc(&b.adj, sizeof(uint32_t) * kAdjMax * (size_t)c)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&b.roff, sizeof(uint32_t) * ((size_t)c + (size_t)c / kRecChunk + 4))) != cudaSuccess) return e;
    b.v_cap = c;
  }
  return cudaSuccess;
}

static cudaError_t ensure_triangle_buffers(MeshBuffers& b, int64_t nt) {
  cudaError_t e;
  if (b.t_cap < nt || b.T == nullptr) {
    cudaFree(b.T); cudaFree(b.row0); cudaFree(b.rec);
    b.T = b.row0 = nullptr;
    b.rec = nullptr;
    b.t_cap = 0;
    const int64_t c = nt + nt / 4 + 1024;
    if ((e = cudaMalloc(&b.T, sizeof(uint32_t) * 3 * (size_t)c)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&b.row0, sizeof(uint32_t) * 3 * (size_t)c)) != cudaSuccess) return e;
    if ((e = cudaMalloc(&b.rec, sizeof(uint2) * 6 * (size_t)c)) != cudaSuccess) return e;
    b.t_cap = c;
  }
  return cudaSuccess;
}

static cudaError_t ensure_entries(MeshBuffers& b, int64_t n) {
  if (b.entries_cap >= n && b.entries != nullptr) return cudaSuccess;
  cudaFree(b.entries);
  b.entries = nullptr;
  b.entries_cap = 0;
  const int64_t c = n + n / 4 + 1024;
  const cudaError_t e = cudaMalloc(&b.entries, sizeof(uint4) * (size_t)c);
  if (e == cudaSuccess) b.entries_cap = c;
  return e;
}

cudaError_t mesh_reserve(MeshBuffers& b, int res, int64_t nv, int64_t nt) {
  const int d[3] = {res, res, res};
  cudaError_t e = ensure_grid_buffers(b, (int64_t)res * res * res, brick_count(d));
  if (e == cudaSuccess) e = ensure_vertex_buffers(b, nv);
  if (e == cudaSuccess) e = ensure_triangle_buffers(b, nt);
  if (e == cudaSuccess) e = ensure_entries(b, nv + nv / 2);
  return e;
}

cudaError_t mesh_count_launch(const MeshArgs& a, MeshBuffers& b, cudaStream_t st, KernelCounter* kc,
                              uint32_t* h_tot4) {
  int d[3];
  grid_dims(a, d);
  const GDims gd{d[0], d[1], d[2]};
  const int64_t cells = (int64_t)d[0] * d[1] * d[2];
  const int nb = brick_count(d);
  cudaError_t e = ensure_grid_buffers(b, cells, nb);
  if (e != cudaSuccess) return e;
  GM_LAUNCH(kc, "k_mc_count", st, k_mc_count<<<nb, kMcThreads, 0, st>>>(a.C, gd, window_of(a), b.brick_tot,
                                                                          b.brick_mask, b.cells));
  {
    const int nchunks = (nb + kBrickChunk - 1) / kBrickChunk;
    if (nchunks > kBrickChunk) return cudaErrorInvalidValue;
    if (nchunks > 1)  // (one chunk's scan reads no sums)
      GM_LAUNCH(kc, "k_brick_sums", st, k_brick_sums<<<nchunks, kBrickChunk, 0, st>>>(b.brick_tot, nb));
    GM_LAUNCH(kc, "k_scan_bricks", st, k_scan_bricks<<<nchunks, kBrickChunk, 0, st>>>(b.brick_tot, nb));
  }
  return cudaMemcpyAsync(h_tot4, b.brick_tot + 4 * (size_t)nb, 4 * sizeof(uint32_t), cudaMemcpyDeviceToHost, st);
}

cudaError_t mesh_prepare_grid(const MeshArgs& a, MeshBuffers& b) {
  int d[3];
  grid_dims(a, d);
  return ensure_grid_buffers(b, (int64_t)d[0] * d[1] * d[2], brick_count(d));
}

cudaError_t mesh_count_finish(MeshBuffers& b, const uint32_t* tot, int64_t* nv, int64_t* nt) {
  b.n_cells = tot[0];
  *nv = tot[1];
  *nt = tot[2];
  const int need_fix = b.n_fix = (int)tot[3];
  if (need_fix + 1 > b.fix_cap || b.fix == nullptr) {
    if (b.fix) cudaFree(b.fix);
    b.fix = nullptr;
    const int c = need_fix + 64;
    cudaError_t e = cudaMalloc(&b.fix, sizeof(uint32_t) * (1 + 4 * (size_t)c));
    if (e != cudaSuccess) return e;
    b.fix_cap = c;
  }
  return cudaSuccess;
}

cudaError_t mesh_count(const MeshArgs& a, MeshBuffers& b, cudaStream_t st, KernelCounter* kc, int64_t* nv,
                       int64_t* nt) {
  uint32_t tot[4];
  cudaError_t e = mesh_count_launch(a, b, st, kc, tot);
  if (e != cudaSuccess) return e;
  e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) return e;
  e = mesh_count_finish(b, tot, nv, nt);
  if (e != cudaSuccess) return e;
  return cudaGetLastError();
}

cudaError_t mesh_emit(const MeshArgs& a, MeshBuffers& b, int64_t nv, int64_t nt, cudaStream_t st,
                      KernelCounter* kc) {
  int d[3];
  grid_dims(a, d);
  const GDims gd{d[0], d[1], d[2]};
  const int nb = brick_count(d);
  const McWin w = window_of(a);
  cudaError_t e;
  // per-vertex buffers share one capacity, per-triangle buffers another
  if ((e = ensure_vertex_buffers(b, nv)) != cudaSuccess) return e;
  if ((e = ensure_triangle_buffers(b, nt)) != cudaSuccess) return e;
  const float cs = 0.5f * a.cell_size;  // exact: scaling by a power of two
  if (b.n_fix > 0) cudaMemsetAsync(b.fix, 0, sizeof(uint32_t), st);
  if ((e = ensure_entries(b, b.n_cells)) != cudaSuccess) return e;
  GM_LAUNCH(kc, "k_mc_vertices", st,
            k_mc_vertices<<<nb, kMcThreads, 0, st>>>(gd, w, b.brick_tot, b.brick_mask, b.cells, b.entries, b.V,
                                                     a.bbox_min[0], a.bbox_min[1], a.bbox_min[2], cs, a.isovalue));
  if (b.n_cells > 0)
    GM_LAUNCH(kc, "k_mc_triangles", st,
              k_mc_triangles<<<gs_blocks(8 * b.n_cells, kMcThreads, a.num_sms), kMcThreads, 0, st>>>(
                  gd, w, b.cells, b.entries, (uint32_t)b.n_cells, b.T, (uint32_t)nt, b.fix, b.fix_cap));
  if (b.n_fix > 0) GM_LAUNCH(kc, "k_mc_fix91", st, k_mc_fix91<<<1, 256, 0, st>>>(b.fix, b.fix_cap, b.T));
  if (a.geometry_done) cudaEventRecord(a.geometry_done, st);
  if (nv == 0 || nt == 0) return cudaGetLastError();
  // normals
  const int sms = a.num_sms;
  uint32_t* adj_more = b.adj + (size_t)kAdjRow * b.v_cap;
  uint32_t* counters = b.cursor + nv;
  const int iters = a.bilateral_iters;
  const int zi = a.zero_isolated;
  uint2* rec = iters > 0 ? b.rec : nullptr;
  float* n3 = iters == 0 ? b.N : nullptr;
  cudaMemsetAsync(b.cursor, 0, sizeof(uint32_t) * (size_t)(nv + kCntWords), st);
  GM_LAUNCH(kc, "k_adj_slots", st,
            k_adj_slots<<<gs_blocks(3 * nt, 256, sms), 256, 0, st>>>(b.T, nt, b.cursor, b.adj, adj_more, b.row0));
  GM_LAUNCH(kc, "k_adj_finish", st,
            k_adj_finish<<<(unsigned)((nv + kRecChunk - 1) / kRecChunk), kRecChunk, 0, st>>>(
                b.V, b.T, b.cursor, b.adj, adj_more, nv, zi, b.N4a, n3, rec, b.roff, counters));
  GM_LAUNCH(kc, "k_row0_finish", st,
            k_row0_finish<<<1, 1024, 0, st>>>(b.V, b.T, b.cursor, b.row0, nt, b.N4a, n3, rec, b.roff));
  if (a.defer_filter) return cudaGetLastError();
  float4* nin = b.N4a;
  float4* nout = b.N4b;
  const int64_t share = nv / (sms > 0 ? sms : 152) / 32 * 32 + 32;  // vertices of an SM, whole warps
  const int res_threads = (int)(share < 128 ? 128 : share);
  if (iters > 1 && res_threads <= kResThreads) {
    uint32_t nv32 = (uint32_t)nv, *arrived = counters + kCntArrived;
    uint32_t missing = a.stall_filter ? 1u : 0u, polls = a.stall_filter ? kResPollsStalled : kResPolls;
    uint32_t* gave_up = a.gave_up;
    unsigned int* errors = kernel_error_word();
    void* args[] = {&b.N4a, &b.N4b, &b.rec, &b.roff, &nv32, const_cast<int*>(&iters), const_cast<int*>(&zi),
                    &arrived, &missing, &polls, &b.N, &errors, &gave_up};
    const size_t res_smem = 2 * kResGathers * sizeof(uint32_t) * (size_t)res_threads;
    cudaError_t le = ensure_dynamic_smem(reinterpret_cast<const void*>(k_bilateral_resident), res_smem);
    if (le != cudaSuccess) return le;
    GM_LAUNCH(kc, "k_bilateral", st,
              le = cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_bilateral_resident),
                                               dim3((unsigned)((nv + res_threads - 1) / res_threads)),
                                               dim3((unsigned)res_threads), args, res_smem, st));
    if (le == cudaSuccess) return cudaGetLastError();
    if (le != cudaErrorCooperativeLaunchTooLarge) return le;
    cudaGetLastError();  // fewer SMs than the device has: an iteration per launch
  }
  const int bil_blocks = wave_blocks(reinterpret_cast<const void*>(k_bilateral), nv, sms);
  for (int it = 0; it < iters; it++) {
    const float sn = it < 2 ? 1e10f : 0.2f;  // GMorpho.cu:6959-6969
    GM_LAUNCH(kc, "k_bilateral", st,
              k_bilateral<<<bil_blocks, 256, 0, st>>>(nin, b.rec, b.roff, (uint32_t)nv, sn * sn, zi, nout,
                                                      it == iters - 1 ? b.N : nullptr));
    float4* t = nin; nin = nout; nout = t;
  }
  return cudaGetLastError();
}

size_t mesh_filter_table_bytes(int n) {
  return ((sizeof(BilMesh) * (size_t)n + 15) / 16) * 16 + sizeof(int64_t) * ((size_t)n + 1);
}

cudaError_t mesh_filter_group(MeshBuffers* const* meshes, const int64_t* nv, const int* zero_isolated, int n,
                              int iters, void* table, void* h_table, int sms, cudaStream_t st, KernelCounter* kc) {
  if (iters <= 0 || n <= 0) return cudaSuccess;
  BilMesh* hm = static_cast<BilMesh*>(h_table);
  int64_t* hs = reinterpret_cast<int64_t*>(static_cast<uint8_t*>(h_table) + ((sizeof(BilMesh) * (size_t)n + 15) / 16) * 16);
  hs[0] = 0;
  for (int i = 0; i < n; i++) {
    const MeshBuffers& b = *meshes[i];
    hm[i] = BilMesh{b.N4a, b.N4b, b.rec, b.roff, b.N, (uint32_t)nv[i], zero_isolated[i]};
    hs[i + 1] = hs[i] + (nv[i] + 255) / 256;
  }
  const int64_t total = hs[n];
  cudaError_t e = cudaMemcpyAsync(table, h_table, mesh_filter_table_bytes(n), cudaMemcpyHostToDevice, st);
  if (e != cudaSuccess || total == 0) return e;
  const BilMesh* dm = static_cast<const BilMesh*>(table);
  const int64_t* ds = reinterpret_cast<const int64_t*>(static_cast<const uint8_t*>(table) +
                                                       ((sizeof(BilMesh) * (size_t)n + 15) / 16) * 16);
  const int grp_blocks = wave_blocks(reinterpret_cast<const void*>(k_bilateral_group), 256 * total, sms);
  for (int it = 0; it < iters; it++) {
    const float sn = it < 2 ? 1e10f : 0.2f;  // GMorpho.cu:6959-6969
    GM_LAUNCH(kc, "k_bilateral", st,
              k_bilateral_group<<<grp_blocks, 256, 0, st>>>(dm, ds, n, it & 1, it == iters - 1, sn * sn));
  }
  return cudaGetLastError();
}

}  // namespace gm
