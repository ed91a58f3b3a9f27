// framefield.cu — the frame field's biharmonic quaternion system (reference:
// FrameField::Generate with BiHarmonicSystem, GMorpho/FrameField.cu:556-575;
// FrameField::BuildSparseLTLMatrix, BuildSparseSMatrix,
// BuildSparseBiharmonicSystem, SolveSparseBiharmonicSystem,
// GMorpho/FrameFieldSparseBiharmonic.cu:170-647).
//
// System, per quaternion component k (x, y, z, w) on the res^3 lattice:
//   (L^T L + S) q_k = b_k
// L: the degree-normalised 6-neighbour Laplacian, row i = 1 on the diagonal
// and -1/deg(i) on each in-bounds neighbour (the reference builds these
// entries in float: -(1.f / deg) is used here too); S: 1 on the diagonal
// of every hard-constrained node; b_k: the constraint quaternion's
// component at those nodes.
//
// The reference factors L^T L + S with a float sparse Cholesky
// (cusolverSp).  Here the system is solved directly, in double precision,
// up to the float rounding of L's entries, and refined:
//   * with exact entries L = D^-1 G, D the degrees and G the lattice's
//     graph Laplacian, which the cosine transform of each axis (DCT-II)
//     diagonalises: G^+ f = C^T (C f / lambda), lambda the sum of the three
//     axes' eigenvalues 2 - 2 cos(pi k / res);
//   * L^T L z = f, f of zero sum, is then z = H f + alpha with
//     H f = G^+ D^2 (G^+ f + beta), beta making D^2 (..) sum to zero;
//   * S has at most 20 nodes (E: their unit vectors), so S is a small dense
//     correction: z = H (f - E lambda) + alpha with lambda = E^T z gives
//     (I + E^T H E) lambda - alpha 1 = E^T H f, sum lambda = sum f;
//   * b = E q lies in those nodes, so the first solution needs no transform
//     beyond those of the columns H E;
//   * the residual of the real system (7-point stencils, float entries) is
//     solved for again until it is below tol * |b_k|: the entries' rounding
//     is about 3e-8 against eigenvalues of L down to 1e-3 (res 32) or 2e-5
//     (res 256), so each round gains at least two digits, usually four.
// Transforms are dense products along an axis, folded by the cosine
// matrix's even and odd symmetry.  Two or three solutions of nine transform
// kernels (five on small lattices) each replace thousands of conjugate-gradient
// iterations of six dependent launches: 32^3 nodes, 4 constraints 124.9 ->
// 0.24 ms, and 1.6 ms at 64^3, 21 ms at 128^3; 1.3 s at 256^3 with 20.
#include <math.h>

#include <vector>

#include "gm_common.cuh"
#include "gm_internal.h"

namespace gm {

namespace {

constexpr int kFfThreads = 256;
constexpr int kFfCols = 16;     // lattice lines per block of a transform
constexpr int kFfMaxRounds = 40;

// the constrained nodes and their quaternions
struct FfPoints {
  int m;
  int node[kFrameFieldMaxPoints];
  double q[kFrameFieldMaxPoints][4];
};

__device__ __forceinline__ int ff_deg(int x, int y, int z, int n) {
  return (x > 0) + (x < n - 1) + (y > 0) + (y < n - 1) + (z > 0) + (z < n - 1);
}

// the reference's off-diagonal entry -(1.f / deg), in float, widened
__device__ __forceinline__ double ff_w(int deg) { return (double)(-(1.f / (float)deg)); }

struct V4 {
  double v[4];
};

__device__ __forceinline__ V4 ld4(const double* a, int64_t i) {
  const double2 lo = reinterpret_cast<const double2*>(a)[2 * i], hi = reinterpret_cast<const double2*>(a)[2 * i + 1];
  return V4{{lo.x, lo.y, hi.x, hi.y}};
}
__device__ __forceinline__ void st4(double* a, int64_t i, const V4& x) {
  reinterpret_cast<double2*>(a)[2 * i] = make_double2(x.v[0], x.v[1]);
  reinterpret_cast<double2*>(a)[2 * i + 1] = make_double2(x.v[2], x.v[3]);
}

// ---- transforms along an axis
//
// v holds nc components per node, in place.  A block takes kFfCols lines
// whole: line q of the axis has its elements at stride inner = nc * (nodes
// before the axis).  Forward: the line is folded into sums (even wave
// numbers) and differences (odd ones) of mirrored elements; inverse: each
// thread builds an element and its mirror from the even and the odd half.
// Either way res / 2 multiply-adds an output.  Bound by FP64 issue (two
// multiply-adds a clock and SM on this part), which is why the lines stay
// in shared memory through what lies between two transforms of an axis:
//   FF_SOLVE  (axis z): forward, divide by lambda, inverse
//   FF_WEIGHT (axis x): inverse, multiply by deg^2, forward
enum FfMode { FF_FWD = 0, FF_INV = 1, FF_SOLVE = 2, FF_WEIGHT = 3 };

__device__ __forceinline__ void ff_forward(const double* __restrict__ C, int n, double* src, double* dst, int col,
                                           int kg) {
  for (int i = kg; i < n / 2; i += 8) {
    const double a = src[i * kFfCols + col], b = src[(n - 1 - i) * kFfCols + col];
    src[i * kFfCols + col] = a + b;
    src[(n - 1 - i) * kFfCols + col] = a - b;
  }
  __syncthreads();
  const bool odd = kg & 1;  // the parity of every wave number kg + 8 m
  const int cnt = odd ? n / 2 : (n + 1) / 2;
  const double* s = src + (odd ? (n - 1) * kFfCols : 0) + col;
  const int step = odd ? -kFfCols : kFfCols;
  for (int k0 = kg; k0 < n; k0 += 32) {
    double acc[4] = {0, 0, 0, 0};
    const double* row[4];
#pragma unroll
    for (int m = 0; m < 4; m++) row[m] = C + (size_t)(k0 + 8 * m < n ? k0 + 8 * m : k0) * n;
    for (int i = 0; i < cnt; i++) {
      const double x = s[i * step];
#pragma unroll
      for (int m = 0; m < 4; m++) acc[m] = fma(__ldg(row[m] + i), x, acc[m]);
    }
#pragma unroll
    for (int m = 0; m < 4; m++)
      if (k0 + 8 * m < n) dst[(k0 + 8 * m) * kFfCols + col] = acc[m];
  }
  __syncthreads();
}

__device__ __forceinline__ void ff_inverse(const double* __restrict__ C, int n, const double* src, double* dst,
                                           int col, int kg) {
  const int nh = (n + 1) / 2;
  for (int i0 = kg; i0 < nh; i0 += 16) {
    const int i1 = i0 + 8 < nh ? i0 + 8 : i0;
    double e0 = 0, o0 = 0, e1 = 0, o1 = 0;
    int k = 0;
    for (; k + 1 < n; k += 2) {
      const double ye = src[k * kFfCols + col], yo = src[(k + 1) * kFfCols + col];
      const double* c = C + (size_t)k * n;
      e0 = fma(__ldg(c + i0), ye, e0);
      o0 = fma(__ldg(c + n + i0), yo, o0);
      e1 = fma(__ldg(c + i1), ye, e1);
      o1 = fma(__ldg(c + n + i1), yo, o1);
    }
    if (k < n) {
      const double ye = src[k * kFfCols + col];
      e0 = fma(__ldg(C + (size_t)k * n + i0), ye, e0);
      e1 = fma(__ldg(C + (size_t)k * n + i1), ye, e1);
    }
    // (the middle of an odd line: the odd wave numbers vanish there)
    dst[(n - 1 - i0) * kFfCols + col] = e0 - o0;
    dst[i0 * kFfCols + col] = e0 + o0;
    if (i1 != i0) {
      dst[(n - 1 - i1) * kFfCols + col] = e1 - o1;
      dst[i1 * kFfCols + col] = e1 + o1;
    }
  }
  __syncthreads();
}

template <int MODE>
__global__ void __launch_bounds__(128) k_ff_line(double* __restrict__ v, int n, int axis, int nc,
                                                 const double* __restrict__ C, const double* __restrict__ lam,
                                                 double* __restrict__ dc) {
  extern __shared__ double ff_sm[];
  double* a = ff_sm;
  double* b = ff_sm + (size_t)n * kFfCols;
  const int col = threadIdx.x & (kFfCols - 1), kg = threadIdx.x / kFfCols;  // 8 groups
  const int64_t inner = (int64_t)nc * (axis == 0 ? 1 : (axis == 1 ? n : n * n));
  const int64_t q = (int64_t)blockIdx.x * kFfCols + col;
  const bool ok = q < (int64_t)n * n * nc;
  const int64_t o = q / inner, j = q - o * inner;
  double* line = v + o * n * inner + j;
  for (int i = kg; i < n; i += 8) a[i * kFfCols + col] = ok ? line[i * inner] : 0.0;
  __syncthreads();
  double* out = b;
  if (MODE == FF_FWD) {
    ff_forward(C, n, a, b, col, kg);
  } else if (MODE == FF_INV) {
    ff_inverse(C, n, a, b, col, kg);
  } else if (MODE == FF_SOLVE) {
    ff_forward(C, n, a, b, col, kg);
    if (ok) {
      const int c = (int)(j % nc), kx = (int)((j / nc) % n), ky = (int)(j / ((int64_t)nc * n));
      const double lxy = lam[kx] + lam[ky];
      for (int k = kg; k < n; k += 8) {
        if ((kx | ky | k) == 0) {
          dc[c] = b[col];  // the sum over the nodes / n^1.5
          b[col] = 0.0;
        } else {
          b[k * kFfCols + col] /= lxy + lam[k];
        }
      }
    }
    __syncthreads();
    ff_inverse(C, n, b, a, col, kg);
    out = a;
  } else {
    ff_inverse(C, n, a, b, col, kg);
    if (ok) {
      const int y = (int)(o % n), z = (int)(o / n);
      for (int i = kg; i < n; i += 8) {
        const double d = (double)ff_deg(i, y, z, n);
        b[i * kFfCols + col] *= d * d;
      }
    }
    __syncthreads();
    ff_forward(C, n, b, a, col, kg);
    out = a;
  }
  if (ok)
    for (int i = kg; i < n; i += 8) line[i * inner] = out[i * kFfCols + col];
}

// g = deg^2 per node (one component), before its transforms
__global__ void __launch_bounds__(kFfThreads) k_ff_deg2(double* __restrict__ g, int n) {
  const int64_t total = (int64_t)n * n * n;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= total) return;
  const double d = (double)ff_deg((int)(i % n), (int)((i / n) % n), (int)(i / ((int64_t)n * n)), n);
  g[i] = d * d;
}

// The transforms of the unit vectors of the constrained nodes are products of
// three cosines: the columns' forward transforms, their division by lambda
// and the inverse along z in one kernel that reads nothing but the cosines.
__global__ void __launch_bounds__(128) k_ff_units(double* __restrict__ v, int n, int nc, const double* __restrict__ C,
                                                  const double* __restrict__ lam, double* __restrict__ dc,
                                                  const __grid_constant__ FfPoints pts) {
  extern __shared__ double ff_sm[];
  double* a = ff_sm;
  double* b = ff_sm + (size_t)n * kFfCols;
  const int col = threadIdx.x & (kFfCols - 1), kg = threadIdx.x / kFfCols;
  const int64_t inner = (int64_t)nc * n * n, q = (int64_t)blockIdx.x * kFfCols + col;
  const bool ok = q < inner;
  const int c = (int)(q % nc), kx = (int)((q / nc) % n), ky = (int)(q / ((int64_t)nc * n));
  const bool on = ok && c < pts.m;
  const int node = on ? pts.node[c] : 0, px = node % n, py = (node / n) % n, pz = node / (n * n);
  const double cxy = on ? C[(size_t)kx * n + px] * C[(size_t)ky * n + py] : 0.0, lxy = on ? lam[kx] + lam[ky] : 0.0;
  for (int k = kg; k < n; k += 8) {
    double s = on ? cxy * C[(size_t)k * n + pz] : 0.0;
    if (ok && (kx | ky | k) == 0) {
      dc[c] = s;  // the sum over the nodes / n^1.5
      s = 0.0;
    } else if (on) {
      s /= lxy + lam[k];
    }
    b[k * kFfCols + col] = s;
  }
  __syncthreads();
  ff_inverse(C, n, b, a, col, kg);
  if (ok)
    for (int i = kg; i < n; i += 8) v[(int64_t)i * inner + q] = a[i * kFfCols + col];
}

// ---- transforms of an xy plane
//
// On small lattices a launch per axis waits longer than it computes: a block
// takes one plane of one component whole in shared memory, with the cosines,
// through what lies between two transforms along z:
//   FF_FWD: along x and y; FF_INV: inverse along both;
//   FF_WEIGHT: inverse along both, multiply by deg^2, along both
// (16 warps; lane: the line, warp: wave number or element mod 16.  E: ceil of
// n / 16.)  Taken up to 32 nodes an axis, where a solve of 4 constraints went
// from 0.317 to 0.243 ms (32) and 0.232 to 0.174 (16) together with
// k_ff_units.  Above, the second round of lines leaves lanes idle and a plane
// leaves an SM few blocks: 48: 0.78 ms with a launch per axis, 1.02 with
// planes; 64: no difference.
constexpr int kFfPlaneThreads = 512;

// element i of line l at i es + l ls
template <int E>
__device__ __forceinline__ void plane_forward(const double* C, int n, double* src, double* dst, int es, int ls) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  for (int l = lane; l < n; l += 32)
    for (int i = wid; i < n / 2; i += 16) {
      double *p = src + i * es + l * ls, *q = src + (n - 1 - i) * es + l * ls;
      const double a = *p, b = *q;
      *p = a + b;
      *q = a - b;
    }
  __syncthreads();
  const bool odd = wid & 1;  // the parity of every wave number wid + 16 m
  const int cnt = odd ? n / 2 : (n + 1) / 2, step = odd ? -es : es;
  const double* row[E];
#pragma unroll
  for (int m = 0; m < E; m++) row[m] = C + (wid + 16 * m < n ? wid + 16 * m : 0) * n;
  for (int l = lane; l < n; l += 32) {
    const double* s = src + l * ls + (odd ? (n - 1) * es : 0);
    double acc[E];
#pragma unroll
    for (int m = 0; m < E; m++) acc[m] = 0;
    for (int i = 0; i < cnt; i++) {
      const double x = s[i * step];
#pragma unroll
      for (int m = 0; m < E; m++) acc[m] = fma(row[m][i], x, acc[m]);
    }
#pragma unroll
    for (int m = 0; m < E; m++)
      if (wid + 16 * m < n) dst[(wid + 16 * m) * es + l * ls] = acc[m];
  }
  __syncthreads();
}

template <int E>
__device__ __forceinline__ void plane_inverse(const double* C, int n, const double* src, double* dst, int es, int ls) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nh = (n + 1) / 2;
  constexpr int H = (E + 1) / 2;  // elements of a half line a thread
  for (int l = lane; l < n; l += 32) {
    const double* s = src + l * ls;
    double e[H], o[H];
#pragma unroll
    for (int m = 0; m < H; m++) e[m] = o[m] = 0;
    for (int k = 0; k < n; k += 2) {
      const double ye = s[k * es], yo = k + 1 < n ? s[(k + 1) * es] : 0.0;
      const double *ce = C + k * n, *co = C + (k + 1 < n ? k + 1 : k) * n;
#pragma unroll
      for (int m = 0; m < H; m++) {
        const int i = wid + 16 * m < nh ? wid + 16 * m : 0;
        e[m] = fma(ce[i], ye, e[m]);
        o[m] = fma(co[i], yo, o[m]);
      }
    }
#pragma unroll
    for (int m = 0; m < H; m++) {
      const int i = wid + 16 * m;
      if (i < nh) {  // (the middle of an odd line: the odd wave numbers vanish there)
        dst[(n - 1 - i) * es + l * ls] = e[m] - o[m];
        dst[i * es + l * ls] = e[m] + o[m];
      }
    }
  }
  __syncthreads();
}

template <int MODE, int E>
__global__ void __launch_bounds__(kFfPlaneThreads) k_ff_plane(double* __restrict__ v, int n, int nc,
                                                              const double* __restrict__ cosines) {
  extern __shared__ double ff_sm[];
  const int pitch = n + 1;  // (lines along either axis without bank conflicts)
  double* C = ff_sm;
  double* a = C + n * n;
  double* b = a + n * pitch;
  const int z = (int)(blockIdx.x / nc), c = (int)(blockIdx.x % nc);
  double* plane = v + (int64_t)z * n * n * nc + c;
  for (int i = threadIdx.x; i < n * n; i += kFfPlaneThreads) {
    C[i] = cosines[i];
    a[i / n * pitch + i % n] = plane[(int64_t)i * nc];
  }
  __syncthreads();
  if (MODE != FF_FWD) {
    plane_inverse<E>(C, n, a, b, pitch, 1);
    plane_inverse<E>(C, n, b, a, 1, pitch);
  }
  if (MODE == FF_WEIGHT) {
    for (int i = threadIdx.x; i < n * n; i += kFfPlaneThreads) {
      const double d = (double)ff_deg(i % n, i / n, z, n);
      a[i / n * pitch + i % n] *= d * d;
    }
    __syncthreads();
  }
  if (MODE != FF_INV) {
    plane_forward<E>(C, n, a, b, 1, pitch);
    plane_forward<E>(C, n, b, a, pitch, 1);
  }
  for (int i = threadIdx.x; i < n * n; i += kFfPlaneThreads) plane[(int64_t)i * nc] = a[i / n * pitch + i % n];
}

// ---- the small dense correction (one block)
//
// sm (doubles): the inverse of A = I + E^T H E, its row sums and their sum,
// the columns' beta; then the update's coefficients: of the columns of H E,
// of g, and the constant.
struct FfSmall {
  double inv[kFrameFieldMaxPoints][kFrameFieldMaxPoints];
  double rows[kFrameFieldMaxPoints], total;
  double beta[kFrameFieldMaxPoints];
  double coef[kFrameFieldMaxPoints][4], gcoef[4], alpha[4];
};

// lambda from h (in sh[m][4]) and the right-hand side's sum; then the
// coefficients: first solution q - lambda, later ones -lambda
__device__ void ff_lambda(FfSmall* __restrict__ sm, const FfPoints& pts, double (*sh)[4], const double* rho,
                          const double* beta_r, bool first) {
  const int t = threadIdx.x, m = pts.m;
  __shared__ double lp[kFrameFieldMaxPoints][4], al[4], co[kFrameFieldMaxPoints][4];
  if (t < 4 * m) {
    double s = 0;
    for (int j = 0; j < m; j++) s = fma(sm->inv[t / 4][j], sh[j][t % 4], s);
    lp[t / 4][t % 4] = s;
  }
  __syncthreads();
  if (t < 4) {
    double s = rho[t];
    for (int j = 0; j < m; j++) s -= lp[j][t];
    al[t] = s / sm->total;
    sm->alpha[t] = al[t];
  }
  __syncthreads();
  if (t < 4 * m) {
    const int j = t / 4, c = t % 4;
    const double l = fma(al[c], sm->rows[j], lp[j][c]);
    co[j][c] = first ? pts.q[j][c] - l : -l;
    sm->coef[j][c] = co[j][c];
  }
  __syncthreads();
  if (t < 4) {
    double s = beta_r[t];
    for (int j = 0; j < m; j++) s = fma(sm->beta[j], co[j][t], s);
    sm->gcoef[t] = s;
  }
}

// A and its inverse (Gauss-Jordan; A is symmetric positive definite), and
// the coefficients of the first solution
__global__ void __launch_bounds__(512) k_ff_small_first(const double* __restrict__ HE, int nc,
                                                        const double* __restrict__ g, const double* __restrict__ dc,
                                                        double dc_to_beta, const __grid_constant__ FfPoints pts,
                                                        FfSmall* __restrict__ sm) {
  constexpr int M = kFrameFieldMaxPoints;
  __shared__ double A[M][M], B[M][M], h[M][4], rho[4], zero[4];
  const int t = threadIdx.x, m = pts.m, i = t / M, j = t % M;
  const bool on = i < m && j < m;
  if (on) {
    const double beta = dc[j] * dc_to_beta;
    if (i == 0) sm->beta[j] = beta;
    A[i][j] = fma(beta, g[pts.node[i]], HE[(int64_t)pts.node[i] * nc + j]);  // E^T H E
    B[i][j] = i == j ? 1.0 : 0.0;
  }
  __syncthreads();
  if (t < 4 * m) {  // h = E^T H E q
    double s = 0;
    for (int k = 0; k < m; k++) s = fma(A[t / 4][k], pts.q[k][t % 4], s);
    h[t / 4][t % 4] = s;
  }
  if (t < 4) {
    double s = 0;
    for (int k = 0; k < m; k++) s += pts.q[k][t];
    rho[t] = s;
    zero[t] = 0;
  }
  __syncthreads();
  if (on && i == j) A[i][i] += 1.0;
  __syncthreads();
  for (int p = 0; p < m; p++) {
    double d = 1, f = 0, ap = 0, bp = 0;
    if (on) d = 1.0 / A[p][p], f = A[i][p], ap = A[p][j] * d, bp = B[p][j] * d;
    __syncthreads();
    if (on) {
      A[i][j] = i == p ? ap : fma(-f, ap, A[i][j]);
      B[i][j] = i == p ? bp : fma(-f, bp, B[i][j]);
    }
    __syncthreads();
  }
  if (on) sm->inv[i][j] = B[i][j];
  if (t < m) {
    double s = 0;
    for (int k = 0; k < m; k++) s += B[t][k];
    sm->rows[t] = s;
    A[0][t] = s;
  }
  __syncthreads();
  if (t == 0) {
    double s = 0;
    for (int k = 0; k < m; k++) s += A[0][k];
    sm->total = s;
  }
  __threadfence_block();
  __syncthreads();
  ff_lambda(sm, pts, h, rho, zero, true);
}

// the coefficients of a later solution: tr = H0 r (H without its beta)
__global__ void __launch_bounds__(128) k_ff_small(const double* __restrict__ tr, const double* __restrict__ g,
                                                  const double* __restrict__ dc_sum, const double* __restrict__ dc,
                                                  double dc_to_sum, double dc_to_beta,
                                                  const __grid_constant__ FfPoints pts, FfSmall* __restrict__ sm) {
  __shared__ double h[kFrameFieldMaxPoints][4], rho[4], beta[4];
  const int t = threadIdx.x, m = pts.m;
  if (t < 4) {
    rho[t] = dc_sum[t] * dc_to_sum;
    beta[t] = dc[t] * dc_to_beta;
  }
  __syncthreads();
  if (t < 4 * m) h[t / 4][t % 4] = fma(beta[t % 4], g[pts.node[t / 4]], tr[4 * (int64_t)pts.node[t / 4] + t % 4]);
  __syncthreads();
  ff_lambda(sm, pts, h, rho, beta, false);
}

// x (+)= [tr] + H0 E coef + g gcoef + alpha
template <bool FIRST>
__global__ void __launch_bounds__(kFfThreads) k_ff_apply(double* __restrict__ x, const double* __restrict__ tr,
                                                         const double* __restrict__ HE, int nc, int m,
                                                         const double* __restrict__ g,
                                                         const FfSmall* __restrict__ sm, int64_t total) {
  __shared__ double coef[kFrameFieldMaxPoints][4];
  for (int k = threadIdx.x; k < 4 * m; k += blockDim.x) coef[k / 4][k % 4] = sm->coef[k / 4][k % 4];
  __syncthreads();
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= total) return;
  V4 s;
  const double gi = g[i];
#pragma unroll
  for (int k = 0; k < 4; k++) s.v[k] = fma(gi, sm->gcoef[k], sm->alpha[k]);
  for (int j = 0; j < m; j++) {
    const double e = HE[i * nc + j];
#pragma unroll
    for (int k = 0; k < 4; k++) s.v[k] = fma(e, coef[j][k], s.v[k]);
  }
  if (!FIRST) {
    const V4 t = ld4(tr, i), xv = ld4(x, i);
#pragma unroll
    for (int k = 0; k < 4; k++) s.v[k] = xv.v[k] + (s.v[k] + t.v[k]);
  }
  st4(x, i, s);
}

// ---- the real system (float entries), matrix-free

// block sum of 4 doubles per thread into part[4 * blockIdx.x + k]
__device__ void ff_block_sum(const double (&s)[4], double* part) {
  __shared__ double red[kFfThreads / 32][4];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 4; k++) {
    double v = s[k];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[wid][k] = v;
  }
  __syncthreads();
  if (threadIdx.x < 4) {
    double t = 0;
    for (int w = 0; w < kFfThreads / 32; w++) t += red[w][threadIdx.x];
    part[4 * blockIdx.x + threadIdx.x] = t;
  }
}

// y = L p
__global__ void __launch_bounds__(kFfThreads) k_ff_lap(const double* __restrict__ p, double* __restrict__ y, int n) {
  const int64_t total = (int64_t)n * n * n;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= total) return;
  const int x = (int)(i % n), yy = (int)((i / n) % n), z = (int)(i / ((int64_t)n * n));
  const double w = ff_w(ff_deg(x, yy, z, n));
  V4 s{{0, 0, 0, 0}};
  auto add = [&](int64_t j) {
    const V4 a = ld4(p, j);
#pragma unroll
    for (int k = 0; k < 4; k++) s.v[k] += a.v[k];
  };
  const int64_t sy = n, sz = (int64_t)n * n;
  if (z > 0) add(i - sz);
  if (yy > 0) add(i - sy);
  if (x > 0) add(i - 1);
  if (x < n - 1) add(i + 1);
  if (yy < n - 1) add(i + sy);
  if (z < n - 1) add(i + sz);
  const V4 c = ld4(p, i);
  V4 o;
#pragma unroll
  for (int k = 0; k < 4; k++) o.v[k] = c.v[k] + w * s.v[k];
  st4(y, i, o);
}

// r = b - (L^T y + S p), y = L p, and the block partials of r . r
__global__ void __launch_bounds__(kFfThreads) k_ff_residual(const double* __restrict__ y,
                                                            const double* __restrict__ p, double* __restrict__ r,
                                                            double* __restrict__ part, int n,
                                                            const __grid_constant__ FfPoints pts) {
  const int64_t total = (int64_t)n * n * n;
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  double dot[4] = {0, 0, 0, 0};
  if (i < total) {
    const int x = (int)(i % n), yy = (int)((i / n) % n), z = (int)(i / ((int64_t)n * n));
    V4 o = ld4(y, i);
    auto add = [&](int64_t j, int jx, int jy, int jz) {
      const double w = ff_w(ff_deg(jx, jy, jz, n));
      const V4 a = ld4(y, j);
#pragma unroll
      for (int k = 0; k < 4; k++) o.v[k] += w * a.v[k];
    };
    const int64_t sy = n, sz = (int64_t)n * n;
    if (z > 0) add(i - sz, x, yy, z - 1);
    if (yy > 0) add(i - sy, x, yy - 1, z);
    if (x > 0) add(i - 1, x - 1, yy, z);
    if (x < n - 1) add(i + 1, x + 1, yy, z);
    if (yy < n - 1) add(i + sy, x, yy + 1, z);
    if (z < n - 1) add(i + sz, x, yy, z + 1);
    int at = -1;
    for (int c = 0; c < pts.m; c++)
      if (pts.node[c] == (int)i) at = c;
    V4 rv;
#pragma unroll
    for (int k = 0; k < 4; k++) rv.v[k] = -o.v[k];
    if (at >= 0) {
      const V4 pc = ld4(p, i);
#pragma unroll
      for (int k = 0; k < 4; k++) rv.v[k] = pts.q[at][k] - (o.v[k] + pc.v[k]);
    }
    st4(r, i, rv);
#pragma unroll
    for (int k = 0; k < 4; k++) dot[k] = rv.v[k] * rv.v[k];
  }
  ff_block_sum(dot, part);
}

// one block: the partials of `nb` blocks summed in a fixed order
__global__ void __launch_bounds__(kFfThreads) k_ff_sum(const double* __restrict__ part, int nb,
                                                       double* __restrict__ rr) {
  __shared__ double red[kFfThreads][4];
  double s[4] = {0, 0, 0, 0};
  for (int b = threadIdx.x; b < nb; b += blockDim.x)
#pragma unroll
    for (int k = 0; k < 4; k++) s[k] += part[4 * b + k];
#pragma unroll
  for (int k = 0; k < 4; k++) red[threadIdx.x][k] = s[k];
  __syncthreads();
  for (int h = kFfThreads / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h)
#pragma unroll
      for (int k = 0; k < 4; k++) red[threadIdx.x][k] += red[threadIdx.x + h][k];
    __syncthreads();
  }
  if (threadIdx.x < 4) rr[threadIdx.x] = red[0][threadIdx.x];
}

__global__ void k_ff_store(const double* __restrict__ x, float4* __restrict__ q, int64_t total) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x) {
    const V4 v = ld4(x, i);
    q[i] = make_float4((float)v.v[0], (float)v.v[1], (float)v.v[2], (float)v.v[3]);
  }
}

__global__ void k_ff_fill(float4* __restrict__ q, float4 v, int64_t total) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += (int64_t)gridDim.x * blockDim.x)
    q[i] = v;
}

int ff_blocks(int64_t total) { return (int)((total + kFfThreads - 1) / kFfThreads); }

template <int MODE>
cudaError_t ff_line(FrameFieldGpu& f, double* v, int axis, int nc, double* dc, cudaStream_t st, KernelCounter* kc) {
  const int n = f.res;
  const int64_t lines = (int64_t)n * n * nc;
  const size_t smem = sizeof(double) * 2 * kFfCols * (size_t)n;
  cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(k_ff_line<MODE>), smem);
  if (e != cudaSuccess) return e;
  GM_LAUNCH(kc, "k_ff_line", st,
            k_ff_line<MODE><<<(unsigned)((lines + kFfCols - 1) / kFfCols), 128, smem, st>>>(v, n, axis, nc, f.cosines,
                                                                                          f.lambda, dc));
  return cudaGetLastError();
}

// the transforms of an xy plane of MODE (see k_ff_plane), one launch or one per axis
template <int MODE, int E>
cudaError_t ff_plane_e(FrameFieldGpu& f, double* v, int nc, cudaStream_t st, KernelCounter* kc) {
  const int n = f.res;
  const size_t smem = sizeof(double) * ((size_t)n * n + 2 * (size_t)n * (n + 1));
  cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(k_ff_plane<MODE, E>), smem);
  if (e != cudaSuccess) return e;
  GM_LAUNCH(kc, "k_ff_plane", st,
            k_ff_plane<MODE, E><<<(unsigned)(n * nc), kFfPlaneThreads, smem, st>>>(v, n, nc, f.cosines));
  return cudaGetLastError();
}
template <int MODE>
cudaError_t ff_plane(FrameFieldGpu& f, double* v, int nc, cudaStream_t st, KernelCounter* kc) {
  const int n = f.res;
  if (n <= 16) return ff_plane_e<MODE, 1>(f, v, nc, st, kc);
  if (n <= 32) return ff_plane_e<MODE, 2>(f, v, nc, st, kc);
  cudaError_t e;
  if (MODE == FF_FWD) {
    if ((e = ff_line<FF_FWD>(f, v, 0, nc, nullptr, st, kc)) != cudaSuccess) return e;
    return ff_line<FF_FWD>(f, v, 1, nc, nullptr, st, kc);
  }
  if ((e = ff_line<FF_INV>(f, v, 1, nc, nullptr, st, kc)) != cudaSuccess) return e;
  if (MODE == FF_INV) return ff_line<FF_INV>(f, v, 0, nc, nullptr, st, kc);
  if ((e = ff_line<FF_WEIGHT>(f, v, 0, nc, nullptr, st, kc)) != cudaSuccess) return e;
  return ff_line<FF_FWD>(f, v, 1, nc, nullptr, st, kc);
}

// v = G^+ D^2 G^+ v without beta, the sums' coefficients into dc[0 .. nc)
// (of v) and dc[nc ..) (of D^2 G^+ v); with pts, v starts as their nodes'
// unit vectors (and need not hold anything)
cudaError_t ff_h0(FrameFieldGpu& f, double* v, int nc, const FfPoints* pts, double* dc, cudaStream_t st,
                  KernelCounter* kc) {
  cudaError_t e;
  if (pts) {
    const int n = f.res;
    const size_t smem = sizeof(double) * 2 * kFfCols * (size_t)n;
    if ((e = ensure_dynamic_smem(reinterpret_cast<const void*>(k_ff_units), smem)) != cudaSuccess) return e;
    GM_LAUNCH(kc, "k_ff_units", st,
              k_ff_units<<<(unsigned)(((int64_t)n * n * nc + kFfCols - 1) / kFfCols), 128, smem, st>>>(
                  v, n, nc, f.cosines, f.lambda, dc, *pts));
  } else {
    if ((e = ff_plane<FF_FWD>(f, v, nc, st, kc)) != cudaSuccess) return e;
    if ((e = ff_line<FF_SOLVE>(f, v, 2, nc, dc, st, kc)) != cudaSuccess) return e;
  }
  if ((e = ff_plane<FF_WEIGHT>(f, v, nc, st, kc)) != cudaSuccess) return e;
  if ((e = ff_line<FF_SOLVE>(f, v, 2, nc, dc + nc, st, kc)) != cudaSuccess) return e;
  return ff_plane<FF_INV>(f, v, nc, st, kc);
}

// The field's plan, on its first solve: cosine matrix, eigenvalues, G^+ of
// the squared degrees (they depend on res only).
cudaError_t ff_plan(FrameFieldGpu& f, cudaStream_t st, KernelCounter* kc) {
  const int n = f.res;
  const int64_t total = (int64_t)n * n * n;
  cudaError_t e;
  const double pi = 3.14159265358979323846;
  std::vector<double> c((size_t)n * n + n);
  std::vector<double> quarter(4 * (size_t)n);  // cos(pi j / 2n), j mod 4n
  for (int j = 0; j < 4 * n; j++) quarter[j] = cos(pi * j / (2.0 * n));
  for (int k = 0; k < n; k++)
    for (int i = 0; i < n; i++)
      c[(size_t)k * n + i] = sqrt((k == 0 ? 1.0 : 2.0) / n) * quarter[(size_t)k * (2 * i + 1) % (4 * n)];
  for (int k = 0; k < n; k++) {
    const double s = sin(pi * k / (2.0 * n));
    c[(size_t)n * n + k] = 4.0 * s * s;  // 2 - 2 cos(pi k / n)
  }
  if (!f.cosines && (e = cudaMalloc(&f.cosines, sizeof(double) * c.size())) != cudaSuccess) return e;
  if (!f.g && (e = cudaMalloc(&f.g, sizeof(double) * total)) != cudaSuccess) return e;
  f.lambda = f.cosines + (size_t)n * n;
  // (the copy reads pageable memory: it has left c when the call returns)
  if ((e = cudaMemcpyAsync(f.cosines, c.data(), sizeof(double) * c.size(), cudaMemcpyHostToDevice, st)) != cudaSuccess)
    return e;
  GM_LAUNCH(kc, "k_ff_deg2", st, k_ff_deg2<<<ff_blocks(total), kFfThreads, 0, st>>>(f.g, n));
  if ((e = ff_plane<FF_FWD>(f, f.g, 1, st, kc)) != cudaSuccess) return e;
  if ((e = ff_line<FF_SOLVE>(f, f.g, 2, 1, f.dc, st, kc)) != cudaSuccess) return e;
  if ((e = ff_plane<FF_INV>(f, f.g, 1, st, kc)) != cudaSuccess) return e;
  // sum of deg^2 over the lattice: end nodes of an axis count 1, others 2
  f.sum_deg2 = 0;
  for (int ends = 0; ends < 8; ends++) {
    double count = 1, d = 0;
    for (int a = 0; a < 3; a++) {
      count *= (ends >> a) & 1 ? 2.0 : (double)(n - 2);
      d += (ends >> a) & 1 ? 1.0 : 2.0;
    }
    f.sum_deg2 += count * d * d;
  }
  f.planned = true;
  return cudaSuccess;
}

}  // namespace

cudaError_t frame_field_alloc(FrameFieldGpu& f, int res) {
  frame_field_free(f);
  const int64_t total = (int64_t)res * res * res;
  const int nb = ff_blocks(total);
  f.res = res;
  cudaError_t e;
  if ((e = cudaMalloc(&f.quats, sizeof(float4) * total)) != cudaSuccess) return e;
  if ((e = cudaMalloc(&f.x, sizeof(double) * 4 * total * 3)) != cudaSuccess) return e;
  f.r = f.x + 4 * total;
  f.y = f.r + 4 * total;
  if ((e = cudaMalloc(&f.part, sizeof(double) * 4 * nb)) != cudaSuccess) return e;
  // sums' coefficients, residual norms, the small system
  if ((e = cudaMalloc(&f.dc, sizeof(double) * (2 * kFrameFieldMaxPoints + 8) + sizeof(FfSmall))) != cudaSuccess) return e;
  f.rr = f.dc + 2 * kFrameFieldMaxPoints + 4;
  f.small = f.rr + 4;
  if ((e = cudaMallocHost(&f.h_rr, sizeof(double) * 4)) != cudaSuccess) return e;
  return cudaSuccess;
}

void frame_field_free(FrameFieldGpu& f) {
  cudaFree(f.quats);
  cudaFree(f.x);
  cudaFree(f.part);
  cudaFree(f.dc);
  cudaFree(f.cosines);
  cudaFree(f.g);
  cudaFree(f.HE);
  if (f.h_rr) cudaFreeHost(f.h_rr);
  f = FrameFieldGpu{};
}

cudaError_t frame_field_fill(FrameFieldGpu& f, float qx, float qy, float qz, float qw, cudaStream_t st,
                             KernelCounter* kc) {
  const int64_t total = (int64_t)f.res * f.res * f.res;
  int b = ff_blocks(total);
  if (b > 152 * 8) b = 152 * 8;
  GM_LAUNCH(kc, "k_ff_fill", st, k_ff_fill<<<b, kFfThreads, 0, st>>>(f.quats, make_float4(qx, qy, qz, qw), total));
  return cudaGetLastError();
}

cudaError_t frame_field_solve(FrameFieldGpu& f, const int64_t* nodes, const float* rhs4, int npts, double tol,
                              int* rounds_out, cudaStream_t st, KernelCounter* kc) {
  const int n = f.res;
  const int64_t total = (int64_t)n * n * n;
  const int nb = ff_blocks(total);
  cudaError_t e;
  // distinct nodes: points in order, the last one on a node wins
  FfPoints pts;
  pts.m = 0;
  double bb[4] = {0, 0, 0, 0};
  for (int c = 0; c < npts; c++) {
    int at = 0;
    while (at < pts.m && pts.node[at] != (int)nodes[c]) at++;
    if (at == kFrameFieldMaxPoints) return cudaErrorInvalidValue;
    if (at == pts.m) pts.m++;
    pts.node[at] = (int)nodes[c];
    for (int k = 0; k < 4; k++) pts.q[at][k] = (double)rhs4[4 * c + k];
  }
  for (int c = 0; c < pts.m; c++)
    for (int k = 0; k < 4; k++) bb[k] += pts.q[c][k] * pts.q[c][k];
  const int nc = (pts.m + 3) / 4 * 4;
  if (nc > f.HE_cols) {
    cudaFree(f.HE);
    f.HE = nullptr;
    f.HE_cols = 0;
    if ((e = cudaMalloc(&f.HE, sizeof(double) * total * nc)) != cudaSuccess) return e;
    f.HE_cols = nc;
  }
  // (all memory is there before the first launch: a solve that fails for
  // memory leaves no plan at work on a stream that the next may not be on)
  if (!f.planned && (e = ff_plan(f, st, kc)) != cudaSuccess) return e;
  FfSmall* sm = reinterpret_cast<FfSmall*>(f.small);
  const double dc_to_sum = (double)n * sqrt((double)n), dc_to_beta = -dc_to_sum / f.sum_deg2;
  // the columns H0 E and the first solution
  if ((e = ff_h0(f, f.HE, nc, &pts, f.dc, st, kc)) != cudaSuccess) return e;
  GM_LAUNCH(kc, "k_ff_small", st, k_ff_small_first<<<1, 512, 0, st>>>(f.HE, nc, f.g, f.dc + nc, dc_to_beta, pts, sm));
  GM_LAUNCH(kc, "k_ff_apply", st,
            k_ff_apply<true><<<nb, kFfThreads, 0, st>>>(f.x, nullptr, f.HE, nc, pts.m, f.g, sm, total));
  int rounds = 1;
  for (;;) {
    GM_LAUNCH(kc, "k_ff_lap", st, k_ff_lap<<<nb, kFfThreads, 0, st>>>(f.x, f.y, n));
    GM_LAUNCH(kc, "k_ff_residual", st, k_ff_residual<<<nb, kFfThreads, 0, st>>>(f.y, f.x, f.r, f.part, n, pts));
    if (rounds > 1) {  // the first solution carries the entries' rounding: one refinement at least
      GM_LAUNCH(kc, "k_ff_sum", st, k_ff_sum<<<1, kFfThreads, 0, st>>>(f.part, nb, f.rr));
      if ((e = cudaMemcpyAsync(f.h_rr, f.rr, sizeof(double) * 4, cudaMemcpyDeviceToHost, st)) != cudaSuccess) return e;
      if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
      bool done = true;
      for (int k = 0; k < 4; k++)
        if (f.h_rr[k] > tol * tol * bb[k]) done = false;
      if (done || rounds >= kFfMaxRounds) break;
    }
    if ((e = ff_h0(f, f.r, 4, nullptr, f.dc, st, kc)) != cudaSuccess) return e;
    GM_LAUNCH(kc, "k_ff_small", st,
              k_ff_small<<<1, 128, 0, st>>>(f.r, f.g, f.dc, f.dc + 4, dc_to_sum, dc_to_beta, pts, sm));
    GM_LAUNCH(kc, "k_ff_apply", st,
              k_ff_apply<false><<<nb, kFfThreads, 0, st>>>(f.x, f.r, f.HE, nc, pts.m, f.g, sm, total));
    rounds++;
  }
  if (rounds_out) *rounds_out = rounds;
  int bs = nb > 152 * 8 ? 152 * 8 : nb;
  GM_LAUNCH(kc, "k_ff_store", st, k_ff_store<<<bs, kFfThreads, 0, st>>>(f.x, f.quats, total));
  return cudaGetLastError();
}

}  // namespace gm
