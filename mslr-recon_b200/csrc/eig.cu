// eig.cu — per-patch Hermitian eigen stage of the patch SVST (sm_100a).
//
// For each patch Gram matrix G (n × n, Hermitian, column-major, FP32 complex)
// and threshold β this computes the scaled eigenvector matrix
//     Ṽ = V diag(√h),   h_i = max(√λ_i − β, 0) / √λ_i,
// over the eigenpairs (λ_i, v_i) of G with λ_i > β², so that the rebuild
// matrix of the patch SVST (src/recon.jl:183-211, expressed through its Gram
// matrix) is W = Ṽ Ṽᴴ — one more Gram product, formed by the batched Gram
// kernels after this launch.  One CTA per patch — 384 threads when n <= 384
// (two patches per SM, so one patch's latency-bound phases overlap the
// other's), else 1024; one launch may cover several segments (the patches of
// several scales, each with its own n and λ_k).  The matrix lives in global
// memory (L2); only its lower triangle is read or written:
//   1. Householder tridiagonalisation G = Q T Qᴴ (FP32).  Each step applies
//      the previous step's rank-2 update on the fly while forming the next
//      Hermitian matrix-vector product over 32 × 32 tiles of the trailing
//      lower triangle (one warp per tile: row sums per lane, column sums by a
//      shuffle transpose-reduction, both stored per tile and summed per row
//      in a fixed order, so results are bit-reproducible), streaming the
//      trailing triangle once per step; the working set of ~300 resident
//      patches stays in L2.  The pass also leaves the next column in shared
//      memory, and every thread computes the reflector scalars and the next
//      pivot row's (v, w) itself, so a step has four block barriers.
//   2. Eigenvalues of T above β² by bisection on FP64 Sturm counts, one
//      thread per eigenvalue.
//   3. Eigenvectors of T by FP64 twisted factorisation, one thread per
//      eigenvector; eigenvalues equal to working precision (true
//      degeneracies) are re-orthogonalised cooperatively by Gram–Schmidt.
//   4. V = Q Z with the reflectors applied 16 at a time in compact WY form
//      (Q_b = I − Y T Yᴴ); thread i keeps vector i's block coefficients in
//      registers, so the update needs no cross-thread reduction.
//   5. Ṽ written as conj(V) diag(√h) in row-major order ([row][vector]),
//      columns beyond the rank set to zero.
// Zero patches give no eigenvalue above β² and Ṽ = 0, hence W = 0 (the
// reference's zero-norm skip, src/recon.jl:185).
//
// Split stage (9 <= n <= 384): three launches (two for the values alone) instead
// of one, so that each phase has the shape it needs — phase 1 and the WY
// blocks' T factors (k_tri_reg: the matrix in registers, n <= 128; k_tri_big:
// panels), phases 2–3 (k_pairs: two, four or eight CTAs per SM by side and
// number of patches), and phases 4–5 as k_wy_apply: 64 eigenvectors of one patch
// per CTA, held in registers through every block update.  Phase 1 measured
// against k_eig's: one patch of side 64 351 → 71 µs, 40 of 128 834 → 219 µs, 2250
// of 128 8.0 → 3.5 ms, 486 of 300 12.7 → 8.7 ms.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <vector>

#include "internal.h"

namespace mslr {

namespace {

constexpr int kT = 1024;   // most threads per CTA (one row / eigenvalue per thread)
constexpr int kSmallT = 384;   // CTA size for n <= 384: two patches share an SM
constexpr int kNb = 16;    // reflectors per WY block
constexpr int kCW = 16;    // eigenvectors per back-transform pass

__device__ __forceinline__ float warp_sum(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_sum_d(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block sums; every thread gets the result.  Consecutive calls must alternate
// between two scratch buffers (one barrier per call).
__device__ __forceinline__ float block_sum(float v, float* red) {
  v = warp_sum(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  float r = 0.f;
  const int nw = (int)(blockDim.x >> 5);
  for (int i = 0; i < nw; ++i) r += red[i];
  return r;
}
__device__ __forceinline__ double block_sum_d(double v, double* red) {
  v = warp_sum_d(v);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  double r = 0.0;
  const int nw = (int)(blockDim.x >> 5);
  for (int i = 0; i < nw; ++i) r += red[i];
  return r;
}

// eigenvalues of the symmetric tridiagonal (d, e²) strictly below x
__device__ __forceinline__ int sturm_less(const double* d, const double* e2, int n, double x,
                                          double pivmin) {
  int cnt = 0;
  double q = d[0] - x;
  if (fabs(q) < pivmin) q = -pivmin;
  cnt += (q < 0.0);
  for (int i = 1; i < n; ++i) {
    q = d[i] - x - e2[i - 1] / q;
    if (fabs(q) < pivmin) q = -pivmin;
    cnt += (q < 0.0);
  }
  return cnt;
}

// sturm_less in FP32 on a copy of T scaled to norm ~1 (d / ‖T‖, e² / ‖T‖²),
// with the fast reciprocal division: the count is exact for a matrix within a
// few FP32 roundings of T (the Sturm sequence is backward stable), which is
// all the first rounds of bracketing need
__device__ __forceinline__ int sturm_less_f(const float* d, const float* e2, int n, float x) {
  constexpr float pivmin = 1e-30f;
  int cnt = 0;
  float q = d[0] - x;
  if (fabsf(q) < pivmin) q = -pivmin;
  cnt += (q < 0.f);
  for (int i = 1; i < n; ++i) {
    q = d[i] - x - __fdividef(e2[i - 1], q);
    if (fabsf(q) < pivmin) q = -pivmin;
    cnt += (q < 0.f);
  }
  return cnt;
}

// Which of several equal eigenvalues (to ctol) number e is, counted from the
// first, or -1 when it stands alone; lam[0 … r) descending.
__device__ __forceinline__ int tie_of(const double* lam, int r, int e, double ctol) {
  int t = 0;
  while (t < e && lam[e - t - 1] - lam[e - t] <= ctol) ++t;
  return t > 0 || (e + 1 < r && lam[e] - lam[e + 1] <= ctol) ? t : -1;
}

// Twist of the vector of the t-th of several equal eigenvalues.  They come from
// blocks of T that nothing couples (an unreduced T has none: a diagonal Gram, a
// patch with zero voxels), so the smallest |γ| of all rows is the same row for
// each of them.  The t-th takes the t-th block that has the eigenvalue, the row
// of the smallest |γ| in it, and rows b0 … b1 of that block alone.  How far the
// block's own eigenvalue is from λ̂ is the Rayleigh correction γ / ‖z‖², z its
// vector: z_j = −up(j) z_{j+1} above the twist, −down(j) z_{j−1} below.
struct Twist {
  int k, b0, b1;
};
template <class Gamma, class Up, class Down>
__device__ __noinline__ Twist tied_twist(int n, int t, const double* ee, double tnorm, Gamma gamma, Up up, Down down) {
  const double tau = 2e-12 * tnorm, cut = 1e-15 * tnorm;
  double best = 1e308;
  int bk = 0, b0 = 0;
  for (int k = 0; k < n; ++k) {
    const double g = gamma(k);
    if (g < best) {
      best = g;
      bk = k;
    }
    if (k == n - 1 || fabs(ee[k]) <= cut) {
      if (best <= tau * n) {   // ‖z‖² <= n at the row of the largest |z_j|
        double z = 1.0, s = 1.0;
        for (int j = bk - 1; j >= b0; --j) {
          z *= -up(j);
          s = fma(z, z, s);
        }
        z = 1.0;
        for (int j = bk + 1; j <= k; ++j) {
          z *= -down(j);
          s = fma(z, z, s);
        }
        if (best <= tau * s && t-- == 0) return {bk, b0, k};
      }
      best = 1e308;
      b0 = k + 1;
    }
  }
  return {-1, 0, n - 1};
}

struct Seg {
  int n;
  int64_t first;   // first block of the segment
  int64_t np;      // patches
  cf* gram;        // np × n × n: G in (lower triangle), Householder vectors out
  cf* zv;          // np × n × n: eigenvectors, [row j][vector i], i fastest; Ṽ out
  double* aux;     // np × n × n: FP64 pivots of the twisted factorisations
  int* rank;       // np
  double lam;      // threshold multiplier of the segment (λ_k)
  double* nuc;     // values-only mode when set: np sums Σ √λ_i over λ_i above β², no vectors
  double* lam_out; // full mode when set: all n eigenpairs, V unscaled in zv, λ (descending) here
  double* side;    // split stage: np × 6n — d, e (FP64), λ, h of the tridiagonal (k_eig modes 1, 2)
};

constexpr int kMaxSeg = 8;

struct EigArgs {
  int nseg;
  Seg seg[kMaxSeg];
  const double* thr;   // device: threshold scale (ζ or β), or per patch
  int thr_per_patch;
  int rz;              // eigenvectors staged in shared memory (more: global slots)
};

// vectors are padded to n + 32 entries (zero tails) so 32-wide tiles read them in bounds
// Per-tile partial sums of the tridiagonalisation's matvec: 64 values for
// each 32 × 32 tile of the largest trailing triangle (side n − 1).
size_t part_bytes(int n) {
  const size_t T = (size_t)(n - 1 + 31) / 32;
  return T * (T + 1) / 2 * 64 * sizeof(cf);
}

size_t vec_bytes(int n) {
  const size_t np = (size_t)n + 32;
  return np * sizeof(float4) + 5 * np * sizeof(cf) + 4 * (size_t)n * sizeof(double) +
         3 * (size_t)n * sizeof(float) + 64 * sizeof(float) + 64 * sizeof(double);
}

// Buffers of the back-transform besides the vector stage: Y (n × kNb), T and
// YᴴY (kNb × kNb each), S and T·S (kNb × kCW each), one partial sum per thread.
size_t wy_bytes(int n, int threads) {
  return ((size_t)n * kNb + 2 * kNb * kNb + 2 * kNb * kCW + (size_t)threads + 1) * sizeof(cf);
}

// The region after the vectors, by phase: the matvec partial sums (phase 1,
// 384-thread variant), the FP64 twisted-factorisation columns of up to rz
// eigenvectors (phase 3: z and D+, n × rz doubles each), the complex
// eigenvector stage (n × rz) followed by the back-transform buffers (phase 4).
size_t smem_bytes(int n, int threads, int rz) {
  const size_t stage = (size_t)n * rz * sizeof(cf);
  size_t region = std::max(2 * stage, stage + wy_bytes(n, threads));
  if (threads <= kSmallT) region = std::max(region, part_bytes(n));
  return vec_bytes(n) + region + 128;
}

// Dynamic shared memory one CTA may use: two CTAs per SM for the 384-thread
// variant (228 KB per SM, 1 KB reserved per CTA), one for the large variant;
// both leave room for the kernel's static shared variables.
size_t smem_budget(int threads) { return threads <= kSmallT ? 112 * 1024 : 227 * 1024 - 1024; }

// eigenvectors staged in shared memory: the most that fit beside everything else
int stage_cols(int n, int threads) {
  int rz = 0;
  while (rz < n && smem_bytes(n, threads, rz + 1) <= smem_budget(threads)) ++rz;
  return rz;
}

// Eight columns of a tile row: the pending rank-2 update of element
// (row, jb + b), its contribution to the row sum y_row and to the column
// partials (cr, ci), written back.
__device__ __forceinline__ void tile_group(cf* a, const float4* pw, const float4* vv, cf vpr, cf wpr, cf vr,
                                           float& yr, float& yim, float* cr, float* ci) {
#pragma unroll
  for (int b = 0; b < 8; ++b) {
    const float4 p = pw[b];   // (vp_j, wp_j)
    const float4 v2 = vv[b >> 1];
    const float vjx = (b & 1) ? v2.z : v2.x, vjy = (b & 1) ? v2.w : v2.y;
    cf e = a[b];
    e.x -= (vpr.x * p.z + vpr.y * p.w) + (wpr.x * p.x + wpr.y * p.y);
    e.y -= (vpr.y * p.z - vpr.x * p.w) + (wpr.y * p.x - wpr.x * p.y);
    a[b] = e;
    yr += e.x * vjx - e.y * vjy;
    yim += e.x * vjy + e.y * vjx;
    cr[b] = e.x * vr.x + e.y * vr.y;
    ci[b] = e.x * vr.y - e.y * vr.x;
  }
}

// Column sums of eight columns over the 32 lanes (a shuffle transpose): lane l
// ends with the sum of column l / 4 in cr[0], ci[0].
__device__ __forceinline__ void col_sums(float* cr, float* ci, int lane) {
  const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const float sr_ = h16 ? cr[q] : cr[q + 4], si_ = h16 ? ci[q] : ci[q + 4];
    const float kr = h16 ? cr[q + 4] : cr[q], ki = h16 ? ci[q + 4] : ci[q];
    cr[q] = kr + __shfl_xor_sync(0xffffffffu, sr_, 16);
    ci[q] = ki + __shfl_xor_sync(0xffffffffu, si_, 16);
  }
#pragma unroll
  for (int q = 0; q < 2; ++q) {
    const float sr_ = h8 ? cr[q] : cr[q + 2], si_ = h8 ? ci[q] : ci[q + 2];
    const float kr = h8 ? cr[q + 2] : cr[q], ki = h8 ? ci[q + 2] : ci[q];
    cr[q] = kr + __shfl_xor_sync(0xffffffffu, sr_, 8);
    ci[q] = ki + __shfl_xor_sync(0xffffffffu, si_, 8);
  }
  {
    const float sr_ = h4 ? cr[0] : cr[1], si_ = h4 ? ci[0] : ci[1];
    const float kr = h4 ? cr[1] : cr[0], ki = h4 ? ci[1] : ci[0];
    cr[0] = kr + __shfl_xor_sync(0xffffffffu, sr_, 4);
    ci[0] = ki + __shfl_xor_sync(0xffffffffu, si_, 4);
  }
  cr[0] += __shfl_xor_sync(0xffffffffu, cr[0], 2);
  ci[0] += __shfl_xor_sync(0xffffffffu, ci[0], 2);
  cr[0] += __shfl_xor_sync(0xffffffffu, cr[0], 1);
  ci[0] += __shfl_xor_sync(0xffffffffu, ci[0], 1);
}

// The power of two that takes a matrix's largest diagonal entry, which bounds a
// Gram's entries, into [1, 2), and its inverse, with which d and e are scaled
// back; reflectors and τ do not depend on it.  As it is when the entry is zero
// or not finite.
struct PowerOfTwo {
  float up;
  double down;
  __device__ __forceinline__ explicit PowerOfTwo(float dmax) {
    const int ex = __float_as_int(dmax) >> 23;   // (dmax >= 0)
    const int k = dmax > 0.f && ex < 255 ? min(max(ex, 1), 253) : 127;
    up = __int_as_float((254 - k) << 23);
    down = __hiloint2double((k - 127 + 1023) << 20, 0);
  }
};

// What is left of a column below its subdiagonal (and the subdiagonal's
// imaginary part) is dropped, the column taken as it is, when its square is
// at most this: 1e-16 of the scaled matrix, far below FP32's rounding of it.
// Above, neither |u₁|² nor the sums with u lose bits to denormals.
constexpr float kNoColumn = 1e-32f;

// An off-diagonal tile (I, J), J < I, whose 32 columns all lie inside the
// matrix (rows past n, in the last tile row, are masked per lane): the same
// arithmetic as the general tile path without its per-element tests; the
// column values come from the re-based vectors as
// 16-byte loads, and each group's loads are issued before the previous
// group is updated and stored (they address other columns) when PIPE (the
// 384-thread variant; the 1024-thread variant's 64 registers do not hold
// the second group).
template <bool PIPE>
__device__ __noinline__ void full_tile(cf* A, int n, int o, int I, int J, int t, int lane, const float4* spw,
                                       const cf* svr, const cf* svp, const cf* swp, const cf* sv, cf* part,
                                       cf* scol) {
  const int row = o + I * 32 + lane;
  const bool rowok = row < n;   // the last tile row may reach past n (its vectors are zero there)
  const cf vpr = svp[row], wpr = swp[row], vr = sv[row];
  float yr = 0.f, yim = 0.f;
  const int jo = J * 32;   // first column − o
  cf* col0 = A + (int64_t)(o + jo) * n + row;
  const float4* pw = spw + jo;
  const float4* vv = reinterpret_cast<const float4*>(svr + jo);
  cf a[8];
  if constexpr (PIPE) {
#pragma unroll
    for (int b = 0; b < 8; ++b) a[b] = rowok ? __ldcg(col0 + (int64_t)b * n) : make_float2(0.f, 0.f);
  }
#pragma unroll 1
  for (int g8 = 0; g8 < 4; ++g8) {
    cf nx[8];
    if constexpr (PIPE) {
      if (g8 < 3) {
#pragma unroll
        for (int b = 0; b < 8; ++b)
          nx[b] = rowok ? __ldcg(col0 + (int64_t)((g8 + 1) * 8 + b) * n) : make_float2(0.f, 0.f);
      }
    } else {
#pragma unroll
      for (int b = 0; b < 8; ++b) a[b] = rowok ? __ldcg(col0 + (int64_t)(g8 * 8 + b) * n) : make_float2(0.f, 0.f);
    }
    float cr[8], ci[8];
    tile_group(a, pw + g8 * 8, vv + g8 * 4, vpr, wpr, vr, yr, yim, cr, ci);
    if (scol && g8 == 0) scol[row] = a[0];   // column o, the next step's
    if (rowok) {
#pragma unroll
      for (int b = 0; b < 8; ++b) col0[(int64_t)(g8 * 8 + b) * n] = a[b];
    }
    col_sums(cr, ci, lane);
    if ((lane & 3) == 0) part[(2 * t + 1) * 32 + g8 * 8 + (lane >> 2)] = make_float2(cr[0], ci[0]);
    if constexpr (PIPE) {
#pragma unroll
      for (int b = 0; b < 8; ++b) a[b] = nx[b];
    }
  }
  part[2 * t * 32 + lane] = make_float2(yr, yim);
}

// One eigenvector in global memory (column `col` of Z, row stride n) through
// one WY block of kNb reflectors starting at row k0 + 1: S = Yᴴ z, S ← T S,
// z −= Y S.  Y's rows are read as 16-byte pairs (sYb is 16-byte aligned) and
// the vector's elements kB rows ahead of their use.
__device__ __noinline__ void bt_vector(cf* Z, int n, int col, int k0, const cf* sYb, const cf* sT) {
  cf Sv[kNb];
#pragma unroll
  for (int jj = 0; jj < kNb; ++jj) Sv[jj] = make_float2(0.f, 0.f);
  constexpr int kB = 4;
  auto accum = [&](int row, const cf z) {
    const float4* y4 = reinterpret_cast<const float4*>(sYb + row * kNb);
#pragma unroll
    for (int q = 0; q < kNb / 2; ++q) {
      const float4 yy = y4[q];
      Sv[2 * q].x += yy.x * z.x + yy.y * z.y;
      Sv[2 * q].y += yy.x * z.y - yy.y * z.x;
      Sv[2 * q + 1].x += yy.z * z.x + yy.w * z.y;
      Sv[2 * q + 1].y += yy.z * z.y - yy.w * z.x;
    }
  };
  {
    int row = k0 + 1;
    for (; row + kB <= n; row += kB) {
      cf z[kB];
#pragma unroll
      for (int b = 0; b < kB; ++b) z[b] = __ldcg(Z + (int64_t)(row + b) * n + col);
#pragma unroll
      for (int b = 0; b < kB; ++b) accum(row + b, z[b]);
    }
    for (; row < n; ++row) accum(row, __ldcg(Z + (int64_t)row * n + col));
  }
  // T upper-triangular: S[a] is last needed by row a itself (in place)
#pragma unroll
  for (int a = 0; a < kNb; ++a) {
    cf sacc = make_float2(0.f, 0.f);
#pragma unroll
    for (int b = a; b < kNb; ++b) sacc = cadd(sacc, cmul(sT[a * kNb + b], Sv[b]));
    Sv[a] = sacc;
  }
  auto upd = [&](int row, cf z) {
    const float4* y4 = reinterpret_cast<const float4*>(sYb + row * kNb);
#pragma unroll
    for (int q = 0; q < kNb / 2; ++q) {
      const float4 yy = y4[q];
      z = csub(z, cmul(make_float2(yy.x, yy.y), Sv[2 * q]));
      z = csub(z, cmul(make_float2(yy.z, yy.w), Sv[2 * q + 1]));
    }
    return z;
  };
  int row = k0 + 1;
  for (; row + kB <= n; row += kB) {
    cf z[kB];
#pragma unroll
    for (int b = 0; b < kB; ++b) z[b] = __ldcg(Z + (int64_t)(row + b) * n + col);
#pragma unroll
    for (int b = 0; b < kB; ++b) z[b] = upd(row + b, z[b]);
#pragma unroll
    for (int b = 0; b < kB; ++b) Z[(int64_t)(row + b) * n + col] = z[b];
  }
  for (; row < n; ++row) Z[(int64_t)row * n + col] = upd(row, Z[(int64_t)row * n + col]);
}

// Upper-triangle slot q (column by column, column c holding rows 0..c−1) of a
// column-major n × n matrix: the split stage keeps the WY blocks' T factors in
// the strictly upper triangle of the patch's Gram buffer, which nothing reads
// between the tridiagonalisation and the back-transform (the W Gram rewrites
// the whole buffer afterwards).
__device__ __forceinline__ int64_t upper_slot(int n, int q) {
  int c = (int)((1.f + sqrtf(1.f + 8.f * (float)q)) * 0.5f);
  while (c > 1 && c * (c - 1) / 2 > q) --c;
  while ((c + 1) * c / 2 <= q) ++c;
  return (int64_t)c * n + (q - c * (c - 1) / 2);
}

// Entry (a, b), a <= b, of block blk's T factor: the blocks' upper triangles
// packed by columns.  Only the last block may have fewer than kNb columns, so
// all of them take n (n − 1) / 2 slots at most, what the upper triangle has.
__device__ __forceinline__ int64_t t_slot(int n, int blk, int a, int b) {
  return upper_slot(n, blk * (kNb * (kNb + 1) / 2) + b * (b + 1) / 2 + a);
}

// T factors (zlarft, forward columnwise) of the WY blocks of kNb reflectors,
// taken from the last reflector down as the back-transform applies them;
// block blk = (n − 1 − kend) / kNb goes to its slots of the upper triangle.
// sYb: n × kNb complex scratch followed by two kNb × kNb blocks.
__device__ void wy_factors(cf* A, int n, const float* taur, const float* taui, cf* sYb, int tid, int kT) {
  cf* sT = sYb + (int64_t)n * kNb;
  cf* sYY = sT + kNb * kNb;
  const int nref = n - 1;
  for (int kend = nref; kend > 0; kend -= kNb) {
    const int k0 = max(0, kend - kNb);
    const int nb = kend - k0;
    const int blk = (nref - kend) / kNb;
    const int m = n - k0 - 1;
    for (int q = tid; q < m * kNb; q += kT) {   // rows k0+1 .. n−1 of reflectors k0 .. k0+nb−1
      const int jj = q / m, row = k0 + 1 + (q - jj * m);
      const int k = k0 + jj;
      cf y = make_float2(0.f, 0.f);
      if (jj < nb) {
        if (row == k + 1) y = make_float2(1.f, 0.f);
        else if (row > k + 1) y = __ldcg(A + (int64_t)k * n + row);
      }
      sYb[row * kNb + jj] = y;
    }
    __syncthreads();
    for (int t = tid; t < kNb * kNb; t += kT) {   // Yᴴ Y
      const int a = t / kNb, b = t - a * kNb;
      float sr = 0.f, si = 0.f;
      for (int row = k0 + 1; row < n; ++row) {
        const cf ya = sYb[row * kNb + a], yb = sYb[row * kNb + b];
        sr += ya.x * yb.x + ya.y * yb.y;
        si += ya.x * yb.y - ya.y * yb.x;
      }
      sYY[t] = make_float2(sr, si);
    }
    __syncthreads();
    if (tid < 32) {   // lane a owns row a of T
      const int a = tid;
      for (int jj = 0; jj < kNb; ++jj) {
        const cf tj = (jj < nb) ? make_float2(taur[k0 + jj], taui[k0 + jj]) : make_float2(0.f, 0.f);
        if (a < jj) {
          cf sacc = make_float2(0.f, 0.f);
          for (int b = a; b < jj; ++b) sacc = cadd(sacc, cmul(sT[a * kNb + b], sYY[b * kNb + jj]));
          const cf v = cmul(tj, sacc);
          sT[a * kNb + jj] = make_float2(-v.x, -v.y);
        } else if (a < kNb) {
          sT[a * kNb + jj] = (a == jj) ? tj : make_float2(0.f, 0.f);
        }
        __syncwarp();
      }
    }
    __syncthreads();
    for (int t = tid; t < kNb * kNb; t += kT) {
      const int a = t / kNb, b = t - a * kNb;
      if (a <= b && b < nb) A[t_slot(n, blk, a, b)] = sT[t];
    }
    __syncthreads();
  }
}

// MODE 0: the whole stage in one launch.  MODE 1: phase 1 of the split stage
// (1024-thread variant) — d and e to the side buffer and the WY blocks' T
// factors to the Gram's upper triangle.
template <int MAXT, int MINB, int MODE>
__global__ void __launch_bounds__(MAXT, MINB) k_eig(EigArgs g) {
  extern __shared__ __align__(16) unsigned char smraw[];
  int s = 0;
  while (s + 1 < g.nseg && (int64_t)blockIdx.x >= g.seg[s + 1].first) ++s;
  const Seg& S = g.seg[s];
  const int n = S.n;
  const int64_t ip = (int64_t)blockIdx.x - S.first;
  const int tid = threadIdx.x;
  const int kT = blockDim.x;   // n <= blockDim.x
  cf* A = S.gram + ip * (int64_t)n * n;
  cf* Z = S.zv + ip * (int64_t)n * n;
  double* AUX = S.aux + ip * (int64_t)n * n;

  // shared layout (8-byte aligned pieces first); complex vectors hold n + 32 entries
  const int npad = n + 32;
  double* dd = reinterpret_cast<double*>(smraw);   // diagonal        [n]
  double* ee = dd + n;                              // off-diagonal    [n]
  double* ee2 = ee + n;                             // e²              [n]
  double* lam = ee2 + n;                            // eigenvalues     [n]
  double* redd = lam + n;                           // 64 doubles
  // the step's vectors again, indexed from the trailing block's first row o =
  // k + 1 (16-byte aligned, so a tile's eight columns load as vectors):
  // spw[j − o] = (vp_j, wp_j), svr[j − o] = v_j
  float4* spw = reinterpret_cast<float4*>(redd + 64);   //             [npad]
  cf* svr = reinterpret_cast<cf*>(spw + npad);           //             [npad]
  cf* sv = svr + npad;                              // v of this step  [npad]
  cf* svp = sv + npad;                              // previous v      [npad]
  cf* swp = svp + npad;                             // previous w      [npad]
  cf* scol = swp + npad;                            // next column     [npad]
  float* hv = reinterpret_cast<float*>(scol + npad); // h              [n]
  float* taur = hv + n;                             // τ               [n]
  float* taui = taur + n;                           //                 [n]
  float* red0 = taui + n;                           // 2 × 32 floats
  float* red1 = red0 + 32;
  cf* sY = reinterpret_cast<cf*>((reinterpret_cast<uintptr_t>(red1 + 32) + 15) & ~(uintptr_t)15);
  __shared__ cf s_x;
  __shared__ double s_bd[4];
  __shared__ int s_r;

  const bool full = S.lam_out != nullptr;
  const double beta_d = full ? 0.0 : g.thr[g.thr_per_patch ? (int64_t)blockIdx.x : 0] * S.lam;
  const float beta = (float)beta_d;
  (void)beta;

  const int i = tid;   // row owned by this thread (n <= kT)
  const int warp = tid >> 5, lane = tid & 31, nwarp = kT >> 5;
  // ---- 1. tridiagonalisation with delayed rank-2 updates ---------------------
  // The matrix scaled by a power of two first (PowerOfTwo): columns of an unscaled
  // one, squared, leave FP32 from 1e19 up and below 1e-19, where a pass over the
  // triangle costs one step of n.
  double down;
  {
    float q = i < n ? fabsf(__ldcg(&A[(int64_t)i * n + i].x)) : 0.f;
    for (int o = 16; o > 0; o >>= 1) q = fmaxf(q, __shfl_xor_sync(0xffffffffu, q, o));
    if (lane == 0) red1[warp] = q;
    __syncthreads();
    float dmax = 0.f;
    for (int w = 0; w < nwarp; ++w) dmax = fmaxf(dmax, red1[w]);
    const PowerOfTwo p(dmax);
    down = p.down;
    for (int c = warp; c < n; c += nwarp)
      for (int r = c + lane; r < n; r += 32) A[(int64_t)c * n + r] = cscale(__ldcg(A + (int64_t)c * n + r), p.up);
  }
  for (int q = tid; q < npad; q += kT) {
    sv[q] = make_float2(0.f, 0.f);
    svp[q] = make_float2(0.f, 0.f);
    swp[q] = make_float2(0.f, 0.f);
    svr[q] = make_float2(0.f, 0.f);
    spw[q] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
  __syncthreads();
  // per-tile row / column sums of the Hermitian matvec of a step: shared
  // memory (sharing the WY blocks' storage) for the 384-thread variant, the
  // patch's FP64 pivot scratch (idle until phase 3) for the large variant
  cf* part = (MAXT <= kSmallT) ? sY : reinterpret_cast<cf*>(AUX);
  // (vp, wp) of the pivot row k, known to every thread: row k's entries of the
  // previous step's v (1 when it reflected) and w (τ y_k − c), the latter from
  // the row sums every thread adds up itself, so no barrier publishes them
  cf vpk = make_float2(0.f, 0.f), wpk = make_float2(0.f, 0.f);
  for (int k = 0; k < n - 1; ++k) {
    // current column k and diagonal k: stored − (vp wpᴴ + wp vpᴴ); after the
    // first step the previous pass left the stored column in scol
    cf x = make_float2(0.f, 0.f);
    cf vpi = make_float2(0.f, 0.f), wpi = make_float2(0.f, 0.f);
    if (i < n) {
      vpi = svp[i];
      wpi = swp[i];
    }
    if (i >= k && i < n) {
      x = (k == 0) ? __ldcg(A + i) : scol[i];
      x = csub(x, cadd(cmul(vpi, cconj(wpk)), cmul(wpi, cconj(vpk))));
      if (i == k) dd[k] = (double)x.x * down;
    }
    if (i == k + 1) s_x = x;
    const float xn = block_sum((i >= k + 2 && i < n) ? cabs2(x) : 0.f, red0);
    // zlarfg, by every thread on the same values: Hᴴ (α, x) = (β, 0), H = I − τ v vᴴ, β real
    float tr, ti, sr, si;
    {
      const float ar = s_x.x, ai = s_x.y;
      float bt;
      if (xn + ai * ai <= kNoColumn) {   // (false for NaN)
        bt = ar;
        tr = ti = 0.f;
        sr = 1.f;
        si = 0.f;
      } else {
        bt = -copysignf(sqrtf(ar * ar + ai * ai + xn), ar);
        tr = (bt - ar) / bt;
        ti = -ai / bt;
        const float zr = ar - bt, zi = ai;
        const float den = zr * zr + zi * zi;
        sr = zr / den;
        si = -zi / den;
      }
      if (i == k + 1) {
        ee[k] = (double)bt * down;
        ee2[k] = ee[k] * ee[k];
        taur[k] = tr;
        taui[k] = ti;
      }
    }
    const cf tau = make_float2(tr, ti);
    const cf scal = make_float2(sr, si);
    const bool refl = (tau.x != 0.f || tau.y != 0.f);
    cf vi = make_float2(0.f, 0.f);
    if (i == k + 1) {
      vi = make_float2(1.f, 0.f);
    } else if (i >= k + 2 && i < n) {
      vi = cmul(x, scal);
      A[(int64_t)k * n + i] = vi;   // reflector kept below the subdiagonal
    }
    if (i < n) sv[i] = vi;
    if (i > k && i < n) svr[i - k - 1] = vi;
    __syncthreads();
    // fused over the trailing lower triangle [o, n)²: A22 ← A22 − (vp wpᴴ + wp vpᴴ)
    // and y = A22 v (Hermitian: element (r, c), r > c, also gives y_c += conj(a) v_r).
    {
      const int o = k + 1;
      const int T = (n - o + 31) >> 5;
      const int ntile = T * (T + 1) / 2;
      // work order: the T diagonal tiles (the costlier general path) first,
      // one per warp, then the off-diagonal tiles row by row; t is the
      // tile's slot in the partial sums (row-major over the triangle)
      for (int u = warp; u < ntile; u += nwarp) {
        int I, J;
        if (u < T) {
          I = J = u;
        } else {
          const int q = u - T;   // q-th tile strictly below the diagonal
          I = (int)((1.f + sqrtf(8.f * (float)q + 1.f)) * 0.5f);
          while (I > 1 && I * (I - 1) / 2 > q) --I;
          while ((I + 1) * I / 2 <= q) ++I;
          J = q - I * (I - 1) / 2;
        }
        const int t = I * (I + 1) / 2 + J;
        if (I != J) {   // off-diagonal tiles: every column inside the matrix
          full_tile<(MAXT <= kSmallT)>(A, n, o, I, J, t, lane, spw, svr, svp, swp, sv, part,
                                       J == 0 ? scol : nullptr);
          continue;
        }
        const bool diag = (I == J);
        const int row = o + I * 32 + lane;
        const bool rowok = row < n;
        const int rr = rowok ? row : n - 1;
        const cf vpr = svp[rr], wpr = swp[rr];
        const cf vr = rowok ? sv[rr] : make_float2(0.f, 0.f);
        float yr = 0.f, yim = 0.f;
        const int j0 = o + J * 32;
        cf* col0 = A + (int64_t)j0 * n + rr;
        for (int g8 = 0; g8 < 4; ++g8) {
          const int jb = j0 + g8 * 8;
          if (jb >= n) break;
          cf a[8];
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            const int j = jb + b;
            const bool ok = rowok && j < n && (!diag || row >= j);
            a[b] = ok ? __ldcg(col0 + (int64_t)(g8 * 8 + b) * n) : make_float2(0.f, 0.f);
          }
          float cr[8], ci[8];
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            const int j = jb + b;
            const bool ok = rowok && j < n && (!diag || row >= j);
            const cf vpj = svp[j], wpj = swp[j], vj = sv[j];
            cf e = a[b];
            e.x -= (vpr.x * wpj.x + vpr.y * wpj.y) + (wpr.x * vpj.x + wpr.y * vpj.y);
            e.y -= (vpr.y * wpj.x - vpr.x * wpj.y) + (wpr.y * vpj.x - wpr.x * vpj.y);
            if (!ok) e = make_float2(0.f, 0.f);
            a[b] = e;
            yr += e.x * vj.x - e.y * vj.y;
            yim += e.x * vj.y + e.y * vj.x;
            const bool low = !diag || row > j;   // strictly below the diagonal
            cr[b] = low ? (e.x * vr.x + e.y * vr.y) : 0.f;
            ci[b] = low ? (e.x * vr.y - e.y * vr.x) : 0.f;
          }
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            const int j = jb + b;
            if (rowok && j < n && (!diag || row >= j)) col0[(int64_t)(g8 * 8 + b) * n] = a[b];
          }
          if (J == 0 && g8 == 0 && rowok) scol[row] = a[0];   // column o, the next step's
          // column sums over the 32 lanes: lane l ends with the sum of column l/4
          const bool h16 = lane & 16, h8 = lane & 8, h4 = lane & 4;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float sr_ = h16 ? cr[q] : cr[q + 4], si_ = h16 ? ci[q] : ci[q + 4];
            const float kr = h16 ? cr[q + 4] : cr[q], ki = h16 ? ci[q + 4] : ci[q];
            cr[q] = kr + __shfl_xor_sync(0xffffffffu, sr_, 16);
            ci[q] = ki + __shfl_xor_sync(0xffffffffu, si_, 16);
          }
#pragma unroll
          for (int q = 0; q < 2; ++q) {
            const float sr_ = h8 ? cr[q] : cr[q + 2], si_ = h8 ? ci[q] : ci[q + 2];
            const float kr = h8 ? cr[q + 2] : cr[q], ki = h8 ? ci[q + 2] : ci[q];
            cr[q] = kr + __shfl_xor_sync(0xffffffffu, sr_, 8);
            ci[q] = ki + __shfl_xor_sync(0xffffffffu, si_, 8);
          }
          {
            const float sr_ = h4 ? cr[0] : cr[1], si_ = h4 ? ci[0] : ci[1];
            const float kr = h4 ? cr[1] : cr[0], ki = h4 ? ci[1] : ci[0];
            cr[0] = kr + __shfl_xor_sync(0xffffffffu, sr_, 4);
            ci[0] = ki + __shfl_xor_sync(0xffffffffu, si_, 4);
          }
          cr[0] += __shfl_xor_sync(0xffffffffu, cr[0], 2);
          ci[0] += __shfl_xor_sync(0xffffffffu, ci[0], 2);
          cr[0] += __shfl_xor_sync(0xffffffffu, cr[0], 1);
          ci[0] += __shfl_xor_sync(0xffffffffu, ci[0], 1);
          if ((lane & 3) == 0 && jb + (lane >> 2) < n)
            part[(2 * t + 1) * 32 + g8 * 8 + (lane >> 2)] = make_float2(cr[0], ci[0]);
        }
        part[2 * t * 32 + lane] = make_float2(yr, yim);
      }
    }
    __syncthreads();
    // y_i in a fixed order: the row sums of tiles (I, 0..I), then the column
    // sums of tiles (I..T-1, I) — the same bits on every run; every thread
    // also adds up y of row k + 1 (the next pivot row) in the same order
    float yr = 0.f, yi = 0.f, y1r = 0.f, y1i = 0.f;
    {
      const int o = k + 1, T = (n - o + 31) >> 5;
      if (i >= k + 1 && i < n) {
        const int I = (i - o) >> 5, l = (i - o) & 31;
        const int t0 = I * (I + 1) / 2;
        for (int J = 0; J <= I; ++J) {
          const cf v = part[2 * (t0 + J) * 32 + l];
          yr += v.x;
          yi += v.y;
        }
        for (int I2 = I; I2 < T; ++I2) {
          const cf v = part[(2 * (I2 * (I2 + 1) / 2 + I) + 1) * 32 + l];
          yr += v.x;
          yi += v.y;
        }
      }
      {
        const cf v = part[0];
        y1r += v.x;
        y1i += v.y;
      }
      for (int I2 = 0; I2 < T; ++I2) {
        const cf v = part[(2 * (I2 * (I2 + 1) / 2)) * 32 + 32];
        y1r += v.x;
        y1i += v.y;
      }
    }
    // vᴴ y (real for Hermitian A)
    const float vy = block_sum((i >= k + 1 && i < n) ? (vi.x * yr + vi.y * yi) : 0.f, red1);
    const float c = 0.5f * (tau.x * tau.x + tau.y * tau.y) * vy;
    // the next pivot row's (vp, wp); thread k + 1 stores these same values
    if (refl) {
      const cf ty = cmul(tau, make_float2(y1r, y1i));
      vpk = make_float2(1.f, 0.f);
      wpk = make_float2(ty.x - c, ty.y);
    } else {
      vpk = wpk = make_float2(0.f, 0.f);
    }
    if (i < n) {
      cf w = make_float2(0.f, 0.f);
      if (i == k + 1) {
        w = wpk;
      } else if (i > k + 1 && refl) {
        const cf ty = cmul(tau, make_float2(yr, yi));
        w = make_float2(ty.x - c * vi.x, ty.y - c * vi.y);
      }
      swp[i] = w;
      svp[i] = refl ? vi : make_float2(0.f, 0.f);
      if (i > k + 1) {
        const cf vq = refl ? vi : make_float2(0.f, 0.f);
        spw[i - k - 2] = make_float4(vq.x, vq.y, w.x, w.y);
      }
    }
    // no barrier here: the next step reads only this thread's own svp/swp
    // entries before its first block sum, and the reduction buffers of the
    // two sums differ
  }
  if (i == n - 1) {
    cf x = __ldcg(A + (int64_t)(n - 1) * n + (n - 1));
    const cf vpk = svp[n - 1], wpk = swp[n - 1];
    x = csub(x, cadd(cmul(vpk, cconj(wpk)), cmul(wpk, cconj(vpk))));
    dd[n - 1] = (double)x.x * down;
    ee[n - 1] = 0.0;
    ee2[n - 1] = 0.0;
  }
  __syncthreads();
  if constexpr (MODE == 1) {
    double* side = S.side + ip * 6 * (int64_t)n;
    for (int q = tid; q < n; q += kT) {
      side[q] = dd[q];
      side[n + q] = ee[q];
    }
    wy_factors(A, n, taur, taui, sY, tid, kT);
    return;
  }

  // ---- 2. eigenvalues above β² (FP64 multisection) ----------------------------
  if (tid == 0) {
    double gl = dd[0], gu = dd[0], emax2 = 0.0;
    for (int q = 0; q < n; ++q) {
      const double rr = (q > 0 ? fabs(ee[q - 1]) : 0.0) + (q < n - 1 ? fabs(ee[q]) : 0.0);
      gl = fmin(gl, dd[q] - rr);
      gu = fmax(gu, dd[q] + rr);
      if (q < n - 1) emax2 = fmax(emax2, ee2[q]);
    }
    const double tnorm = fmax(fabs(gl), fabs(gu));
    const double pivmin = fmax(2.2250738585072014e-308 * fmax(emax2, 1.0), 1e-290);
    const double pad = 2.0 * 2.220446049250313e-16 * tnorm * n + pivmin;
    gl -= pad;
    gu += pad;
    s_bd[0] = gl;
    s_bd[1] = gu;
    s_bd[2] = pivmin;
    s_bd[3] = tnorm;
    const double thr2 = beta_d * beta_d;
    s_r = full ? n : (thr2 >= gu) ? 0 : n - sturm_less(dd, ee2, n, thr2, pivmin);
  }
  __syncthreads();
  const int r = s_r;
  const double gl = full ? s_bd[0] : fmax(s_bd[0], beta_d * beta_d), gu = s_bd[1],
               pivmin = s_bd[2], tnorm = s_bd[3];
  if (tid == 0) S.rank[ip] = r;
  // FP32 copy of T scaled by 1/‖T‖ (in the phase-1 vector buffers, free now)
  const double tsc = fmax(tnorm, 1e-300);
  float* ddf = reinterpret_cast<float*>(sv);
  float* e2f = ddf + n;
  for (int q = tid; q < n; q += kT) {
    ddf[q] = (float)(dd[q] / tsc);
    e2f[q] = (float)(ee2[q] / tsc / tsc);
  }
  __syncthreads();
  {
    // A group of gsz threads (a power of two, at most a warp) per eigenvalue:
    // each round counts the eigenvalues below gsz evenly spaced interior
    // points of the bracket and keeps the sub-interval holding the
    // eigenvalue, a factor gsz + 1 per round of Sturm sequences instead of
    // bisection's 2.  The first rounds run on the FP32 copy; the bracket is
    // then widened by 4e-6·‖T‖ (far beyond the FP32 counts' error), checked
    // with two FP64 counts (the whole interval again if the check fails) and
    // narrowed in FP64 to 4e-13·‖T‖ — enough for the twisted factorisations'
    // vectors, whose error scales with |λ̂ − λ| / gap.
    int gsz = 1;
    while (gsz < 32 && 2 * gsz * r <= kT) gsz <<= 1;
    const int e = tid / gsz, sl = tid & (gsz - 1);
    if (warp * 32 < r * gsz) {   // whole warps, for the shuffles
      const int kth = n - 1 - e;   // e-th largest = kth smallest
      const double frac = (double)(sl + 1) / (double)(gsz + 1);
      double lo = gl, hi = gu;
      bool done = e >= r;
      if (tnorm > 0.0) {
        const float fracf = (float)frac;
        float lof = (float)(gl / tsc), hif = (float)(gu / tsc);
        bool fdone = done;
        for (int it = 0; it < 64; ++it) {
          if (!__any_sync(0xffffffffu, !fdone)) break;
          const float x = lof + (hif - lof) * fracf;
          const bool ok = !fdone && x > lof && x < hif;
          const bool up = ok && sturm_less_f(ddf, e2f, n, x) > kth;
          float nlo = (ok && !up) ? x : lof;
          float nhi = (ok && up) ? x : hif;
          int any = ok ? 1 : 0;
          for (int o = 1; o < gsz; o <<= 1) {
            nlo = fmaxf(nlo, __shfl_xor_sync(0xffffffffu, nlo, o));
            nhi = fminf(nhi, __shfl_xor_sync(0xffffffffu, nhi, o));
            any |= __shfl_xor_sync(0xffffffffu, any, o);
          }
          if (!fdone) {
            if (!any || !(nlo < nhi)) {
              fdone = true;
            } else {
              lof = nlo;
              hif = nhi;
            }
          }
        }
        lo = fmax(gl, ((double)lof - 4e-6) * tsc);
        hi = fmin(gu, ((double)hif + 4e-6) * tsc);
        // check the widened bracket in FP64: #{λ < lo} <= kth < #{λ < hi}
        int c = 0;
        if (!done) {
          if (gsz >= 2) c = (sl == 0) ? sturm_less(dd, ee2, n, lo, pivmin)
                          : (sl == 1) ? sturm_less(dd, ee2, n, hi, pivmin) : 0;
          else c = sturm_less(dd, ee2, n, lo, pivmin);
        }
        const int base = (lane & ~(gsz - 1));
        const int cl = (gsz >= 2) ? __shfl_sync(0xffffffffu, c, base) : c;
        int ch = (gsz >= 2) ? __shfl_sync(0xffffffffu, c, base + 1) : 0;
        if (gsz < 2 && !done) ch = sturm_less(dd, ee2, n, hi, pivmin);
        if (!done && !(cl <= kth && ch > kth)) {
          lo = gl;
          hi = gu;
        }
      }
      const double tol = 4e-13 * tnorm;
      for (int it = 0; it < 200; ++it) {
        if (!done && !(hi - lo > tol)) done = true;
        if (!__any_sync(0xffffffffu, !done)) break;
        const double x = lo + (hi - lo) * frac;
        const bool ok = !done && x > lo && x < hi;
        const bool up = ok && sturm_less(dd, ee2, n, x, pivmin) > kth;   // eigenvalue below x
        double nlo = (ok && !up) ? x : lo;
        double nhi = (ok && up) ? x : hi;
        int any = ok ? 1 : 0;
        for (int o = 1; o < gsz; o <<= 1) {
          nlo = fmax(nlo, __shfl_xor_sync(0xffffffffu, nlo, o));
          nhi = fmin(nhi, __shfl_xor_sync(0xffffffffu, nhi, o));
          any |= __shfl_xor_sync(0xffffffffu, any, o);
        }
        if (!done) {
          if (!any || !(nlo < nhi)) {
            done = true;
          } else {
            lo = nlo;
            hi = nhi;
          }
        }
      }
      if (e < r && sl == 0) {
        const double lm = 0.5 * (lo + hi);
        lam[e] = lm;
        const double sg = sqrt(fmax(lm, 0.0));
        hv[e] = (sg > beta_d && sg > 0.0) ? (float)((sg - beta_d) / sg) : 0.f;
      }
    }
  }
  __syncthreads();
  if (S.nuc) {   // nuclear norm of the patch (src/recon.jl:138-146): Σ σ_i = Σ √λ_i
    const double sq = (tid < r) ? sqrt(fmax(lam[tid], 0.0)) : 0.0;
    const double tot = block_sum_d(sq, redd);
    if (tid == 0) S.nuc[ip] = tot;
    return;
  }
  if (r == 0) {
    for (int64_t q = tid; q < (int64_t)n * n; q += kT) Z[q] = make_float2(0.f, 0.f);
    return;
  }

  // Up to g.rz eigenvectors live in shared memory from here to the output
  // ([row][vector], row stride rz); more use the patch's global slots (row
  // stride n).  zb / zs address them either way.
  const bool stg = r <= g.rz;
  const int64_t zs = stg ? g.rz : n;
  cf* zb = stg ? sY : Z;

  // ---- 3. eigenvectors of T (FP64 twisted factorisation) --------------------
  // z_j in the vector slots read as doubles, D+ after them (shared) or in
  // AUX (global); finally converted in place to complex float.
  if (tid < r) {
    const double lm = lam[tid];
    double* zd = reinterpret_cast<double*>(zb) + tid;
    double* dp = (stg ? reinterpret_cast<double*>(zb) + (int64_t)n * zs : AUX) + tid;
    double q = dd[0] - lm;
    if (fabs(q) < pivmin) q = -pivmin;
    dp[0] = q;
    for (int j = 0; j + 1 < n; ++j) {
      q = dd[j + 1] - lm - ee2[j] / q;
      if (fabs(q) < pivmin) q = -pivmin;
      dp[(int64_t)(j + 1) * zs] = q;
    }
    q = dd[n - 1] - lm;
    if (fabs(q) < pivmin) q = -pivmin;
    zd[(int64_t)(n - 1) * zs] = q;
    int kb = n - 1;
    double gb = fabs(dp[(int64_t)(n - 1) * zs] + q - (dd[n - 1] - lm));
    for (int j = n - 2; j >= 0; --j) {
      q = dd[j] - lm - ee2[j] / q;
      if (fabs(q) < pivmin) q = -pivmin;
      zd[(int64_t)j * zs] = q;
      const double gm = fabs(dp[(int64_t)j * zs] + q - (dd[j] - lm));
      if (gm < gb) {
        gb = gm;
        kb = j;
      }
    }
    int b0 = 0, b1 = n - 1;
    if (const int t = tie_of(lam, r, tid, 1e-12 * fmax(tnorm, 1e-300)); t >= 0) {
      const Twist w = tied_twist(
          n, t, ee, tnorm,
          [=](int k) { return fabs(dp[(int64_t)k * zs] + zd[(int64_t)k * zs] - (dd[k] - lm)); },
          [=](int j) { return ee[j] / dp[(int64_t)j * zs]; }, [=](int j) { return ee[j - 1] / zd[(int64_t)j * zs]; });
      if (w.k >= 0) {
        kb = w.k;
        b0 = w.b0;
        b1 = w.b1;
      }
    }
    double nrm = 1.0, zp = 1.0;
    for (int j = kb - 1; j >= 0; --j) {   // z_j = −e_j z_{j+1} / D+_j
      zp = j < b0 ? 0.0 : -ee[j] * zp / dp[(int64_t)j * zs];
      zd[(int64_t)j * zs] = zp;
      nrm += zp * zp;
    }
    zd[(int64_t)kb * zs] = 1.0;
    zp = 1.0;
    for (int j = kb + 1; j < n; ++j) {    // z_j = −e_{j−1} z_{j−1} / D−_j
      zp = j > b1 ? 0.0 : -ee[j - 1] * zp / zd[(int64_t)j * zs];
      zd[(int64_t)j * zs] = zp;
      nrm += zp * zp;
    }
    const double inv = 1.0 / sqrt(nrm);
    cf* zc = zb + tid;
    for (int j = 0; j < n; ++j) {
      const double zj = zd[(int64_t)j * zs];
      zc[(int64_t)j * zs] = make_float2((float)(zj * inv), 0.f);
    }
  }
  __syncthreads();
  // Eigenvalues equal to working precision: Gram–Schmidt inside the cluster,
  // cooperatively (every thread walks the same clusters).
  {
    const double ctol = 1e-12 * fmax(tnorm, 1e-300);
    int s0 = 0;
    int rb = 0;
    while (s0 < r) {
      int t = s0 + 1;
      while (t < r && lam[t - 1] - lam[t] <= ctol) ++t;
      for (int qv = s0 + 1; qv < t; ++qv) {
        for (int attempt = 0; attempt < 4; ++attempt) {
          for (int pv = s0; pv < qv; ++pv) {
            double dot = 0.0;
            for (int j = tid; j < n; j += kT) dot += (double)zb[j * zs + pv].x * zb[j * zs + qv].x;
            dot = block_sum_d(dot, redd + 32 * (rb++ & 1));
            for (int j = tid; j < n; j += kT) zb[j * zs + qv].x -= (float)dot * zb[j * zs + pv].x;
            __syncthreads();
          }
          double nr = 0.0;
          for (int j = tid; j < n; j += kT) nr += (double)zb[j * zs + qv].x * zb[j * zs + qv].x;
          nr = sqrt(block_sum_d(nr, redd + 32 * (rb++ & 1)));
          if (nr > 0.1) {
            for (int j = tid; j < n; j += kT) zb[j * zs + qv].x /= (float)nr;
            __syncthreads();
            break;
          }
          // collapsed onto earlier vectors: restart from a unit vector
          for (int j = tid; j < n; j += kT)
            zb[j * zs + qv].x = (j == (qv + attempt * 7919) % n) ? 1.f : 0.f;
          __syncthreads();
        }
      }
      s0 = t;
    }
  }
  // ---- 4. V = H_0 ⋯ H_{n-2} Z, blocks of kNb reflectors from the last ---------
  // Staged vectors (few): every thread takes part — S = Yᴴ Z by (output, row
  // group) partial sums added in a fixed order, S ← T S, then Z −= Y S by
  // (row, vector) element, in passes of kCW vectors.  Vectors in global
  // memory (many): thread i updates vector i with its block coefficients in
  // registers.
  // Y: n × kNb, [row][reflector], after the vector stage (16-byte aligned)
  cf* sYb = sY + (((int64_t)n * g.rz + 1) & ~(int64_t)1);
  cf* sT = sYb + (int64_t)n * kNb;    // kNb × kNb, T[a][b] at a*kNb + b
  cf* sYY = sT + kNb * kNb;           // Yᴴ Y
  cf* sS = sYY + kNb * kNb;           // kNb × kCW
  cf* sS2 = sS + kNb * kCW;           // T S
  cf* sP = sS2 + kNb * kCW;           // partial sums, one per thread
  const int nref = n - 1;
  for (int kend = nref; kend > 0; kend -= kNb) {
    const int k0 = max(0, kend - kNb);
    const int nb = kend - k0;
    for (int q = tid; q < n * kNb; q += kT) {   // Y: column jj = reflector k0 + jj
      const int row = q / kNb, jj = q - row * kNb;
      const int k = k0 + jj;
      cf y = make_float2(0.f, 0.f);
      if (jj < nb) {
        if (row == k + 1) y = make_float2(1.f, 0.f);
        else if (row > k + 1) y = A[(int64_t)k * n + row];
      }
      sYb[q] = y;
    }
    __syncthreads();
    if (tid < kNb * kNb) {   // Yᴴ Y
      const int a = tid / kNb, b = tid - a * kNb;
      float sr = 0.f, si = 0.f;
      for (int row = k0 + 1; row < n; ++row) {
        const cf ya = sYb[row * kNb + a], yb = sYb[row * kNb + b];
        sr += ya.x * yb.x + ya.y * yb.y;
        si += ya.x * yb.y - ya.y * yb.x;
      }
      sYY[tid] = make_float2(sr, si);
    }
    __syncthreads();
    if (tid < 32) {   // zlarft (forward, columnwise); lane a owns row a of T
      const int a = tid;
      for (int jj = 0; jj < kNb; ++jj) {
        const cf tj = (jj < nb) ? make_float2(taur[k0 + jj], taui[k0 + jj]) : make_float2(0.f, 0.f);
        if (a < jj) {
          cf sacc = make_float2(0.f, 0.f);
          for (int b = a; b < jj; ++b) sacc = cadd(sacc, cmul(sT[a * kNb + b], sYY[b * kNb + jj]));
          const cf v = cmul(tj, sacc);
          sT[a * kNb + jj] = make_float2(-v.x, -v.y);
        } else if (a < kNb) {
          sT[a * kNb + jj] = (a == jj) ? tj : make_float2(0.f, 0.f);
        }
        __syncwarp();
      }
    }
    __syncthreads();
    if (!stg) {   // vectors in global memory: thread tid updates vector tid (S = Yᴴ z; S ← T S; z −= Y S)
      if (tid < r) bt_vector(Z, n, tid, k0, sYb, sT);
      __syncthreads();
      continue;
    }
    // vectors staged in shared memory: every thread takes part
    for (int c0 = 0; c0 < r; c0 += kCW) {
      const int cw = min(kCW, r - c0);
      const int no = kNb * cw;   // outputs of S = Yᴴ Z (at most 256 <= threads)
      const int ng = kT / no;    // row groups
      if (tid < no * ng) {
        const int o = tid % no, grp = tid / no;
        const int jj = o / cw, c = c0 + (o - jj * cw);
        float sr = 0.f, si = 0.f;
        for (int row = k0 + 1 + grp; row < n; row += ng) {
          const cf y = sYb[row * kNb + jj], z = zb[row * zs + c];   // conj(y)·z
          sr += y.x * z.x + y.y * z.y;
          si += y.x * z.y - y.y * z.x;
        }
        sP[tid] = make_float2(sr, si);
      }
      __syncthreads();
      if (tid < no) {
        float sr = 0.f, si = 0.f;
        for (int gq = 0; gq < ng; ++gq) {
          sr += sP[gq * no + tid].x;
          si += sP[gq * no + tid].y;
        }
        sS[tid] = make_float2(sr, si);
      }
      __syncthreads();
      if (tid < no) {   // T upper-triangular
        const int a = tid / cw, c = tid - a * cw;
        cf sacc = make_float2(0.f, 0.f);
        for (int b = a; b < kNb; ++b) sacc = cadd(sacc, cmul(sT[a * kNb + b], sS[b * cw + c]));
        sS2[tid] = sacc;
      }
      __syncthreads();
      const int rows = n - (k0 + 1);
      for (int q = tid; q < rows * cw; q += kT) {
        const int rr = q / cw, c = q - rr * cw;
        const int row = k0 + 1 + rr;
        cf* zp = zb + row * zs + c0 + c;
        cf z = *zp;
#pragma unroll
        for (int jj = 0; jj < kNb; ++jj) z = csub(z, cmul(sYb[row * kNb + jj], sS2[jj * cw + c]));
        *zp = z;
      }
      __syncthreads();
    }
  }

  // ---- 5. Ṽ = conj(V) diag(√h), columns >= r zero ------------------------------
  if (full) {   // V itself and the eigenvalues
    for (int c = tid; c < n; c += kT) S.lam_out[ip * n + c] = lam[c];
    for (int row = 0; row < n; ++row)
      for (int c = tid; c < n; c += kT) Z[(int64_t)row * n + c] = zb[row * zs + c];
    return;
  }
  for (int row = 0; row < n; ++row) {
    for (int c = tid; c < n; c += kT) {
      cf v = make_float2(0.f, 0.f);
      if (c < r) {
        const cf z = zb[row * zs + c];
        const float sh = sqrtf(hv[c]);
        v = make_float2(z.x * sh, -z.y * sh);
      }
      Z[(int64_t)row * n + c] = v;
    }
  }
}

// ---- tridiagonalisation with the matrix in registers (n <= 128) -------------------
// Phase 1 for Gram sides up to 32·NT: the warps hold the whole Hermitian
// matrix, one tile of 32 rows × 4·CU columns per warp, lane (rg, cg) rows rg +
// 8t and columns cg + 4u of it.  A step is what k_eig's is — the previous
// rank-2 update applied on the fly while y = A v is formed — but nothing but
// vectors moves: the tile pass is six packed FMAs per value on registers with
// the column's (v, w) from shared memory, and both triangles are stored, so a
// row's sum is a thread's own and needs no transposed partial sums.
// Two barriers a step: the column x and its norm's partial sums before the
// tile pass (which works on the unscaled reflector u = (α − β, x), v = u / (α
// − β), so no second round publishes v), and the partial sums of A u and of
// uᴴ A u after it (so no third one reduces vᴴ y).
// That sum is of the third power of the matrix, so the matrix is scaled to
// order one first (PowerOfTwo): unscaled, in FP32, it overflowed for entries
// from 1e11 on (n = 300) and lost its bits below 2e-13.
// With the matrix in L2 a step cost 5.6 µs whatever n was (n = 64, one
// patch: 351 µs), the latency of its round trips and four barriers.
// A warp's tile column is rotated by its tile row, so that the tiles left in
// play when the leading ones are done stay spread over the SM's schedulers.
// The tile pass is as much shared-memory loads as FMAs: a 16-byte load takes
// the pipe four cycles, so (v, w) of a row or column come in one, without the
// doubled components that a packed FMA would take directly (those are moves,
// for which the FMAs leave issue slots), and the reflector's scalars that only
// the vector phases need are worked out by their warps alone: 148 matrices of
// side 128 252 -> 227 us, 216 of side 64 99 -> 94 (by the profiler now 221 and 89,
// 218 and 89 without the scaling).
// CU columns per lane: tiles of 32 rows × 4·CU columns, one per warp.  Eight is
// what 16 warps' registers hold at NT = 4; with four the smaller sides have
// twice the warps, so the latencies of a tile pass overlap.
constexpr int tri_cu(int nt) { return nt == 4 ? 8 : 4; }
template <int NT>
struct TriVec {
  static constexpr int NP = 32 * NT, LD = NP + 1, CU = tri_cu(NT), TC = 4 * CU, NTC = NP / TC;
  static constexpr int kThreads = NT * NTC * 32;
  float4 vw[NP];          // the pending update, by row: (vp, wp)
  cf sx[NP];              // this step's column x below the subdiagonal
  cf scol[NP];            // next column, before the pending update
  cf part[NTC][NP];       // per tile column: partial sums of A u
  float red0[4], redt[NT * NTC];
  cf x1;
};

// zlarfg with α = (ar, ai) and ‖x‖² = xn: Hᴴ (α, x) = (β, 0), H = I − τ v vᴴ, β
// real, v = (1, x / u₁), u₁ = α − β.  The root and its reciprocal come from one
// approximation, each refined to the last bit by a Newton step (shorter than a
// root followed by a division by it).
struct Reflector {
  float b, ib;   // β, 1/β
  __device__ __forceinline__ Reflector(float ar, float ai, float xn) {
    const float s = ar * ar + ai * ai + xn;
    float r = rsqrtf(s);
    r = fmaf(0.5f * r, fmaf(-s * r, r, 1.f), r);
    float q = s * r;
    q = fmaf(0.5f * r, fmaf(-q, q, s), q);
    b = -copysignf(q, ar);
    ib = -copysignf(r, ar);
  }
  __device__ __forceinline__ cf u1(float ar, float ai) const { return make_float2(ar - b, ai); }
  __device__ __forceinline__ cf tau(float ar, float ai) const { return make_float2((b - ar) * ib, -ai * ib); }
};
// 1 / u₁
__device__ __forceinline__ cf inverse(cf u) {
  const float id = __frcp_rn(u.x * u.x + u.y * u.y);
  return make_float2(u.x * id, -u.y * id);
}

// The n steps of the n × n Hermitian matrix at A (column stride ld, n <= 32·NT,
// lower triangle read): d, e and τ; reflectors below A's subdiagonal and, when
// given, in Y (unit entry and zeros included).  TriVec<NT>::kThreads threads.
// SCALE: the matrix is scaled here (PowerOfTwo), else it has been; d and e are
// scaled back by `down`, which SCALE sets.
template <int NT, bool SCALE>
__device__ __forceinline__ void tri_steps(cf* A, int ld, int n, TriVec<NT>& m, double* dd, double* ee, cf* taus,
                                          cf* Y, double down) {
  constexpr int NP = 32 * NT, LD = TriVec<NT>::LD, CU = TriVec<NT>::CU, TC = TriVec<NT>::TC, NTC = TriVec<NT>::NTC;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int I = warp / NTC, J = (warp + I) % NTC;
  const int rg = lane >> 2, cg = lane & 3;

  // the tile, from the lower triangle
  cf a[4][CU];
#pragma unroll
  for (int t = 0; t < 4; ++t)
#pragma unroll
    for (int u = 0; u < CU; ++u) {
      const int r = I * 32 + rg + 8 * t, c = J * TC + cg + 4 * u;
      cf v = make_float2(0.f, 0.f);
      if (r < n && c < n) {
        v = r >= c ? __ldcg(A + (int64_t)c * ld + r) : __ldcg(A + (int64_t)r * ld + c);
        if (r < c) v.y = -v.y;
        if (r == c) v.y = 0.f;
      }
      a[t][u] = v;
    }
  const int i = tid;                 // row of the vector phases
  const bool own = tid < NP;         // (the first NT warps)
  float up = 1.f;
  if constexpr (SCALE) {
    if (own) {
      float q = i < n ? fabsf(__ldcg(&A[(int64_t)i * ld + i].x)) : 0.f;
      for (int o = 16; o > 0; o >>= 1) q = fmaxf(q, __shfl_xor_sync(0xffffffffu, q, o));
      if (lane == 0) m.redt[warp] = q;   // (next written after the first step's barrier)
    }
    __syncthreads();
    float dmax = 0.f;
#pragma unroll
    for (int q = 0; q < NT; ++q) dmax = fmaxf(dmax, m.redt[q]);
    const PowerOfTwo p(dmax);
    up = p.up;
    down = p.down;
#pragma unroll
    for (int t = 0; t < 4; ++t)
#pragma unroll
      for (int u = 0; u < CU; ++u) a[t][u] = cscale(a[t][u], up);
  }
  if (own) {
    m.vw[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    m.scol[i] = (i < n) ? cscale(__ldcg(A + i), up) : make_float2(0.f, 0.f);
  }
  const int row = I * 32 + rg + 8 * cg;   // row whose sum this lane ends with
  cf vpi = make_float2(0.f, 0.f), wpi = vpi, vpk = vpi, wpk = vpi;
  for (int k = 0; k < n - 1; ++k) {
    // column k with the pending update; its norm below the subdiagonal
    cf x = make_float2(0.f, 0.f);
    if (own) {
      if (i >= k && i < n) x = csub(m.scol[i], cadd(cmul(vpi, cconj(wpk)), cmul(wpi, cconj(vpk))));
      if (i == k) dd[k] = (double)x.x * down;
      if (i == k + 1) m.x1 = x;
      if (i <= k + 1) x = make_float2(0.f, 0.f);
      m.sx[i] = x;
      const float q = warp_sum(cabs2(x));
      if (lane == 0) m.red0[warp] = q;
    }
    __syncthreads();
    float xn = 0.f;
#pragma unroll
    for (int q = 0; q < NT; ++q) xn += m.red0[q];
    // the reflector, by every thread on the same values: all need u1, those
    // of the vector phases the rest, worked out here, under the tiles' work
    const float ar = m.x1.x, ai = m.x1.y;
    float bt = ar;
    cf tau = make_float2(0.f, 0.f), scal = tau, u1 = tau;
    const bool refl = !(xn + ai * ai <= kNoColumn);   // (true for NaN)
    if (refl) {
      const Reflector h(ar, ai, xn);
      u1 = h.u1(ar, ai);
      if (own) {
        bt = h.b;
        tau = h.tau(ar, ai);
        scal = inverse(u1);
        asm volatile("" : "+f"(scal.x), "+f"(scal.y), "+f"(tau.x), "+f"(tau.y));
      }
    }
    // A ← A − (vp wpᴴ + wp vpᴴ), A u on the tiles still in play
    float tq = 0.f;
    if (I * 32 + 31 > k && J * TC + TC - 1 > k) {
      const int c0 = J * TC + cg;
      {
        cf r1[4], r2[4], r3[4], r4[4];   // −(vp), −(vp rotated), −(wp), −(wp rotated) of the rows
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float4 q = m.vw[I * 32 + rg + 8 * t];
          r1[t] = make_float2(-q.x, -q.y);
          r2[t] = make_float2(-q.y, q.x);
          r3[t] = make_float2(-q.z, -q.w);
          r4[t] = make_float2(-q.w, q.z);
        }
#pragma unroll
        for (int u = 0; u < CU; ++u) {   // a −= vp conj(wp_j) + wp conj(vp_j)
          const float4 q = m.vw[c0 + 4 * u];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            cf e = a[t][u];
            e = __ffma2_rn(r1[t], make_float2(q.z, q.z), e);
            e = __ffma2_rn(r2[t], make_float2(q.w, q.w), e);
            e = __ffma2_rn(r3[t], make_float2(q.x, q.x), e);
            a[t][u] = __ffma2_rn(r4[t], make_float2(q.y, q.y), e);
          }
        }
      }
      cf y[4];
      {
        cf P[4], Q[4];   // (Σ a.x x.x, Σ a.y x.y), (Σ a.x x.y, Σ a.y x.x)
#pragma unroll
        for (int t = 0; t < 4; ++t) P[t] = Q[t] = make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < CU; ++u) {
          const cf v = m.sx[c0 + 4 * u];
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            P[t] = __ffma2_rn(a[t][u], v, P[t]);
            Q[t] = __ffma2_rn(a[t][u], make_float2(v.y, v.x), Q[t]);
          }
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) y[t] = make_float2(P[t].x - P[t].y, Q[t].x + Q[t].y);
      }
      if (J == (k + 1) / TC) {   // column k + 1: entry u1 of u, and the next step's column
        const int us = ((k + 1) % TC) >> 2;
        cf nx[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) nx[t] = a[t][0];
#pragma unroll
        for (int u = 1; u < CU; ++u)
          if (u == us) {
#pragma unroll
            for (int t = 0; t < 4; ++t) nx[t] = a[t][u];
          }
        if (cg == ((k + 1) & 3)) {
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            m.scol[I * 32 + rg + 8 * t] = nx[t];
            y[t] = cadd(y[t], cmul(nx[t], u1));
          }
        }
      }
      // sums over the four column groups; lane cg ends with row t = cg
      const bool h2 = cg & 2, h1 = cg & 1;
      cf z0 = h2 ? y[2] : y[0], z1 = h2 ? y[3] : y[1];
      const cf o0 = h2 ? y[0] : y[2], o1 = h2 ? y[1] : y[3];
      z0.x += __shfl_xor_sync(0xffffffffu, o0.x, 2);
      z0.y += __shfl_xor_sync(0xffffffffu, o0.y, 2);
      z1.x += __shfl_xor_sync(0xffffffffu, o1.x, 2);
      z1.y += __shfl_xor_sync(0xffffffffu, o1.y, 2);
      cf z = h1 ? z1 : z0;
      const cf o = h1 ? z0 : z1;
      z.x += __shfl_xor_sync(0xffffffffu, o.x, 1);
      z.y += __shfl_xor_sync(0xffffffffu, o.y, 1);
      m.part[J][row] = z;
      const cf ur = row == k + 1 ? u1 : m.sx[row];
      tq = warp_sum(ur.x * z.x + ur.y * z.y);   // uᴴ A u is real
    }
    if (lane == 0) m.redt[warp] = tq;
    __syncthreads();
    if (own) {
      // y = A v of this row and of row k + 1 (the next pivot row), in tile order
      cf y = make_float2(0.f, 0.f), y1 = y;
      const int q0 = (k + 1) / TC;
#pragma unroll
      for (int q = 0; q < NTC; ++q)
        if (q >= q0) {
          y = cadd(y, m.part[q][i]);
          y1 = cadd(y1, m.part[q][k + 1]);
        }
      float t = 0.f;
#pragma unroll
      for (int q = 0; q < NT * NTC; ++q) t += m.redt[q];
      const float c = 0.5f * (tau.x * tau.x + tau.y * tau.y) * (scal.x * scal.x + scal.y * scal.y) * t;
      const cf vi = i == k + 1 ? make_float2(1.f, 0.f) : cmul(x, scal);   // 0 for i <= k and i >= n
      if (i == k + 1) {
        ee[k] = (double)bt * down;
        taus[k] = tau;
      }
      if (Y) Y[k * LD + i] = vi;
      if (i >= k + 2 && i < n) A[(int64_t)k * ld + i] = vi;   // reflector kept below the subdiagonal
      vpi = vpk = wpi = wpk = make_float2(0.f, 0.f);
      if (refl) {
        const cf ts = cmul(tau, scal);
        const cf t1 = cmul(ts, y1), ty = cmul(ts, y);
        vpk = make_float2(1.f, 0.f);
        wpk = make_float2(t1.x - c, t1.y);
        if (i > k && i < n) {
          vpi = vi;
          wpi = make_float2(ty.x - c * vi.x, ty.y - c * vi.y);
        }
      }
      m.vw[i] = make_float4(vpi.x, vpi.y, wpi.x, wpi.y);
    }
    // what the next step's first phase reads was written before the last
    // barrier or is this thread's own
  }
  if (own && i == n - 1) {
    const cf x = csub(m.scol[i], cadd(cmul(vpi, cconj(wpi)), cmul(wpi, cconj(vpi))));
    dd[n - 1] = (double)x.x * down;
    ee[n - 1] = 0.0;
  }
  __syncthreads();
}

// Row `lane` of the T factor (zlarft, forward columnwise) of one WY block by
// one warp: tau of its nb reflectors, G the products Yᴴ Y above the diagonal,
// column by column; into the block's upper slots of A.
__device__ __forceinline__ void wy_tfactor(cf* A, int n, int blk, const cf* tau, int nb, const cf* G) {
  const int lane = threadIdx.x & 31;
  cf t[kNb];
#pragma unroll
  for (int jj = 0; jj < kNb; ++jj) {
    const cf tj = jj < nb ? tau[jj] : make_float2(0.f, 0.f);
    cf sacc = make_float2(0.f, 0.f);
#pragma unroll
    for (int b = 0; b < jj; ++b) sacc = cadd(sacc, cmul(t[b], G[jj * (jj - 1) / 2 + b]));
    const cf v = cmul(tj, sacc);
    t[jj] = lane == jj ? tj : lane < jj ? make_float2(-v.x, -v.y) : make_float2(0.f, 0.f);
  }
  if (lane < kNb) {
#pragma unroll
    for (int jj = 0; jj < kNb; ++jj)
      if (lane <= jj && jj < nb) A[t_slot(n, blk, lane, jj)] = t[jj];
  }
}
// entry e of a block's G: column jj, row b < jj
__device__ __forceinline__ void g_entry(int e, int* jj, int* b) {
  int j = 1;
  while ((j + 1) * j / 2 <= e) ++j;
  *jj = j;
  *b = e - j * (j - 1) / 2;
}

template <int NT>
struct TriSmem {
  TriVec<NT> v;
  double dd[32 * NT], ee[32 * NT];
  cf tau[32 * NT];
  cf Y[32 * NT * TriVec<NT>::LD];   // reflectors, Y[k·LD + i]
  cf G[NT * 2][120];                // per WY block: Yᴴ Y above the diagonal
};

template <int NT>
__global__ void __launch_bounds__(TriVec<NT>::kThreads, NT == 1 ? 8 : NT == 2 ? 2 : 1) k_tri_reg(EigArgs g) {
  extern __shared__ __align__(16) unsigned char smraw[];
  TriSmem<NT>& m = *reinterpret_cast<TriSmem<NT>*>(smraw);
  int s = 0;
  while (s + 1 < g.nseg && (int64_t)blockIdx.x >= g.seg[s + 1].first) ++s;
  const Seg& S = g.seg[s];
  const int n = S.n;
  const int64_t ip = (int64_t)blockIdx.x - S.first;
  constexpr int kThreads = TriVec<NT>::kThreads, LD = TriVec<NT>::LD;
  const int tid = threadIdx.x, warp = tid >> 5;
  cf* A = S.gram + ip * (int64_t)n * n;
  tri_steps<NT, true>(A, n, n, m.v, m.dd, m.ee, m.tau, m.Y, 1.0);
  double* side = S.side + ip * 6 * (int64_t)n;
  for (int q = tid; q < n; q += kThreads) {
    side[q] = m.dd[q];
    side[n + q] = m.ee[q];
  }
  // the T factors of all WY blocks, from the last reflector down: the products
  // Yᴴ Y of every block at once, then one warp per block
  const int nref = n - 1, nblk = (nref + kNb - 1) / kNb;
  for (int q = tid; q < nblk * 120; q += kThreads) {
    const int blk = q / 120, e = q - blk * 120;
    int jj, b;
    g_entry(e, &jj, &b);
    const int kend = nref - blk * kNb, k0 = max(0, kend - kNb);
    float sr = 0.f, si = 0.f;
    if (jj < kend - k0) {
      const cf* ya = m.Y + (k0 + b) * LD;
      const cf* yb = m.Y + (k0 + jj) * LD;
#pragma unroll 8
      for (int row = k0 + jj + 1; row < n; ++row) {
        sr += ya[row].x * yb[row].x + ya[row].y * yb[row].y;
        si += ya[row].x * yb[row].y - ya[row].y * yb[row].x;
      }
    }
    m.G[blk][e] = make_float2(sr, si);
  }
  __syncthreads();
  for (int blk = warp; blk < nblk; blk += kThreads / 32) {
    const int kend = nref - blk * kNb, k0 = max(0, kend - kNb);
    wy_tfactor(A, n, blk, m.tau + k0, kend - k0, m.G[blk]);
  }
}

// ---- blocked tridiagonalisation (128 < n <= 384) --------------------------------------
// The leading n − 128 columns in panels of eight with the matrix in L2, the
// trailing 128 × 128 block in registers (tri_steps).  Within a panel the
// matrix is only read: column k gets its pending updates from the panel's V
// and W in shared memory, and y = A u − V (Wᴴ u) − W (Vᴴ u); the rank-16 update
// of the trailing lower triangle follows at the panel's end.  k_eig reads and
// writes the triangle every step instead, and spends most of its time on
// per-tile bookkeeping (486 patches of side 300: 12.7 ms).
// The matrix–vector product reads the lower triangle once, in groups of 64
// rows × 8 columns (lane = two rows, eight 16-byte loads in flight): each value
// serves its row (kept in the lane while the warp's groups stay in one 64-row
// chunk) and its column (a shuffle transpose of the group's eight sums).
// So that no value needs a test, the diagonal 64 × 64 blocks are kept with
// zeros above the diagonal and half the diagonal (each half counts once in the
// row's and once in the column's sum).  The matrix is scaled as tri_steps does
// it: by the first panel as it reads, by its update for good.
// Each warp takes an equal share of the groups, chunk by chunk, and every
// partial sum has its own slot, added up in a fixed order.  One 512-thread CTA
// per SM, so that the working set, 148 triangles, stays in L2.
constexpr int kPb = 8;            // panel width
constexpr int kBigT = 512;
constexpr int kBigW = kBigT / 32;
constexpr int kTail = 128;        // trailing block in registers
constexpr int kChunks = kSmallT / 64;

struct BigSmem {
  union {
    struct {
      float4 vw[kPb][kSmallT];                      // the panel's (v, w), by row
      cf rowp[kChunks][kBigW][64];                  // row sums: chunk, warp
      cf colp[kChunks][kSmallT];                    // column sums: chunk
      float4 sx[kSmallT];                           // u: (x.x, x.y, x.y, x.x)
      float4 g[kPb];                                // (Vᴴ u, Wᴴ u)
      float red0[kBigW], redt[kBigW];
      cf x1;
    } p;
    TriVec<4> t;
    struct {
      cf Y[4][kSmallT * kNb];                       // four WY blocks' reflectors, [row][reflector]
      cf G[4][120];
    } y;
  };
  double dd[kSmallT], ee[kSmallT];
  cf tau[kSmallT];
};

// Groups of 64 rows × 8 columns of the lower triangle from column o on, chunk
// by chunk (chunk q: rows 64q …), the first chunk being the one of row o.
__device__ __forceinline__ int groups_of(int o, int q, int n) {   // of chunk q
  return min(8 * (q + 1), (n + 7) >> 3) - (o >> 3);
}
__device__ __forceinline__ int groups_before(int o, int q) {   // of the chunks before q (none of them the last)
  const int q0 = o >> 6;
  return 4 * (q * (q + 1) - q0 * (q0 + 1)) - (q - q0) * (o >> 3);
}
__device__ __forceinline__ int groups_all(int o, int n) {
  const int ql = (n - 1) >> 6;
  return groups_before(o, ql) + groups_of(o, ql, n);
}
struct GroupIt {
  int q, base, cnt;
  // moves on to the chunk of group gi; the group's first column
  __device__ __forceinline__ int col(int o, int n, int gi) {
    while (gi >= base + cnt) {
      base += cnt;
      ++q;
      cnt = groups_of(o, q, n);
    }
    return (o & ~7) + 8 * (gi - base);
  }
};

// rows r (even) and r + 1 of a column; rows at or beyond n read the last ones
template <bool EVEN>
__device__ __forceinline__ void load2(cf* a0, cf* a1, const cf* col, int r, int n) {
  if constexpr (EVEN) {
    const float4 v = __ldcg(reinterpret_cast<const float4*>(col + min(r, n - 2)));
    *a0 = make_float2(v.x, v.y);
    *a1 = make_float2(v.z, v.w);
  } else {
    *a0 = __ldcg(col + min(r, n - 1));
    *a1 = __ldcg(col + min(r + 1, n - 1));
  }
}

template <bool EVEN>
__global__ void __launch_bounds__(kBigT, 1) k_tri_big(EigArgs g) {
  extern __shared__ __align__(16) unsigned char smraw[];
  BigSmem& m = *reinterpret_cast<BigSmem*>(smraw);
  int s = 0;
  while (s + 1 < g.nseg && (int64_t)blockIdx.x >= g.seg[s + 1].first) ++s;
  const Seg& S = g.seg[s];
  const int n = S.n;
  const int64_t ip = (int64_t)blockIdx.x - S.first;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  cf* A = S.gram + ip * (int64_t)n * n;
  const int i = tid;   // row of the vector phases
  const int nchunk = (n + 63) >> 6;
  float dmax = 0.f;   // (lane 0)
  for (int c = warp; c < n; c += kBigW) {   // the diagonal blocks (see above)
    cf* col = A + (int64_t)c * n;
    for (int r = (c & ~63) + lane; r < c; r += 32) col[r] = make_float2(0.f, 0.f);
    if (lane == 0) {
      const float d = __ldcg(&col[c].x);
      dmax = fmaxf(dmax, fabsf(d));
      col[c] = make_float2(0.5f * d, 0.f);
    }
  }
  if (lane == 0) m.p.redt[warp] = dmax;   // (next written after the first column's barriers)
  __syncthreads();
#pragma unroll
  for (int q = 0; q < kBigW; ++q) dmax = fmaxf(dmax, m.p.redt[q]);
  const PowerOfTwo pw(dmax);
  float up = pw.up;   // of the matrix in memory: 1 from the first update on
  int k = 0;
  while (n - k > kTail) {
    const int p0 = k, pe = min(p0 + kPb, n - kTail);   // this panel's columns
    cf xraw = (i >= p0 && i < n) ? __ldcg(A + (int64_t)p0 * n + i) : make_float2(0.f, 0.f);
    for (; k < pe; ++k) {
      const int np = k - p0;
      // column k with the panel's updates so far
      cf x = make_float2(0.f, 0.f);
      if (i >= k && i < n) {
        x = cscale(xraw, up);
        if (i == k) x.x *= 2.f;
#pragma unroll 4
        for (int p = 0; p < np; ++p) {
          const float4 a = m.p.vw[p][i], b = m.p.vw[p][k];   // − v conj(w_k) − w conj(v_k)
          x.x -= a.x * b.z + a.y * b.w + a.z * b.x + a.w * b.y;
          x.y -= a.y * b.z - a.x * b.w + a.w * b.x - a.z * b.y;
        }
      }
      if (k + 1 < pe && i > k && i < n) xraw = __ldcg(A + (int64_t)(k + 1) * n + i);   // the next column
      if (i == k) m.dd[k] = (double)x.x * pw.down;
      if (i == k + 1) m.p.x1 = x;
      if (i <= k + 1) x = make_float2(0.f, 0.f);
      if (i < kSmallT) m.p.sx[i] = make_float4(x.x, x.y, x.y, x.x);
      {
        const float q = warp_sum(cabs2(x));
        if (lane == 0) m.p.red0[warp] = q;
      }
      __syncthreads();
      float xn = 0.f;
#pragma unroll
      for (int q = 0; q < kBigW; ++q) xn += m.p.red0[q];
      // zlarfg as in tri_steps: u = (α − β, x), v = scal · u
      const float ar = m.p.x1.x, ai = m.p.x1.y;
      float bt = ar;
      cf tau = make_float2(0.f, 0.f), scal = tau, u1 = tau;
      const bool refl = !(xn + ai * ai <= kNoColumn);   // (true for NaN)
      if (refl) {
        const Reflector h(ar, ai, xn);
        bt = h.b;
        tau = h.tau(ar, ai);
        u1 = h.u1(ar, ai);
        scal = inverse(u1);
      }
      const int o = k + 1;
      if (i == o) m.p.sx[o] = make_float4(u1.x, u1.y, u1.y, u1.x);
      __syncthreads();
      // Wᴴ u and Vᴴ u of the panel's earlier columns, one per warp
      if (warp < np) {
        cf gw = make_float2(0.f, 0.f), gv = gw;
        for (int r = o + lane; r < n; r += 32) {
          const float4 q = m.p.sx[r];
          const cf u = make_float2(q.x, q.y);
          const float4 a = m.p.vw[warp][r];
          const cf v = make_float2(a.x, a.y), w = make_float2(a.z, a.w);
          gw.x += w.x * u.x + w.y * u.y;
          gw.y += w.x * u.y - w.y * u.x;
          gv.x += v.x * u.x + v.y * u.y;
          gv.y += v.x * u.y - v.y * u.x;
        }
        gw.x = warp_sum(gw.x);
        gw.y = warp_sum(gw.y);
        gv.x = warp_sum(gv.x);
        gv.y = warp_sum(gv.y);
        if (lane == 0) m.p.g[warp] = make_float4(gv.x, gv.y, gw.x, gw.y);
      }
      // A u over this warp's groups, the next group's values on their way
      float tq = 0.f;
      {
        const int G = groups_all(o, n);
        const int ge = (warp + 1) * G / kBigW;
        int gi = warp * G / kBigW;
        GroupIt it{o >> 6, 0, groups_of(o, o >> 6, n)};
        int c0 = it.col(o, n, gi), q = it.q, cur = -1, r = 0;
        cf u0 = make_float2(0.f, 0.f), uu = u0;         // u of the lane's two rows
        cf P0 = u0, Q0 = u0, P1 = u0, Q1 = u0;           // row sums (Σ a.x u.x, Σ a.y u.y), (Σ a.x u.y, Σ a.y u.x)
        cf a0[8], a1[8];
        if (gi < ge) {
#pragma unroll
          for (int b = 0; b < 8; ++b)
            load2<EVEN>(&a0[b], &a1[b], A + (int64_t)min(c0 + b, n - 1) * n, 64 * q + 2 * lane, n);
        }
        auto flush = [&]() {
          if (cur < 0) return;
          const cf y0 = make_float2((P0.x - P0.y) * up, (Q0.x + Q0.y) * up);
          const cf y1 = make_float2((P1.x - P1.y) * up, (Q1.x + Q1.y) * up);
          *reinterpret_cast<float4*>(&m.p.rowp[cur][warp][2 * lane]) = make_float4(y0.x, y0.y, y1.x, y1.y);
          tq += u0.x * y0.x + u0.y * y0.y + uu.x * y1.x + uu.y * y1.y;
        };
        for (; gi < ge; ++gi) {
          if (q != cur) {
            flush();
            cur = q;
            r = 64 * q + 2 * lane;
            const float4 q0 = r < n ? m.p.sx[r] : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 q1 = r + 1 < n ? m.p.sx[r + 1] : make_float4(0.f, 0.f, 0.f, 0.f);
            u0 = make_float2(q0.x, q0.y);
            uu = make_float2(q1.x, q1.y);
            P0 = Q0 = P1 = Q1 = make_float2(0.f, 0.f);
          }
          int nq = q, nc0 = c0;
          if (gi + 1 < ge) {
            nc0 = it.col(o, n, gi + 1);
            nq = it.q;
          }
          const cf* nxt = A + (int64_t)nc0 * n;
          const int nr = 64 * nq + 2 * lane;
          float cr[8], ci[8];
          const cf s0 = make_float2(u0.y, u0.x), s1 = make_float2(uu.y, uu.x);
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            // u of columns before o, of columns at or beyond n and of such rows is zero
            const float4 v = m.p.sx[c0 + b];
            const cf e0 = a0[b], e1 = a1[b];
            load2<EVEN>(&a0[b], &a1[b], nxt + (int64_t)min(b, n - 1 - nc0) * n, nr, n);
            P0 = __ffma2_rn(e0, make_float2(v.x, v.y), P0);
            Q0 = __ffma2_rn(e0, make_float2(v.z, v.w), Q0);
            P1 = __ffma2_rn(e1, make_float2(v.x, v.y), P1);
            Q1 = __ffma2_rn(e1, make_float2(v.z, v.w), Q1);
            const cf pc = __ffma2_rn(e1, uu, __fmul2_rn(e0, u0)), qc = __ffma2_rn(e1, s1, __fmul2_rn(e0, s0));
            cr[b] = pc.x + pc.y;   // conj(a) u
            ci[b] = qc.x - qc.y;
          }
          col_sums(cr, ci, lane);
          if ((lane & 3) == 0) {
            const int c = c0 + (lane >> 2);
            const cf y = make_float2(cr[0] * up, ci[0] * up);
            m.p.colp[q][c] = y;
            const float4 v = m.p.sx[c];
            tq += v.x * y.x + v.y * y.y;
          }
          q = nq;
          c0 = nc0;
        }
        flush();
      }
      tq = warp_sum(tq);
      if (lane == 0) m.p.redt[warp] = tq;
      __syncthreads();
      // y = A u − V (Wᴴ u) − W (Vᴴ u); uᴴ y; w
      {
        float t = 0.f;
#pragma unroll
        for (int q = 0; q < kBigW; ++q) t += m.p.redt[q];
        for (int p = 0; p < np; ++p) {
          const float4 a = m.p.g[p];
          t -= 2.f * (a.x * a.z + a.y * a.w);
        }
        const float c = 0.5f * (tau.x * tau.x + tau.y * tau.y) * (scal.x * scal.x + scal.y * scal.y) * t;
        cf vi = make_float2(0.f, 0.f), wi = vi;
        if (i > k && i < n) {
          cf y = make_float2(0.f, 0.f);
          // group x belongs to warp ⌈16 (x + 1) / G⌉ − 1 (G >= 16: no warp is without groups)
          const int q = i >> 6, G = groups_all(o, n), gb = groups_before(o, q);
          const int w0 = (kBigW * (gb + 1) + G - 1) / G - 1;
          const int w1 = (kBigW * (gb + groups_of(o, q, n)) + G - 1) / G - 1;
          for (int w = w0; w <= w1; ++w) y = cadd(y, m.p.rowp[q][w][i & 63]);
          for (int q2 = q; q2 < nchunk; ++q2) y = cadd(y, m.p.colp[q2][i]);
#pragma unroll 4
          for (int p = 0; p < np; ++p) {
            const float4 a = m.p.vw[p][i], b = m.p.g[p];
            y = csub(y, cadd(cmul(make_float2(a.x, a.y), make_float2(b.z, b.w)),
                             cmul(make_float2(a.z, a.w), make_float2(b.x, b.y))));
          }
          vi = i == o ? make_float2(1.f, 0.f) : cmul(x, scal);
          if (i == o) {
            m.ee[k] = (double)bt * pw.down;
            m.tau[k] = tau;
          } else {
            A[(int64_t)k * n + i] = vi;   // reflector kept below the subdiagonal
          }
          if (refl) {
            const cf ty = cmul(cmul(tau, scal), y);
            wi = make_float2(ty.x - c * vi.x, ty.y - c * vi.y);
          }
          if (!refl) vi = make_float2(0.f, 0.f);
        }
        if (i < kSmallT) {
          m.p.vw[np][i] = make_float4(vi.x, vi.y, wi.x, wi.y);
        }
      }
      __syncthreads();
    }
    // A ← A − V Wᴴ − W Vᴴ on the trailing lower triangle, groups as above
    {
      const int np = pe - p0, o = pe;
      const int G = groups_all(o, n);
      const float dh = n - pe == kTail ? 1.f : 0.5f;   // the trailing block goes on with its whole diagonal
      GroupIt it{o >> 6, 0, groups_of(o, o >> 6, n)};
      for (int gi = warp; gi < G; gi += kBigW) {
        const int c0 = it.col(o, n, gi), r = 64 * it.q + 2 * lane;
        cf a0[8], a1[8];
#pragma unroll
        for (int b = 0; b < 8; ++b) load2<EVEN>(&a0[b], &a1[b], A + (int64_t)min(c0 + b, n - 1) * n, r, n);
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          a0[b] = cscale(a0[b], up);
          a1[b] = cscale(a1[b], up);
        }
        if (c0 + 8 > 64 * it.q) {   // the whole diagonal
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            if (r == c0 + b) a0[b].x *= 2.f;
            if (r + 1 == c0 + b) a1[b].x *= 2.f;
          }
        }
        const int rs = min(r, kSmallT - 2);
#pragma unroll 2
        for (int p = 0; p < np; ++p) {
          const float4 x0 = m.p.vw[p][rs], x1 = m.p.vw[p][rs + 1];
#pragma unroll
          for (int b = 0; b < 8; ++b) {
            const float4 c = m.p.vw[p][min(c0 + b, kSmallT - 1)];
            auto upd = [&](cf& e, const float4& x) {   // e −= v conj(w_c) + w conj(v_c)
              e.x = fmaf(-x.x, c.z, e.x);
              e.y = fmaf(-x.y, c.z, e.y);
              e.x = fmaf(-x.y, c.w, e.x);
              e.y = fmaf(x.x, c.w, e.y);
              e.x = fmaf(-x.z, c.x, e.x);
              e.y = fmaf(-x.w, c.x, e.y);
              e.x = fmaf(-x.w, c.y, e.x);
              e.y = fmaf(x.z, c.y, e.y);
            };
            upd(a0[b], x0);
            upd(a1[b], x1);
          }
        }
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          const int c = c0 + b;
          if (c < o || c >= n) continue;
          if (r == c) a0[b] = make_float2(dh * a0[b].x, 0.f);
          if (r + 1 == c) a1[b] = make_float2(dh * a1[b].x, 0.f);
          cf* d = A + (int64_t)c * n + r;
          if (EVEN && r >= c && r + 1 < n) {
            *reinterpret_cast<float4*>(d) = make_float4(a0[b].x, a0[b].y, a1[b].x, a1[b].y);
          } else {
            if (r >= c && r < n) d[0] = a0[b];
            if (r + 1 >= c && r + 1 < n) d[1] = a1[b];
          }
        }
      }
    }
    up = 1.f;
    __syncthreads();
  }
  tri_steps<4, false>(A + (int64_t)k * n + k, n, n - k, m.t, m.dd + k, m.ee + k, m.tau + k, nullptr, pw.down);
  double* side = S.side + ip * 6 * (int64_t)n;
  for (int q = tid; q < n; q += kBigT) {
    side[q] = m.dd[q];
    side[n + q] = m.ee[q];
  }
  // T factors, four WY blocks at a time
  const int nref = n - 1, nblk = (nref + kNb - 1) / kNb;
  for (int b0 = 0; b0 < nblk; b0 += 4) {
    const int nb4 = min(4, nblk - b0);
    __syncthreads();
    for (int q = warp; q < nb4 * kNb; q += kBigW) {   // one reflector per warp
      const int bl = q >> 4, jj = q & 15;
      const int kend = nref - (b0 + bl) * kNb, k0 = max(0, kend - kNb), kk = k0 + jj;
      cf* y = m.y.Y[bl] + jj;
      for (int r = k0 + lane; r < n; r += 32) {
        cf v = make_float2(0.f, 0.f);
        if (kk < kend) {
          if (r == kk + 1) v = make_float2(1.f, 0.f);
          else if (r > kk + 1) v = __ldcg(A + (int64_t)kk * n + r);
        }
        y[r * kNb] = v;
      }
    }
    __syncthreads();
    if (tid < nb4 * 120) {
      const int bl = tid / 120, e = tid - bl * 120;
      int jj, b;
      g_entry(e, &jj, &b);
      const int kend = nref - (b0 + bl) * kNb, k0 = max(0, kend - kNb);
      const cf* y = m.y.Y[bl];
      float sr = 0.f, si = 0.f;
#pragma unroll 8
      for (int r = k0 + jj + 1; r < n; ++r) {
        const cf ya = y[r * kNb + b], yb = y[r * kNb + jj];
        sr += ya.x * yb.x + ya.y * yb.y;
        si += ya.x * yb.y - ya.y * yb.x;
      }
      m.y.G[bl][e] = make_float2(sr, si);
    }
    __syncthreads();
    if (warp < nb4) {
      const int blk = b0 + warp, kend = nref - blk * kNb, k0 = max(0, kend - kNb);
      wy_tfactor(A, n, blk, m.tau + k0, kend - k0, m.y.G[warp]);
    }
  }
}

template <int NT>
void tri_reg_launch(const EigArgs& a, unsigned grid, cudaStream_t st) {
  k_tri_reg<NT><<<grid, TriVec<NT>::kThreads, sizeof(TriSmem<NT>), st>>>(a);
}

// ---- split stage, second launch: eigenpairs of T --------------------------------------
// Phases 2–3 from d and e of the side buffer.
//   Eigenvalues: multisection on FP64 Sturm counts of T scaled by a power of two
// to norm at most 1.  The count is the number of sign changes of the leading
// minors p_i = (d_i − x) p_{i−1} − e²_{i−1} p_{i−2} (Givens' sequence; computed
// it is that of a T with a few relative roundings, as the quotient form is),
// rescaled every eight steps: three FP64 operations a step and one of them on
// the critical path, where the quotients p_i / p_{i−1} need a division each.
// Couplings are kept at or above 1e-30 of the norm so that no two consecutive
// minors vanish.  A group of g threads per eigenvalue counts below g points of
// its bracket a round (two or three points a thread measured no faster).
//   Vectors: twisted factorisation T − λ = L₊D₊L₊ᵀ = U₋D₋U₋ᵀ with the
// multipliers l_j = e_j / D₊_j and m_j = e_{j−1} / D₋_j kept (two divisions a
// row instead of four); γ_k = d_k − λ − e_{k−1} l_{k−1} − e_k m_{k+1}, z_k = 1 at
// the smallest |γ_k|, z_j = −l_j z_{j+1} above it and −m_j z_{j−1} below.
// Against the quotient form with FP32 first rounds: 486 full-rank sides of 300
// 3.60 → 1.68 ms, one of 64 87 → 24 µs, 40 of 128 493 → 119 µs.

// the reciprocal by two Newton steps from the hardware's approximation (|q| >= 1e-290)
__device__ __forceinline__ double recip(double q) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(q));
  y = fma(y, fma(-q, y, 1.0), y);
  return fma(y, fma(-q, y, 1.0), y);
}

// eigenvalues below x: de[i] = (d_i, e²_{i−1}) of the scaled T
__device__ __forceinline__ int sturm_count(const double2* de, int n, double x) {
  double p0 = 1.0, p1 = de[0].x - x;
  int cnt = (unsigned)__double2hiint(p1) >> 31;
  auto step = [&](double2 t) {
    const double p2 = fma(t.x - x, p1, -(t.y * p0));
    cnt += (unsigned)(__double2hiint(p2) ^ __double2hiint(p1)) >> 31;
    p0 = p1;
    p1 = p2;
  };
  int i = 1;
  for (; i + 8 <= n; i += 8) {
#pragma unroll
    for (int u = 0; u < 8; ++u) step(de[i + u]);
    // the larger of the two back to [1, 2)
    const int e0 = (__double2hiint(p0) >> 20) & 0x7ff, e1 = (__double2hiint(p1) >> 20) & 0x7ff;
    const double sc = __hiloint2double((2046 - max(max(e0, e1), 1)) << 20, 0);
    p0 *= sc;
    p1 *= sc;
  }
  for (; i < n; ++i) step(de[i]);
  return cnt;
}

// TH threads, n <= TH, MINB CTAs per SM
template <int TH, int MINB>
__global__ void __launch_bounds__(TH, MINB) k_pairs(EigArgs g) {
  extern __shared__ __align__(16) unsigned char smraw[];
  int s = 0;
  while (s + 1 < g.nseg && (int64_t)blockIdx.x >= g.seg[s + 1].first) ++s;
  const Seg& S = g.seg[s];
  const int n = S.n;
  const int64_t ip = (int64_t)blockIdx.x - S.first;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  constexpr int kThr = TH;
  cf* Z = S.zv + ip * (int64_t)n * n;
  double* AUX = S.aux + ip * (int64_t)n * n;
  double* side = S.side + ip * 6 * (int64_t)n;
  const bool full = S.lam_out != nullptr;
  const double beta = full ? 0.0 : g.thr[g.thr_per_patch ? (int64_t)blockIdx.x : 0] * S.lam;

  double2* de = reinterpret_cast<double2*>(smraw);   // scaled (d_i, e²_{i−1})
  double* dd = reinterpret_cast<double*>(de + n);
  double* ee = dd + n;
  double* lam = ee + n;
  double* redd = lam + n;                            // 64 doubles
  float* hv = reinterpret_cast<float*>(redd + 64);
  __shared__ int s_r;
  for (int q = tid; q < n; q += kThr) {
    dd[q] = side[q];
    ee[q] = side[n + q];
  }
  __syncthreads();
  // Gershgorin's interval; fmin and fmax pass a NaN by, so it is looked for by itself
  double gl = 1e300, gu = -1e300;
  bool bad = false;
  for (int q = tid; q < n; q += kThr) {
    const double rr = (q > 0 ? fabs(ee[q - 1]) : 0.0) + (q < n - 1 ? fabs(ee[q]) : 0.0);
    bad = bad || !(fabs(dd[q]) + rr < 1e300);
    gl = fmin(gl, dd[q] - rr);
    gu = fmax(gu, dd[q] + rr);
  }
  for (int o = 16; o > 0; o >>= 1) {
    gl = fmin(gl, __shfl_xor_sync(0xffffffffu, gl, o));
    gu = fmax(gu, __shfl_xor_sync(0xffffffffu, gu, o));
  }
  if (lane == 0) {
    redd[warp] = gl;
    redd[32 + warp] = gu;
  }
  if (__syncthreads_or(bad)) {
    // a NaN or Inf among the patch's values: all eigenpairs, NaN, so that the
    // patch comes out NaN and not as the zeros of an empty spectrum
    const float nan = __int_as_float(0x7fc00000);
    if (tid == 0) {
      S.rank[ip] = n;
      if (S.nuc) S.nuc[ip] = nan;
    }
    if (S.nuc) return;
    for (int q = tid; q < n * n; q += kThr) Z[q] = make_float2(nan, nan);
    for (int q = tid; q < n; q += kThr) {
      side[3 * n + q] = nan;
      reinterpret_cast<float*>(side + 4 * (int64_t)n)[q] = 1.f;
      if (full) S.lam_out[ip * n + q] = nan;
    }
    return;
  }
  for (int w = 0; w < kThr / 32; ++w) {
    gl = fmin(gl, redd[w]);
    gu = fmax(gu, redd[32 + w]);
  }
  const double tnorm = fmax(fabs(gl), fabs(gu));
  // power of two with norm · sc in [1/2, 1) (1 for a zero T)
  const int tex = (__double2hiint(tnorm) >> 20) & 0x7ff;
  const bool sane = tex > 64 && tex < 1983;
  const double sc = sane ? __hiloint2double((2045 - tex) << 20, 0) : 1.0;
  const double isc = sane ? __hiloint2double((tex + 1) << 20, 0) : 1.0;
  const double pad = 2.0 * 2.220446049250313e-16 * n;
  gl = gl * sc - pad;
  gu = gu * sc + pad;
  for (int q = tid; q < n; q += kThr) {
    const double e = q > 0 ? ee[q - 1] * sc : 0.0;
    de[q] = make_double2(dd[q] * sc, fmax(e * e, 1e-60));
  }
  __syncthreads();
  const double thr2 = beta * beta * sc;
  if (tid == 0) {
    s_r = full ? n : !(tnorm > 0.0) || thr2 >= gu ? 0 : n - sturm_count(de, n, thr2);
    S.rank[ip] = s_r;
  }
  __syncthreads();
  const int r = s_r;
  {
    if (!full) gl = fmax(gl, thr2);
    int gsz = 1;
    while (gsz < 32 && 2 * gsz * r <= kThr) gsz <<= 1;
    const int e = tid / gsz, sl = tid & (gsz - 1);
    if (warp * 32 < r * gsz) {   // whole warps, for the shuffles
      const int kth = n - 1 - e;   // e-th largest = kth smallest
      const double frac = (double)(sl + 1) / (double)(gsz + 1);
      double lo = gl, hi = gu;
      bool done = e >= r;
      for (int it = 0; it < 200; ++it) {
        // 4e-13 of the norm is well below what the vectors need (their error is |λ̂ − λ| / gap)
        if (!done && !(hi - lo > 4e-13)) done = true;
        if (!__any_sync(0xffffffffu, !done)) break;
        const double x = lo + (hi - lo) * frac;
        double nlo = lo, nhi = hi;
        const int c = sturm_count(de, n, x);
        if (x > lo && x < hi) {
          if (c > kth) nhi = x;   // the eigenvalue is below x
          else nlo = x;
        }
        for (int o = 1; o < gsz; o <<= 1) {
          nlo = fmax(nlo, __shfl_xor_sync(0xffffffffu, nlo, o));
          nhi = fmin(nhi, __shfl_xor_sync(0xffffffffu, nhi, o));
        }
        if (!done) {
          if (!(nhi - nlo < hi - lo) || !(nlo < nhi)) {
            done = true;
          } else {
            lo = nlo;
            hi = nhi;
          }
        }
      }
      if (e < r && sl == 0) {
        const double lm = 0.5 * (lo + hi) * isc;
        lam[e] = lm;
        const double sg = sqrt(fmax(lm, 0.0));
        hv[e] = (sg > beta && sg > 0.0) ? (float)((sg - beta) / sg) : 0.f;
      }
    }
  }
  __syncthreads();
  if (S.nuc) {   // nuclear norm of the patch (src/recon.jl:138-146): Σ σ_i = Σ √λ_i
    const double sq = (tid < r) ? sqrt(fmax(lam[tid], 0.0)) : 0.0;
    const double tot = block_sum_d(sq, redd);
    if (tid == 0) S.nuc[ip] = tot;
    return;
  }
  if (r == 0) return;   // the back-transform writes the zero columns itself

  // eigenvectors of T: l in AUX, m in the vector's slots read as doubles
  // ([row][vector], row stride n), replaced by z in place
  const int64_t zs = n;
  if (tid < r) {
    const double lm = lam[tid];
    const double pivmin = fmax(2.2250738585072014e-308 * fmax(tnorm * tnorm, 1.0), 1e-290);
    double* zd = reinterpret_cast<double*>(Z) + tid;
    double* dp = AUX + tid;
    auto piv = [&](double q) { return fabs(q) < pivmin ? -pivmin : q; };
    {   // both factorisations, one from either end
      double qf = piv(dd[0] - lm), qb = piv(dd[n - 1] - lm);
      for (int j = 0; j + 1 < n; ++j) {
        const int jb = n - 1 - j;
        const double ef = ee[j], eb = ee[jb - 1];
        const double l = ef * recip(qf), m = eb * recip(qb);
        dp[(int64_t)j * zs] = l;
        zd[(int64_t)jb * zs] = m;
        qf = piv(fma(-ef, l, dd[j + 1] - lm));
        qb = piv(fma(-eb, m, dd[jb - 1] - lm));
      }
    }
    int kb = 0;
    double gb = 1e308;
    {
      double el = 0.0;   // e_{k−1} l_{k−1}
#pragma unroll 4
      for (int k = 0; k < n; ++k) {
        const double em = k + 1 < n ? ee[k] * zd[(int64_t)(k + 1) * zs] : 0.0;
        const double gm = fabs(dd[k] - lm - el - em);
        if (gm <= gb) {
          gb = gm;
          kb = k;
        }
        if (k + 1 < n) el = ee[k] * dp[(int64_t)k * zs];
      }
    }
    if (const int t = tie_of(lam, r, tid, 1e-12 * fmax(tnorm, 1e-300)); t >= 0) {
      const Twist w = tied_twist(
          n, t, ee, tnorm,
          [=](int k) {
            const double em = k + 1 < n ? ee[k] * zd[(int64_t)(k + 1) * zs] : 0.0;
            const double el = k > 0 ? ee[k - 1] * dp[(int64_t)(k - 1) * zs] : 0.0;
            return fabs(dd[k] - lm - el - em);
          },
          [=](int j) { return dp[(int64_t)j * zs]; }, [=](int j) { return zd[(int64_t)j * zs]; });
      if (w.k >= 0) {   // nothing goes past the block's ends
        kb = w.k;
        if (w.b0 > 0) dp[(int64_t)(w.b0 - 1) * zs] = 0.0;
        if (w.b1 + 1 < n) zd[(int64_t)(w.b1 + 1) * zs] = 0.0;
      }
    }
    double nrm = 1.0;
    {
      double z = 1.0;
#pragma unroll 8
      for (int j = kb - 1; j >= 0; --j) {
        z *= -dp[(int64_t)j * zs];
        nrm = fma(z, z, nrm);
      }
      z = 1.0;
#pragma unroll 8
      for (int j = kb + 1; j < n; ++j) {
        z *= -zd[(int64_t)j * zs];
        nrm = fma(z, z, nrm);
      }
    }
    const double inv = 1.0 / sqrt(nrm);
    cf* zc = Z + tid;
    double z = inv;
    for (int j = kb + 1; j < n; j += 4) {   // (the slots that hold the multipliers first)
      double mv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) mv[q] = j + q < n ? zd[(int64_t)(j + q) * zs] : 0.0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        z *= -mv[q];
        if (j + q < n) zc[(int64_t)(j + q) * zs] = make_float2((float)z, 0.f);
      }
    }
    zc[(int64_t)kb * zs] = make_float2((float)inv, 0.f);
    z = inv;
    for (int j = kb - 1; j >= 0; j -= 4) {
      double lv[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) lv[q] = j - q >= 0 ? dp[(int64_t)(j - q) * zs] : 0.0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        z *= -lv[q];
        if (j - q >= 0) zc[(int64_t)(j - q) * zs] = make_float2((float)z, 0.f);
      }
    }
  }
  __syncthreads();
  // Eigenvalues equal to working precision: Gram–Schmidt inside the cluster,
  // cooperatively (every thread walks the same clusters).
  {
    const double ctol = 1e-12 * fmax(tnorm, 1e-300);
    int s0 = 0, rb = 0;
    while (s0 < r) {
      int t = s0 + 1;
      while (t < r && lam[t - 1] - lam[t] <= ctol) ++t;
      for (int qv = s0 + 1; qv < t; ++qv) {
        for (int attempt = 0; attempt < 4; ++attempt) {
          for (int pv = s0; pv < qv; ++pv) {
            double dot = 0.0;
            for (int j = tid; j < n; j += kThr) dot += (double)Z[j * zs + pv].x * Z[j * zs + qv].x;
            dot = block_sum_d(dot, redd + 32 * (rb++ & 1));
            for (int j = tid; j < n; j += kThr) Z[j * zs + qv].x -= (float)dot * Z[j * zs + pv].x;
            __syncthreads();
          }
          double nr = 0.0;
          for (int j = tid; j < n; j += kThr) nr += (double)Z[j * zs + qv].x * Z[j * zs + qv].x;
          nr = sqrt(block_sum_d(nr, redd + 32 * (rb++ & 1)));
          if (nr > 0.1) {
            for (int j = tid; j < n; j += kThr) Z[j * zs + qv].x /= (float)nr;
            __syncthreads();
            break;
          }
          // collapsed onto earlier vectors: restart from a unit vector
          for (int j = tid; j < n; j += kThr)
            Z[j * zs + qv].x = (j == (qv + attempt * 7919) % n) ? 1.f : 0.f;
          __syncthreads();
        }
      }
      s0 = t;
    }
  }
  float* sh = reinterpret_cast<float*>(side + 4 * (int64_t)n);
  for (int q = tid; q < r; q += kThr) {
    side[3 * n + q] = lam[q];
    sh[q] = hv[q];
    if (full) S.lam_out[ip * n + q] = lam[q];
  }
}

size_t pairs_smem(int n) { return (size_t)n * (2 + 3) * sizeof(double) + 64 * sizeof(double) + n * sizeof(float) + 16; }

// A patch's chain of Sturm rounds and divisions wants no spills and threads for
// several points per eigenvalue while patches are few; with more patches than
// SMs, CTAs of about n threads keep more of them resident.  320 threads, two
// CTAs per SM (96 registers, none spilled): 40 patches of 128 168 -> 119 us
// against four CTAs (48 registers), 486 of 300 1.76 -> 1.68 ms; 160 threads, four
// CTAs: 240 patches of 50 36 -> 30 us against that; 128 threads, eight CTAs:
// 2250 patches of 128 0.30 -> 0.26 ms against the four (0.52 against the two).
void pairs_launch(const EigArgs& a, int nmax, int64_t total, cudaStream_t st) {
  constexpr int kSms = 148;
  const size_t sm = pairs_smem(nmax);
  const unsigned grid = (unsigned)total;
  if (nmax <= 128 && total > 4 * kSms) k_pairs<128, 8><<<grid, 128, sm, st>>>(a);
  else if (nmax <= 160 && total > kSms) k_pairs<160, 4><<<grid, 160, sm, st>>>(a);
  else if (nmax <= 320) k_pairs<320, 2><<<grid, 320, sm, st>>>(a);
  else k_pairs<kSmallT, 2><<<grid, kSmallT, sm, st>>>(a);
}

// ---- split stage, third launch: Ṽ = conj(Q Z) diag(√h) -------------------------
// One CTA per 64 eigenvectors of a patch (32 when no more are left, or above
// side 320); warp w holds rows w, w + 16, … of its vectors in registers (lane
// = vectors lane and lane + 32) through all WY blocks, taken from the last
// reflector down.  Each block's Y (rows k0+1 … n−1, kYS-strided so a row's 16
// reflector entries load as warp-wide broadcasts) and T arrive by cp.async
// into one of two buffers while the previous block is applied: S = Yᴴ Z by
// per-warp partial sums added in warp order, eight reflectors at a time, S ← T
// S, then Z −= Y S.  The complex products run as packed FP32x2 FMAs on
// lane-wise products, (y.re·z.re, y.im·z.im) and (y.re·z.im, y.im·z.re),
// combined once per row or per reflector.  A 16-byte broadcast of Y takes the
// shared-memory pipe four cycles whatever it feeds: with one vector per lane
// (four FMAs) the kernel waited for it at twice the FMAs' time, two vectors
// balance the two (486 full-rank patches of side 300: 5.3 → 4.5 ms).
// Columns at or beyond the patch's rank are written as zeros.
constexpr int kYS = 18;        // row stride of the staged Y (16-byte aligned rows)
constexpr int kWyThreads = 512;
constexpr int kWyCols = 64;
constexpr int kWyWarps = kWyThreads / 32;

size_t wy_apply_smem(int nmax) {
  const int rows = (nmax + 63) / 64 * 64;   // 16 · rows per warp
  return ((size_t)2 * rows * kYS + kWyWarps * 8 * kWyCols + 2 * kNb * kWyCols + 2 * kNb * kNb) * sizeof(cf);
}

__device__ __forceinline__ void cpa8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
__device__ __forceinline__ void cpa_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
__device__ __forceinline__ void cpa_wait_all() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

// Y rows k0+1 … n−1 of reflectors k0 … k0+nb−1 (the unit entry and the zeros
// above it written directly) and the block's T into (ys, ts); thread t owns
// row k0+1+t (m <= n − 1 < kWyThreads).
__device__ __forceinline__ void wy_stage(const cf* A, int n, int kend, cf* ys, cf* ts, int tid) {
  const int k0 = max(0, kend - kNb), nb = kend - k0;
  const int blk = (n - 1 - kend) / kNb;
  const int m = n - k0 - 1;
  if (tid < m) {
    const int row = k0 + 1 + tid;
    cf* dst = ys + row * kYS;
#pragma unroll
    for (int jj = 0; jj < kNb; ++jj) {
      const int k = k0 + jj;
      if (jj < nb && row > k + 1) cpa8(dst + jj, A + (int64_t)k * n + row);
      else dst[jj] = make_float2((jj < nb && row == k + 1) ? 1.f : 0.f, 0.f);
    }
  }
  if (tid < kNb * kNb) {
    const int a = tid / kNb, b = tid - a * kNb;
    if (a <= b && b < nb) cpa8(ts + tid, A + t_slot(n, blk, a, b));
    else ts[tid] = make_float2(0.f, 0.f);
  }
  cpa_commit();
}

// NV vectors per lane: columns cb + lane + 32 v of the patch's n × n matrix Z
template <int RPW, int NV>
__device__ __forceinline__ void wy_apply_body(const Seg& S, const cf* A, cf* Z, const float* hw, int n, int r, int cb,
                                              cf* smem) {
  const int tid = threadIdx.x, w = tid >> 5, lane = tid & 31;
  // two buffers of Y, zero in the rows no block has reached yet (they are taken
  // from the last reflector down) and beyond n, so that rows go untested in fours
  cf* Ybuf = smem;
  constexpr int ystride = 16 * RPW * kYS;
  cf* part = Ybuf + 2 * ystride;                 // 16 warps × 8 × 64
  cf* Ss = part + kWyWarps * 8 * kWyCols;        // kNb × 64
  cf* S2 = Ss + kNb * kWyCols;                   // kNb × 64
  cf* Tbuf = S2 + kNb * kWyCols;                 // two buffers of kNb × kNb
  cf z[RPW][NV];
#pragma unroll
  for (int q = 0; q < RPW; ++q) {
    const int row = w + 16 * q;
#pragma unroll
    for (int v = 0; v < NV; ++v) {
      const int c = cb + lane + 32 * v;
      z[q][v] = make_float2((c < r && row < n) ? __ldcg(&Z[(int64_t)row * n + c].x) : 0.f, 0.f);
    }
  }
  const int nref = n - 1;
  for (int q = tid; q < ystride; q += kWyThreads) reinterpret_cast<float4*>(Ybuf)[q] = make_float4(0.f, 0.f, 0.f, 0.f);
  __syncthreads();
  if (nref > 0) wy_stage(A, n, nref, Ybuf, Tbuf, tid);
  cpa_wait_all();
  __syncthreads();
  int buf = 0;
  for (int kend = nref; kend > 0; kend -= kNb, buf ^= 1) {
    const int k0 = max(0, kend - kNb);
    const cf* Ys = Ybuf + buf * ystride;
    const cf* Ts = Tbuf + buf * kNb * kNb;
    if (kend - kNb > 0)   // the next block, into the other buffers
      wy_stage(A, n, kend - kNb, Ybuf + (buf ^ 1) * ystride, Tbuf + (buf ^ 1) * kNb * kNb, tid);
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      // partial S = Yᴴ Z over this warp's rows, reflectors 8h … 8h + 7 in passes of four
#pragma unroll
      for (int a4 = 0; a4 < 2; ++a4) {
        cf P[4][NV], Q[4][NV];
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int v = 0; v < NV; ++v) P[a][v] = Q[a][v] = make_float2(0.f, 0.f);
#pragma unroll
        for (int q4 = 0; q4 < RPW; q4 += 4) {
          if (w + 16 * (q4 + 3) <= k0) continue;
#pragma unroll
          for (int q = q4; q < q4 + 4; ++q) {
            const int row = w + 16 * q;
            const float4* yr = reinterpret_cast<const float4*>(Ys + row * kYS) + 4 * h + 2 * a4;
            const float4 y01 = yr[0], y23 = yr[1];
#pragma unroll
            for (int v = 0; v < NV; ++v) {
              const cf z1 = z[q][v], z2 = make_float2(z1.y, z1.x);
              P[0][v] = __ffma2_rn(make_float2(y01.x, y01.y), z1, P[0][v]);
              Q[0][v] = __ffma2_rn(make_float2(y01.x, y01.y), z2, Q[0][v]);
              P[1][v] = __ffma2_rn(make_float2(y01.z, y01.w), z1, P[1][v]);
              Q[1][v] = __ffma2_rn(make_float2(y01.z, y01.w), z2, Q[1][v]);
              P[2][v] = __ffma2_rn(make_float2(y23.x, y23.y), z1, P[2][v]);
              Q[2][v] = __ffma2_rn(make_float2(y23.x, y23.y), z2, Q[2][v]);
              P[3][v] = __ffma2_rn(make_float2(y23.z, y23.w), z1, P[3][v]);
              Q[3][v] = __ffma2_rn(make_float2(y23.z, y23.w), z2, Q[3][v]);
            }
          }
        }
        // conj(y)·z = (Σ y.re z.re + y.im z.im, Σ y.re z.im − y.im z.re)
#pragma unroll
        for (int a = 0; a < 4; ++a)
#pragma unroll
          for (int v = 0; v < NV; ++v)
            part[(w * 8 + 4 * a4 + a) * kWyCols + 32 * v + lane] =
                make_float2(P[a][v].x + P[a][v].y, Q[a][v].x - Q[a][v].y);
      }
      __syncthreads();
      if (NV == 2 || w < 8) {   // one sum per thread: reflector 8h + a, vector c
        const int a = NV == 2 ? w >> 1 : w, c = NV == 2 ? 32 * (w & 1) + lane : lane;
        cf sum = make_float2(0.f, 0.f);
#pragma unroll
        for (int w2 = 0; w2 < kWyWarps; ++w2) sum = cadd(sum, part[(w2 * 8 + a) * kWyCols + c]);
        Ss[(8 * h + a) * kWyCols + c] = sum;
      }
      __syncthreads();
    }
    {
      const int a = w;
      cf acc[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) acc[v] = make_float2(0.f, 0.f);
      for (int b = a; b < kNb; ++b) {
        const cf t = Ts[a * kNb + b];
#pragma unroll
        for (int v = 0; v < NV; ++v) acc[v] = cadd(acc[v], cmul(t, Ss[b * kWyCols + 32 * v + lane]));
      }
#pragma unroll
      for (int v = 0; v < NV; ++v) S2[a * kWyCols + 32 * v + lane] = acc[v];
    }
    __syncthreads();
    // Z −= Y (T S) on this warp's rows, four reflectors per pass
#pragma unroll 1
    for (int a4 = 0; a4 < 4; ++a4) {
      cf sa[4][NV], sb[4][NV];
#pragma unroll
      for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int v = 0; v < NV; ++v) {
          sa[a][v] = S2[(4 * a4 + a) * kWyCols + 32 * v + lane];
          sb[a][v] = make_float2(sa[a][v].y, sa[a][v].x);
        }
#pragma unroll
      for (int q4 = 0; q4 < RPW; q4 += 4) {
        if (w + 16 * (q4 + 3) <= k0) continue;
#pragma unroll
        for (int q = q4; q < q4 + 4; ++q) {
          const int row = w + 16 * q;
          const float4* yr = reinterpret_cast<const float4*>(Ys + row * kYS) + 2 * a4;
          const float4 y01 = yr[0], y23 = yr[1];
#pragma unroll
          for (int v = 0; v < NV; ++v) {
            cf U = __fmul2_rn(make_float2(y01.x, y01.y), sa[0][v]), V = __fmul2_rn(make_float2(y01.x, y01.y), sb[0][v]);
            U = __ffma2_rn(make_float2(y01.z, y01.w), sa[1][v], U);
            V = __ffma2_rn(make_float2(y01.z, y01.w), sb[1][v], V);
            U = __ffma2_rn(make_float2(y23.x, y23.y), sa[2][v], U);
            V = __ffma2_rn(make_float2(y23.x, y23.y), sb[2][v], V);
            U = __ffma2_rn(make_float2(y23.z, y23.w), sa[3][v], U);
            V = __ffma2_rn(make_float2(y23.z, y23.w), sb[3][v], V);
            // y·s = (Σ y.re s.re − y.im s.im, Σ y.re s.im + y.im s.re)
            z[q][v].x -= U.x - U.y;
            z[q][v].y -= V.x + V.y;
          }
        }
      }
    }
    cpa_wait_all();
    __syncthreads();
  }
  // Ṽ, or V itself when every eigenpair is wanted
#pragma unroll
  for (int v = 0; v < NV; ++v) {
    const int c = cb + lane + 32 * v;
    const float sh = S.lam_out ? 1.f : (c < r) ? sqrtf(hw[c]) : 0.f, sc = S.lam_out ? 1.f : -sh;
#pragma unroll
    for (int q = 0; q < RPW; ++q) {
      const int row = w + 16 * q;
      if (row < n && c < n) Z[(int64_t)row * n + c] = make_float2(z[q][v].x * sh, z[q][v].y * sc);
    }
  }
}

// One block per patch and group of 32·NV columns, the groups of a patch in a
// row; one grid dimension, since all scales' patches may pass 65 535
template <int RPW, int NV>
__global__ void __launch_bounds__(kWyThreads, 1) k_wy_apply(EigArgs g, int groups) {
  extern __shared__ __align__(16) unsigned char smraw[];
  const int64_t patch = blockIdx.x / groups;
  int s = 0;
  while (s + 1 < g.nseg && patch >= g.seg[s + 1].first) ++s;
  const Seg& S = g.seg[s];
  const int n = S.n;
  const int64_t ip = patch - S.first;
  const int cb = (int)(blockIdx.x - patch * groups) * 32 * NV;
  if (cb >= n) return;   // the grid covers the launch's largest n
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const cf* A = S.gram + ip * (int64_t)n * n;
  cf* Z = S.zv + ip * (int64_t)n * n;
  const int r = S.rank[ip];
  const float* hw = reinterpret_cast<const float*>(S.side + ip * 6 * (int64_t)n + 4 * (int64_t)n);
  cf* smem = reinterpret_cast<cf*>(smraw);
  // columns from the next group of 32 on that have no vector
  const int z0 = max(cb, (r + 31) / 32 * 32);
  for (int c = z0 + lane; c < min(n, cb + 32 * NV); c += 32)
    for (int row = w; row < n; row += kWyWarps) Z[(int64_t)row * n + c] = make_float2(0.f, 0.f);
  if (cb >= r) return;
  if (NV == 2 && r - cb > 32) wy_apply_body<RPW, NV>(S, A, Z, hw, n, r, cb, smem);
  else wy_apply_body<RPW, 1>(S, A, Z, hw, n, r, cb, smem);
}

const void* wy_kernel(int rows_per_warp) {
  return rows_per_warp <= 4    ? reinterpret_cast<const void*>(&k_wy_apply<4, 2>)
         : rows_per_warp <= 8  ? reinterpret_cast<const void*>(&k_wy_apply<8, 2>)
         : rows_per_warp <= 12 ? reinterpret_cast<const void*>(&k_wy_apply<12, 2>)
         : rows_per_warp <= 16 ? reinterpret_cast<const void*>(&k_wy_apply<16, 2>)
         : rows_per_warp <= 20 ? reinterpret_cast<const void*>(&k_wy_apply<20, 2>)
                               : reinterpret_cast<const void*>(&k_wy_apply<24, 1>);
}

}  // namespace

int eig2_prepare(int nmax) {
  if (nmax > kT) return fail(MSLR_ERR_UNSUPPORTED, "Gram side above 1024");
  if (smem_bytes(nmax, kT, 0) > smem_budget(kT))
    return fail(MSLR_ERR_UNSUPPORTED, "Gram side too large for the eigen stage");
  const int big = (int)smem_budget(kT), small = (int)smem_budget(kSmallT);
  MSLR_CUDA_TRY(cudaFuncSetAttribute(k_eig<kT, 1, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  MSLR_CUDA_TRY(cudaFuncSetAttribute(k_eig<kSmallT, 2, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, small));
  MSLR_CUDA_TRY(cudaFuncSetAttribute(k_eig<kT, 1, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize, big));
  MSLR_CUDA_TRY(cudaFuncSetAttribute(k_tri_reg<3>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TriSmem<3>)));
  MSLR_CUDA_TRY(cudaFuncSetAttribute(k_tri_reg<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(TriSmem<4>)));
  MSLR_CUDA_TRY(cudaFuncSetAttribute(k_tri_big<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BigSmem)));
  MSLR_CUDA_TRY(cudaFuncSetAttribute(k_tri_big<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BigSmem)));
  static_assert(sizeof(BigSmem) <= 227 * 1024, "shared memory of the blocked tridiagonalisation");
  const int wy = (int)wy_apply_smem(kSmallT);
  for (const void* k : {wy_kernel(4), wy_kernel(8), wy_kernel(12), wy_kernel(16), wy_kernel(20), wy_kernel(24)})
    MSLR_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, wy));
  return MSLR_OK;
}

namespace {

// The split stage applies to stages with a side buffer and 9 <= n <= 384 (the
// back-transform's register tile); the autotuner's 1024 threads from 33 on.
// Sides up to 32 in three launches instead of one: the SVST of 5 matrices 118 ×
// 22 229 → 133 µs, patchSVST of 4³ patches at stride 3 of 35 × 35 × 26 × 21 (1296
// of side 21) 1165 → 569.  Below 9 a matrix has no more than a few steps, and no
// room for the side values of the all-pairs mode below 6: one launch.
// MSLR_EIG_SPLIT=0 keeps the one-launch stage everywhere (for comparisons).
bool split_ok(const EigSegment& e) {
  static const bool off = [] {
    const char* v = std::getenv("MSLR_EIG_SPLIT");
    return v && v[0] == '0';
  }();
  return !off && e.side && e.n >= (e.big ? 33 : 9) && e.n <= kSmallT;
}

int wy_apply_launch(const EigArgs& a, int nmax, int64_t total, cudaStream_t st) {
  const int rpw = (nmax + 15) / 16, cols = rpw <= 20 ? 64 : 32;   // columns per CTA
  int groups = (nmax + cols - 1) / cols;
  EigArgs arg = a;
  void* args[] = {&arg, &groups};
  MSLR_CUDA_TRY(cudaLaunchKernel(wy_kernel(rpw), dim3((unsigned)(total * groups)), dim3(kWyThreads), args,
                                 wy_apply_smem(nmax), st));
  return MSLR_OK;
}

// Phase 1 of the split stage for one segment: the matrix in registers up to
// 128, the blocked form above (16-byte loads need an even side and a 16-byte
// aligned buffer); the autotuner's 1024-thread variant keeps the step-by-step form.
void tri_launch(const EigArgs& a, bool big, cudaStream_t st) {
  const Seg& S = a.seg[0];
  const int n = S.n;
  const unsigned grid = (unsigned)S.np;
  if (big) {
    k_eig<kT, 1, 1><<<grid, kT, vec_bytes(n) + wy_bytes(n, kT) + 128, st>>>(a);
  } else if (n <= 32) {
    tri_reg_launch<1>(a, grid, st);
  } else if (n <= 64) {
    tri_reg_launch<2>(a, grid, st);
  } else if (n <= 96) {
    tri_reg_launch<3>(a, grid, st);
  } else if (n <= kTail) {
    tri_reg_launch<4>(a, grid, st);
  } else if (n % 2 == 0 && (reinterpret_cast<uintptr_t>(S.gram) & 15) == 0) {
    k_tri_big<true><<<grid, kBigT, sizeof(BigSmem), st>>>(a);
  } else {
    k_tri_big<false><<<grid, kBigT, sizeof(BigSmem), st>>>(a);
  }
}

// One launch (or, for the split stage, two and one per segment) over segments that all take the
// same CTA variant.
int eig_launch_group(const std::vector<const EigSegment*>& segs, const double* thr, int thr_per_patch,
                     cudaStream_t st, uint64_t* launches) {
  EigArgs a;
  a.nseg = (int)segs.size();
  a.thr = thr;
  a.thr_per_patch = thr_per_patch;
  int64_t total = 0;
  int nmax = 1;
  bool split = true;
  for (int s = 0; s < a.nseg; ++s) {
    Seg& S = a.seg[s];
    const EigSegment& e = *segs[s];
    S.n = e.n;
    S.first = total;
    S.np = e.np;
    S.gram = e.gram;
    S.zv = e.zv;
    S.aux = e.aux;
    S.rank = e.rank;
    S.lam = e.lam;
    S.nuc = e.nuc;
    S.lam_out = e.lam_out;
    S.side = e.side;
    total += e.np;
    nmax = std::max(nmax, e.n);
    split = split && split_ok(e);
  }
  bool big = nmax > kSmallT;
  for (const EigSegment* e : segs) big = big || e->big;
  const int threads = big ? kT : kSmallT;
  if (split) {
    a.rz = 0;
    for (int q = 0; q < a.nseg; ++q) {   // phase 1, per segment: the kernel follows its n
      EigArgs one = a;
      one.nseg = 1;
      one.seg[0] = a.seg[q];
      one.seg[0].first = 0;
      tri_launch(one, threads == kT, st);
      if (launches) *launches += 1;
    }
    pairs_launch(a, nmax, total, st);
    const bool values = segs[0]->nuc != nullptr;   // (such calls have one segment)
    if (!values)
      if (int rc = wy_apply_launch(a, nmax, total, st)) return rc;
    MSLR_CUDA_TRY(cudaGetLastError());
    if (launches) *launches += values ? 1 : 2;
    return MSLR_OK;
  }
  a.rz = stage_cols(nmax, threads);
  const size_t sm = smem_bytes(nmax, threads, a.rz);
  if (threads == kSmallT)
    k_eig<kSmallT, 2, 0><<<(unsigned)total, kSmallT, sm, st>>>(a);
  else
    k_eig<kT, 1, 0><<<(unsigned)total, kT, sm, st>>>(a);
  MSLR_CUDA_TRY(cudaGetLastError());
  if (launches) *launches += 1;
  return MSLR_OK;
}

}  // namespace

// Segments with Gram side <= 384 run in the 384-thread variant (two patches per
// SM), larger ones in the 1024-thread variant: one launch per variant present.
// Per-patch thresholds (thr_per_patch) index patches across all segments, so
// such calls keep every segment in one launch.
int eig_launch_multi(int nseg, const EigSegment* segs, const double* thr, int thr_per_patch,
                     cudaStream_t st, uint64_t* launches) {
  if (nseg < 1 || nseg > kMaxSeg) return fail(MSLR_ERR_UNSUPPORTED, "too many scales in one launch");
  std::vector<const EigSegment*> small, big, all;
  for (int s = 0; s < nseg; ++s) {
    (segs[s].n <= kSmallT && !segs[s].big ? small : big).push_back(&segs[s]);
    all.push_back(&segs[s]);
  }
  if (thr_per_patch || small.empty() || big.empty())
    return eig_launch_group(all, thr, thr_per_patch, st, launches);
  int rc = eig_launch_group(big, thr, 0, st, launches);
  if (!rc) rc = eig_launch_group(small, thr, 0, st, launches);
  return rc;
}

int eig2_launch(int n, int64_t np, cf* gram, cf* zv, float* aux, int* rank, const double* thr,
                int thr_per_patch, double lam, cudaStream_t st, int big, double* side, uint64_t* launches) {
  EigSegment s;
  s.n = n;
  s.np = np;
  s.gram = gram;
  s.zv = zv;
  s.aux = reinterpret_cast<double*>(aux);
  s.rank = rank;
  s.lam = lam;
  s.big = big;
  s.nuc = nullptr;
  s.side = side;
  return eig_launch_multi(1, &s, thr, thr_per_patch, st, launches);
}

}  // namespace mslr
