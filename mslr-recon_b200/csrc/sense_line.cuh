// sense_line.cuh — SENSE kernels whose 1-D transforms are whole lines in one
// thread's registers (fft_line.cuh).  T[f][cc][z][y][x] is the per-coil
// k-space of a chunk of frames and a group of coils.
//
// Columns (y and z lines) need no shared memory: neighbouring threads hold
// neighbouring x, so every load and store of a line element is a run of 256
// bytes per warp.  Rows (x lines) pass through shared memory once.
//   k_lcol   z line per thread: DFT_z, mask, bDFT_z in registers (or one
//            direction alone), in place on T; y line per thread: S'·x̄ → DFT_y
//            → T, or bDFT_y in place
//   k_lrow   x line per thread through a shared tile, in place on T
//   k_pfwd, k_padj (sense_line.cu, images with a compiled plane): the x and y
//            passes of a plane in one kernel, turned in shared memory in between
// What bounds them: the z pass moves T once in and once out of L2 (measured
// 13.5 TB/s for a read-modify-write of 24–96 MB) and computes in between, so
// its waves alternate between the two; the plane passes are bound by latency
// with 9 warps per SM (issue slots 35–45% busy, barrier, shared-memory and
// load stalls), for which packed FP32 pairs cut the instructions by a third.
// Measured at 90×90×60, 18 coils, 300 frames: 54.0 → 30.9 ms for the normal
// operator against two Stockham passes per axis through shared memory
// (per 24 coil images: plane passes 80 / 83 → 50 / 46 µs, z pass 86 → 41 µs,
// coil sum 25 → 30 µs with the maps' product moved into it); 75×64×45, 12
// coils, 40 frames: 11.0 → 1.47 ms against generic passes.
#pragma once
#include "fft_line.cuh"
#include "internal.h"

namespace mslr {
namespace line {

// ---- launch shapes ------------------------------------------------------------
constexpr int kColThreads = 128;
// resident CTAs of a 128-thread column kernel: a line of N values needs 2·N
// registers and about 20 more, of the 512 that each of an SM sub-partition's
// 32 lanes has for its warps (one per CTA).  With 8 more, one CTA more was
// resident and some of the line spilled: normal operator at 75 × 64 × 45 × 12 ×
// 40 1.55 -> 1.43 ms, at 90 × 90 × 60 × 18 × 300 30.5 -> 30.0; with 32 or 48
// more it is no faster or slower (1.43 / 1.50 and 30.1 / 30.1 ms).
constexpr int col_ctas(int n) {
  const int c = 512 / (2 * n + 20);
  return c < 1 ? 1 : c > 8 ? 8 : c;
}
// rows per CTA of the x pass: a shared tile of at most about 50 KB
constexpr int row_threads(int n) { return n > 48 ? 64 : 128; }
constexpr int row_ctas(int n) {
  const int c = (n > 48 ? 2 : 1) * (512 / (2 * n + 16));
  return c < 1 ? 1 : c > 8 ? 8 : c;
}
// row stride of a shared tile: even for 16-byte accesses, with an odd number
// of 16-byte units (a quarter-warp's rows then fall on distinct banks); odd
// lengths use 8-byte accesses, for which an odd stride has the same effect
constexpr int row_stride(int n) { return n % 2 ? n : (n / 2) % 2 ? n : n + 2; }
constexpr size_t row_smem(int n) { return (size_t)row_threads(n) * row_stride(n) * sizeof(cf); }

enum ColMode { kZMask = 0, kZFwd = 1, kZInv = 2, kYFwdMul = 3, kYInv = 4 };

struct ColArgs {
  cf* T;                  // chunk k-space
  const cf* xs;           // kYFwdMul: image of frame t0 + f at xs + (t0 + f)·nvox
  const cf* smod;         // modulated coil maps (cc0 + cc)·nvox
  const uint32_t* mz;     // kZMask: sample bits over z, (t, word, y·NX + x)
  int64_t nvox;
  int nlines;             // lines of one image
  int nx, pl;             // NX, NX·NY
  int ch, cc0, t0;
};

// One line per thread, blockIdx.y = f·ch + cc.  z lines: line i = (y, x) at
// offset i, element stride pl.  y lines: line i = (z, x) at z·pl + x, element
// stride nx.  Bound by L2 / HBM traffic (one read and one write of T); the
// whole line's loads are in flight at once.
// SE: element stride when known at compile time (plain immediates), else 0.
template <int N, int MODE, int SE>
__global__ void __launch_bounds__(kColThreads, col_ctas(N)) k_lcol(const ColArgs a) {
  const int i = blockIdx.x * kColThreads + threadIdx.x;
  if (i >= a.nlines) return;
  const int f = blockIdx.y / a.ch, cc = blockIdx.y - f * a.ch;
  constexpr bool kY = MODE == kYFwdMul || MODE == kYInv;
  int64_t off = i;
  if constexpr (kY) {
    const int z = i / a.nx;
    off = (int64_t)z * a.pl + (i - z * a.nx);
  }
  int se = SE ? SE : kY ? a.nx : a.pl;
  cf* p = a.T + (int64_t)blockIdx.y * a.nvox + off;
  cf v[N];
  if constexpr (MODE == kYFwdMul) {
    const cf* x = a.xs + (int64_t)(a.t0 + f) * a.nvox + off;
    const cf* s = a.smod + (int64_t)(a.cc0 + cc) * a.nvox + off;
#pragma unroll
    for (int e = 0; e < N; ++e) v[e] = cmul(__ldg(x + e * se), __ldg(s + e * se));
  } else {
#pragma unroll
    for (int e = 0; e < N; ++e) v[e] = p[e * se];
  }
  if constexpr (MODE == kZMask) {
    constexpr int NW = (N + 31) / 32;
    uint32_t w[NW];
    const uint32_t* m = a.mz + (int64_t)(a.t0 + f) * NW * a.pl + i;
#pragma unroll
    for (int q = 0; q < NW; ++q) w[q] = __ldg(m + (int64_t)q * a.pl);
    LD<N, false>::run(v);
#pragma unroll
    for (int e = 0; e < N; ++e)
      if (!((w[e >> 5] >> (e & 31)) & 1u)) v[e] = make_float2(0.f, 0.f);
    LD<N, true>::run(v);
  } else {
    LD<N, MODE == kZInv || MODE == kYInv>::run(v);
  }
  // with a runtime stride: store addresses computed anew instead of the N load
  // addresses kept in registers through the transform
  if constexpr (SE == 0) asm volatile("" : "+l"(p), "+r"(se));
#pragma unroll
  for (int e = 0; e < N; ++e) p[e * se] = v[e];
}

// x lines: rows [b·R, b·R + R) of the chunk's rows (all contiguous), one per
// thread, through a shared tile: coalesced in, the line in registers,
// coalesced out.
template <int N, bool INV>
__global__ void __launch_bounds__(row_threads(N), row_ctas(N)) k_lrow(cf* __restrict__ T, int64_t rows) {
  constexpr int R = row_threads(N), RS = row_stride(N);
  extern __shared__ __align__(16) unsigned char smraw[];
  cf* W = reinterpret_cast<cf*>(smraw);
  const int tid = threadIdx.x;
  const int64_t r0 = (int64_t)blockIdx.x * R;
  const int nr = (int)(rows - r0 < R ? rows - r0 : R);
  cf* g = T + r0 * N;
  if constexpr (N % 2 == 0) {
    constexpr int H = N / 2;
    const float4* g4 = reinterpret_cast<const float4*>(g);
#pragma unroll 8
    for (int i = tid; i < nr * H; i += R) {
      const int r = i / H;
      *reinterpret_cast<float4*>(W + r * RS + 2 * (i - r * H)) = g4[i];
    }
  } else {
#pragma unroll 8
    for (int i = tid; i < nr * N; i += R) {
      const int r = i / N;
      W[r * RS + (i - r * N)] = g[i];
    }
  }
  __syncthreads();
  if (tid < nr) {
    cf v[N];
    cf* w = W + tid * RS;
    if constexpr (N % 2 == 0) {
#pragma unroll
      for (int e = 0; e < N; e += 2) {
        const float4 q = *reinterpret_cast<const float4*>(w + e);
        v[e] = make_float2(q.x, q.y);
        v[e + 1] = make_float2(q.z, q.w);
      }
    } else {
#pragma unroll
      for (int e = 0; e < N; ++e) v[e] = w[e];
    }
    LD<N, INV>::run(v);
    if constexpr (N % 2 == 0) {
#pragma unroll
      for (int e = 0; e < N; e += 2)
        *reinterpret_cast<float4*>(w + e) = make_float4(v[e].x, v[e].y, v[e + 1].x, v[e + 1].y);
    } else {
#pragma unroll
      for (int e = 0; e < N; ++e) w[e] = v[e];
    }
  }
  __syncthreads();
  if constexpr (N % 2 == 0) {
    constexpr int H = N / 2;
    float4* g4 = reinterpret_cast<float4*>(g);
#pragma unroll 8
    for (int i = tid; i < nr * H; i += R) {
      const int r = i / H;
      g4[i] = *reinterpret_cast<const float4*>(W + r * RS + 2 * (i - r * H));
    }
  } else {
#pragma unroll 8
    for (int i = tid; i < nr * N; i += R) {
      const int r = i / N;
      g[i] = W[r * RS + (i - r * N)];
    }
  }
}

// ---- kernel table of one axis length ---------------------------------------------
struct LineOps {
  int n = 0;
  const void* col[5] = {};    // by ColMode, runtime element stride
  const void* row[2] = {};    // forward, inverse
};

template <int N>
LineOps line_ops_of() {
  LineOps o;
  o.n = N;
  o.col[kZMask] = reinterpret_cast<const void*>(&k_lcol<N, kZMask, 0>);
  o.col[kZFwd] = reinterpret_cast<const void*>(&k_lcol<N, kZFwd, 0>);
  o.col[kZInv] = reinterpret_cast<const void*>(&k_lcol<N, kZInv, 0>);
  o.col[kYFwdMul] = reinterpret_cast<const void*>(&k_lcol<N, kYFwdMul, 0>);
  o.col[kYInv] = reinterpret_cast<const void*>(&k_lcol<N, kYInv, 0>);
  o.row[0] = reinterpret_cast<const void*>(&k_lrow<N, false>);
  o.row[1] = reinterpret_cast<const void*>(&k_lrow<N, true>);
  return o;
}

// the lengths are spread over several translation units (sense_line_*.cu)
const LineOps* line_ops_a(int n);
const LineOps* line_ops_b(int n);
const LineOps* line_ops_c(int n);
const LineOps* line_ops_d(int n);

template <int... N>
const LineOps* line_ops_pick(int n) {
  static const LineOps table[] = {line_ops_of<N>()...};
  for (const LineOps& o : table)
    if (o.n == n) return &o;
  return nullptr;
}

}  // namespace line
}  // namespace mslr
