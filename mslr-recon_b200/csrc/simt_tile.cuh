// simt_tile.cuh — 64 × 64 complex FP32 matrix product tiles on the CUDA cores,
// shared by the plain form's Gram and rebuild (svst.cu) and by the products of
// the gradient (grad.cu).
//
// Bound by the FP32 pipes (8 flops per complex product).  What a tile needs
// beside them is kept below their time:
//  * 128 threads with 4 × 8 outputs each: per step of the contraction 64
//    packed FFMA (128 pipe cycles a warp) against six 16-byte shared loads
//    (a warp's load takes four LSU cycles, the LSU serves four schedulers: 96
//    cycles).  4 × 4 outputs with 8-byte loads were bound by those.
//  * Two real sums per output, P = Σ x_a (x_b, y_b) and Q = Σ y_a (x_b, y_b),
//    whose recombination at the end gives any conjugation: no sign or swap
//    inside the loop, and a sum takes one rounding per step, as the sum of
//    the products formed first did.
//  * The next 16 steps' operands are loaded to registers while the current
//    ones are multiplied, into the other of two buffers: one barrier per 16.
//  * Addresses: an operand is a pointer, a stride and an offset function of
//    its contiguous index that a thread evaluates once per 16 steps (or once).
// Measured on 144 patches of 512 × 128 and one of 73728 × 128, mean of both
// (one product is 9.7 GFLOP, 130 us of the FP32 pipes): M̄ = W Ō + K M 831 ->
// 446 us, Ō Mᴴ 611 -> 208, M Mᴴ (three of four tiles) 456 -> 184, a batch of
// 128 × 128 products 58-65 -> 35; before are 256 threads with 4 × 4 outputs,
// products formed with separate additions and addresses from two divisions
// per element.
#pragma once
#include "patchmap.cuh"

namespace mslr {
namespace simt {

constexpr int kTile = 64;
constexpr int kKc = 16;
constexpr int kThreads = 128;
constexpr int kPitch = kTile + 2;   // 16-byte rows, 4 banks apart

struct Smem {
  cf a[2][kKc][kPitch];
  cf b[2][kKc][kPitch];
};

// How a thread's outputs lie in the tile: rows row(i), i < 4, columns col(j), j < 8
// (pairs, so that a warp's 16-byte loads are contiguous).
__device__ __forceinline__ int row(int i) { return (threadIdx.x >> 3) * 2 + (i & 1) + 32 * (i >> 1); }
__device__ __forceinline__ int col(int j) { return (threadIdx.x & 7) * 2 + (j & 1) + 16 * (j >> 1); }

struct Acc {
  cf p[4][8], q[4][8];
  __device__ __forceinline__ void zero() {
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) p[i][j] = q[i][j] = make_float2(0.f, 0.f);
  }
  // Σ a b;  Σ conj(a) b;  Σ a conj(b)
  __device__ __forceinline__ cf ab(int i, int j) const {
    return make_float2(p[i][j].x - q[i][j].y, p[i][j].y + q[i][j].x);
  }
  __device__ __forceinline__ cf cab(int i, int j) const {
    return make_float2(p[i][j].x + q[i][j].y, p[i][j].y - q[i][j].x);
  }
  __device__ __forceinline__ cf acb(int i, int j) const {
    return make_float2(p[i][j].x + q[i][j].y, q[i][j].x - p[i][j].y);
  }
};

// An operand's 64 × 16 slices, loaded with the index that is contiguous in
// memory fastest across threads.  Elements (r, k), r < rlim, k < the loop's
// end; others are 0.
//   KF (k contiguous): base[koff(k) + r · step]
//   !KF (r contiguous): base[roff(r) + k · step]
template <bool KF, class Off>
struct Operand {
  const cf* base;
  int64_t step;
  bool rok;      // !KF: this thread's r is in range
  int rlim;      // KF
  Off off;
  __device__ __forceinline__ Operand(const cf* img, int64_t stp, int r0, int rl, Off o) : step(stp), off(o) {
    if (KF) {
      rlim = rl - r0;
      rok = true;
      base = img + (r0 + (int)(threadIdx.x >> 4)) * stp;
    } else {
      const int r = r0 + (threadIdx.x & 63);
      rok = r < rl;
      rlim = 0;
      base = img + (rok ? off(r) : 0);
    }
  }
  __device__ __forceinline__ void load(cf (&v)[8], int k0, int kend) const {
    if (KF) {
      const int k = k0 + (threadIdx.x & 15);
      const bool ok = k < kend;
      const cf* q = base + (ok ? off(k) : 0);
      const int r = threadIdx.x >> 4;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        v[j] = (ok && r + 8 * j < rlim) ? q[8 * j * step] : make_float2(0.f, 0.f);
    } else {
      const int k = k0 + (threadIdx.x >> 6);
      const cf* q = base + k * step;
#pragma unroll
      for (int j = 0; j < 8; ++j)
        v[j] = (rok && k + 2 * j < kend) ? q[2 * j * step] : make_float2(0.f, 0.f);
    }
  }
  static __device__ __forceinline__ void store(const cf (&v)[8], cf (*s)[kPitch]) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (KF) s[threadIdx.x & 15][(threadIdx.x >> 4) + 8 * j] = v[j];
      else s[(threadIdx.x >> 6) + 2 * j][threadIdx.x & 63] = v[j];
    }
  }
};

__device__ __forceinline__ void slice(const cf (*as)[kPitch], const cf (*bs)[kPitch], Acc& c) {
  const int ty = threadIdx.x >> 3, tx = threadIdx.x & 7;
#pragma unroll
  for (int k = 0; k < kKc; ++k) {
    const float4* ar = reinterpret_cast<const float4*>(as[k]);
    const float4* br = reinterpret_cast<const float4*>(bs[k]);
    const float4 a0 = ar[ty], a1 = ar[ty + 16];
    const cf a[4] = {make_float2(a0.x, a0.y), make_float2(a0.z, a0.w), make_float2(a1.x, a1.y),
                     make_float2(a1.z, a1.w)};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float4 b4 = br[tx + 8 * j];
      const cf b0 = make_float2(b4.x, b4.y), b1 = make_float2(b4.z, b4.w);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const cf ax = make_float2(a[i].x, a[i].x), ay = make_float2(a[i].y, a[i].y);
        c.p[i][2 * j] = __ffma2_rn(ax, b0, c.p[i][2 * j]);
        c.q[i][2 * j] = __ffma2_rn(ay, b0, c.q[i][2 * j]);
        c.p[i][2 * j + 1] = __ffma2_rn(ax, b1, c.p[i][2 * j + 1]);
        c.q[i][2 * j + 1] = __ffma2_rn(ay, b1, c.q[i][2 * j + 1]);
      }
    }
  }
}

// c += Σ_{k in [kb, ke)} a(·, k) ⊗ b(·, k); same: b's slices are a's.  Ends
// with a barrier, so that the buffers can be used again.
template <class A, class B>
__device__ __forceinline__ void accumulate(Smem& s, const A& a, const B& b, int kb, int ke, bool same, Acc& c) {
  cf va[8], vb[8];
  a.load(va, kb, ke);
  if (!same) b.load(vb, kb, ke);
  int cur = 0;
  for (int k0 = kb; k0 < ke; k0 += kKc) {
    A::store(va, s.a[cur]);
    if (!same) B::store(vb, s.b[cur]);
    __syncthreads();
    if (k0 + kKc < ke) {
      a.load(va, k0 + kKc, ke);
      if (!same) b.load(vb, k0 + kKc, ke);
    }
    slice(s.a[cur], same ? s.a[cur] : s.b[cur], c);
    cur ^= 1;
  }
  __syncthreads();
}

struct Linear {
  __device__ __forceinline__ int64_t operator()(int l) const { return l; }
};
struct InPatch {
  const PatchMap& m;
  __device__ __forceinline__ int64_t operator()(int l) const { return patch_off(m, l); }
};

// Rows M[·][l] (without the conjugation of a tall patch's M) as an operand
// whose contraction runs over l: tall patches are contiguous in l, wide in a.
template <bool TALL>
__device__ __forceinline__ Operand<TALL, InPatch> rows_of(const PatchMap& m, const cf* img, int64_t org, int a0) {
  return Operand<TALL, InPatch>(img + org, tstride(m), a0, m.n, InPatch{m});
}

// The same image as the right operand of W M: columns l, contraction over a.
template <bool TALL>
__device__ __forceinline__ Operand<!TALL, InPatch> cols_of(const PatchMap& m, const cf* img, int64_t org, int l0) {
  return Operand<!TALL, InPatch>(img + org, tstride(m), l0, m.L, InPatch{m});
}

// Writes the tile of M_out at (a0, l0): into the image when direct, else into
// the per-patch buffer (p, Nt, Np).  W's conjugation for tall patches is taken here.
template <bool TALL>
__device__ __forceinline__ void put_tile(const PatchMap& m, const Acc& c, int64_t org, int64_t ip, int a0, int l0,
                                         cf* out, int direct) {
  const int64_t vs = direct ? tstride(m) : (int64_t)m.p;
  cf* o = direct ? out + org : out + ip * m.Nt * (int64_t)m.p;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      const int a = a0 + row(i), l = l0 + col(j);
      if (a >= m.n || l >= m.L) continue;
      const int pv = TALL ? l : a, tt = TALL ? a : l;
      o[(direct ? patch_off(m, pv) : (int64_t)pv) + tt * vs] = TALL ? c.cab(i, j) : c.ab(i, j);
    }
  }
}

}  // namespace simt
}  // namespace mslr
