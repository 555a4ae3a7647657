// gram_umma.cu — patch Grams and rebuilds on the 5th-generation tensor cores
// (tcgen05.mma, accumulators in tensor memory) for the tuned form.
//
// Patch Grams and rebuilds as complex GEMMs over rows with the
// contraction index K contiguous:
//   Gram     G[a][b]      = Σ_l M[a][l] conj(M[b][l])      (A = B = rows of M)
//   rebuild  M_out[a][l]  = Σ_b W[a][b] M[b][l]            (A = rows of W, B = columns of M)
// with M = Pᴴ for tall patches (p >= Nt), M = P otherwise.  Complex values are
// split into planar real / imaginary BF16 tiles, each FP32 value v carried as
// hi = bf16(v) and lo = bf16(v − hi); a real product x·y is hi·hi + hi·lo +
// lo·hi with FP32 accumulation.  Per 16-element K step one thread issues 12
// M=128 × N=128 × K=16 MMAs into two accumulators (real, imaginary; 256 TMEM
// columns):
//   Gram     Re += Ar·Brᵀ + Ai·Biᵀ      Im += Ai·Brᵀ − Ar·Biᵀ
//   rebuild  Re += Ar·Brᵀ − Ai·Biᵀ      Im += Ar·Biᵀ + Ai·Brᵀ
// (negation through the instruction descriptor).
//
// The TF32 form runs the same products with TF32 operands (one FP32 plane per
// part, rounded to TF32) and four M=128 × N=128 × K=8 kind::tf32 MMAs per
// 8-element K step: Gram Re += Ar·Brᵀ + Ai·Biᵀ, Im += Ai·Brᵀ − Ar·Biᵀ (the
// rebuild's signs as above).
//
// One CTA of 8 warps per 128 × 128 output tile, two CTAs per SM (all of its
// tensor memory).  K advances 16 elements per chunk: every thread loads its
// share of the next chunk from global memory into registers (patch element
// addresses from per-row / per-K offset tables; a diagonal Gram tile, which
// has one operand, the next two chunks) while the tensor core works on the
// current chunk, then converts it into the K-major, unswizzled core-matrix
// layout of a free stage (two stages, 8 tiles of 4 KB each).  What bounds the
// kernels is the chain load → convert → barrier → MMA of a tile and its
// epilogue, not a pipe (LSU 47 %, issue 21 %, tensor cores below that): the
// two CTAs run one tile's chain under the other's.  With chunks of 32 and one
// CTA per SM, and tall rebuilds stored a row per lane (32 lines a store), 486
// patches of 1000 × 300 took 3.34 ms to rebuild, 1.78 for their Grams and 0.60
// for W; now 1.93, 1.42 and 0.44.  Grams whose tiles have an SM each still go in
// chunks of 32 (gram_umma_launch).  A Gram of at most 64 rows takes half of each
// operand and half the columns of an MMA (one 216 × 64: 17.4 -> 15.2 us, its rebuild
// 12.8 -> 10.7; 240 of 343 × 50: 48 -> 31 and 65 -> 42).
// A stage is reused only after the tcgen05.commit of
// the MMAs that read it has arrived on the stage's mbarrier.  The epilogue
// reads the accumulators with tcgen05.ld (warp w: TMEM lanes 32·(w mod 4),
// columns 64·(w / 4)); stores along a row's columns go through shared memory so
// that 16 lanes share a line.  Every wait is bounded (DevWait::polls polls).  On a
// time-out the kernel stops issuing work, thread 0 waits (with the default
// poll count) for the MMAs it has already committed, the output tile is
// written as zeros, the tensor memory is freed and kErrMmaWait is raised in
// the caller's error word.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <mutex>
#include <type_traits>

#include "internal.h"
#include "patchmap.cuh"

namespace mslr {

namespace {

constexpr int kTM = 128;          // output rows per CTA (TMEM lanes)
constexpr int kTN = 128;          // output columns per CTA
constexpr int kThr = 256;
constexpr int kTmemCols = 256;
// K elements per chunk (KC): 16, two CTAs per SM, or 32, one CTA (see gram_umma_launch)
constexpr int tile_words(int KC) { return kTM * KC / 2; }         // bf16 pairs of a planar tile
constexpr int pairs_of(int KC) { return tile_words(KC) / kThr; }   // per thread and operand: 4 or 8
constexpr int ctas_of(int KC) { return KC == 16 ? 2 : 1; }

enum { AR_H, AR_L, AI_H, AI_L, BR_H, BR_L, BI_H, BI_L, NOPS };

template <int KC>
struct USmem {
  uint32_t op[2][NOPS][tile_words(KC)];   // two stages × 8 tiles of 128 × KC bf16 (as bf16 pairs)
  int rowA[kTM], rowB[kTN];
  int kof[2][KC];
  uint64_t bar[2];
  uint32_t tmem;
};

__device__ __forceinline__ unsigned su32(const void* p) {
  return (unsigned)__cvta_generic_to_shared(p);
}

// word index of the bf16 pair (r, k..k+1), k even, in a K-major unswizzled tile:
// 8-row × 8-element core matrices of 128 bytes, k-adjacent cores 128 B apart
// (LBO), 8-row groups KC / 8 of them apart (SBO)
template <int KC>
__device__ __forceinline__ int pair_word(int r, int k) {
  return ((r >> 3) * (KC / 8) + (k >> 3)) * 32 + (r & 7) * 4 + ((k & 7) >> 1);
}

// shared-memory matrix descriptor (sm_100 layout): start, LBO = 128 B, SBO =
// KC / 8 · 128 B, version 1, no swizzle
template <int KC>
__device__ __forceinline__ uint64_t sdesc(const void* p) {
  const uint64_t a = su32(p);
  return ((a >> 4) & 0x3FFFull) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)((KC / 8 * 128) >> 4) << 32) |
         (1ull << 46);
}

// Operand modes.  kF16 serves operands whose values are at most 1 (the scaled
// eigenvectors), times 2¹⁰: hi = bf16(v), exact in FP16, and lo = fp16(v − hi),
// three bits more than a BF16 lo at the same number of MMAs, so that what is
// left out of v shrinks from 2⁻¹⁷ to 2⁻²⁰ of it; the product is scaled back by
// 2⁻²⁰.  Fixed range, so not for image data.
enum Mode { kBf16 = 0, kTf32 = 1, kF16 = 2 };
constexpr float kF16Scale = 1024.f;

// instruction descriptor: BF16 × BF16 (F16 × F16) → F32, both K-major, M = 128; N is added by with_n
__host__ __device__ constexpr uint32_t idesc(bool negA, bool f16 = false) {
  return (1u << 4) | (f16 ? 0u : (1u << 7) | (1u << 10)) | ((negA ? 1u : 0u) << 13) | ((uint32_t)(kTM >> 4) << 24);
}
// N columns, rounded up to the 16 that M = 128 takes
__device__ __forceinline__ uint32_t with_n(uint32_t id, int N) { return id | (uint32_t)((N + 15) >> 4 << 1) << 17; }

__device__ __forceinline__ void umma(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t id, bool acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
      "l"(a), "l"(b), "r"(id), "r"(acc ? 1u : 0u));
}
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(
                   su32(bar))
               : "memory");
}
__device__ __forceinline__ void tc_fence_after() {
  asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void tc_fence_before() {
  asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
}
__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(su32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity, int polls) {
  const unsigned a = su32(bar);
  for (int it = 0; it < polls; ++it) {
    unsigned ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(a), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// 16 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float (&v)[16]) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, "
      "%12, %13, %14, %15}, [%16];\n"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// hi/lo split of two consecutive values into packed bf16 pairs (k in the low half)
__device__ __forceinline__ void split_pair(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  const __nv_bfloat162 h = __floats2bfloat162_rn(x0, x1);
  const float2 hf = __bfloat1622float2(h);
  const __nv_bfloat162 l = __floats2bfloat162_rn(x0 - hf.x, x1 - hf.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

__device__ __forceinline__ void split_pair_f16(float x0, float x1, uint32_t& hi, uint32_t& lo) {
  x0 *= kF16Scale;
  x1 *= kF16Scale;
  const float2 hf = __bfloat1622float2(__floats2bfloat162_rn(x0, x1));
  const __half2 h = __floats2half2_rn(hf.x, hf.y);
  const __half2 l = __floats2half2_rn(x0 - hf.x, x1 - hf.y);
  hi = *reinterpret_cast<const uint32_t*>(&h);
  lo = *reinterpret_cast<const uint32_t*>(&l);
}

// TF32 operands (the TF32 form): one FP32 plane per real / imaginary part,
// each value rounded to TF32 (to nearest, ties away), in K-major unswizzled
// core matrices of 8 rows × 4 values (128 bytes): k-adjacent cores 128 B apart
// (LBO), 8-row groups KC / 4 of them apart (SBO).  A chunk of KC values is KC / 8
// 8-value MMA steps.  Planes per stage: Ar, Ai, Br, Bi of 128 · KC words each.
constexpr int tf_plane(int KC) { return kTM * KC; }   // words per TF32 plane

__device__ __forceinline__ uint32_t to_tf32(float x) {
  uint32_t r;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(r) : "f"(x));
  return r;
}
template <int KC>
__device__ __forceinline__ int tf_word(int r, int k) {
  return ((r >> 3) * (KC / 4) + (k >> 2)) * 32 + (r & 7) * 4 + (k & 3);
}
template <int KC>
__device__ __forceinline__ uint64_t sdesc_tf(const void* p) {
  const uint64_t a = su32(p);
  return ((a >> 4) & 0x3FFFull) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)((KC / 4 * 128) >> 4) << 32) |
         (1ull << 46);
}
// instruction descriptor: TF32 × TF32 → F32, both K-major, M = 128; N is added by with_n
__host__ __device__ constexpr uint32_t idesc_tf(bool negA) {
  return (1u << 4) | (2u << 7) | (2u << 10) | ((negA ? 1u : 0u) << 13) | ((uint32_t)(kTM >> 4) << 24);
}
__device__ __forceinline__ void umma_tf(uint32_t dtmem, uint64_t a, uint64_t b, uint32_t id, bool acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, p;\n}\n" ::"r"(dtmem),
      "l"(a), "l"(b), "r"(id), "r"(acc ? 1u : 0u));
}

// Registers of one operand chunk: thread t holds pairs q = t + 256 i, i < KC / 4,
// of the 128 × KC tile; pair q is (row r, k..k+1) of core c = q / 32, so pair i
// lies in the i-th of KC / 4 equal groups of rows.  A Gram's tile of at most 64
// rows takes the first half only (NI = KC / 8): what the stage holds beyond
// reaches no output.
template <int KC>
struct Chunk {
  cf v[pairs_of(KC)][2];
};

template <int KC>
__device__ __forceinline__ void pair_rk(int i, int& r, int& k) {
  constexpr int CK = KC / 8;   // cores along K
  const int q = threadIdx.x + kThr * i;
  const int c = q >> 5, w = q & 31;
  r = (c / CK) * 8 + (w >> 2);
  k = (c % CK) * 8 + (w & 3) * 2;
}

template <int KC, int NI>
__device__ __forceinline__ void load_chunk(Chunk<KC>& ch, const cf* __restrict__ base, const int* row,
                                           const int* kof) {
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    int r, k;
    pair_rk<KC>(i, r, k);
    const int ro = row[r];
#pragma unroll
    for (int d = 0; d < 2; ++d) {
      const int ko = kof[k + d];
      ch.v[i][d] = (ro >= 0 && ko >= 0) ? __ldg(base + (int64_t)ro + ko) : make_float2(0.f, 0.f);
    }
  }
}

// chunk → planar hi / lo tiles (re_h, re_l, im_h, im_l), conjugated when conj
template <int KC, bool F16, int NI>
__device__ __forceinline__ void store_chunk(const Chunk<KC>& ch, uint32_t* rh, uint32_t* rl,
                                            uint32_t* ih, uint32_t* il, bool conj) {
#pragma unroll
  for (int i = 0; i < NI; ++i) {
    int r, k;
    pair_rk<KC>(i, r, k);
    const int w = pair_word<KC>(r, k);
    const cf a = ch.v[i][0], b = ch.v[i][1];
    const float ai = conj ? -a.y : a.y, bi = conj ? -b.y : b.y;
    uint32_t h, l;
    if constexpr (F16) split_pair_f16(a.x, b.x, h, l);
    else split_pair(a.x, b.x, h, l);
    rh[w] = h;
    rl[w] = l;
    if constexpr (F16) split_pair_f16(ai, bi, h, l);
    else split_pair(ai, bi, h, l);
    ih[w] = h;
    il[w] = l;
  }
}

// One operand chunk into stage `stage` (B operand when isB), conjugated when conj.
template <int KC, int MODE, int NI>
__device__ __forceinline__ void store_operand(const Chunk<KC>& ch, uint32_t* stage, bool isB, bool conj) {
  if constexpr (MODE == kTf32) {
    uint32_t* re = stage + (isB ? 2 : 0) * tf_plane(KC);
    uint32_t* im = stage + (isB ? 3 : 1) * tf_plane(KC);
#pragma unroll
    for (int i = 0; i < NI; ++i) {
      int r, k;
      pair_rk<KC>(i, r, k);
      const int w = tf_word<KC>(r, k);
      const cf a = ch.v[i][0], b = ch.v[i][1];
      *reinterpret_cast<uint2*>(re + w) = make_uint2(to_tf32(a.x), to_tf32(b.x));
      *reinterpret_cast<uint2*>(im + w) = make_uint2(to_tf32(conj ? -a.y : a.y), to_tf32(conj ? -b.y : b.y));
    }
  } else {
    uint32_t* o = stage + (isB ? BR_H : AR_H) * tile_words(KC);
    store_chunk<KC, MODE == kF16, NI>(ch, o, o + tile_words(KC), o + 2 * tile_words(KC), o + 3 * tile_words(KC), conj);
  }
}

// The 12 MMAs of a 16-element K step of stage st.
template <int KC, bool GRAM, bool F16>
__device__ __forceinline__ void issue_step(const USmem<KC>& s, int st, int step, uint32_t dre, uint32_t dim, bool acc,
                                           bool bSameAsA, int cols) {
  const uint32_t* o = &s.op[st][0][0] + step * 64;   // two cores a step
  auto A = [&](int k) { return sdesc<KC>(o + k * tile_words(KC)); };
  const int bro = bSameAsA ? AR_H : BR_H;   // B operands: same tiles as A on diagonal Gram tiles
  auto B = [&](int k) { return sdesc<KC>(o + (bro + (k - BR_H)) * tile_words(KC)); };
  const uint32_t P = with_n(idesc(false, F16), cols), N = with_n(idesc(true, F16), cols);
  // real part
  umma(dre, A(AR_H), B(BR_H), P, acc);
  umma(dre, A(AR_H), B(BR_L), P, true);
  umma(dre, A(AR_L), B(BR_H), P, true);
  umma(dre, A(AI_H), B(BI_H), GRAM ? P : N, true);
  umma(dre, A(AI_H), B(BI_L), GRAM ? P : N, true);
  umma(dre, A(AI_L), B(BI_H), GRAM ? P : N, true);
  // imaginary part
  if (GRAM) {
    umma(dim, A(AI_H), B(BR_H), P, acc);
    umma(dim, A(AI_H), B(BR_L), P, true);
    umma(dim, A(AI_L), B(BR_H), P, true);
    umma(dim, A(AR_H), B(BI_H), N, true);
    umma(dim, A(AR_H), B(BI_L), N, true);
    umma(dim, A(AR_L), B(BI_H), N, true);
  } else {
    umma(dim, A(AR_H), B(BI_H), P, acc);
    umma(dim, A(AR_H), B(BI_L), P, true);
    umma(dim, A(AR_L), B(BI_H), P, true);
    umma(dim, A(AI_H), B(BR_H), P, true);
    umma(dim, A(AI_H), B(BR_L), P, true);
    umma(dim, A(AI_L), B(BR_H), P, true);
  }
}

// All MMAs of the chunk in stage st (first: the accumulators start from zero).
template <int KC, bool GRAM, int MODE>
__device__ __forceinline__ void issue_chunk(const USmem<KC>& s, int st, uint32_t dre, uint32_t dim,
                                            bool first, bool bSameAsA, int cols) {
  if constexpr (MODE == kTf32) {
    const uint32_t* o = &s.op[st][0][0];
    const int br = bSameAsA ? 0 : 2, bi = bSameAsA ? 1 : 3;
    const uint32_t P = with_n(idesc_tf(false), cols), N = with_n(idesc_tf(true), cols);
#pragma unroll
    for (int t = 0; t < KC / 8; ++t) {
      auto D = [&](int pl) { return sdesc_tf<KC>(o + pl * tf_plane(KC) + t * 64); };   // +2 cores = 256 B
      const bool acc = !first || t > 0;
      // Gram:    Re += Ar·Brᵀ + Ai·Biᵀ   Im += Ai·Brᵀ − Ar·Biᵀ
      // rebuild: Re += Ar·Brᵀ − Ai·Biᵀ   Im += Ar·Biᵀ + Ai·Brᵀ
      umma_tf(dre, D(0), D(br), P, acc);
      umma_tf(dre, D(1), D(bi), GRAM ? P : N, true);
      if (GRAM) {
        umma_tf(dim, D(1), D(br), P, acc);
        umma_tf(dim, D(0), D(bi), N, true);
      } else {
        umma_tf(dim, D(0), D(bi), P, acc);
        umma_tf(dim, D(1), D(br), P, true);
      }
    }
  } else {
#pragma unroll
    for (int t = 0; t < KC / 16; ++t)
      issue_step<KC, GRAM, MODE == kF16>(s, st, t, dre, dim, !first || t > 0, bSameAsA, cols);
  }
}

// Commits of thread 0 that it has not yet seen arrive: at most one per stage
// barrier, since a stage is refilled (and committed again) only after its
// previous commit has been observed.
struct Pending {
  int c0 = -1, c1 = -1;   // chunk committed on bar[0] / bar[1], -1 when none is pending
  __device__ void committed(int ch) {
    if (ch & 1) c1 = ch;
    else c0 = ch;
  }
  __device__ void observed(int ch) {
    if (ch & 1) c1 = -1;
    else c0 = -1;
  }
  // After a timed-out wait: thread 0 waits, with the default poll count, for
  // every commit still pending, so that no MMA reads shared memory or writes
  // tensor memory after the kernel frees them and returns.
  template <int KC>
  __device__ void drain(USmem<KC>& s) const {
    if (c0 >= 0) mbar_wait(&s.bar[0], (unsigned)((c0 >> 1) & 1), kWaitPolls);
    if (c1 >= 0) mbar_wait(&s.bar[1], (unsigned)((c1 >> 1) & 1), kWaitPolls);
  }
};

// Main loop shared by both kernels: nch chunks; kofs(c, buf) fills s.kof[buf]
// for chunk c (threads < KC; chunks 0 and 1 are in place).  Returns false when
// a wait timed out.
//
// One chunk of the main loop: its operands, already in registers, into stage
// c mod 2; the loads that `next` issues run under its MMAs.
template <int KC, bool GRAM, int MODE, class Store, class Next>
__device__ __forceinline__ void chunk_step(USmem<KC>& s, int c, bool& ok, Pending& pend, bool bSameAsA, int cols, int polls,
                                           const Store& store, const Next& next) {
  const int st = c & 1;
  if (c >= 2 && ok) {
    if (mbar_wait(&s.bar[st], (unsigned)(((c - 2) >> 1) & 1), polls)) pend.observed(c - 2);
    else ok = false;
  }
  if (ok) store(&s.op[st][0][0]);
  fence_async_smem();
  // the only barrier of a chunk: while thread 0 issues its MMAs the others fill
  // the other stage; s.kof's slots are rewritten two barriers after being read
  ok = __syncthreads_and(ok);
  next();
  if (threadIdx.x == 0 && ok) {
    tc_fence_after();
    issue_chunk<KC, GRAM, MODE>(s, st, s.tmem, s.tmem + kTN, c == 0, bSameAsA, cols);
    umma_commit(&s.bar[st]);
    pend.committed(c);
  }
}

template <int KC>
__device__ __forceinline__ bool mainloop_end(USmem<KC>& s, int nch, bool ok, Pending& pend, int polls) {
  if (nch > 0 && ok) {
    const int l = nch - 1;
    if (mbar_wait(&s.bar[l & 1], (unsigned)((l >> 1) & 1), polls)) pend.observed(l);
    else ok = false;
  }
  ok = __syncthreads_and(ok);
  if (!ok && threadIdx.x == 0) pend.drain(s);
  tc_fence_after();
  __syncthreads();
  return ok;
}

// Two operands, cols rows of B; load(c, buf) brings chunk c of both to registers.
template <int KC, bool GRAM, int MODE, class KOfs, class Load>
__device__ __forceinline__ bool mainloop(USmem<KC>& s, int nch, Chunk<KC>& ca, Chunk<KC>& cb, bool conjA, bool conjB,
                                         int cols, const KOfs& kofs, const Load& load, int polls) {
  bool ok = true;
  Pending pend;
  if (nch > 0) load(0, 0);
  __syncthreads();
  for (int c = 0; c < nch; ++c) {
    if (c > 0 && c + 1 < nch) kofs(c + 1, (c + 1) & 1);
    chunk_step<KC, GRAM, MODE>(
        s, c, ok, pend, false, cols, polls,
        [&](uint32_t* stage) {
          store_operand<KC, MODE, pairs_of(KC)>(ca, stage, false, conjA);
          store_operand<KC, MODE, pairs_of(KC)>(cb, stage, true, conjB);
        },
        [&] {
          if (c + 1 < nch) load(c + 1, (c + 1) & 1);
        });
  }
  return mainloop_end(s, nch, ok, pend, polls);
}

// One operand on both sides (a Gram's diagonal tiles): with the registers of
// the second, two chunks of loads are under way.  load(x, c, buf): chunk c into x.
template <int KC, int MODE, int NI, class KOfs, class Load>
__device__ __forceinline__ bool mainloop_same(USmem<KC>& s, int nch, Chunk<KC>& c0, Chunk<KC>& c1, bool conj, int rows,
                                              const KOfs& kofs, const Load& load, int polls) {
  bool ok = true;
  Pending pend;
  if (nch > 0) load(c0, 0, 0);
  if (nch > 1) load(c1, 1, 1);
  __syncthreads();
  auto step = [&](Chunk<KC>& x, int c) {
    if (c + 2 < nch) kofs(c + 2, c & 1);
    chunk_step<KC, true, MODE>(
        s, c, ok, pend, true, rows, polls,
        [&](uint32_t* stage) { store_operand<KC, MODE, NI>(x, stage, false, conj); },
        [&] {
          if (c + 2 < nch) load(x, c + 2, c & 1);
        });
  };
  for (int c = 0; c < nch; c += 2) {
    step(c0, c);
    if (c + 1 < nch) step(c1, c + 1);
  }
  return mainloop_end(s, nch, ok, pend, polls);
}

template <int KC>
__device__ __forceinline__ void tmem_alloc(USmem<KC>& s) {
  if ((threadIdx.x >> 5) == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(
                     su32(&s.tmem)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
  }
  if (threadIdx.x == 0) {
    mbar_init(&s.bar[0]);
    mbar_init(&s.bar[1]);
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
}

template <int KC>
__device__ __forceinline__ void tmem_free(USmem<KC>& s) {
  tc_fence_before();
  __syncthreads();
  if ((threadIdx.x >> 5) == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(s.tmem),
                 "r"(kTmemCols)
                 : "memory");
}

// A warp's 32 rows × 16 columns of a tile, from lane = row to 16 lanes along a
// row and two rows per access: 16 consecutive columns leave in one store where
// lane = row would touch 32 lines.  Uses the operand stages, which no MMA reads
// any more; put(row, column, value) for this lane's share.
template <int KC, class Put>
__device__ __forceinline__ void by_columns(USmem<KC>& s, const cf (&v)[16], const Put& put) {
  cf* t = reinterpret_cast<cf*>(&s.op[0][0][0]) + (threadIdx.x >> 5) * (32 * 17);
  const int lane = threadIdx.x & 31;
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 16; ++j) t[lane * 17 + j] = v[j];
  __syncwarp();
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int r = 2 * i + (lane >> 4), j = lane & 15;
    put(r, j, t[r * 17 + j]);
  }
}

// ---------------------------------------------------------------------------
// kcols (or null): the patch's contraction stops at kcols[ip] values (the
// eigenvectors beyond the rank are zero).
template <int MODE, int KC>
__global__ void __launch_bounds__(kThr, ctas_of(KC))
    k_gram_umma(const cf* __restrict__ img, PatchMap m, cf* __restrict__ out, int nsplit,
                int lchunk, const int* __restrict__ kcols, DevWait dw) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  USmem<KC>& s = *reinterpret_cast<USmem<KC>*>(smraw);
  constexpr int kPairs = pairs_of(KC);
  int t = blockIdx.x, ta = 0;
  while (t > ta) {
    t -= ta + 1;
    ++ta;
  }
  const int tb = t;
  const bool diag = (ta == tb);
  const int64_t ip = blockIdx.y;
  const int split = blockIdx.z;
  const int64_t org = patch_origin(m, ip);
  const int64_t ts = tstride(m);
  const int a0 = ta * kTM, b0 = tb * kTN;
  const int l_begin = split * lchunk;
  const int l_end = min(kcols ? kcols[ip] : m.L, l_begin + lchunk);
  const int n = m.n;
  const int nch = l_end > l_begin ? (l_end - l_begin + KC - 1) / KC : 0;
  tmem_alloc(s);
  for (int r = threadIdx.x; r < kTM; r += kThr) {
    const int a = a0 + r, b = b0 + r;
    s.rowA[r] = (a < n) ? (int)(m.tall ? (int64_t)a * ts : patch_off(m, a)) : -1;
    s.rowB[r] = (b < n) ? (int)(m.tall ? (int64_t)b * ts : patch_off(m, b)) : -1;
  }
  auto kofs = [&](int c, int buf) {
    if (threadIdx.x < KC) {
      const int l = l_begin + c * KC + threadIdx.x;
      s.kof[buf][threadIdx.x] = (l < l_end) ? (int)(m.tall ? patch_off(m, l) : (int64_t)l * ts) : -1;
    }
  };
  kofs(0, 0);
  kofs(1, 1);
  __syncthreads();
  tc_fence_after();
  const cf* base = img + org;
  const bool cj = m.tall != 0;
  Chunk<KC> ca, cb;
  const int ra = min(kTM, n - a0);
  bool ok;
  if (diag) {
    auto one = [&](auto ni) {
      constexpr int NI = decltype(ni)::value;
      return mainloop_same<KC, MODE, NI>(
          s, nch, ca, cb, cj, ra, kofs,
          [&](Chunk<KC>& x, int, int buf) { load_chunk<KC, NI>(x, base, s.rowA, s.kof[buf]); }, dw.polls);
    };
    ok = ra <= kTM / 2 ? one(std::integral_constant<int, kPairs / 2>{}) : one(std::integral_constant<int, kPairs>{});
  } else {
    auto load = [&](int, int buf) {
      load_chunk<KC, kPairs>(ca, base, s.rowA, s.kof[buf]);
      load_chunk<KC, kPairs>(cb, base, s.rowB, s.kof[buf]);
    };
    ok = mainloop<KC, true, MODE>(s, nch, ca, cb, cj, cj, kTN, kofs, load, dw.polls);
  }
  cf* G = out + ((nsplit > 1) ? (int64_t)split * n * n : ip * (int64_t)n * n);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a = a0 + (warp & 3) * 32 + lane;
  // on a time-out the tile is written as zeros (a zero Gram: the eigen stage
  // then finds no singular value above the threshold) and the error raised
  if (!ok && threadIdx.x == 0 && dw.err) atomicOr(dw.err, kErrMmaWait);
  {
    for (int cb = 0; cb < 4; ++cb) {
      const int col = (warp >> 2) * 64 + cb * 16;
      const uint32_t taddr = s.tmem + ((uint32_t)((warp & 3) * 32) << 16) + col;
      float re[16], im[16];
      if (ok && nch > 0) {
        tmem_ld16(taddr, re);
        tmem_ld16(taddr + kTN, im);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) re[j] = im[j] = 0.f;
      }
      constexpr float sc = MODE == kF16 ? 1.f / (kF16Scale * kF16Scale) : 1.f;
      cf v[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        const int b = b0 + col + j;
        v[j] = make_float2(re[j] * sc, im[j] * sc);
        if (a < n && b < n) G[(int64_t)b * n + a] = v[j];
      }
      if (!diag)
        by_columns(s, v, [&](int r, int j, cf x) {
          const int ar = a0 + (warp & 3) * 32 + r, b = b0 + col + j;
          if (ar < n && b < n) G[(int64_t)ar * n + b] = cconj(x);
        });
    }
  }
  tmem_free(s);
}

// ---------------------------------------------------------------------------
template <int MODE>
__global__ void __launch_bounds__(kThr, 2)
    k_rebuild_umma(const cf* __restrict__ img, const cf* __restrict__ W, PatchMap m,
                   cf* __restrict__ out, int direct, DevWait dw) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  constexpr int KC = 16, kPairs = pairs_of(KC);
  USmem<KC>& s = *reinterpret_cast<USmem<KC>*>(smraw);
  const int a0 = blockIdx.x * kTM, l0 = blockIdx.y * kTN;
  const int64_t ip = blockIdx.z;
  const int n = m.n;
  const cf* Wp = W + ip * (int64_t)n * n;
  const int64_t org = patch_origin(m, ip);
  const int64_t ts = tstride(m);
  const int nch = (n + KC - 1) / KC;
  tmem_alloc(s);
  // A rows a: the stored W column a holds conj(W[a][·]); conjugated back on conversion.
  // B rows l: M[·][l] — tall: conj(img[b·ts + org + off(l)]); wide: img[l·ts + org + off(b)]
  for (int r = threadIdx.x; r < kTM; r += kThr) {
    const int a = a0 + r, l = l0 + r;
    s.rowA[r] = (a < n) ? a * n : -1;
    s.rowB[r] = (l < m.L) ? (int)(m.tall ? patch_off(m, l) : (int64_t)l * ts) : -1;
  }
  // the K offsets of A (b) and B (frame or voxel of b) differ: A uses kof + its own rows
  auto kofs = [&](int c, int buf) {
    if (threadIdx.x < KC) {
      const int b = c * KC + threadIdx.x;
      s.kof[buf][threadIdx.x] = (b < n) ? (int)(m.tall ? (int64_t)b * ts : patch_off(m, b)) : -1;
    }
  };
  kofs(0, 0);
  kofs(1, 1);
  __syncthreads();
  tc_fence_after();
  // A's element (a, b) is at Wp[a·n + b] (rows a·n in rowA, K offset b itself);
  // B's element (l, b) at org + rowB[l] + kof[b].
  Chunk<KC> ca, cb;
  auto load = [&](int c, int buf) {
#pragma unroll
    for (int i = 0; i < kPairs; ++i) {
      int r, k;
      pair_rk<KC>(i, r, k);
      const int ro = s.rowA[r];
#pragma unroll
      for (int d = 0; d < 2; ++d) {
        const int b = c * KC + k + d;
        ca.v[i][d] = (ro >= 0 && b < n) ? __ldg(Wp + ro + b) : make_float2(0.f, 0.f);
      }
    }
    load_chunk<KC, kPairs>(cb, img + org, s.rowB, s.kof[buf]);
  };
  const bool ok = mainloop<KC, false, MODE>(s, nch, ca, cb, true, m.tall != 0, min(kTN, m.L - l0), kofs, load, dw.polls);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int a = a0 + (warp & 3) * 32 + lane;
  // on a time-out the output tile is written as zeros and the error raised
  if (!ok && threadIdx.x == 0 && dw.err) atomicOr(dw.err, kErrMmaWait);
  {
    const int64_t offa = (a < n && !m.tall) ? patch_off(m, a) : 0;
    for (int cb = 0; cb < 4; ++cb) {
      const int col = (warp >> 2) * 64 + cb * 16;
      const uint32_t taddr = s.tmem + ((uint32_t)((warp & 3) * 32) << 16) + col;
      float re[16], im[16];
      if (ok && nch > 0) {
        tmem_ld16(taddr, re);
        tmem_ld16(taddr + kTN, im);
      } else {
#pragma unroll
        for (int j = 0; j < 16; ++j) re[j] = im[j] = 0.f;
      }
      if (m.tall) {   // frame a, voxel l: conj(M_out[a][l])
        cf v[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) v[j] = make_float2(re[j], -im[j]);
        const int l = l0 + col + (lane & 15);
        const int64_t rs = direct ? ts : (int64_t)m.p;
        cf* o = direct ? out + org + (l < m.L ? s.rowB[col + (lane & 15)] : 0)
                       : out + ip * m.Nt * (int64_t)m.p + l;
        by_columns(s, v, [&](int r, int, cf x) {
          const int f = a0 + (warp & 3) * 32 + r;
          if (f < n && l < m.L) o[f * rs] = x;
        });
      } else if (a < n) {   // frame l, voxel a
#pragma unroll
        for (int j = 0; j < 16; ++j) {
          const int l = l0 + col + j;
          if (l >= m.L) continue;
          const cf v = make_float2(re[j], im[j]);
          if (direct) out[org + offa + (int64_t)l * ts] = v;
          else out[(ip * m.Nt + l) * (int64_t)m.p + a] = v;
        }
      }
    }
  }
  tmem_free(s);
}

}  // namespace

// The 32-bit row and K offset tables of the tcgen05 kernels cover this map.
bool umma_supported(const PatchMap& m) {
  const int64_t span = m.batch ? m.mstride : (int64_t)m.Nt * m.nvox;
  return span < (int64_t)0x7fffffff && (int64_t)m.n * m.n < (int64_t)0x7fffffff;
}

int umma_prepare() {
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  MSLR_CUDA_TRY(cudaGetDevice(&dev));
  std::lock_guard<std::mutex> lk(mu);
  if (dev < 64 && done[dev]) return MSLR_OK;
  for (const void* k : {reinterpret_cast<const void*>(&k_gram_umma<kBf16, 16>), reinterpret_cast<const void*>(&k_gram_umma<kTf32, 16>),
                        reinterpret_cast<const void*>(&k_gram_umma<kF16, 16>), reinterpret_cast<const void*>(&k_rebuild_umma<kBf16>),
                        reinterpret_cast<const void*>(&k_rebuild_umma<kTf32>)})
    MSLR_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(USmem<16>)));
  for (const void* k : {reinterpret_cast<const void*>(&k_gram_umma<kBf16, 32>), reinterpret_cast<const void*>(&k_gram_umma<kTf32, 32>)})
    MSLR_CUDA_TRY(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(USmem<32>)));
  if (dev < 64) done[dev] = true;
  return MSLR_OK;
}

int gram_umma_launch(const cf* img, const PatchMap& m, int64_t np, cf* out_or_part, int nsplit,
                     int lchunk, const DevWait& dw, cudaStream_t st, bool tf32, const int* kcols) {
  if (int rc = umma_prepare()) return rc;
  const int T = (m.n + kTM - 1) / kTM;
  const int ntri = T * (T + 1) / 2;
  const dim3 grid(ntri, (unsigned)np, nsplit);
  // No more tiles than SMs: each has its SM to itself, and nothing runs under
  // its chain of chunks, which should then be the shorter one of 32 elements, half
  // the barriers and waits (the sums are the same, bit for bit).  One of 216 × 64
  // 16.9 -> 14.7 us, 140 of 1000 × 64 71 -> 50, 140 of 512 × 128 48 -> 39, one of
  // 1000 × 300 89 -> 78, 49 of 1000 × 200 (147 tiles) 93.6 -> 89.3, one of 100 000 ×
  // 128 7.03 -> 5.11 ms, of 500 000 × 300 43.0 -> 36.1.  With two tiles per SM the
  // shorter chunks are faster (486 of 1000 × 300: see above).
  constexpr int kSms = 148;
  if (!kcols && (int64_t)ntri * np * nsplit <= kSms) {
    if (tf32) k_gram_umma<kTf32, 32><<<grid, kThr, sizeof(USmem<32>), st>>>(img, m, out_or_part, nsplit, lchunk, kcols, dw);
    else k_gram_umma<kBf16, 32><<<grid, kThr, sizeof(USmem<32>), st>>>(img, m, out_or_part, nsplit, lchunk, kcols, dw);
  } else if (tf32) {
    k_gram_umma<kTf32, 16><<<grid, kThr, sizeof(USmem<16>), st>>>(img, m, out_or_part, nsplit, lchunk, kcols, dw);
  } else if (kcols) {
    k_gram_umma<kF16, 16><<<grid, kThr, sizeof(USmem<16>), st>>>(img, m, out_or_part, nsplit, lchunk, kcols, dw);
  } else {
    k_gram_umma<kBf16, 16><<<grid, kThr, sizeof(USmem<16>), st>>>(img, m, out_or_part, nsplit, lchunk, nullptr, dw);
  }
  MSLR_CUDA_TRY(cudaGetLastError());
  return MSLR_OK;
}

int rebuild_umma_launch(const cf* img, const cf* W, const PatchMap& m, int64_t np, cf* out,
                        int direct, const DevWait& dw, cudaStream_t st, bool tf32) {
  if (int rc = umma_prepare()) return rc;
  const dim3 grid((m.n + kTM - 1) / kTM, (m.L + kTN - 1) / kTN, (unsigned)np);
  if (tf32)
    k_rebuild_umma<kTf32><<<grid, kThr, sizeof(USmem<16>), st>>>(img, W, m, out, direct, dw);
  else
    k_rebuild_umma<kBf16><<<grid, kThr, sizeof(USmem<16>), st>>>(img, W, m, out, direct, dw);
  MSLR_CUDA_TRY(cudaGetLastError());
  return MSLR_OK;
}

}  // namespace mslr
