// sense_line.cu — tuned SENSE operators on whole-line register DFTs
// (sense_line.cuh): every image whose three axes are 5-smooth numbers of 8 to
// 96.  A = M F S' per frame and coil; the centring identity is in the header
// of sense.cu.  The work goes coil group by coil group and chunk by chunk of
// frames, sized so that a chunk's per-coil k-space T stays in L2; consecutive
// chunks alternate between two streams ("lanes", each with its own T).
//
// Normal operator, per chunk and coil group:
//   images with a compiled plane  k_pfwd | z pass with mask | k_padj | k_csum (× conj(S'), coil sum)
//   other images                  y, x pass | z pass with mask | x, y pass | k_csum
// The encoding operator and its adjoint use the same passes around a gather
// of, or a scatter from, the samples.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <string>

#include "sense_line.cuh"

namespace mslr {

using line::ColArgs;
using line::LineOps;

namespace {

// ---- fused plane passes (compiled planes) ------------------------------------------
// Both passes of a plane in one kernel, one line per thread, P planes per CTA
// (consecutive units u = (cc fastest, then z, then frame)).  The k-space plane
// is kept transposed in T, [z][kx][ky]: a row thread (fixed ky) then reads and
// writes T with its neighbours in one run, as a column thread (fixed x) does
// the image, so the only shared-memory traffic is the turn of the plane
// between the two passes.  Rows of RS values, odd: the row threads' accesses
// fall on distinct banks.
template <int NX_, int NY_, int NZ_, int P_, int CTAS_>
struct Plane {
  static constexpr int NX = NX_, NY = NY_, NZ = NZ_, P = P_, CTAS = CTAS_;
  static constexpr int RS = NX | 1, RT = NY | 1, PL = NX * NY;   // row strides, upright and turned
  static constexpr int64_t NVOX = (int64_t)PL * NZ;
  static constexpr int THREADS = ((NX > NY ? NX : NY) * P + 31) / 32 * 32;
  static constexpr size_t smem = sizeof(cf) * P * (NY * RS > NX * RT ? NY * RS : NX * RT);
};

// element e of a line at w[e·S]
template <int S>
struct Line {
  cf* w;
  __device__ __forceinline__ cf operator()(int e) const { return w[e * S]; }
  __device__ __forceinline__ void operator()(int e, cf v) const { w[e * S] = v; }
};
template <int SX, int SS>
struct LineMul {   // x̄ (shared) · S' (global)
  const cf *x, *s;
  __device__ __forceinline__ cf operator()(int e) const { return cmul(x[e * SX], __ldg(s + e * SS)); }
};
template <int S>
__device__ __forceinline__ Line<S> shifted(const Line<S>& l, int e) { return {l.w + e * S}; }

// One line, ld → DFT → st, with `tmp` the line's own slots in shared memory.
// Lengths N = 2·H, H odd and above 40, would leave a thread no registers to
// load ahead with (90 points: 243 registers, two CTAs of three warps per SM,
// against three CTAs at 168).  They go in two halves: the sums of the pairs
// (n, n + H mod N) stay in registers, the differences wait in the pair's odd
// slot of tmp; one H-point transform gives the even outputs, the same code
// run again on the differences the odd ones.
template <int N, bool INV, class Ld, class Tmp, class St>
__device__ __forceinline__ void line_dft(const Ld& ld, const Tmp& tmp, const St& st) {
  if constexpr (N % 4 == 2 && N > 80) {
    constexpr int H = N / 2;
    cf v[H];
#pragma unroll
    for (int n = 0; n < H; ++n) {
      const cf a = ld((2 * n) % N), b = ld((H + 2 * n) % N);
      v[n] = line::add2(a, b);
      tmp((H + 2 * n) % N, line::sub2(a, b));
    }
    // output k ≡ k2 (mod H) of parity h: at k2 when k2 has that parity, else at k2 + H
#pragma unroll 1
    for (int h = 0; h < 2; ++h) {
      if (h) {
        asm volatile("" ::: "memory");   // the differences come back from shared memory, not from registers
#pragma unroll
        for (int n = 0; n < H; ++n) v[n] = tmp((H + 2 * n) % N);
      }
      line::LD<H, INV>::run(v);
      const auto se = shifted(st, h ? H : 0), so = shifted(st, h ? 0 : H);
#pragma unroll
      for (int k = 0; k < H; ++k) {
        if (k % 2) so(k, v[k]);
        else se(k, v[k]);
      }
    }
  } else {
    cf v[N];
#pragma unroll
    for (int e = 0; e < N; ++e) v[e] = ld(e);
    line::LD<N, INV>::run(v);
#pragma unroll
    for (int e = 0; e < N; ++e) st(e, v[e]);
  }
}

// The plane [rows][cols] of g into shared memory with rows of RS values, every
// copy in flight at once (8-byte copies: odd row strides); waits for the thread's
// own copies, so that a barrier has to follow.
template <int ROWS, int COLS, int RS, int THREADS>
__device__ __forceinline__ void plane_in(cf* W, const cf* g) {
  constexpr int NW = THREADS / 32;
  const int lane = threadIdx.x & 31;
  const cf* src = g + lane;
  unsigned dst = spec::su32(W + lane);
#pragma unroll 2
  for (int r = threadIdx.x >> 5; r < ROWS; r += NW) {
#pragma unroll
    for (int c = 0; c < COLS; c += 32)
      if (c + 32 <= COLS || lane < COLS - c)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(dst + (r * RS + c) * 8),
                     "l"(src + r * COLS + c));
  }
  asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;\n" ::: "memory");
}

// S'_c ⊙ x̄ → DFT_y (columns) → DFT_x (rows) → T
template <class Sh>
__global__ void __launch_bounds__(Sh::THREADS, Sh::CTAS)
    k_pfwd(const cf* __restrict__ xs, int t0, int units, int cc0, int ch, const cf* __restrict__ smod,
           cf* __restrict__ T) {
  constexpr int NX = Sh::NX, NY = Sh::NY, NZ = Sh::NZ, PL = Sh::PL, RS = Sh::RS;
  constexpr int64_t NVOX = Sh::NVOX;
  extern __shared__ __align__(128) unsigned char smraw[];
  cf* W = reinterpret_cast<cf*>(smraw);
#pragma unroll 1
  for (int p = 0; p < Sh::P; ++p) {
    const int u = blockIdx.x * Sh::P + p, r = u / ch, z = r % NZ, f = r / NZ;
    if (u < units)
      plane_in<NY, NX, RS, Sh::THREADS>(W + p * NY * RS, xs + (t0 + f) * NVOX + (int64_t)z * PL);
  }
  __syncthreads();
  {
    const int pl = threadIdx.x / NX, x = threadIdx.x - pl * NX;
    const int u = blockIdx.x * Sh::P + pl;
    if (pl < Sh::P && u < units) {
      const int cc = u % ch, z = (u / ch) % NZ;
      const Line<RS> w{W + pl * NY * RS + x};
      line_dft<NY, false>(LineMul<RS, NX>{w.w, smod + (cc0 + cc) * NVOX + (int64_t)z * PL + x}, w, w);
    }
  }
  __syncthreads();
  const int pl = threadIdx.x / NY, y = threadIdx.x - pl * NY;
  const int u = blockIdx.x * Sh::P + pl;
  if (pl < Sh::P && u < units) {
    const int cc = u % ch, r = u / ch, z = r % NZ, f = r / NZ;
    const Line<1> w{W + (pl * NY + y) * RS};
    line_dft<NX, false>(w, w, Line<NY>{T + ((int64_t)f * ch + cc) * NVOX + (int64_t)z * PL + y});
  }
}

// T → bDFT_x (rows) → bDFT_y (columns) → T as images [z][y][x], in place (a
// plane is read whole before its first result is written).  The plane stays
// turned in shared memory, [x][ky].
template <class Sh>
__global__ void __launch_bounds__(Sh::THREADS, Sh::CTAS) k_padj(cf* T, int units) {
  constexpr int NX = Sh::NX, NY = Sh::NY, PL = Sh::PL, RS = Sh::RT;
  extern __shared__ __align__(128) unsigned char smraw[];
  cf* W = reinterpret_cast<cf*>(smraw);
  cf* g = T + (int64_t)blockIdx.x * Sh::P * PL;   // planes of the chunk in order
  const int np = min(Sh::P, units - (int)blockIdx.x * Sh::P);
#pragma unroll 1
  for (int p = 0; p < np; ++p) plane_in<NX, NY, RS, Sh::THREADS>(W + p * NX * RS, g + p * PL);
  __syncthreads();
  {
    const int pl = threadIdx.x / NY, y = threadIdx.x - pl * NY;
    if (pl < np) {
      const Line<RS> w{W + pl * NX * RS + y};
      line_dft<NX, true>(w, w, w);
    }
  }
  __syncthreads();
  const int pl = threadIdx.x / NX, x = threadIdx.x - pl * NX;
  if (pl < np) {
    const Line<1> w{W + (pl * NX + x) * RS};
    line_dft<NY, true>(w, w, Line<NX>{g + pl * PL + x});
  }
}

struct PlaneOps {
  int nx, ny, nz, planes, threads;
  size_t smem;
  const void* pfwd;
  const void* padj;
  const void* z[3];   // z passes with the plane stride compiled in: mask, forward, inverse
};
template <class Sh>
PlaneOps plane_ops_of() {
  return {Sh::NX, Sh::NY, Sh::NZ, Sh::P, Sh::THREADS, Sh::smem,
          reinterpret_cast<const void*>(&k_pfwd<Sh>),
          reinterpret_cast<const void*>(&k_padj<Sh>),
          {reinterpret_cast<const void*>(&line::k_lcol<Sh::NZ, line::kZMask, Sh::PL>),
           reinterpret_cast<const void*>(&line::k_lcol<Sh::NZ, line::kZFwd, Sh::PL>),
           reinterpret_cast<const void*>(&line::k_lcol<Sh::NZ, line::kZInv, Sh::PL>)}};
}
// the shapes of sense_spec.cu
const PlaneOps* plane_ops(int nx, int ny, int nz) {
  static const PlaneOps table[] = {plane_ops_of<Plane<90, 90, 60, 1, 3>>(),
                                   plane_ops_of<Plane<48, 48, 32, 2, 5>>(),
                                   plane_ops_of<Plane<32, 32, 24, 2, 8>>()};
  for (const PlaneOps& o : table)
    if (o.nx == nx && o.ny == ny && o.nz == nz) return &o;
  return nullptr;
}

const LineOps* line_ops(int n) {
  if (!line::line_ok(n) || n < 8) return nullptr;
  const LineOps* o = line::line_ops_a(n);
  if (!o) o = line::line_ops_b(n);
  if (!o) o = line::line_ops_c(n);
  if (!o) o = line::line_ops_d(n);
  return o;
}

// ---- coil combine ----------------------------------------------------------------------
// out[t0 + f] (=, −A'y, or +=) scale·Σ_c conj(S'_c)·T[f][c], coils in order;
// VEC values per access; CH coils (0: `ch`, any number).  A thread keeps its
// voxels' maps in registers over its frames, so they are read once per chunk
// and not once per frame, as a multiplication in the plane pass would have it.
template <int VEC> struct Vals;
template <> struct Vals<1> { using type = float2; };
template <> struct Vals<2> { using type = float4; };
// a += conj(s)·v, the product formed first: the running sum is then rounded once
// a coil and not twice (normal operator at 32 × 32 × 24 × 8 × 64: 1.49e-6 -> 1.40e-6
// against 64 bits, 0.2 to 0.5 % of its time)
__device__ __forceinline__ void mac_c(float2& a, const float2 s, const float2 v) {
  a.x += fmaf(s.x, v.x, s.y * v.y);
  a.y += fmaf(s.x, v.y, -(s.y * v.x));
}
__device__ __forceinline__ void mac_c(float4& a, const float4 s, const float4 v) {
  a.x += fmaf(s.x, v.x, s.y * v.y);
  a.y += fmaf(s.x, v.y, -(s.y * v.x));
  a.z += fmaf(s.z, v.z, s.w * v.w);
  a.w += fmaf(s.z, v.w, -(s.w * v.z));
}
__device__ __forceinline__ float2 axpy(float k, float2 a, float2 b) { return make_float2(fmaf(k, a.x, b.x), fmaf(k, a.y, b.y)); }
__device__ __forceinline__ float4 axpy(float k, float4 a, float4 b) {
  return make_float4(fmaf(k, a.x, b.x), fmaf(k, a.y, b.y), fmaf(k, a.z, b.z), fmaf(k, a.w, b.w));
}
__device__ __forceinline__ void zero(float2& v) { v = make_float2(0.f, 0.f); }
__device__ __forceinline__ void zero(float4& v) { v = make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ float2 minus(float2 v) { return make_float2(-v.x, -v.y); }
__device__ __forceinline__ float4 minus(float4 v) { return make_float4(-v.x, -v.y, -v.z, -v.w); }

template <int VEC, int CH>
__global__ void __launch_bounds__(256, 4) k_csum(const cf* __restrict__ T_, const cf* __restrict__ smod_, int nf, int ch,
                                              int64_t nvox, cf* __restrict__ out_, const cf* __restrict__ ahy_,
                                              int t0, float scale, int add) {
  using V = typename Vals<VEC>::type;
  const int64_t n = nvox / VEC, i = blockIdx.x * (int64_t)256 + threadIdx.x;
  if (i >= n) return;
  const V* s = reinterpret_cast<const V*>(smod_) + i;
  V m[CH ? CH : 1];
  if constexpr (CH > 0) {
#pragma unroll
    for (int c = 0; c < CH; ++c) m[c] = __ldg(s + c * n);
  }
  for (int f = blockIdx.y; f < nf; f += gridDim.y) {
    const V* t = reinterpret_cast<const V*>(T_) + (int64_t)f * ch * n + i;
    V* o = reinterpret_cast<V*>(out_) + (int64_t)(t0 + f) * n + i;
    V a, r;
    zero(a);
    if (add) r = *o;
    else if (ahy_) r = minus(__ldg(reinterpret_cast<const V*>(ahy_) + (int64_t)(t0 + f) * n + i));
    else zero(r);
    if constexpr (CH > 0) {
      V v[CH];
#pragma unroll
      for (int c = 0; c < CH; ++c) v[c] = t[c * n];
#pragma unroll
      for (int c = 0; c < CH; ++c) mac_c(a, m[c], v[c]);
    } else {
#pragma unroll 4
      for (int c = 0; c < ch; ++c) mac_c(a, __ldg(s + c * n), t[c * n]);
    }
    *o = axpy(scale, a, r);
  }
}
template <int VEC>
const void* coil_sum_of(int ch) {
  switch (ch) {
    case 1: return reinterpret_cast<const void*>(&k_csum<VEC, 1>);
    case 2: return reinterpret_cast<const void*>(&k_csum<VEC, 2>);
    case 3: return reinterpret_cast<const void*>(&k_csum<VEC, 3>);
    case 4: return reinterpret_cast<const void*>(&k_csum<VEC, 4>);
    case 5: return reinterpret_cast<const void*>(&k_csum<VEC, 5>);
    case 6: return reinterpret_cast<const void*>(&k_csum<VEC, 6>);
    case 7: return reinterpret_cast<const void*>(&k_csum<VEC, 7>);
    case 8: return reinterpret_cast<const void*>(&k_csum<VEC, 8>);
    default: return reinterpret_cast<const void*>(&k_csum<VEC, 0>);
  }
}
const void* coil_sum_kernel(int ch, bool pairs) { return pairs ? coil_sum_of<2>(ch) : coil_sum_of<1>(ch); }

// ---- sample bits over z --------------------------------------------------------------
// mz[(t·NW + q)·PL + i]: bit z − 32q set when (z, i) is sampled in frame t, i the
// position within a plane of T (turned: kx·Ny + ky, else ky·Nx + kx)
__global__ void k_mask_z(const uint32_t* __restrict__ mask, int nwords, uint32_t* __restrict__ mz,
                         int nx, int ny, int turned, int nz, int nw, int nt) {
  const int q = blockIdx.y, pl = nx * ny;
  for (int t = blockIdx.z; t < nt; t += gridDim.z) {
    const uint32_t* m = mask + (int64_t)t * nwords;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < pl; i += gridDim.x * blockDim.x) {
      uint32_t w = 0;
      const int j = turned ? (i % nx) * ny + i / nx : i;
      for (int z = 32 * q; z < min(nz, 32 * q + 32); ++z) {
        const int64_t k = (int64_t)z * pl + i;
        w |= ((__ldg(m + (k >> 5)) >> (k & 31)) & 1u) << (z - 32 * q);
      }
      mz[((int64_t)t * nw + q) * pl + j] = w;
    }
  }
}

// ---- samples ----------------------------------------------------------------------------
struct SampArgs {
  const int32_t* idx;
  int64_t K, nvox;
  const cf *px, *py, *pz;   // φ of each axis
  int nx, ny, nc, ch, cc0, t0, turned;
  float s;
};
// weight s·φ(k) of grid position k, and *j its position in T
__device__ __forceinline__ cf sample_at(int k, const SampArgs& a, int* j) {
  const int r = k / a.nx, x = k - r * a.nx, z = r / a.ny, y = r - z * a.ny;
  *j = a.turned ? (z * a.nx + x) * a.ny + y : k;
  return cscale(cmul(__ldg(a.px + x), cmul(__ldg(a.py + y), __ldg(a.pz + z))), a.s);
}
// y[t][c][i] = s·φ(idx)·T[f][cc][idx]; blockIdx.y = frame; a thread serves all coils of the group
__global__ void k_take(const cf* __restrict__ T, cf* __restrict__ y, const SampArgs a) {
  const int t = a.t0 + blockIdx.y;
  const cf* tf = T + (int64_t)blockIdx.y * a.ch * a.nvox;
  cf* yo = y + ((int64_t)t * a.nc + a.cc0) * a.K;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.K;
       i += (int64_t)gridDim.x * blockDim.x) {
    int k;
    const cf w = sample_at(__ldg(a.idx + (int64_t)t * a.K + i), a, &k);
#pragma unroll 4
    for (int c = 0; c < a.ch; ++c) yo[c * a.K + i] = cmul(w, tf[c * a.nvox + k]);
  }
}
// its adjoint: T[f][cc][idx] = s·conj(φ)·y[t][c][i] (T zeroed before)
__global__ void k_put(cf* __restrict__ T, const cf* __restrict__ y, const SampArgs a) {
  const int t = a.t0 + blockIdx.y;
  cf* tf = T + (int64_t)blockIdx.y * a.ch * a.nvox;
  const cf* yi = y + ((int64_t)t * a.nc + a.cc0) * a.K;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.K;
       i += (int64_t)gridDim.x * blockDim.x) {
    int k;
    const cf w = sample_at(__ldg(a.idx + (int64_t)t * a.K + i), a, &k);
#pragma unroll 4
    for (int c = 0; c < a.ch; ++c) tf[c * a.nvox + k] = cmulc(w, __ldg(yi + c * a.K + i));
  }
}

// ---- launches -----------------------------------------------------------------------------
int launch(const void* fn, dim3 grid, int threads, size_t smem, cudaStream_t st, void** args) {
  MSLR_CUDA_TRY(cudaLaunchKernel(fn, grid, dim3(threads), args, smem, st));
  return MSLR_OK;
}

struct Pass {   // one chunk of one coil group
  Ctx* c;
  cf* T;
  int ch, cc0, t0, f;
  cudaStream_t st;
  int imgs() const { return ch * f; }
  ColArgs col(int nlines) const {
    ColArgs a{};
    a.T = T;
    a.smod = c->d_smaps_mod;
    a.mz = c->d_mz;
    a.nvox = c->nvox;
    a.nlines = nlines;
    a.nx = c->N[0];
    a.pl = c->N[0] * c->N[1];
    a.ch = ch;
    a.cc0 = cc0;
    a.t0 = t0;
    return a;
  }
  int columns(const void* fn, ColArgs a) const {
    void* args[] = {&a};
    const dim3 grid((a.nlines + line::kColThreads - 1) / line::kColThreads, imgs());
    c->launches += 1;
    return launch(fn, grid, line::kColThreads, 0, st, args);
  }
  int z_pass(int mode) const {
    const PlaneOps* po = plane_ops(c->N[0], c->N[1], c->N[2]);
    return columns(po ? po->z[mode] : line_ops(c->N[2])->col[mode], col(c->N[0] * c->N[1]));
  }
  int rows(bool inv) const {
    const int n = c->N[0];
    int64_t nrows = (int64_t)imgs() * c->N[1] * c->N[2];
    cf* t = T;
    void* args[] = {&t, &nrows};
    const int R = line::row_threads(n);
    c->launches += 1;
    return launch(line_ops(n)->row[inv ? 1 : 0], dim3((unsigned)((nrows + R - 1) / R)), R, line::row_smem(n), st,
                  args);
  }
  // S'·x̄ → DFT over planes → T
  int planes_fwd(const cf* xs) const {
    if (const PlaneOps* po = plane_ops(c->N[0], c->N[1], c->N[2])) {
      int units = imgs() * c->N[2], t = t0, cc = cc0, h = ch;
      const cf* smod = c->d_smaps_mod;
      cf* tp = T;
      void* args[] = {&xs, &t, &units, &cc, &h, &smod, &tp};
      c->launches += 1;
      return launch(po->pfwd, dim3((units + po->planes - 1) / po->planes), po->threads, po->smem, st, args);
    }
    ColArgs a = col(c->N[0] * c->N[2]);
    a.xs = xs;
    if (int rc = columns(line_ops(c->N[1])->col[line::kYFwdMul], a)) return rc;
    return rows(false);
  }
  // T → inverse DFT over planes → T
  int planes_inv() const {
    if (const PlaneOps* po = plane_ops(c->N[0], c->N[1], c->N[2])) {
      int units = imgs() * c->N[2];
      cf* tp = T;
      void* args[] = {&tp, &units};
      c->launches += 1;
      return launch(po->padj, dim3((units + po->planes - 1) / po->planes), po->threads, po->smem, st, args);
    }
    if (int rc = rows(true)) return rc;
    return columns(line_ops(c->N[1])->col[line::kYInv], col(c->N[0] * c->N[2]));
  }
  // out (=, −A'y, or +=) scale·Σ_cc conj(S')·T
  int coil_sum(cf* out, float scale, const cf* ahy) const {
    const int64_t n = c->nvox;
    const cf* sm = c->d_smaps_mod + (int64_t)cc0 * n;
    const bool pairs = n % 2 == 0 && ((reinterpret_cast<uintptr_t>(out) | reinterpret_cast<uintptr_t>(ahy)) & 15) == 0;
    const int64_t items = pairs ? n / 2 : n;
    const int bx = (int)((items + 255) / 256);
    // frames per thread: the maps are loaded once per thread, but the grid should fill the GPU
    const int by = std::max(1, std::min(f, (8 * c->nsm + bx - 1) / bx));
    int nf = f, t = t0, h = ch, add = cc0 > 0;
    cf* o = out;
    const cf* tp = T;
    void* args[] = {&tp, &sm, &nf, &h, (void*)&n, &o, &ahy, &t, &scale, &add};
    c->launches += 1;
    return launch(coil_sum_kernel(ch, pairs), dim3(bx, by), 256, 0, st, args);
  }
  SampArgs samples(float s) const {
    SampArgs a{};
    a.idx = c->d_idx;
    a.K = c->K;
    a.nvox = c->nvox;
    a.px = c->d_phase[0];
    a.py = c->d_phase[1];
    a.pz = c->d_phase[2];
    a.nx = c->N[0];
    a.ny = c->N[1];
    a.nc = c->Nc;
    a.ch = ch;
    a.cc0 = cc0;
    a.t0 = t0;
    a.turned = plane_ops(c->N[0], c->N[1], c->N[2]) != nullptr;
    a.s = s;
    return a;
  }
  dim3 sample_grid() const { return dim3((unsigned)std::min<int64_t>((c->K + 255) / 256, 512), f); }
};

// Bytes of k-space in one unit of spec_fr (two units by default).  Measured at 90×90×60
// (60 frames, 18 coils, two lanes): 24 / 48 / 72 / 96 MB per launch 6.23 / 6.05
// / 6.19 / 6.24 ms — smaller launches do not fill the GPU, larger ones leave
// L2.  Small images take several units of spec_fr frames per launch.
constexpr double kChunkBytes = 24e6;

// Up to this much k-space in all, every coil and frame goes in one launch a pass
// on one stream: a launch is then little more than its latency, and three groups
// of coils, or two lanes of which each has half the frames, are as many times
// that.  16³, normal operator: 16 coils × 1 frame 74.5 → 28.2 us (three groups of
// 6), 32 coils 147.5 → 28.1; 4 coils × 15 frames (2 MB, four chunks) 82.9 → 29.5;
// 32 × 32 × 24 × 8 × 10 (16 MB) 34.2 → 29.5, at 32 MB 38.2 → 42.9.  With more than
// one group, 12 coils at 64 MB 108.2 → 91.7, 16 coils 133.7 → 88, at 128 MB 146 →
// 225 and 194 → 223.
constexpr double kOneLaunchBytes = 16e6, kOneLaunchBytesGroups = 64e6;
int coil_groups(int nc) { return nc <= 8 ? 1 : (nc + 5) / 6; }   // of equal size, at most 6 coils (8 when that is all)
bool one_launch(const Ctx* c) {   // (the buffer holds it: F = Nt)
  const double most = coil_groups(c->Nc) > 1 ? kOneLaunchBytesGroups : kOneLaunchBytes;
  return (double)c->nvox * sizeof(cf) * c->Nc * c->Nt <= most;
}

// Coils per group and frames per launch of the next operator: within the
// k-space buffer, which two lanes share when both fit; the launches of a
// group equally large, and an even number of them on two lanes.
void chunk_of(const Ctx* c, int* ch, int* fr, bool* lanes) {
  if (one_launch(c)) {
    *ch = c->Nc;
    *fr = c->Nt;
    *lanes = false;
    return;
  }
  *ch = std::max(1, std::min(c->Nc, c->spec_ch));
  const int64_t cap = (int64_t)c->F * c->Nc;
  const double img = (double)c->nvox * sizeof(cf) * *ch;
  const int unit = std::max(1, (int)(kChunkBytes / img));   // frames per unit of spec_fr
  const bool two = c->spec_lanes == 2 && !c->prof_on;
  int64_t f = std::max(1, std::min(c->Nt, c->spec_fr * unit));
  f = std::max<int64_t>(1, std::min(f, cap / *ch));
  if (two && 2 * f * *ch > cap && c->Nt > 1 && cap >= 2 * *ch) f = cap / (2 * *ch);
  int64_t n = (c->Nt + f - 1) / f;
  if (two && n > 1) n += n & 1;
  f = (c->Nt + n - 1) / n;
  *fr = (int)f;
  *lanes = two && 2 * f * *ch <= cap && c->Nt > f;
}

// Runs fn(pass, mode) over every coil group and chunk; chunk j of every group
// on lane j % 2, so that what a group adds to a frame's result follows the
// earlier groups' additions.
template <class Fn>
int for_chunks(Ctx* c, cudaStream_t st, Fn&& fn) {
  int ch, fr;
  bool lanes;
  chunk_of(c, &ch, &fr, &lanes);
  if (lanes) {
    MSLR_CUDA_TRY(cudaEventRecord(c->sn_fork, st));
    MSLR_CUDA_TRY(cudaStreamWaitEvent(c->sn_stream, c->sn_fork, 0));
  }
  for (int cc0 = 0; cc0 < c->Nc; cc0 += ch)
    for (int t0 = 0, j = 0; t0 < c->Nt; t0 += fr, ++j) {
      const int lane = lanes ? (j & 1) : 0;
      Pass p{c, c->d_T + (int64_t)lane * ch * fr * c->nvox, std::min(ch, c->Nc - cc0), cc0, t0,
             std::min(fr, c->Nt - t0), lane ? c->sn_stream : st};
      if (int rc = fn(p)) return rc;
    }
  if (lanes) {
    MSLR_CUDA_TRY(cudaEventRecord(c->sn_join, c->sn_stream));
    MSLR_CUDA_TRY(cudaStreamWaitEvent(st, c->sn_join, 0));
  }
  return MSLR_OK;
}

// Whether the normal operator reads a copy or the sum of its images.  One image
// is read where it is, unless the result lies over it and a second coil group
// would read what the first has written (with one group, a chunk's frames are
// read before they are written, and by no other chunk).
bool needs_sum(const Ctx* c, const cf* X, int ns, const cf* g) {
  if (ns > 1) return true;
  int ch, fr;
  bool lanes;
  chunk_of(c, &ch, &fr, &lanes);
  const int64_t series = (int64_t)c->Nt * c->nvox;
  return X < g + series && g < X + series && (ch < c->Nc || g != X);
}

// One frame of a small image without a compiled plane: six launches here, three
// in sense_fast.cu, each little more than its latency (that form takes three a
// frame, so from two frames on this one is no slower).  Normal operator here and
// there: 8³, one coil 37.7 and 26.6 us; 16³, 4 coils 29.3 and 27.3; 24 × 20 × 18, 8
// coils 31 and 28; 48 × 45 × 40, 2 coils 33 and 30; but 32 × 30 × 27, 8 coils 31 and
// 48, 48 × 45 × 40, 4 coils 34 and 46, 12³, 16 coils 28 and 32 (8³ 28 and 25), and
// large planes, 96 × 96 × 8, one coil 29 and 143.
bool few_launches_win(const Ctx* c) {
  const int64_t points = c->nvox * c->Nc;
  return c->Nt == 1 && c->fast && c->N[0] * c->N[1] <= 4096 &&
         points <= (c->Nc <= 2 ? 330000 : c->Nc <= 8 ? 105000 : 12000);
}

}  // namespace

bool sense_line_setup(Ctx* c) {
  for (int d = 0; d < 3; ++d)
    if (!line_ops(c->N[d])) return false;
  const PlaneOps* po = plane_ops(c->N[0], c->N[1], c->N[2]);
  if (!po && few_launches_win(c)) return false;
  if (po) {
    if (raise_dyn_smem(po->pfwd, (int)po->smem) || raise_dyn_smem(po->padj, (int)po->smem)) {
      cudaGetLastError();
      return false;
    }
  } else {
    const LineOps* ox = line_ops(c->N[0]);
    for (const void* k : ox->row)
      if (raise_dyn_smem(k, (int)line::row_smem(c->N[0]))) {
        cudaGetLastError();
        return false;
      }
  }
  int dev = 0, nsm = 0;
  if (!cudaGetDevice(&dev) && !cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) && nsm > 0)
    c->nsm = nsm;
  const int nw = (c->N[2] + 31) / 32;
  if (dalloc(c, (void**)&c->d_mz, (size_t)c->Nt * nw * c->N[0] * c->N[1] * sizeof(uint32_t))) {
    cudaGetLastError();
    return false;
  }
  if (!c->spec_three && !c->xy_tc) {
    const int groups = one_launch(c) ? 1 : coil_groups(c->Nc);
    c->spec_ch = (c->Nc + groups - 1) / groups;
    c->spec_fr = 2;
  }
  const char* ln = std::getenv("MSLR_SENSE_LANES");
  if (!c->sn_stream && !(ln && std::string(ln) == "1") &&
      !cudaStreamCreateWithFlags(&c->sn_stream, cudaStreamNonBlocking) &&
      !cudaEventCreateWithFlags(&c->sn_fork, cudaEventDisableTiming) &&
      !cudaEventCreateWithFlags(&c->sn_join, cudaEventDisableTiming))
    c->spec_lanes = 2;
  cudaGetLastError();
  return true;
}

bool sense_line_fixed(const Ctx* c) { return one_launch(c); }

int sense_line_bind(Ctx* c, cudaStream_t st) {
  const int pl = c->N[0] * c->N[1], nw = (c->N[2] + 31) / 32;
  const dim3 grid((pl + 255) / 256, nw, std::min(c->Nt, 65535));
  k_mask_z<<<grid, 256, 0, st>>>(c->d_mask, c->nwords, c->d_mz, c->N[0], c->N[1],
                                 plane_ops(c->N[0], c->N[1], c->N[2]) != nullptr, c->N[2], nw, c->Nt);
  MSLR_CUDA_TRY(cudaGetLastError());
  return MSLR_OK;
}

int normal_op_line(Ctx* c, const cf* X, int ns, int64_t sstride, cf* g, bool subtract, cudaStream_t st) {
  const float scale = (float)(1.0 / (double)c->nvox);
  const cf* xs = X;
  if (needs_sum(c, X, ns, g)) {
    // Into a buffer of the POGM state that holds nothing between calls: the
    // gradient, or, when that is the result, z, which a step writes after it.
    // (Whatever uses those two also uses T, so calls that may overlap on the
    // GPU are none fewer.)
    cf* sum = g == c->d_G ? c->d_Z : c->d_G;
    if (int rc = image_sum(c, X, ns, sstride, sum, st)) return rc;
    xs = sum;
  }
  c->prof_kernels = 4;
  return for_chunks(c, st, [&](const Pass& p) {
    int rc = prof_mark(c, p.st);
    if (!rc) rc = p.planes_fwd(xs);
    if (!rc) rc = prof_mark(c, p.st);
    if (!rc) rc = p.z_pass(line::kZMask);
    if (!rc) rc = prof_mark(c, p.st);
    if (!rc) rc = p.planes_inv();
    if (!rc) rc = prof_mark(c, p.st);
    if (!rc) rc = p.coil_sum(g, scale, subtract ? c->d_ahy : nullptr);
    if (!rc) rc = prof_mark(c, p.st);
    return rc;
  });
}

int sense_forward_line(Ctx* c, const cf* x, cf* y, cudaStream_t st) {
  const float s = (float)(1.0 / std::sqrt((double)c->nvox));
  return for_chunks(c, st, [&](const Pass& p) {
    int rc = p.planes_fwd(x);
    if (!rc) rc = p.z_pass(line::kZFwd);
    if (rc) return rc;
    k_take<<<p.sample_grid(), 256, 0, p.st>>>(p.T, y, p.samples(s));
    c->launches += 1;
    MSLR_CUDA_TRY(cudaGetLastError());
    return MSLR_OK;
  });
}

int sense_adjoint_line(Ctx* c, const cf* y, cf* x, cudaStream_t st) {
  const float s = (float)(1.0 / std::sqrt((double)c->nvox));
  return for_chunks(c, st, [&](const Pass& p) {
    MSLR_CUDA_TRY(cudaMemsetAsync(p.T, 0, (size_t)p.imgs() * c->nvox * sizeof(cf), p.st));
    k_put<<<p.sample_grid(), 256, 0, p.st>>>(p.T, y, p.samples(s));
    c->launches += 1;
    MSLR_CUDA_TRY(cudaGetLastError());
    int rc = p.z_pass(line::kZInv);
    if (!rc) rc = p.planes_inv();
    if (!rc) rc = p.coil_sum(x, 1.0f, nullptr);
    return rc;
  });
}

}  // namespace mslr
