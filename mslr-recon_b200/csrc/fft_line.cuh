// fft_line.cuh — whole-line DFTs in one thread's registers.
//
// A line of N = 2^a 3^b 5^c values (N <= 96) is transformed by one thread with
// no shared memory, no twiddle loads and no synchronisation: every index is a
// compile-time constant, coprime factors are combined by the prime-factor map
// (no twiddles at all: 90 = 9·10, 10 = 2·5, 60 = 3·4·5 ...), powers of one
// prime by Cooley–Tukey with literal twiddles.  90 points take about 1700
// FP32 instructions, 19 per point; two Stockham passes through shared memory
// cost about twice as many instructions plus four shared accesses per point.
//
// Prime-factor map, N = A·B coprime (Good 1958): input n = (B·n1 + A·n2) mod N,
// output k with k ≡ k1 (mod A), k ≡ k2 (mod B); then
// X[k] = Σ_{n1} ω_A^{n1 k1} Σ_{n2} ω_B^{n2 k2} x[n].
// Forward ω_N = e^{−2πi/N}; INV gives the unnormalised backward transform.
#pragma once
#include "fft_spec.cuh"

namespace mslr {
namespace line {

using spec::cmul_w;
using spec::sfor;

constexpr int kMaxLine = 96;   // two registers a value: 192 of a thread's 255

// lengths with a register plan: 5-smooth numbers
constexpr bool line_ok(int n) {
  if (n < 2 || n > kMaxLine) return false;
  while (n % 2 == 0) n /= 2;
  while (n % 3 == 0) n /= 3;
  while (n % 5 == 0) n /= 5;
  return n == 1;
}

constexpr int ppow(int n, int p) {   // the power of p in n
  int r = 1;
  while (n % p == 0) {
    n /= p;
    r *= p;
  }
  return r;
}
constexpr bool prime_power(int n) { return ppow(n, 2) == n || ppow(n, 3) == n || ppow(n, 5) == n; }
// factor A of N = A·B: coprime parts first, else the radix of a Cooley–Tukey step
constexpr int split_of(int n) {
  if (!prime_power(n)) {
    const int t = ppow(n, 3);
    return t > 1 ? t : ppow(n, 2);
  }
  switch (n) {
    case 8: return 2;
    case 16: return 4;
    case 32: return 4;
    case 64: return 8;
    case 9: return 3;
    case 27: return 3;
    case 81: return 9;
    case 25: return 5;
    default: return n;
  }
}

template <int N, bool INV, bool PP = prime_power(N)>
struct LD;

// ---- complex arithmetic, a pair per instruction -----------------------------------------
// sm_100a adds, multiplies and multiply-adds two FP32 values per instruction
// (register pairs; each half rounded as the scalar instruction would).  The
// pipe's rate per value is that of the scalar forms, but the transforms here
// are bound by issue and latency with two to four warps per scheduler, so
// fewer instructions are time.  A multiplication by ∓i is folded into the
// subtraction before it, which writes its halves swapped (two scalar
// instructions) with the sign left to the packed multiply-add after it.
__device__ __forceinline__ cf add2(cf a, cf b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ cf sub2(cf a, cf b) { return __ffma2_rn(b, make_float2(-1.f, -1.f), a); }
__device__ __forceinline__ cf mad2(cf a, float k, cf c) { return __ffma2_rn(a, make_float2(k, k), c); }
__device__ __forceinline__ cf mul2(cf a, float k) { return __fmul2_rn(a, make_float2(k, k)); }
// swapped difference: (a.y − b.y, a.x − b.x); with the factors (k, −k) it is −i·k·(a − b)
__device__ __forceinline__ cf sub_swap(cf a, cf b) { return make_float2(a.y - b.y, a.x - b.x); }
template <bool INV>
__device__ __forceinline__ cf rot_k(float k) { return INV ? make_float2(-k, k) : make_float2(k, -k); }

template <bool INV>
struct LD<2, INV, true> {
  static __device__ __forceinline__ void run(cf* v) {
    const cf a = v[0], b = v[1];
    v[0] = add2(a, b);
    v[1] = sub2(a, b);
  }
};
template <bool INV>
struct LD<3, INV, true> {
  static __device__ __forceinline__ void run(cf* v) {
    constexpr float s3 = 0.86602540378443864676f;   // sin(2π/3)
    const cf a = v[0], t = add2(v[1], v[2]), d = sub_swap(v[1], v[2]);
    const cf m = mad2(t, -0.5f, a);
    v[0] = add2(a, t);
    v[1] = __ffma2_rn(d, rot_k<INV>(s3), m);
    v[2] = __ffma2_rn(d, rot_k<INV>(-s3), m);
  }
};
template <bool INV>
struct LD<4, INV, true> {
  static __device__ __forceinline__ void run(cf* v) {
    const cf s0 = add2(v[0], v[2]), d0 = sub2(v[0], v[2]), s1 = add2(v[1], v[3]), d1 = sub_swap(v[1], v[3]);
    v[0] = add2(s0, s1);
    v[1] = __ffma2_rn(d1, rot_k<INV>(1.f), d0);
    v[2] = sub2(s0, s1);
    v[3] = __ffma2_rn(d1, rot_k<INV>(-1.f), d0);
  }
};
template <bool INV>
struct LD<5, INV, true> {
  static __device__ __forceinline__ void run(cf* v) {
    constexpr float c1 = 0.30901699437494742410f;    // cos(2π/5)
    constexpr float c2 = -0.80901699437494742410f;   // cos(4π/5)
    constexpr float s1 = 0.95105651629515357212f;    // sin(2π/5)
    constexpr float s2 = 0.58778525229247312917f;    // sin(4π/5)
    const cf x0 = v[0], t1 = add2(v[1], v[4]), t2 = add2(v[2], v[3]);
    const cf t3 = sub_swap(v[1], v[4]), t4 = sub_swap(v[2], v[3]);
    const cf a1 = mad2(t2, c2, mad2(t1, c1, x0)), a2 = mad2(t2, c1, mad2(t1, c2, x0));
    const cf b1 = __ffma2_rn(t4, rot_k<INV>(s2), __fmul2_rn(t3, rot_k<INV>(s1)));
    const cf b2 = __ffma2_rn(t4, rot_k<INV>(-s1), __fmul2_rn(t3, rot_k<INV>(s2)));
    v[0] = add2(x0, add2(t1, t2));
    v[1] = add2(a1, b1);
    v[4] = sub2(a1, b1);
    v[2] = add2(a2, b2);
    v[3] = sub2(a2, b2);
  }
};

// prime powers: N = A·B, r = r1 + A·r2, q = q2 + B·q1 (Cooley–Tukey, literal twiddles)
template <int N, bool INV>
struct LD<N, INV, true> {
  static __device__ __forceinline__ void run(cf* v) {
    constexpr int A = split_of(N), B = N / A;
    static_assert(A > 1 && B > 1, "no plan for this length");
    cf t[A][B];
    sfor<0, A>([&](auto r1) {
      sfor<0, B>([&](auto r2) { t[r1][r2] = v[r1 + A * r2]; });
      LD<B, INV>::run(t[r1]);
      sfor<1, B>([&](auto q2) {
        constexpr int K = decltype(r1)::value * decltype(q2)::value;
        t[r1][q2] = cmul_w<N, K, INV>(t[r1][q2]);
      });
    });
    sfor<0, B>([&](auto q2) {
      cf u[A];
      sfor<0, A>([&](auto r1) { u[r1] = t[r1][q2]; });
      LD<A, INV>::run(u);
      sfor<0, A>([&](auto q1) { v[q2 + B * q1] = u[q1]; });
    });
  }
};

// coprime factors: prime-factor map, no twiddles
template <int N, bool INV>
struct LD<N, INV, false> {
  static constexpr int A = split_of(N), B = N / A;
  static constexpr int out(int k1, int k2) {   // k ≡ k1 (mod A), ≡ k2 (mod B)
    for (int k = k2; k < N; k += B)
      if (k % A == k1) return k;
    return -1;
  }
  static __device__ __forceinline__ void run(cf* v) {
    cf t[A][B];
    sfor<0, A>([&](auto n1) {
      sfor<0, B>([&](auto n2) {
        constexpr int n = (B * decltype(n1)::value + A * decltype(n2)::value) % N;
        t[n1][n2] = v[n];
      });
      LD<B, INV>::run(t[n1]);
    });
    sfor<0, B>([&](auto k2) {
      cf u[A];
      sfor<0, A>([&](auto n1) { u[n1] = t[n1][k2]; });
      LD<A, INV>::run(u);
      sfor<0, A>([&](auto k1) {
        constexpr int k = out(decltype(k1)::value, decltype(k2)::value);
        v[k] = u[k1];
      });
    });
  }
};

}  // namespace line
}  // namespace mslr
