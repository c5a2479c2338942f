// Two-factor line FFTs with packed FP32 arithmetic: the transforms of the time
// step, of the Poisson solve and of the plain 3D transform.
//
// N = RA RB; with the points at n = RB n1 + n2 and the frequencies at k = k1 +
// RA k2,
//   X[k] = sum_n2 W_RB^(n2 k2) W_N^(n2 k1) sum_n1 W_RA^(n1 k1) x[n],
// so a transform is two stages: stage A takes, for each n2, the RA points RB n1 +
// n2 of a line, transforms them in registers and puts element (k1, n2) back at
// RB k1 + n2; stage B takes, for each k1, the RB elements (k1, n2), multiplies by
// the twiddles W_N^(n2 k1) and transforms them into the frequencies k1 + RA k2.
// Both work in place: a stage's butterfly reads and writes its own points
// only, so one barrier separates the stages, a thread holds one butterfly
// (at most 32 points) at a time, and a stage is a short loop.  An inverse that
// follows a pointwise operator starts with stage B's transform on the registers
// it just left (IDFT over k2, conjugate twiddles) and ends with stage A's, which
// leaves the points RB n1 + n2.
//
// Against the Stockham plans of fft_engine.cuh (two or three exchanges per
// transform, 12 to 24 points per thread) this takes one exchange, fewer
// twiddles and half the instructions per point.  The adjoint stays on those:
// its derivative by the tidal amplitude is a small difference of large sums,
// and any other order of rounding moves it in the fourth or fifth digit.
#pragma once
#include "fft_engine.cuh"

namespace wdm {
namespace fx {

// Complex arithmetic in packed FP32: a float2 is one aligned register pair, and
// the packed add, multiply and fused multiply-add work on both halves with one
// instruction, each half rounded as the scalar instruction rounds it.  Packed
// instructions do not raise the FMA pipe's rate; they halve the issue slots
// the arithmetic takes, and issue slots are what bounds the x and z passes.  A
// half may be swapped, repeated or negated on the way in at no cost (a radix-8
// stage with its twiddles on two lines, counted by ncu: 158 warp instructions
// against 278 in scalar form, the FMA pipe's share 141 against 265).
__device__ __forceinline__ unsigned long long pack2(float2 a) {
  unsigned long long r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
  return r;
}
__device__ __forceinline__ float2 unpack2(unsigned long long r) {
  float2 a;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a.x), "=f"(a.y) : "l"(r));
  return a;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
  unsigned long long d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(d);
}
__device__ __forceinline__ float2 sub2(float2 a, float2 b) {
  unsigned long long d;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(d);
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
  unsigned long long d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(pack2(a)), "l"(pack2(b)));
  return unpack2(d);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
  unsigned long long d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(pack2(a)), "l"(pack2(b)), "l"(pack2(c)));
  return unpack2(d);
}
__device__ __forceinline__ float2 both(float s) { return make_float2(s, s); }
__device__ __forceinline__ float2 swapped(float2 a) { return make_float2(a.y, a.x); }

__device__ __forceinline__ float2 cadd(float2 a, float2 b) { return add2(a, b); }
__device__ __forceinline__ float2 csub(float2 a, float2 b) { return sub2(a, b); }
__device__ __forceinline__ float2 cscale(float2 a, float s) { return mul2(a, both(s)); }
// a + (-i) b (forward sign) or a + i b (inverse sign), and the same with the
// sign of b reversed: exact products by +-1, so one rounding per half
template <bool INV>
__device__ __forceinline__ float2 cadd_i(float2 a, float2 b) {
  return fma2(swapped(b), INV ? make_float2(-1.f, 1.f) : make_float2(1.f, -1.f), a);
}
template <bool INV>
__device__ __forceinline__ float2 csub_i(float2 a, float2 b) {
  return cadd_i<!INV>(a, b);
}

// ----------------------------------------------------------------------------
// small DFTs in registers (forward: exp(-2 pi i nk/R), inverse: exp(+...)); the
// irrational constants act as two-term products (Const)
// ----------------------------------------------------------------------------
__device__ __forceinline__ float2 mul_r(float2 a) { return fma2(a, both(Const::r_hi), mul2(a, both(Const::r_lo))); }
__device__ __forceinline__ float2 mul_h(float2 a) { return fma2(a, both(Const::h_hi), mul2(a, both(Const::h_lo))); }

template <bool INV>
__device__ __forceinline__ void dft2(float2* v) {
  float2 a = v[0], b = v[1];
  v[0] = cadd(a, b);
  v[1] = csub(a, b);
}

template <bool INV>
__device__ __forceinline__ void dft3(float2* v) {
  float2 a = v[0], b = v[1], c = v[2];
  float2 s = cadd(b, c), d = mul_h(csub(b, c));
  float2 m = fma2(both(-0.5f), s, a);
  v[0] = cadd(a, s);
  v[1] = cadd_i<INV>(m, d);
  v[2] = csub_i<INV>(m, d);
}

template <bool INV>
__device__ __forceinline__ void dft4(float2* v) {
  float2 t0 = cadd(v[0], v[2]), t1 = csub(v[0], v[2]);
  float2 t2 = cadd(v[1], v[3]), d = csub(v[1], v[3]);
  v[0] = cadd(t0, t2);
  v[2] = csub(t0, t2);
  v[1] = cadd_i<INV>(t1, d);
  v[3] = csub_i<INV>(t1, d);
}

template <bool INV>
__device__ __forceinline__ void dft8(float2* v) {
  float2 e[4] = {v[0], v[2], v[4], v[6]};
  float2 o[4] = {v[1], v[3], v[5], v[7]};
  dft4<INV>(e);
  dft4<INV>(o);
  // o[1] W8 and o[3] W8^3 (forward W8 = exp(-i pi/4)): with
  // p = sqrt(2)/2 (x + y, y - x) and q = sqrt(2)/2 (y - x, x + y) of o[1] and
  // o[3], forward W8 o1 = p(o1), W8^3 o3 = (q.x, -q.y); inverse
  // W8 o1 = (-q.x, q.y) with q of o1, W8^3 o3 = -p(o3)
  auto plus = [](float2 a) { return mul_r(fma2(swapped(a), make_float2(1.f, -1.f), a)); };
  auto minus = [](float2 a) { return mul_r(fma2(a, make_float2(-1.f, 1.f), swapped(a))); };
  v[0] = cadd(e[0], o[0]);
  v[4] = csub(e[0], o[0]);
  v[2] = cadd_i<INV>(e[2], o[2]);
  v[6] = csub_i<INV>(e[2], o[2]);
  if constexpr (!INV) {
    const float2 p = plus(o[1]), q = minus(o[3]);
    v[1] = cadd(e[1], p);
    v[5] = csub(e[1], p);
    v[3] = fma2(q, make_float2(1.f, -1.f), e[3]);
    v[7] = fma2(q, make_float2(-1.f, 1.f), e[3]);
  } else {
    const float2 q = minus(o[1]), p = plus(o[3]);
    v[1] = fma2(q, make_float2(-1.f, 1.f), e[1]);
    v[5] = fma2(q, make_float2(1.f, -1.f), e[1]);
    v[3] = csub(e[3], p);
    v[7] = cadd(e[3], p);
  }
}

// 6 = 3 x 2, 12 = 3 x 4 and 24 = 3 x 8 have coprime factors: with the inputs
// at n = B n1 + 3 n2 and the outputs at k = (KA k1 + KB k2) mod 3B (KA = 1 mod 3
// and 0 mod B, KB = 0 mod 3 and 1 mod B) the product n k is B n1 k1 + 3 n2 k2
// mod 3B, so the 3-point and B-point transforms need no twiddles in between
// (Good 1958).
template <int B, bool INV>
__device__ __forceinline__ void dft3xB(float2* v);

// a exp(-+2 pi i M / R) with the constant kept as a (hi, lo) pair like the
// twiddles of the tables (none of those used here has a part of +-1/2).
__host__ __device__ constexpr double cos_2pi(int m, int r);

template <int M, int R, bool INV>
__device__ __forceinline__ float2 const_twiddle(float2 a) {
  static_assert(R == 16 || R == 32, "constants of W16 and W32");
  constexpr int m = M % R;
  if constexpr (m == 0) {
    return a;
  } else if constexpr (4 * m == R) {
    return INV ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
  } else if constexpr (8 * m == R || 8 * m == 3 * R) {
    // sqrt(2)/2 (+-1, -+1): the sum and difference first, exact up to one rounding
    constexpr bool odd3 = 8 * m == 3 * R;
    constexpr float sg = INV ? -1.f : 1.f;
    // forward W8: (x + y, y - x), W8^3: (y - x, -x - y); inverse W8: (x - y, x + y), W8^3: (-x - y, x - y)
    const float2 u = odd3 ? fma2(a, both(-1.f), make_float2(sg * a.y, -sg * a.x))
                          : fma2(swapped(a), make_float2(sg, -sg), a);
    return mul_r(u);
  } else {
    constexpr double c = cos_2pi(m, R), sn = -cos_2pi((m + 3 * R / 4) % R, R);  // cos(x + 3 pi/2) = sin x
    constexpr double s = INV ? -sn : sn;                                          // -sin forward
    constexpr float ch = (float)c, cl = (float)(c - (double)(float)c);
    constexpr float sh = (float)s, sl = (float)(s - (double)(float)s);
    const float2 e = fma2(a, both(cl), mul2(swapped(a), make_float2(-sl, sl)));
    return fma2(a, both(ch), fma2(swapped(a), make_float2(-sh, sh), e));
  }
}

// cos(2 pi m / r) for r = 16 or 32, from the half-angle values of one octant
__host__ __device__ constexpr double cos_2pi(int m, int r) {
  constexpr double c[9] = {1.0,
                           0.98078528040323044913,
                           0.92387953251128675613,
                           0.83146961230254523708,
                           0.70710678118654752440,
                           0.55557023301960222474,
                           0.38268343236508977173,
                           0.19509032201612826785,
                           0.0};
  int k = (m * (32 / r)) % 32;
  if (k > 16) k = 32 - k;
  return k <= 8 ? c[k] : -c[16 - k];
}

template <int... Is>
struct IntSeq {};
template <int N, int... Is>
struct MakeIntSeq : MakeIntSeq<N - 1, N - 1, Is...> {};
template <int... Is>
struct MakeIntSeq<0, Is...> {
  using type = IntSeq<Is...>;
};

template <int A, int B, bool INV, int N2, int K1>
__device__ __forceinline__ void mix_one(float2 (*u)[A]) {
  u[N2][K1] = const_twiddle<N2 * K1, A * B, INV>(u[N2][K1]);
}
template <int A, int B, bool INV, int N2, int... K1>
__device__ __forceinline__ void mix_row(float2 (*u)[A], IntSeq<K1...>) {
  (mix_one<A, B, INV, N2, K1>(u), ...);
}
template <int A, int B, bool INV, int... N2>
__device__ __forceinline__ void mix_all(float2 (*u)[A], IntSeq<N2...>) {
  (mix_row<A, B, INV, N2>(u, typename MakeIntSeq<A>::type{}), ...);
}

template <int R, bool INV>
__device__ __forceinline__ void dftR(float2* v);

// 16 = 4 x 4 and 32 = 4 x 8 Cooley-Tukey with constant twiddles:
// y[k1 + A k2] = sum_n2 W_B^(n2 k2) W_AB^(n2 k1) sum_n1 x[B n1 + n2] W_A^(n1 k1).
template <int A, int B, bool INV>
__device__ __forceinline__ void dftAxB(float2* v) {
  float2 u[B][A];
#pragma unroll
  for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
    for (int n1 = 0; n1 < A; ++n1) u[n2][n1] = v[B * n1 + n2];
    dftR<A, INV>(u[n2]);
  }
  mix_all<A, B, INV>(u, typename MakeIntSeq<B>::type{});
#pragma unroll
  for (int k1 = 0; k1 < A; ++k1) {
    float2 w[B];
#pragma unroll
    for (int n2 = 0; n2 < B; ++n2) w[n2] = u[n2][k1];
    dftR<B, INV>(w);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = w[k2];
  }
}

template <int B, bool INV>
__device__ __forceinline__ void dft3xB(float2* v) {
  constexpr int R = 3 * B;
  constexpr int KA = B % 3 == 1 ? B : 2 * B;  // 1 mod 3, 0 mod B
  constexpr int KB = R + 1 - KA;              // 0 mod 3, 1 mod B
  float2 u[3][B];
#pragma unroll
  for (int n2 = 0; n2 < B; ++n2) {
    float2 w[3];
#pragma unroll
    for (int n1 = 0; n1 < 3; ++n1) w[n1] = v[(B * n1 + 3 * n2) % R];
    dft3<INV>(w);
#pragma unroll
    for (int k1 = 0; k1 < 3; ++k1) u[k1][n2] = w[k1];
  }
#pragma unroll
  for (int k1 = 0; k1 < 3; ++k1) {
    dftR<B, INV>(u[k1]);
#pragma unroll
    for (int k2 = 0; k2 < B; ++k2) v[(KA * k1 + KB * k2) % R] = u[k1][k2];
  }
}

template <int R, bool INV>
__device__ __forceinline__ void dftR(float2* v) {
  if constexpr (R == 2) dft2<INV>(v);
  else if constexpr (R == 3) dft3<INV>(v);
  else if constexpr (R == 4) dft4<INV>(v);
  else if constexpr (R == 6) dft3xB<2, INV>(v);
  else if constexpr (R == 8) dft8<INV>(v);
  else if constexpr (R == 12) dft3xB<4, INV>(v);
  else if constexpr (R == 16) dftAxB<4, 4, INV>(v);
  else if constexpr (R == 24) dft3xB<8, INV>(v);
  else if constexpr (R == 32) dftAxB<4, 8, INV>(v);
  else static_assert(R == 2, "unsupported radix");
}

// ----------------------------------------------------------------------------
// plans and twiddles
// ----------------------------------------------------------------------------
// Plan<N>: the two factors of a line transform and the threads per line T,
// which divides both.
template <int N>
struct Plan;
#define WDM_PLAN(N_, T_, RA_, RB_)                                         \
  template <>                                                              \
  struct Plan<N_> {                                                        \
    static constexpr int N = N_, T = T_, RA = RA_, RB = RB_;               \
    static_assert(RA * RB == N && RA % T == 0 && RB % T == 0, "plan");     \
  };
WDM_PLAN(8, 2, 4, 2)
WDM_PLAN(12, 2, 6, 2)
WDM_PLAN(16, 4, 4, 4)
WDM_PLAN(24, 2, 6, 4)
WDM_PLAN(32, 4, 8, 4)
WDM_PLAN(48, 4, 12, 4)
WDM_PLAN(64, 8, 8, 8)
WDM_PLAN(96, 4, 12, 8)
WDM_PLAN(128, 8, 16, 8)
WDM_PLAN(192, 8, 24, 8)
WDM_PLAN(256, 8, 16, 16)
WDM_PLAN(384, 8, 24, 16)
WDM_PLAN(512, 16, 32, 16)
#undef WDM_PLAN

// a times the twiddle W = (x, y) + (z, w), or its conjugate (pack_twiddle's
// layout and its reasons); ROT: the entry may be stored rotated.
template <bool ROT>
__device__ __forceinline__ float2 twiddle_mul(float2 a, float4 w, bool inv) {
  const bool rot = ROT && (__float_as_uint(w.w) & 1u) != 0;
  const float ax = rot ? (inv ? -a.y : a.y) : a.x;
  const float ay = rot ? (inv ? a.x : -a.x) : a.y;
  const float wy = inv ? -w.y : w.y, ly = inv ? -w.w : w.w;
  const float2 b = make_float2(ax, ay);
  const float2 c = fma2(b, both(w.z), mul2(swapped(b), make_float2(-ly, ly)));
  return fma2(b, both(w.x), fma2(swapped(b), make_float2(-wy, wy), c));
}

struct NoHook {
  __device__ __forceinline__ void operator()() const {}
};

// ----------------------------------------------------------------------------
// two-factor stages (thread t of the T of a line)
// ----------------------------------------------------------------------------
// Stage A: load(p) and store(p, v) access point p of the line.
template <int N, bool INV, class Load, class Store>
__device__ __forceinline__ void factor_a(Load load, Store store, int t) {
  using P = Plan<N>;
#pragma unroll 1
  for (int i = 0; i < P::RB / P::T; ++i) {
    const int n2 = t + P::T * i;
    float2 v[P::RA];
#pragma unroll
    for (int n1 = 0; n1 < P::RA; ++n1) v[n1] = load(P::RB * n1 + n2);
    dftR<P::RA, INV>(v);
#pragma unroll
    for (int k1 = 0; k1 < P::RA; ++k1) store(P::RB * k1 + n2, v[k1]);
  }
}

// Whether some W_N^(n2 k1), k1 < RA, is stored rotated: n2 k1 / N = 1, 5, 7 or
// 11 twelfths (pack_twiddle).
template <int N>
__host__ __device__ constexpr bool factor_rot(int n2) {
  for (int k1 = 0; k1 < Plan<N>::RA; ++k1) {
    const int m = 12 * (n2 * k1 % N);
    if (m == N || m == 5 * N || m == 7 * N || m == 11 * N) return true;
  }
  return false;
}

// W_N^(n2 k1), n2 = 1 .. RB - 1 (or their conjugates), on the elements (k1, n2)
template <int N, bool INV, int N2 = 1>
__device__ __forceinline__ void factor_twiddle(float2* v, const float4* __restrict__ tw, int k1) {
  using P = Plan<N>;
  if constexpr (N2 < P::RB) {
    v[N2] = twiddle_mul<factor_rot<N>(N2)>(v[N2], tw[k1 * (P::RB - 1) + N2 - 1], INV);
    factor_twiddle<N, INV, N2 + 1>(v, tw, k1);
  }
}

// Stage B: use(k1, v) receives the frequencies k1 + RA k2 in v[k2].
template <int N, bool INV, class Load, class Use>
__device__ __forceinline__ void factor_b(Load load, const float4* __restrict__ tw, Use use, int t) {
  using P = Plan<N>;
#pragma unroll 1
  for (int i = 0; i < P::RA / P::T; ++i) {
    const int k1 = t + P::T * i;
    float2 v[P::RB];
#pragma unroll
    for (int n2 = 0; n2 < P::RB; ++n2) v[n2] = load(P::RB * k1 + n2);
    factor_twiddle<N, INV>(v, tw, k1);
    dftR<P::RB, INV>(v);
    use(k1, v);
  }
}

// Host-side builder of the N-entry twiddle table: W_N^(n2 k1) at k1 (RB - 1) + n2
// - 1 (the rest of the N entries is not used).
template <int N, class F>
inline void fill_factor_twiddles(float4* out, F make) {
  using P = Plan<N>;
  for (int q = 0; q < N; ++q) out[q] = make_float4(1.f, 0.f, 0.f, 0.f);
  for (int k1 = 0; k1 < P::RA; ++k1)
    for (int n2 = 1; n2 < P::RB; ++n2) out[k1 * (P::RB - 1) + n2 - 1] = make((long long)k1 * n2);
}

}  // namespace fx
}  // namespace wdm
