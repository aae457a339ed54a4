// dft.cuh -- what the transforms of the two arithmetics share: the in-register inverse DFTs of the
// mixed path's float2 and the FP64 path's double2, and the plans of their Stockham passes.
#pragma once
#include <type_traits>

namespace ermod {

template <class V>
using scalar_of = std::conditional_t<std::is_same_v<V, double2>, double, float>;
template <class V>
__device__ __forceinline__ V cpx(scalar_of<V> x, scalar_of<V> y) {
  V v;
  v.x = x;
  v.y = y;
  return v;
}
template <class V>
__device__ __forceinline__ V cmul(V a, V b) {
  return cpx<V>(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
template <class V>
__device__ __forceinline__ V cadd(V a, V b) { return cpx<V>(a.x + b.x, a.y + b.y); }
template <class V>
__device__ __forceinline__ V csub(V a, V b) { return cpx<V>(a.x - b.x, a.y - b.y); }
template <class V>
__device__ __forceinline__ V mul_i(V a) { return cpx<V>(-a.y, a.x); }  // a * i

// ---- in-register inverse DFTs: Y[q] = sum_r v[r] exp(+2 pi i r q / R) ----------------
template <int R>
struct Dft;

template <>
struct Dft<2> {
  template <class V>
  static __device__ __forceinline__ void run(V* v) {
    const V a = v[0], b = v[1];
    v[0] = cadd(a, b);
    v[1] = csub(a, b);
  }
};
template <>
struct Dft<3> {
  template <class V>
  static __device__ __forceinline__ void run(V* v) {
    const scalar_of<V> c = -0.5, s = (scalar_of<V>)0.86602540378443864676;  // exp(2 pi i / 3)
    const V a = v[0], b = v[1], d = v[2];
    const V t = cadd(b, d), u = csub(b, d);
    v[0] = cadd(a, t);
    const V m = cpx<V>(a.x + c * t.x, a.y + c * t.y);
    const V n = cpx<V>(-s * u.y, s * u.x);  // i s (b - d)
    v[1] = cadd(m, n);
    v[2] = csub(m, n);
  }
};
template <>
struct Dft<4> {
  template <class V>
  static __device__ __forceinline__ void run(V* v) {
    const V a = cadd(v[0], v[2]), b = csub(v[0], v[2]);
    const V c = cadd(v[1], v[3]), d = mul_i(csub(v[1], v[3]));
    v[0] = cadd(a, c);
    v[2] = csub(a, c);
    v[1] = cadd(b, d);
    v[3] = csub(b, d);
  }
};
template <>
struct Dft<5> {
  template <class V>
  static __device__ __forceinline__ void run(V* v) {
    const scalar_of<V> c1 = (scalar_of<V>)0.30901699437494742410, c2 = (scalar_of<V>)-0.80901699437494742410;
    const scalar_of<V> s1 = (scalar_of<V>)0.95105651629515357212, s2 = (scalar_of<V>)0.58778525229247312917;
    const V a = v[0];
    const V t1 = cadd(v[1], v[4]), t2 = cadd(v[2], v[3]);
    const V u1 = csub(v[1], v[4]), u2 = csub(v[2], v[3]);
    v[0] = cadd(a, cadd(t1, t2));
    const V m1 = cpx<V>(a.x + c1 * t1.x + c2 * t2.x, a.y + c1 * t1.y + c2 * t2.y);
    const V m2 = cpx<V>(a.x + c2 * t1.x + c1 * t2.x, a.y + c2 * t1.y + c1 * t2.y);
    const V n1 = cpx<V>(s1 * u1.x + s2 * u2.x, s1 * u1.y + s2 * u2.y);  // (s1 u1 + s2 u2)
    const V n2 = cpx<V>(s2 * u1.x - s1 * u2.x, s2 * u1.y - s1 * u2.y);
    v[1] = cadd(m1, mul_i(n1));
    v[4] = csub(m1, mul_i(n1));
    v[2] = cadd(m2, mul_i(n2));
    v[3] = csub(m2, mul_i(n2));
  }
};

// compile-time cos/sin(pi x) for the in-register twiddles (Taylor series after reduction
// to [-1/2, 1/2]; |error| < 1e-16, folded to constants)
constexpr double ct_pi = 3.14159265358979323846;
constexpr double ct_taylor_cos(double t) {  // cos(t), |t| <= pi/2
  double term = 1.0, sum = 1.0;
  for (int k = 1; k < 16; ++k) {
    term = -term * t * t / ((2.0 * k - 1.0) * (2.0 * k));
    sum += term;
  }
  return sum;
}
constexpr double ct_taylor_sin(double t) {  // sin(t), |t| <= pi/2
  double term = t, sum = t;
  for (int k = 1; k < 16; ++k) {
    term = -term * t * t / ((2.0 * k) * (2.0 * k + 1.0));
    sum += term;
  }
  return sum;
}
constexpr double ct_cospi(double x) {  // cos(pi x)
  while (x > 1.0) x -= 2.0;
  while (x < -1.0) x += 2.0;
  if (x > 0.5) return -ct_taylor_cos(ct_pi * (1.0 - x));
  if (x < -0.5) return -ct_taylor_cos(ct_pi * (1.0 + x));
  return ct_taylor_cos(ct_pi * x);
}
constexpr double ct_sinpi(double x) {  // sin(pi x)
  while (x > 1.0) x -= 2.0;
  while (x < -1.0) x += 2.0;
  if (x > 0.5) return ct_taylor_sin(ct_pi * (1.0 - x));
  if (x < -0.5) return -ct_taylor_sin(ct_pi * (1.0 + x));
  return ct_taylor_sin(ct_pi * x);
}

// composite radix A*B in registers (Cooley-Tukey): B DFTs of size A on stride-B
// subsequences, twiddles exp(+2 pi i a b / R), then A DFTs of size B
template <int A, int B>
struct DftCT {
  static constexpr int R = A * B;
  template <class V>
  static __device__ __forceinline__ void run(V* v) {
    V t[R];
#pragma unroll
    for (int b = 0; b < B; ++b) {
      V s[A];
#pragma unroll
      for (int a = 0; a < A; ++a) s[a] = v[a * B + b];
      Dft<A>::run(s);
#pragma unroll
      for (int a = 0; a < A; ++a) {
        if (a * b != 0) {
          const scalar_of<V> cs = (scalar_of<V>)ct_cospi(2.0 * (double)(a * b) / (double)R);
          const scalar_of<V> sn = (scalar_of<V>)ct_sinpi(2.0 * (double)(a * b) / (double)R);
          s[a] = cmul(s[a], cpx<V>(cs, sn));
        }
        t[a * B + b] = s[a];
      }
    }
    // t[a*B + b]: A-point results (index a) of subsequence b; now B-point DFTs over b
#pragma unroll
    for (int a = 0; a < A; ++a) {
      V s[B];
#pragma unroll
      for (int b = 0; b < B; ++b) s[b] = t[a * B + b];
      Dft<B>::run(s);
#pragma unroll
      for (int b = 0; b < B; ++b) v[b * A + a] = s[b];
    }
  }
};
template <>
struct Dft<6> : DftCT<2, 3> {};
template <>
struct Dft<8> : DftCT<2, 4> {};
template <>
struct Dft<9> : DftCT<3, 3> {};
template <>
struct Dft<10> : DftCT<2, 5> {};
template <>
struct Dft<12> : DftCT<4, 3> {};
template <>
struct Dft<15> : DftCT<3, 5> {};
template <>
struct Dft<16> : DftCT<4, 4> {};

// n / d for n < 2^16 by a multiply-high (m = ceil(2^32 / d)); d = 1 handled apart
struct FastDiv {
  unsigned d, m;
};
__host__ __device__ inline FastDiv make_fastdiv(unsigned d) {
  return FastDiv{d, d <= 1 ? 0u : (unsigned)((0x100000000ull + d - 1) / d)};
}

// radix plan: at most kMaxPasses radices from {16,15,12,10,9,8,6,5,4,3,2}, fewest passes
constexpr int kMaxPasses = 6;
struct FftPlan {
  int n, npass, r[kMaxPasses], ns[kMaxPasses];
  FastDiv fns[kMaxPasses];
};
// the plan of a length with factors 2, 3 and 5 only; false for another one
bool fft_plan(int n, FftPlan& p);

}  // namespace ermod
