// dual.cuh -- forward-mode dual numbers for the local Jacobians of the discrete adjoint.
//
// Dual<N> carries a value and its derivatives along N seed directions.  The adjoint
// kernels evaluate the same templated routines as the forward kernels (reconstruction,
// fluxes, sources, boundary operations) on Dual<N> inputs seeded with the identity, which
// yields the routine's local Jacobian; contracted with the cotangent it gives the routine's
// vector-Jacobian product.  Branches (limiter cases, min/max, upwind direction, clips) are
// taken on the values, as in the forward evaluation, so the derivative is that of the
// branch the forward residual took.  Values are formed without FMA contraction, like the
// reconstruction's uncontracted arithmetic, so that ties at clip bounds resolve the same way.
//
// The direction index of a derivative is always known at compile time (loops over the
// directions unrolled, seeds by comparison).  With an index computed at run time the device
// compiler's full optimisation returned wrong derivatives: cell sources whose first eight
// directions were lost where only the seeds were indexed so, flux gradients of 1e40 where
// every loop was rolled.  The source was not at fault: on the host it reads no uninitialised
// value, stays in range and gives the same bits rolled or unrolled.
#pragma once
#include <cmath>
#include "eos64.cuh"

namespace cfd {

template <int N>
struct Dual {
  double v;
  double d[N];
  __device__ __forceinline__ Dual() {}
  __device__ __forceinline__ Dual(double x) : v(x) {
#pragma unroll
    for (int i = 0; i < N; ++i) d[i] = 0.0;
  }
  __device__ __forceinline__ static Dual seed(double x, int i) {
    Dual r;
    r.v = x;
#pragma unroll
    for (int q = 0; q < N; ++q) r.d[q] = (q == i) ? 1.0 : 0.0;
    return r;
  }
  __device__ __forceinline__ explicit operator double() const { return v; }
};

#define DUAL_LOOP _Pragma("unroll") for (int i = 0; i < N; ++i)

template <int N> __device__ __forceinline__ Dual<N> operator+(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r; r.v = __dadd_rn(a.v, b.v); DUAL_LOOP r.d[i] = a.d[i] + b.d[i]; return r;
}
template <int N> __device__ __forceinline__ Dual<N> operator-(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r; r.v = __dsub_rn(a.v, b.v); DUAL_LOOP r.d[i] = a.d[i] - b.d[i]; return r;
}
template <int N> __device__ __forceinline__ Dual<N> operator-(const Dual<N>& a) {
  Dual<N> r; r.v = -a.v; DUAL_LOOP r.d[i] = -a.d[i]; return r;
}
template <int N> __device__ __forceinline__ Dual<N> operator*(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r; r.v = __dmul_rn(a.v, b.v); DUAL_LOOP r.d[i] = a.d[i] * b.v + a.v * b.d[i]; return r;
}
template <int N> __device__ __forceinline__ Dual<N> operator/(const Dual<N>& a, const Dual<N>& b) {
  Dual<N> r; r.v = a.v / b.v;
  const double ib = 1.0 / b.v;
  DUAL_LOOP r.d[i] = (a.d[i] - r.v * b.d[i]) * ib;
  return r;
}
// mixed operands
template <int N> __device__ __forceinline__ Dual<N> operator+(const Dual<N>& a, double b) { Dual<N> r = a; r.v = __dadd_rn(r.v, b); return r; }
template <int N> __device__ __forceinline__ Dual<N> operator+(double a, const Dual<N>& b) { Dual<N> r = b; r.v = __dadd_rn(a, r.v); return r; }
template <int N> __device__ __forceinline__ Dual<N> operator-(const Dual<N>& a, double b) { Dual<N> r = a; r.v = __dsub_rn(r.v, b); return r; }
template <int N> __device__ __forceinline__ Dual<N> operator-(double a, const Dual<N>& b) {
  Dual<N> r; r.v = __dsub_rn(a, b.v); DUAL_LOOP r.d[i] = -b.d[i]; return r;
}
template <int N> __device__ __forceinline__ Dual<N> operator*(const Dual<N>& a, double b) {
  Dual<N> r; r.v = __dmul_rn(a.v, b); DUAL_LOOP r.d[i] = a.d[i] * b; return r;
}
template <int N> __device__ __forceinline__ Dual<N> operator*(double a, const Dual<N>& b) { return b * a; }
template <int N> __device__ __forceinline__ Dual<N> operator/(const Dual<N>& a, double b) {
  Dual<N> r; r.v = a.v / b;
  const double ib = 1.0 / b;
  DUAL_LOOP r.d[i] = a.d[i] * ib;
  return r;
}
template <int N> __device__ __forceinline__ Dual<N> operator/(double a, const Dual<N>& b) {
  Dual<N> r; r.v = a / b.v;
  const double f = -r.v / b.v;
  DUAL_LOOP r.d[i] = f * b.d[i];
  return r;
}
template <int N> __device__ __forceinline__ Dual<N>& operator+=(Dual<N>& a, const Dual<N>& b) { a = a + b; return a; }
template <int N> __device__ __forceinline__ Dual<N>& operator-=(Dual<N>& a, const Dual<N>& b) { a = a - b; return a; }
template <int N> __device__ __forceinline__ Dual<N>& operator*=(Dual<N>& a, const Dual<N>& b) { a = a * b; return a; }

// comparisons on values
template <int N> __device__ __forceinline__ bool operator<(const Dual<N>& a, const Dual<N>& b) { return a.v < b.v; }
template <int N> __device__ __forceinline__ bool operator>(const Dual<N>& a, const Dual<N>& b) { return a.v > b.v; }
template <int N> __device__ __forceinline__ bool operator<=(const Dual<N>& a, const Dual<N>& b) { return a.v <= b.v; }
template <int N> __device__ __forceinline__ bool operator>=(const Dual<N>& a, const Dual<N>& b) { return a.v >= b.v; }
template <int N> __device__ __forceinline__ bool operator<(const Dual<N>& a, double b) { return a.v < b; }
template <int N> __device__ __forceinline__ bool operator>(const Dual<N>& a, double b) { return a.v > b; }
template <int N> __device__ __forceinline__ bool operator<=(const Dual<N>& a, double b) { return a.v <= b; }
template <int N> __device__ __forceinline__ bool operator>=(const Dual<N>& a, double b) { return a.v >= b; }
template <int N> __device__ __forceinline__ bool operator!=(const Dual<N>& a, double b) { return a.v != b; }
template <int N> __device__ __forceinline__ bool operator!=(const Dual<N>& a, const Dual<N>& b) { return a.v != b.v; }
template <int N> __device__ __forceinline__ bool operator==(const Dual<N>& a, const Dual<N>& b) { return a.v == b.v; }
template <int N> __device__ __forceinline__ bool operator==(const Dual<N>& a, double b) { return a.v == b; }

// elementary functions
template <int N> __device__ __forceinline__ Dual<N> sqrt(const Dual<N>& a) {
  Dual<N> r; r.v = ::sqrt(a.v);
  const double f = (r.v > 0.0) ? 0.5 / r.v : 0.0;
  DUAL_LOOP r.d[i] = f * a.d[i];
  return r;
}
template <int N> __device__ __forceinline__ Dual<N> exp(const Dual<N>& a) {
  Dual<N> r; r.v = ::exp(a.v); DUAL_LOOP r.d[i] = r.v * a.d[i]; return r;
}
template <int N> __device__ __forceinline__ Dual<N> log(const Dual<N>& a) {
  Dual<N> r; r.v = ::log(a.v); const double f = 1.0 / a.v; DUAL_LOOP r.d[i] = f * a.d[i]; return r;
}
template <int N> __device__ __forceinline__ Dual<N> tanh(const Dual<N>& a) {
  Dual<N> r; r.v = ::tanh(a.v); const double f = 1.0 - r.v * r.v; DUAL_LOOP r.d[i] = f * a.d[i]; return r;
}
// x^y with a constant exponent
template <int N> __device__ __forceinline__ Dual<N> pow(const Dual<N>& a, double y) {
  Dual<N> r; r.v = ::pow(a.v, y);
  const double f = (a.v != 0.0) ? y * r.v / a.v : 0.0;
  DUAL_LOOP r.d[i] = f * a.d[i];
  return r;
}
// x^y with both varying: d = x^y (y' log x + y x'/x)
template <int N> __device__ __forceinline__ Dual<N> pow(const Dual<N>& a, const Dual<N>& y) {
  Dual<N> r; r.v = ::pow(a.v, y.v);
  const double lx = (a.v > 0.0) ? ::log(a.v) : 0.0;
  const double f = (a.v != 0.0) ? y.v * r.v / a.v : 0.0;
  DUAL_LOOP r.d[i] = r.v * lx * y.d[i] + f * a.d[i];
  return r;
}
template <int N> __device__ __forceinline__ Dual<N> fabs(const Dual<N>& a) { return (a.v < 0.0) ? -a : a; }
template <int N> __device__ __forceinline__ Dual<N> fmin(const Dual<N>& a, const Dual<N>& b) { return (b.v < a.v) ? b : a; }
template <int N> __device__ __forceinline__ Dual<N> fmax(const Dual<N>& a, const Dual<N>& b) { return (b.v > a.v) ? b : a; }
template <int N> __device__ __forceinline__ Dual<N> fmin(const Dual<N>& a, double b) { return (b < a.v) ? Dual<N>(b) : a; }
template <int N> __device__ __forceinline__ Dual<N> fmax(const Dual<N>& a, double b) { return (b > a.v) ? Dual<N>(b) : a; }
template <int N> __device__ __forceinline__ Dual<N> fmin(double a, const Dual<N>& b) { return (b.v < a) ? b : Dual<N>(a); }
template <int N> __device__ __forceinline__ Dual<N> fmax(double a, const Dual<N>& b) { return (b.v > a) ? b : Dual<N>(a); }
template <int N> __device__ __forceinline__ Dual<N> copysign(double a, const Dual<N>& b) { return Dual<N>(::copysign(a, b.v)); }
template <int N> __device__ __forceinline__ bool isfinite(const Dual<N>& a) { return ::isfinite(a.v); }

// uncontracted arithmetic of the reconstruction: duals have no FMA ambiguity
template <int N> __device__ __forceinline__ Dual<N> nmul(const Dual<N>& a, const Dual<N>& b) { return a * b; }
template <int N> __device__ __forceinline__ Dual<N> nadd(const Dual<N>& a, const Dual<N>& b) { return a + b; }
template <int N> __device__ __forceinline__ Dual<N> nsub(const Dual<N>& a, const Dual<N>& b) { return a - b; }

#undef DUAL_LOOP

// IF97 Gibbs sums on dual arguments: g = sum n x^I y^J with its first three derivatives in
// FP64, by groups of equal I as eos64.cuh sums them, then each derivative g_a becomes a dual
// number with d(g_a) = g_ax dx + g_ay dy.  Exact, and the sums stay plain FP64 code.
struct G64Third {
  double z1 = 0.0, z2 = 0.0, z3 = 0.0;                // I = 0: P1, P2, P3 (Pk = y^k d^k P0 / dy^k)
  double o0 = 0.0, o1 = 0.0, o2 = 0.0, o3 = 0.0;      // I = 1: P0 .. P3
  double t0 = 0.0, t1 = 0.0, t2 = 0.0, t3 = 0.0;      // I = 2
  // I >= 3, X = x^(I-3): X I P0, X I (I-1) P0, X I (I-1) (I-2) P0, X P1, X I P1, X I (I-1) P1,
  // X P2, X I P2, X P3
  double a1 = 0.0, a2 = 0.0, a3 = 0.0, b0 = 0.0, b1 = 0.0, b2 = 0.0, c0 = 0.0, c1 = 0.0, d0 = 0.0;
};
template <const IJN* TAB, size_t K>
__device__ __forceinline__ void g64_term3(double y, double yi, double* p) {
  constexpr int J = TAB[K].j;
  constexpr double n = TAB[K].n, j = J;
  if constexpr (J == 0) p[0] += n;
  else {
    const double q = cpow<J>(y, yi);
    p[0] = fma(n, q, p[0]);
    p[1] = fma(n * j, q, p[1]);
    if constexpr (J != 1) p[2] = fma(n * j * (j - 1.0), q, p[2]);
    if constexpr (J != 1 && J != 2) p[3] = fma(n * j * (j - 1.0) * (j - 2.0), q, p[3]);
  }
}
template <const IJN* TAB, size_t S, size_t... K>
__device__ __forceinline__ void g64_group3(double x, double y, double yi, G64Third& a, std::index_sequence<K...>) {
  constexpr int I = TAB[S].i;
  constexpr double i = I;
  double p[4] = {0.0, 0.0, 0.0, 0.0};
  (g64_term3<TAB, S + K>(y, yi, p), ...);
  if constexpr (I == 0) { a.z1 = p[1]; a.z2 = p[2]; a.z3 = p[3]; }
  else if constexpr (I == 1) { a.o0 = p[0]; a.o1 = p[1]; a.o2 = p[2]; a.o3 = p[3]; }
  else if constexpr (I == 2) { a.t0 = p[0]; a.t1 = p[1]; a.t2 = p[2]; a.t3 = p[3]; }
  else {
    const double X = cpow<I - 3>(x, x), t = X * p[0], u = X * p[1], w = X * p[2];
    a.a1 = fma(i, t, a.a1); a.a2 = fma(i * (i - 1.0), t, a.a2); a.a3 = fma(i * (i - 1.0) * (i - 2.0), t, a.a3);
    a.b0 += u; a.b1 = fma(i, u, a.b1); a.b2 = fma(i * (i - 1.0), u, a.b2);
    a.c0 += w; a.c1 = fma(i, w, a.c1);
    a.d0 = fma(X, p[3], a.d0);
  }
}
template <const IJN* TAB, size_t N, int... G>
__device__ __forceinline__ void g64_groups3(double x, double y, double yi, G64Third& a, std::integer_sequence<int, G...>) {
  (g64_group3<TAB, IGroups<TAB, N>::start(G)>(
       x, y, yi, a, std::make_index_sequence<IGroups<TAB, N>::start(G + 1) - IGroups<TAB, N>::start(G)>{}), ...);
}

template <int N>
struct GibbsByParts<Dual<N>> {
  static constexpr bool value = true;
  template <const IJN* TAB, size_t... K>
  static __device__ __forceinline__ void sum(const Dual<N>& X, const Dual<N>&, const Dual<N>& Y,
                                             const Dual<N>& YI, GAcc<Dual<N>>& a) {
    constexpr size_t M = sizeof...(K);
    const double x = X.v, yi = YI.v, yi2 = yi * yi;
    G64Third g;
    g64_groups3<TAB, M>(x, Y.v, yi, g, std::make_integer_sequence<int, IGroups<TAB, M>::count()>{});
    // S: g_x, g_y, g_xx, g_xy, g_yy, g_xxx, g_xxy, g_xyy, g_yyy
    double S[9];
    S[0] = fma(x, fma(x, g.a1, 2.0 * g.t0), g.o0);
    S[1] = fma(x, fma(x, fma(x, g.b0, g.t1), g.o1), g.z1) * yi;
    S[2] = fma(x, g.a2, 2.0 * g.t0);
    S[3] = fma(x, fma(x, g.b1, 2.0 * g.t1), g.o1) * yi;
    S[4] = fma(x, fma(x, fma(x, g.c0, g.t2), g.o2), g.z2) * yi2;
    S[5] = g.a3;
    S[6] = fma(x, g.b2, 2.0 * g.t1) * yi;
    S[7] = fma(x, fma(x, g.c1, 2.0 * g.t2), g.o2) * yi2;
    S[8] = fma(x, fma(x, fma(x, g.d0, g.t3), g.o3), g.z3) * (yi2 * yi);
    const int from[5][3] = {{0, 2, 3}, {1, 3, 4}, {2, 5, 6}, {3, 6, 7}, {4, 7, 8}};
    Dual<N>* out[5] = {&a.x, &a.y, &a.xx, &a.xy, &a.yy};
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      Dual<N> r(S[from[q][0]]);
#pragma unroll
      for (int i = 0; i < N; ++i) r.d[i] = S[from[q][1]] * X.d[i] + S[from[q][2]] * Y.d[i];
      *out[q] = *out[q] + r;
    }
  }
};

}  // namespace cfd
