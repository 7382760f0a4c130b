// eos64.cuh -- the FP64 form's IF97 phase properties.
//
// A GB300 SM issues one FP64 warp instruction per 16 clocks (1/64 of its FP32 rate) and a
// single warp one per 64, so these routines are bound by the number of FP64 instructions
// alone: in the saturated kernels by the pipe, in the small ones by one warp's chain.  The
// Gibbs sum g = sum n x^I y^J and its derivatives are therefore taken by groups of equal I
// (the tables are sorted by I): a group needs
//   P0 = sum n y^J,   P1 = sum n J y^J = y dP0/dy,   P2 = sum n J (J - 1) y^J = y^2 d2P0/dy2,
// one multiply-add per term and sum with constants formed at compile time, and enters the
// derivatives through one power of x.  Region 1 with all five derivatives takes about 200
// FP64 instructions instead of 550 term by term, rho and h alone about 110 instead of 310.
// The phases' specific volumes follow as gamma_pi t / c without a division, and every
// quotient by t comes from one 1 / t.
#pragma once
#include "iapws.cuh"

namespace cfd {

// runs of equal I in a table sorted by I
template <const IJN* TAB, size_t N>
struct IGroups {
  static constexpr bool head(size_t k) { return k == 0 || TAB[k].i != TAB[k - 1].i; }
  static constexpr int count() {
    int c = 0;
    for (size_t k = 0; k < N; ++k) c += head(k) ? 1 : 0;
    return c;
  }
  static constexpr size_t start(int g) {
    int c = -1;
    for (size_t k = 0; k < N; ++k) {
      if (head(k)) ++c;
      if (c == g) return k;
    }
    return N;
  }
};

// the sums of one table, by the order I of their group: I = 0 (z), I = 1 (o) and the rest,
// whose common factor x (x^2 for the plain y sums) is applied once at the end
struct G64 {
  double z1 = 0.0, z2 = 0.0;               // I = 0: P1, P2
  double o0 = 0.0, o1 = 0.0, o2 = 0.0;     // I = 1: P0, P1, P2
  // I >= 2, X = x^(I-2): sum X I P0, X I (I-1) P0, X P1, X I P1, X P2
  double bx = 0.0, bxx = 0.0, by = 0.0, bxy = 0.0, byy = 0.0;
};

template <const IJN* TAB, size_t K, bool FULL>
__device__ __forceinline__ void g64_term(double y, double yi, double& p0, double& p1, double& p2) {
  constexpr int J = TAB[K].j;
  constexpr double n = TAB[K].n;
  if constexpr (J == 0) p0 += n;
  else {
    const double p = cpow<J>(y, yi);
    p0 = fma(n, p, p0);
    p1 = fma(n * double(J), p, p1);
    if constexpr (FULL && J != 1) p2 = fma(n * double(J) * double(J - 1), p, p2);
  }
}

template <const IJN* TAB, size_t S, bool FULL, size_t... K>
__device__ __forceinline__ void g64_group(double x, double y, double yi, G64& a, std::index_sequence<K...>) {
  constexpr int I = TAB[S].i;
  if constexpr (I >= 2 && sizeof...(K) == 1) {
    // a single term: every sum is a multiple of t = n x^(I-2) y^J
    constexpr int J = TAB[S].j;
    constexpr double i = I, j = J;
    double t;
    if constexpr (J == 0) t = TAB[S].n * cpow<I - 2>(x, x);
    else t = TAB[S].n * cpow<J>(y, yi) * cpow<I - 2>(x, x);
    a.bx = fma(i, t, a.bx);
    if constexpr (J != 0) a.by = fma(j, t, a.by);
    if constexpr (FULL) {
      a.bxx = fma(i * (i - 1.0), t, a.bxx);
      if constexpr (J != 0) a.bxy = fma(i * j, t, a.bxy);
      if constexpr (J != 0 && J != 1) a.byy = fma(j * (j - 1.0), t, a.byy);
    }
  } else {
    double p0 = 0.0, p1 = 0.0, p2 = 0.0;
    (g64_term<TAB, S + K, FULL>(y, yi, p0, p1, p2), ...);
    if constexpr (I == 0) {
      a.z1 = p1; a.z2 = p2;
    } else if constexpr (I == 1) {
      a.o0 = p0; a.o1 = p1; a.o2 = p2;
    } else {
      constexpr double i = I;
      const double X = cpow<I - 2>(x, x);
      if constexpr (FULL) {
        const double t = X * p0, u = X * p1;
        a.bx = fma(i, t, a.bx);
        a.bxx = fma(i * (i - 1.0), t, a.bxx);
        a.by += u;
        a.bxy = fma(i, u, a.bxy);
        a.byy = fma(X, p2, a.byy);
      } else {
        a.bx = fma(i * X, p0, a.bx);
        a.by = fma(X, p1, a.by);
      }
    }
  }
}

template <const IJN* TAB, size_t N, bool FULL, int... G>
__device__ __forceinline__ void g64_groups(double x, double y, double yi, G64& a, std::integer_sequence<int, G...>) {
  (g64_group<TAB, IGroups<TAB, N>::start(G), FULL>(
       x, y, yi, a, std::make_index_sequence<IGroups<TAB, N>::start(G + 1) - IGroups<TAB, N>::start(G)>{}), ...);
}

// g_x, g_y and (FULL) g_xx, g_yy, g_xy of the table's sum; yi = 1 / y
template <const IJN* TAB, size_t N, bool FULL>
__device__ __forceinline__ void g64_sum(double x, double y, double yi, double& gx, double& gxx, double& gy,
                                        double& gyy, double& gxy) {
  G64 a;
  g64_groups<TAB, N, FULL>(x, y, yi, a, std::make_integer_sequence<int, IGroups<TAB, N>::count()>{});
  gx = fma(x, a.bx, a.o0);
  gy = fma(x, fma(x, a.by, a.o1), a.z1) * yi;
  if constexpr (FULL) {
    gxx = a.bxx;
    gxy = fma(x, a.bxy, a.o1) * yi;
    gyy = fma(x, fma(x, a.byy, a.o2), a.z2) * (yi * yi);
  }
}

// c / t from it = RN(1 / t): the product's rounding error taken out by one residual step
// (Markstein 1990), since powers of tau up to the 58th amplify it
__device__ __forceinline__ double over_t(double c, double t, double it) {
  const double q = c * it;
  return fma(fma(-t, q, c), it, q);
}

// region 1 (liquid) at p, t with it = 1 / t: irho = 1 / rho and h; FULL: all of e
template <bool FULL>
__device__ __forceinline__ void if97_liquid(double p, double t, double it, Phase<double>& e, double& irho) {
  const double tau = over_t(1386.0, t, it);
  const double x = 7.1 - p * 0.00000006049607;
  const double y = tau - 1.222, yi = 1.0 / y;
  double gx, gxx, gy, gyy, gxy;
  g64_sum<kR1, 34, FULL>(x, y, yi, gx, gxx, gy, gyy, gxy);
  // d/dpi = -d/dx; rho = c tau / gamma_pi
  constexpr double c = (double)25.841246054191803727f;
  irho = -gx * t * (1.0 / (c * 1386.0));
  e.h = 639675.036 * gy;
  if constexpr (FULL) {
    e.rho = 1.0 / irho;
    const double gp1 = e.rho * t * (1.0 / (c * 1386.0)), gp2 = gp1 * gp1;
    e.drdp = -(gxx * 1.5632937721834122e-6 * tau * gp2);
    e.drdt = -(e.rho * 7.215007215007215e-4 * tau) - (double)0.01864447767257706f * gxy * (tau * tau * tau) * gp2;
    e.dhdp = -(double)0.03869782431941923775f * gxy;
    e.dhdt = -(461.526 * (tau * tau) * gyy);
  }
}

// g_x term by term, n x^I y^J first, in the reference's order of operations and without
// multiply-add contraction (xi = 1 / x)
template <const IJN* TAB, size_t... K>
__device__ __forceinline__ double gx_terms(double x, double xi, double y, double yi, std::index_sequence<K...>) {
  double s = 0.0;
  ((s = __dadd_rn(s, __dmul_rn(double(TAB[K].i) * (TAB[K].n * cpow<TAB[K].i>(x, xi) * cpow<TAB[K].j>(y, yi)), xi))),
   ...);
  return s;
}

// region 2, the metastable set when meta, with pi1 = 1e6 / p (correctly rounded: near the
// metastable limit gamma_pi = pi1 + ... cancels) and it = 1 / t
template <bool FULL>
__device__ __forceinline__ void if97_vapour(double p, double t, double pi1, double it, bool meta, Phase<double>& e,
                                            double& irho) {
  const double pi = p * 1e-6;
  const double tau = over_t(540.0, t, it), taui = t * (1.0 / 540.0);
  const double y = tau - 0.5, yi = 1.0 / y;
  double ix, ixx, iy, iyy, ixy, rx, rxx, ry, ryy, rxy;
  if (meta) {
    g64_sum<kR2MI, 9, FULL>(pi, tau, taui, ix, ixx, iy, iyy, ixy);
    g64_sum<kR2MR, 13, FULL>(pi, y, yi, rx, rxx, ry, ryy, rxy);
    // deep in the metastable range (pressures far above saturation) gamma_pi passes through
    // zero: its sum keeps the reference's order of operations, so that the two round alike
    rx = gx_terms<kR2MR>(pi, pi1, y, yi, std::make_index_sequence<13>{});
  } else {
    g64_sum<kR2I, 9, FULL>(pi, tau, taui, ix, ixx, iy, iyy, ixy);
    g64_sum<kR2R, 43, FULL>(pi, y, yi, rx, rxx, ry, ryy, rxy);
  }
  const double gp = __dadd_rn(pi1, rx);
  // rho before its reciprocal, again the reference's order: the differences 1 / rho_l - 1 / rho_v
  // and the mixture's sums cancel there too
  const double gp1 = 1.0 / gp;
  e.rho = 4.01245401527075799 * tau * gp1;
  irho = 1.0 / e.rho;
  e.h = 249224.04 * (iy + ry);
  if constexpr (FULL) {
    const double gpp = rxx - pi1 * pi1, gtt = iyy + ryy;
    const double gp2 = gp1 * gp1;
    e.drdp = -(gpp * 4.01245401527075799e-6 * tau * gp2);
    e.drdt = -(e.rho * (double)0.00185185185185185185f * tau) +
             (double)0.0074304703986495518f * rxy * (tau * tau * tau) * gp2;
    e.dhdp = 0.24922404 * rxy;
    e.dhdt = -(461.526 * (tau * tau) * gtt);
  }
}

}  // namespace cfd
