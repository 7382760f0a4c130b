// adjoint_flux.cuh -- the inviscid-flux kernel of the discrete adjoint, instantiated by
// adjoint_face.cu (Roe, AUSM+-up: flux_back) and adjoint_duals.cu (Roe-M, AUSMPW+:
// flux_back_duals).  The file comment of adjoint_face.cu describes the face part.
#pragma once
#include "adjoint.cuh"
#include "faces64.cuh"

namespace cfd {

// the gradient of lam . F with respect to a face's states
struct FaceGrad { double pl[NPVM], pr[NPVM], rl, rr, hl, hr, c2l, c2r, uref; };

// the flux reversed: o from the cotangent lam; SENSOR: also the gradient ws[18] with respect to
// the pressure sensor's stencil sdv (the specialisation of each unit)
template <bool SENSOR>
struct FluxBack;

// rho, h of a face state and their derivatives in (p, T, y1, y2): exact derivatives of the
// values' own formulas, from the second derivatives of the Gibbs sums
struct RhoH { double rho, h, drho[4], dh[4]; };

static __device__ __noinline__ RhoH rho_h_jac(int fluid, double p, double t, double y1, double y2) {
  // il, iv, ig: 1 / rho per phase with p and T slopes; hl, hv, hg likewise
  double il, ilp, ilt, hl, hlp, hlt, iv, ivp = 0.0, ivt = 0.0, hv, hvp = 0.0, hvt = 0.0;
  const double it = 1.0 / t, pi1 = 1.0e6 / p, r1 = 0.00348383500557;
  const double ig = t * pi1 * (1.0e-6 / r1), igp = -ig * (pi1 * 1.0e-6), igt = ig * it;
  const double hg = 1004.64 * t, hgt = 1004.64;
  if (fluid == 1) {
    const double q = p + 8.5e8, rl = 0.00037160906726, iq = 1.0 / q;
    il = t * iq * (1.0 / rl); ilp = -il * iq; ilt = il * it;
    hl = 4186.0 * t - 917822.36; hlp = 0.0; hlt = 4186.0;
    iv = ig; ivp = igp; ivt = igt; hv = hg; hvt = hgt;
  } else {
    double gx, gxx, gy, gyy, gxy;
    {
      constexpr double k = 1.0 / ((double)25.841246054191803727f * 1386.0), pip = 0.00000006049607;
      const double tau = over_t(1386.0, t, it), y = tau - 1.222, yi = 1.0 / y, taut = -tau * it;
      g64_sum<kR1, 34, true>(7.1 - p * pip, y, yi, gx, gxx, gy, gyy, gxy);
      il = -gx * t * k; ilp = gxx * pip * t * k; ilt = k * (-gx - gxy * taut * t);
      hl = 639675.036 * gy; hlp = -639675.036 * gxy * pip; hlt = 639675.036 * gyy * taut;
    }
    {
      constexpr double k = 1.0 / (4.01245401527075799 * 540.0);
      const double pi = p * 1e-6, tau = over_t(540.0, t, it), taui = t * (1.0 / 540.0), taut = -tau * it;
      const double y = tau - 0.5, yi = 1.0 / y;
      double jx, jxx, jy, jyy, jxy;
      if (above_psat(p, t)) {
        g64_sum<kR2MI, 9, true>(pi, tau, taui, jx, jxx, jy, jyy, jxy);
        g64_sum<kR2MR, 13, true>(pi, y, yi, gx, gxx, gy, gyy, gxy);
      } else {
        g64_sum<kR2I, 9, true>(pi, tau, taui, jx, jxx, jy, jyy, jxy);
        g64_sum<kR2R, 43, true>(pi, y, yi, gx, gxx, gy, gyy, gxy);
      }
      const double gp = pi1 + gx;
      iv = gp * t * k;
      hv = 249224.04 * (jy + gy);
      if (y1 != 0.0) {
        ivp = (gxx - pi1 * pi1) * 1e-6 * t * k; ivt = k * (gp + gxy * taut * t);
        hvp = 249224.04 * gxy * 1e-6; hvt = 249224.04 * (jyy + gyy) * taut;
      }
    }
  }
  const double yl = 1.0 - y1 - y2;
  RhoH o;
  o.rho = 1.0 / (yl * il + y1 * iv + y2 * ig);
  o.h = yl * hl + y1 * hv + y2 * hg;
  const double r2 = -o.rho * o.rho;
  o.drho[0] = r2 * (yl * ilp + y1 * ivp + y2 * igp);
  o.drho[1] = r2 * (yl * ilt + y1 * ivt + y2 * igt);
  o.drho[2] = r2 * (iv - il);
  o.drho[3] = r2 * (ig - il);
  o.dh[0] = yl * hlp + y1 * hvp;
  o.dh[1] = yl * hlt + y1 * hvt + y2 * hgt;
  o.dh[2] = hv - hl;
  o.dh[3] = hg - hl;
  return o;
}

// the cotangent of a face: face g (between cells g and gr = g + sn) enters the residual of
// g as -F + V and of gr as +F - V
__device__ __forceinline__ bool face_cotangent(const AdjPtr& a, int npv, long long n, long long g, long long gr,
                                               double* lam) {
  bool any = false;
#pragma unroll
  for (int v = 0; v < NPVM; ++v) {
    lam[v] = (v < npv) ? a.lam[v * n + gr] - a.lam[v * n + g] : 0.0;
    any = any || (lam[v] != 0.0);
  }
  return any;
}

// One thread per face.  The gradient with respect to the reconstructed states takes their
// place (d.fi, FS_R) for k_adj_recon; a state reset to its cell's value or clamped sends its
// gradient to that cell or nowhere.  SENSOR: Roe-M and AUSMPW+ (adjoint_duals.cu), else Roe and
// AUSM+-up (adjoint_face.cu).
template <bool SENSOR>
__global__ void __launch_bounds__(64) k_adj_flux(DevPtr d, Par c, AdjPtr a, int dir0) {
  const int slot = blockIdx.z, dir = dir0 + slot, npv = c.npv;
  DirCell f;
  const bool live = dir_cell<0>(d, dir, blockIdx.x * (long long)blockDim.x + threadIdx.x, f);
  double wu = 0.0;
  if (live) {
    const long long n = d.ncell, g = f.g, gr = f.g + f.sn;
    double lam[NPVM];
    const bool any = face_cotangent(a, npv, n, g, gr, lam);
    double* fi = fi_planes(d, dir, npv) + g;
    FaceGrad o{};
    if (any) {
      double nx[3], c9[NPVM], c10[NPVM];
      int fl[NPVM], fr[NPVM];
      face_vec(d, dir == 0 ? GM_CX : (dir == 1 ? GM_EX : GM_TX), g, nx);
      FaceState L, R;
#pragma unroll
      for (int v = 0; v < NPVM; ++v) {
        L.pv[v] = R.pv[v] = c9[v] = c10[v] = 0.0;
        fl[v] = fr[v] = 0;
        if (v >= npv) continue;
        c9[v] = d.pv[v * n + g];
        c10[v] = d.pv[v * n + gr];
        L.pv[v] = (c.nmuscl > 0) ? fi[v * n] : c9[v];
        R.pv[v] = (c.nmuscl > 0) ? fs_plane(d, slot, npv, v, FS_R)[g] : c10[v];
      }
      const int e4[4] = {0, 4, 5, 6};
      EosJac cl{}, cr{};
      RhoH jl{}, jr{};
      if (c.nmuscl > 0) {
        clip_flags(c, c9, c10, L.pv, R.pv, fl, fr);
        if constexpr (SENSOR) {
          cl = eos_jac(c.fluid, L.pv[0] + c.pref, L.pv[4], L.pv[5], L.pv[6]);
          cr = eos_jac(c.fluid, R.pv[0] + c.pref, R.pv[4], R.pv[5], R.pv[6]);
          L.rho = cl.rho; L.h = cl.h; L.c2 = cl.c2; R.rho = cr.rho; R.h = cr.h; R.c2 = cr.c2;
          for (int m = 0; m < 4; ++m) { jl.drho[m] = cl.drho[m]; jl.dh[m] = cl.dh[m]; jr.drho[m] = cr.drho[m]; jr.dh[m] = cr.dh[m]; }
        } else {
          jl = rho_h_jac(c.fluid, L.pv[0] + c.pref, L.pv[4], L.pv[5], L.pv[6]);
          jr = rho_h_jac(c.fluid, R.pv[0] + c.pref, R.pv[4], R.pv[5], R.pv[6]);
          L.rho = jl.rho; L.h = jl.h; R.rho = jr.rho; R.h = jr.h;
          L.c2 = R.c2 = 0.0;
        }
      } else {
        L.rho = d.dv[g]; L.h = d.dv[n + g]; L.c2 = d.dv[5 * n + g];
        R.rho = d.dv[gr]; R.h = d.dv[n + gr]; R.c2 = d.dv[5 * n + gr];
      }
      // the Roe-average state and the derivatives of its sound speed
      double ravg[NPVM];
#pragma unroll
      for (int v = 0; v < NPVM; ++v) ravg[v] = 0.0;
      roe_state<double>(npv, L, R, ravg);
      const EosJac jc = eos_jac(c.fluid, ravg[0] + c.pref, ravg[4], ravg[5], ravg[6]);
      if constexpr (SENSOR) {
        double sdv[18], ws[18];
        for (int l = 0; l < 18; ++l) sdv[l] = d.pv[stencil_cell(l, g, f.sn, f.s1, f.s2)];
        FluxBack<SENSOR>::run(c, nx, L, R, jc, ravg, sdv, lam, o, ws);
        for (int l = 0; l < 18; ++l) aadd(&a.gpv[stencil_cell(l, g, f.sn, f.s1, f.s2)], ws[l]);
      } else {
        FluxBack<SENSOR>::run(c, nx, L, R, jc, ravg, nullptr, lam, o, nullptr);
      }
      wu = o.uref;
      if (c.nmuscl > 0) {
        // face densities, enthalpies (and sound speeds) through the face EOS
        for (int m = 0; m < 4; ++m) {
          o.pl[e4[m]] += o.rl * jl.drho[m] + o.hl * jl.dh[m] + (SENSOR ? o.c2l * cl.dc2[m] : 0.0);
          o.pr[e4[m]] += o.rr * jr.drho[m] + o.hr * jr.dh[m] + (SENSOR ? o.c2r * cr.dc2[m] : 0.0);
        }
#pragma unroll
        for (int v = 0; v < NPVM; ++v) {
          if (v >= npv) continue;
          if (fl[v] == 1) aadd(&a.gpv[v * n + g], o.pl[v]);
          if (fr[v] == 1) aadd(&a.gpv[v * n + gr], o.pr[v]);
          if (fl[v]) o.pl[v] = 0.0;
          if (fr[v]) o.pr[v] = 0.0;
        }
      } else {
        aadd(&a.gdt[GD_RHO * n + g], o.rl); aadd(&a.gdt[GD_H * n + g], o.hl); aadd(&a.gdt[GD_C2 * n + g], o.c2l);
        aadd(&a.gdt[GD_RHO * n + gr], o.rr); aadd(&a.gdt[GD_H * n + gr], o.hr); aadd(&a.gdt[GD_C2 * n + gr], o.c2r);
#pragma unroll
        for (int v = 0; v < NPVM; ++v)
          if (v < npv) { aadd(&a.gpv[v * n + g], o.pl[v]); aadd(&a.gpv[v * n + gr], o.pr[v]); }
      }
    }
    if (c.nmuscl > 0) {
#pragma unroll
      for (int v = 0; v < NPVM; ++v)
        if (v < npv) { fi[v * n] = o.pl[v]; fs_plane(d, slot, npv, v, FS_R)[g] = o.pr[v]; }
    }
  }
  // one atomic per warp for the free-stream-speed gradient
  for (int q = 16; q > 0; q >>= 1) wu += __shfl_down_sync(0xffffffffu, wu, q);
  if ((threadIdx.x & 31) == 0) aadd(&a.gpar[0], wu);
}

}  // namespace cfd
