// flux.cu -- face fluxes of the FP64 form.
//
// Per direction: MUSCL/MLP reconstruction of the 38-cell stencil (src/muscl_module.f90:104-290),
// the face-state EOS, the inviscid flux (src/flux_module.f90:198-641) and the viscous flux
// (src/vsflux_module.f90:182-425), written to fi / fv at the index of the face's left cell
// (rhs_module.f90:282-538).
//
// What bounds it: a GB300 SM issues one FP64 warp instruction -- comparisons included -- per
// 16 clocks, a single warp one per 64, so the face stage costs its FP64 instructions and
// little else (memory traffic, integer work and L1 hits have slack).  So the stage is cut
// where work repeats:
//   k_plane64   per cell, direction and variable what up to four faces share: the minimum and
//               maximum over the 3 x 3 transverse cells (on the integer pipe: order-preserving
//               keys), MLP's transverse ratios, the reciprocal of the normal difference
//   k_recon64   per face and variable: the face states
//   k_flux64    per face: clips, EOS of the two states and of the Roe average on three
//               warps of a CTA side by side, the inviscid flux
//   k_visc64    per face: the viscous flux
// Fused (one thread per face did all of it, 38 loads and 98 FP64 minima and maxima per
// variable) the stage took 13.9 ms on 128x64x64 cells (cavitating, MLP, AUSM+-up) and
// 0.70 ms on 64x32x32 (Euler, TVD, Roe).
#include <algorithm>
#include "faces64.cuh"

namespace cfd {

// ------------------------------------------------------------------ reconstruction
// |num / den| of MLP's transverse ratios; a zero numerator needs no division (and would take
// the quotient's slow path)
__device__ __forceinline__ double abs_ratio(double num, double den) {
  return (is_zero(num) && !is_zero(den)) ? 0.0 : fabs(num / den);
}

__global__ void __launch_bounds__(256) k_plane64(DevPtr d, Par c, int dir0) {
  const int v = blockIdx.y, slot = blockIdx.z, dir = dir0 + slot;
  DirCell f;
  if (!dir_cell<3>(d, dir, blockIdx.x * (long long)blockDim.x + threadIdx.x, f)) return;
  const double* P = d.pv + v * d.ncell + f.g;
  double x[9];   // the 3 x 3 transverse cells, s1 fastest (the stencil's order)
#pragma unroll
  for (int m = 0; m < 9; ++m) x[m] = P[(m % 3 - 1) * f.s1 + (m / 3 - 1) * f.s2];
  long long mn = okey(x[0]), mx = mn;
#pragma unroll
  for (int m = 1; m < 9; ++m) {
    const long long k = okey(x[m]);
    mn = min(mn, k);
    mx = max(mx, k);
  }
  const double eps = 1.0e-30;
  const double xm = P[-f.sn], xp = P[f.sn];
  const double cd = xp - xm + eps;
  const double rxy = abs_ratio(x[5] - x[3], cd), rxz = abs_ratio(x[7] - x[1], cd);
  const bool flat = rxy < 1.0e-3 && rxz < 1.0e-3;
  const double den = 1.0 + rxy + rxz, dq = xp - x[4];
  fs_plane(d, slot, c.npv, v, FS_MN)[f.g] = __longlong_as_double(mn);
  fs_plane(d, slot, c.npv, v, FS_MX)[f.g] = __longlong_as_double(mx);
  fs_plane(d, slot, c.npv, v, FS_DEN)[f.g] = flat ? -den : den;
  fs_plane(d, slot, c.npv, v, FS_IDQ)[f.g] = is_zero(dq) ? 1.0 / 1.0e-30 : 1.0 / (dq + eps);
}

// x / 30 correctly rounded: with y = RN(1 / 30), whose relative error is below 2^-54, the
// quotient x y is faithful and one residual step rounds it correctly (Markstein 1990)
__device__ __forceinline__ double div30(double x) {
  const double y = 1.0 / 30.0, q = x * y;
  return fma(fma(-30.0, q, x), y, q);
}

// muscl_var's limiter on numbers, its minima and maxima on the integer pipe.  The schemes that
// bound their slope by MLP's factor take max(0, min(alp, alp r, cc)) with alp in [1, 2]: where
// r <= 0 that is 0 and where cc <= min(1, r) it is max(0, cc), whatever alp is -- `need` is
// false there and alp is not formed.
struct Lim { double r, cc; bool need; };
__device__ __forceinline__ Lim lim_begin(int nlim, double r, double r1, double r2) {
  Lim o{r, 0.0, false};
  switch (nlim) {
    case 3: o.cc = (r + fabs(r)) / (1.0 + fabs(r)); break;
    case 4: o.cc = (1.0 + r) / 2.0; break;
    case 7: o.cc = nadd(1.0, nmul(2.0, r)) / 3.0; break;
    case 8: o.cc = div30(nsub(nadd(nadd(nmul(-2.0, r1), 11.0), nmul(24.0, r)), nmul(3.0, r2))); break;
    case 9: o.cc = nadd(1.0, nmul(2.0, r)) / 3.0; return o;
    case 10: o.cc = div30(nsub(nadd(nadd(nmul(-2.0, r1), 11.0), nmul(24.0, r)), nmul(3.0, r2))); return o;
    case 5: o.cc = nadd(nmul(r, r), r) / nadd(1.0, nmul(r, r)); return o;
    case 2: case 6: o.need = true; return o;
    default: return o;
  }
  o.need = r > 0.0 && !(o.cc <= kmin(1.0, r));
  return o;
}
__device__ __forceinline__ double lim_end(int nlim, const Lim& o, double alp) {
  const double r = o.r;
  double cc = o.cc;
  switch (nlim) {
    case 0: return 1.0;
    case 1: return kmax(0.0, kmin(1.0, r));
    case 2: return kmax(kmax(0.0, kmin(1.0, alp * r)), kmin(alp, r));
    case 3: case 4: case 7: case 8:
      if (!o.need) return r > 0.0 ? kmax(0.0, cc) : 0.0;
      return kmax(0.0, kmin(kmin(alp, alp * r), cc));
    case 5: return kmax(kmax(0.0, kmin(cc * r, 1.0)), kmin(r, cc));
    case 6: cc = kmin(1.5, alp); return kmax(kmax(0.0, kmin(cc * r, 1.0)), kmin(r, cc));
    default: return cc;
  }
}

// Face states of one variable: muscl_var<double>, step for step in the same roundings (a
// reconstructed state often lands exactly on a clip bound), from the shared per-cell values.
// Valid for stencils of numbers below 1e60 and nonzero denominators, where no intermediate
// overflows or is a NaN; the rest takes muscl_var itself.
__global__ void __launch_bounds__(256) k_recon64(DevPtr d, Par c, int dir0) {
  const int v = blockIdx.y, slot = blockIdx.z, dir = dir0 + slot, npv = c.npv;
  DirCell f;
  if (!dir_cell<0>(d, dir, blockIdx.x * (long long)blockDim.x + threadIdx.x, f)) return;
  const long long n = d.ncell, g = f.g, sn = f.sn;
  const double* P = d.pv + v * n + g;
  double* outL = fi_planes(d, dir, npv) + v * n + g;
  double* outR = fs_plane(d, slot, npv, v, FS_R) + g;
  const double cm2 = P[-2 * sn], cm1 = P[-sn], c0 = P[0], c1 = P[sn], c2 = P[2 * sn], c3 = P[3 * sn];
  const double eps = 1.0e-30;
  const double dq = c1 - c0, dqm = c0 - cm1, dqm1 = cm1 - cm2, dqp = c2 - c1, dqp1 = c3 - c2;
  if (is_zero(dq) && is_zero(dqm) && is_zero(dqm1) && is_zero(dqp) && is_zero(dqp1)) {
    // a constant line (a phase that is absent, a uniform stream): every limiter is finite and
    // multiplies a zero difference
    *outL = c0;
    *outR = c1;
    return;
  }
  const bool mlp = c.nmuscl == 2;
  const long long big = 0x4c63e9e4e4c2f344LL;   // key of 1e60
  double idm, idp, den_l = 1.0, den_r = 1.0;
  long long mnl = 0, mnc0 = 0, mnc1 = 0, mnr = 0, mxl = 0, mxc0 = 0, mxc1 = 0, mxr = 0;
  bool ok;
  if (mlp) {
    const double *MN = fs_plane(d, slot, npv, v, FS_MN) + g, *MX = fs_plane(d, slot, npv, v, FS_MX) + g;
    const double *DN = fs_plane(d, slot, npv, v, FS_DEN) + g, *ID = fs_plane(d, slot, npv, v, FS_IDQ) + g;
    mnl = __double_as_longlong(MN[-sn]); mnc0 = __double_as_longlong(MN[0]);
    mnc1 = __double_as_longlong(MN[sn]); mnr = __double_as_longlong(MN[2 * sn]);
    mxl = __double_as_longlong(MX[-sn]); mxc0 = __double_as_longlong(MX[0]);
    mxc1 = __double_as_longlong(MX[sn]); mxr = __double_as_longlong(MX[2 * sn]);
    den_l = DN[0]; den_r = DN[sn];
    idm = ID[-sn]; idp = ID[sn];
    ok = max(max(mxl, mxc0), max(mxc1, mxr)) < big && min(min(mnl, mnc0), min(mnc1, mnr)) > ~big &&
         finite_bits(den_l) && finite_bits(den_r);
  } else {
    idm = 1.0 / (dqm + eps);
    idp = 1.0 / (dqp + eps);
    const long long a = max(max(okey(cm1), okey(c0)), max(okey(c1), okey(c2)));
    const long long b = min(min(okey(cm1), okey(c0)), min(okey(c1), okey(c2)));
    ok = a < big && b > ~big;
  }
  ok = ok && okey(fabs(cm2)) < big && okey(fabs(c3)) < big && finite_bits(idm) && finite_bits(idp);
  if (!ok) {
    double x[38], xl, xr;
#pragma unroll 1
    for (int l = 0; l < 38; ++l) x[l] = d.pv[v * n + stencil_cell(l, g, sn, f.s1, f.s2)];
    muscl_var<double>(c, x, xl, xr);
    *outL = xl;
    *outR = xr;
    return;
  }
  const double r0 = dq * idm, r10 = dqm1 * idm, r20 = dqp * idm;
  const double r1 = dq * idp, r11 = dqp1 * idp, r21 = dqm * idp;
  const Lim ll = lim_begin(c.nlim, r0, r10, r20), lr = lim_begin(c.nlim, r1, r11, r21);
  double alp0 = 2.0, alp1 = 2.0;
  if (mlp && (ll.need || lr.need)) {
    const long long mnA = min(mnc0, mnc1), mxA = max(mxc0, mxc1);
    if (ll.need) {
      long long qn, qx;
      if (den_l < 0.0) { qn = min(mnA, mnl); qx = max(mxA, mxl); }
      else if (c1 - cm1 > 0.0) { qx = mxA; qn = min(mnc0, mnl); }
      else { qn = mnA; qx = max(mxc0, mxl); }
      const double qml = kmin(fabs(okey_value(qx) - c0), fabs(okey_value(qn) - c0));
      alp0 = 2.0 * kmax(1.0, r0) / (fabs(dq) + eps) / fabs(den_l) * qml;
      alp0 = kmax(1.0, kmin(2.0, alp0));
    }
    if (lr.need) {
      long long qn, qx;
      if (den_r < 0.0) { qn = min(mnA, mnr); qx = max(mxA, mxr); }
      else if (c2 - c0 > 0.0) { qx = max(mxc1, mxr); qn = mnA; }
      else { qn = min(mnc1, mnr); qx = mxA; }
      const double qmr = kmin(fabs(okey_value(qx) - c1), fabs(okey_value(qn) - c1));
      const double q = (fabs(dq) <= eps) ? dqp / eps : 1.0 / r1;
      alp1 = 2.0 * kmax(1.0, q) * fabs(idp) / fabs(den_r) * qmr;
      alp1 = kmax(1.0, kmin(2.0, alp1));
    }
  }
  *outL = nadd(c0, nmul(nmul(0.5, lim_end(c.nlim, ll, alp0)), dqm));
  *outR = nsub(c1, nmul(nmul(0.5, lim_end(c.nlim, lr, alp1)), dqp));
}

// ------------------------------------------------------------------ inviscid flux
// Three roles per face, one per group of F64_FACES threads (so that they run on different
// schedulers): the EOS of the left state, of the right state, and of the Roe average, whose
// p and T are means of the face states' and whose Gibbs sums need nothing else; the last
// role then has the averages' mass fractions from the two densities and forms the flux.  On
// a small case the face costs the longest role's chain, not the sum of the three.
constexpr int F64_FACES = 64;

// the face state's entries the EOS reads (p, T, y1, y2), clipped as muscl_clip clips them
__device__ __forceinline__ void clip_eos_entries(const Par& c, double c5, double c6, double* x) {
  x[0] = fmax(-c.pref + 10.0, x[0]);
  if (x[5] < 0.0 || x[5] > 1.0) x[5] = c5;
  if (x[6] < 0.0 || x[6] > 1.0) x[6] = c6;
  if (x[5] + x[6] > 1.0) { x[5] = c5; x[6] = c6; }
}

__global__ void __launch_bounds__(3 * F64_FACES) k_flux64(DevPtr d, Par c, int dir0) {
  __shared__ double s_eos[2][3][F64_FACES];   // rho, h, c2 of the left and right states
  const int slot = blockIdx.z, dir = dir0 + slot, npv = c.npv;
  const int q = threadIdx.x % F64_FACES, role = threadIdx.x / F64_FACES;
  DirCell f;
  const bool live = dir_cell<0>(d, dir, blockIdx.x * (long long)F64_FACES + q, f);
  const long long n = d.ncell, g = f.g, gr = f.g + f.sn;
  const bool snd = c.nscheme == 2 || c.nscheme == 3;   // Roe-M and AUSMPW+ read the face sound speeds
  double* fi = fi_planes(d, dir, npv);
  if (live && role < 2 && c.nmuscl > 0) {
    const long long cell = role ? gr : g;
    double x[NPVM];
    const int e4[4] = {0, 4, 5, 6};
#pragma unroll
    for (int m = 0; m < 4; ++m) x[e4[m]] = role ? fs_plane(d, slot, npv, e4[m], FS_R)[g] : fi[e4[m] * n + g];
    clip_eos_entries(c, d.pv[5 * n + cell], d.pv[6 * n + cell], x);
    double rho, h, c2 = 0.0;
    if (snd) {
      double dv[NDV];
      deteos_simple(c.fluid, x[0] + c.pref, x[4], x[5], x[6], dv, &d.sc->snd2_fallbacks, x[5] != 0.0);
      rho = dv[0]; h = dv[1]; c2 = dv[5];
    } else {
      eos_rho_h(c.fluid, x[0] + c.pref, x[4], x[5], x[6], rho, h);
    }
    s_eos[role][0][q] = rho; s_eos[role][1][q] = h; s_eos[role][2][q] = c2;
  }
  FaceState L, R;
  Phase<double> pl, pvp, pg;
  double ir[3];
  if (live && role == 2) {
    if (c.nmuscl > 0) {
      double c9[NPVM], c10[NPVM];
#pragma unroll
      for (int v = 0; v < NPVM; ++v) {
        L.pv[v] = R.pv[v] = c9[v] = c10[v] = 0.0;
        if (v >= npv) continue;
        L.pv[v] = fi[v * n + g];
        R.pv[v] = fs_plane(d, slot, npv, v, FS_R)[g];
        if (v >= 5) { c9[v] = d.pv[v * n + g]; c10[v] = d.pv[v * n + gr]; }
      }
      muscl_clip<double>(c, c9, c10, L.pv, R.pv);
    } else {
#pragma unroll
      for (int v = 0; v < NPVM; ++v) {
        L.pv[v] = (v < npv) ? d.pv[v * n + g] : 0.0;
        R.pv[v] = (v < npv) ? d.pv[v * n + gr] : 0.0;
      }
    }
    // (the averaged y1 is zero where both are: its weights are positive)
    phases<true>(c.fluid, 0.5 * (L.pv[0] + R.pv[0]) + c.pref, 0.5 * (L.pv[4] + R.pv[4]), pl, pvp, pg, ir,
                 L.pv[5] != 0.0 || R.pv[5] != 0.0);
  }
  __syncthreads();
  if (!live || role != 2) return;
  if (c.nmuscl > 0) {
    L.rho = s_eos[0][0][q]; L.h = s_eos[0][1][q]; L.c2 = s_eos[0][2][q];
    R.rho = s_eos[1][0][q]; R.h = s_eos[1][1][q]; R.c2 = s_eos[1][2][q];
  } else {
    L.rho = d.dv[g]; L.h = d.dv[n + g]; L.c2 = d.dv[5 * n + g];
    R.rho = d.dv[gr]; R.h = d.dv[n + gr]; R.c2 = d.dv[5 * n + gr];
  }
  if (c.rot) {
    // rothalpy_l / rothalpy_r (src/flux_module.f90:697-721): the face states' total enthalpy
    // less 0.5 |omega x r|^2 at the left and right cells' centroids; h enters the fluxes
    // only through it
    double rl[3], rr[3];
    for (int e = 0; e < 3; ++e) { rl[e] = d.gm[(GM_GRD + 1 + e) * n + g]; rr[e] = d.gm[(GM_GRD + 1 + e) * n + gr]; }
    L.h = L.h - rot_q(c, rl);
    R.h = R.h - rot_q(c, rr);
  }
  double sdst[18];
  if (snd) {
#pragma unroll
    for (int l = 0; l < 18; ++l) sdst[l] = d.pv[stencil_cell(l, g, f.sn, f.s1, f.s2)];
  }
  double nx[3], fx[NPVM];
  face_vec(d, dir == 0 ? GM_CX : (dir == 1 ? GM_EX : GM_TX), g, nx);
  // the Roe-average state; only its sound speed is used (src/flux_module.f90:237,319,461,588)
  double ravg[NPVM], rdv[NDV];
#pragma unroll
  for (int v = 0; v < NPVM; ++v) ravg[v] = 0.0;
  roe_state<double>(npv, L, R, ravg);
  mixture<double>(pl, pvp, pg, ravg[5], ravg[6], rdv, &d.sc->snd2_fallbacks, ir);
  inviscid_flux_core<double>(c, nx, L, R, sdst, ravg, rdv[5], c.uref * c.uref, fx);
#pragma unroll
  for (int v = 0; v < NPVM; ++v)
    if (v < npv) fi[v * n + g] = fx[v];
}

// ------------------------------------------------------------------ viscous flux
// vsflux_laminar / vsflux_turbulent
__global__ void __launch_bounds__(256) k_visc64(DevPtr d, Par c, int dir0) {
  const int dir = dir0 + blockIdx.z, npv = c.npv;
  DirCell f;
  if (!dir_cell<0>(d, dir, blockIdx.x * (long long)blockDim.x + threadIdx.x, f)) return;
  const long long n = d.ncell, g = f.g, sn = f.sn, s1 = f.s1, s2 = f.s2, gr = f.g + f.sn;
  double nx[3];
  face_vec(d, dir == 0 ? GM_CX : (dir == 1 ? GM_EX : GM_TX), g, nx);
  const bool turb = (c.iturb >= -1);
  const int ep = (dir == 0) ? GM_EX : (dir == 1 ? GM_TX : GM_CX);   // faces normal to t1
  const int tp = (dir == 0) ? GM_TX : (dir == 1 ? GM_CX : GM_EX);   // faces normal to t2
  double ev[3], tvv[3];
  for (int q = 0; q < 3; ++q) {
    const double* P = d.gm + (ep + q) * n;
    ev[q] = 0.25 * (P[g - s1] + P[g - s1 + sn] + P[g] + P[g + sn]);
    const double* T = d.gm + (tp + q) * n;
    tvv[q] = 0.25 * (T[g - s2] + T[g - s2 + sn] + T[g] + T[g + sn]);
  }
  double vol = 2.0 / (d.gm[GM_GRD * n + g] + d.gm[GM_GRD * n + gr]);
  double tvl[3] = {0, 0, 0}, tvr[3] = {0, 0, 0};
  for (int q = 0; q < c.ntv; ++q) { tvl[q] = d.tv[q * n + g]; tvr[q] = d.tv[q * n + gr]; }
  double vis = 0.5 * (tvl[0] + tvr[0]);
  double con = 0.5 * (tvl[1] + tvr[1]);
  double emut = 0.0, tcon = 0.0;
  if (turb) {
    emut = 0.5 * (tvl[2] + tvr[2]);
    tcon = 0.5 * (tvl[2] * d.dv[11 * n + g] + tvr[2] * d.dv[11 * n + gr]) / 0.9;
  }
  const int vars[6] = {1, 2, 3, 4, 7, 8};
  double gx[6], gy[6], gz[6], cc[6];
  const int nv = turb ? 6 : 4;
  for (int q = 0; q < nv; ++q) {
    const double* P = d.pv + vars[q] * n;
    double x[18];
#pragma unroll
    for (int l = 0; l < 18; ++l) x[l] = P[stencil_cell(l, g, sn, s1, s2)];
    face_gradient<double>(x, nx, ev, tvv, vol, gx[q], gy[q], gz[q], cc[q]);
  }
  double rho = 0.0, ydns = 0.0;
  if (turb) {
    rho = 0.5 * (d.dv[g] + d.dv[gr]);
    ydns = 0.5 * (d.gm[(GM_GRD + 4) * n + g] + d.gm[(GM_GRD + 4) * n + gr]);
  }
  double fv[NPVM];
  vsflux_core<double>(c, nx, gx, gy, gz, cc, vis, con, emut, tcon, rho, ydns, fv);
  double* fvp = d.fv + (long long)dir * npv * n;
#pragma unroll
  for (int v = 0; v < NPVM; ++v)
    if (v < npv) fvp[v * n + g] = fv[v];
}

// the threads that cover the faces, or the planes, of the directions of one launch
static long long most(const long long* n, int dir, int slots) {
  long long m = 0;
  for (int q = dir; q < dir + slots; ++q) m = std::max(m, n[q]);
  return m;
}
static unsigned nb_of(long long n, int t) { return (unsigned)((n + t - 1) / t); }

void launch_recon64(const Engine& E, const DevPtr& d, int dir, cudaStream_t s) {
  const int T = E.tpb_face;
  const Par& c = E.par;
  const unsigned z = (unsigned)d.fslots, y = (unsigned)c.npv;
  if (c.nmuscl == 2) k_plane64<<<dim3(nb_of(most(E.nplane, dir, d.fslots), T), y, z), T, 0, s>>>(d, c, dir);
  if (c.nmuscl > 0) k_recon64<<<dim3(nb_of(most(E.nface, dir, d.fslots), T), y, z), T, 0, s>>>(d, c, dir);
}

// Three directions per launch where the scratch planes hold them (small cases, whose launches
// would not fill the GPU one direction at a time), else one direction after the other.
void launch_face_flux(const Engine& E, cudaStream_t s) {
  const int T = E.tpb_face;
  const Par& c = E.par;
  const unsigned z = (unsigned)E.d.fslots;
  for (int dir = 0; dir < 3; dir += E.d.fslots) {
    const long long nf = most(E.nface, dir, E.d.fslots);
    launch_recon64(E, E.d, dir, s);
    k_flux64<<<dim3(nb_of(nf, F64_FACES), 1, z), 3 * F64_FACES, 0, s>>>(E.d, c, dir);
    if (c.iturb != -3) k_visc64<<<dim3(nb_of(nf, T), 1, z), T, 0, s>>>(E.d, c, dir);
  }
}

// the launches of one call
int face_flux_launches(const Engine& E) {
  const Par& c = E.par;
  return (3 / E.d.fslots) * (1 + (c.nmuscl > 0) + (c.nmuscl == 2) + (c.iturb != -3));
}

}  // namespace cfd
