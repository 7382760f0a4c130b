// adjoint_face.cu -- the face part of the discrete adjoint: per face, the vector-Jacobian
// product of its inviscid flux (src/flux_module.f90:198-641 with the reconstruction of
// src/muscl_module.f90:104-290) and its viscous flux (src/vsflux_module.f90:182-425) with
// respect to the face's stencil, the face cells' dv / tv and the free-stream speed.  The
// file comment of adjoint.cu describes the whole reverse pass.
//
// What bounds it: FP64 instructions, as in the forward stage (flux.cu).  With forward-mode
// duals over the whole face -- 38 stencil cells a variable and 25 to 43 flux inputs, eight
// directions a pass, the duals in local memory -- a face took some 280000 FP64 issue slots
// (440 of 457 ms on 64^3 SST cells).  A product with one cotangent needs one reverse sweep:
//   k_adj_flux    per face: the face states of the forward kernels, their EOS derivatives in
//                 closed form, the flux reversed; Roe and AUSM+-up keep duals only for the
//                 scalar core that couples the two sides (8 and 9 inputs), Roe-M and AUSMPW+
//                 for the whole flux
//   k_adj_recon   per face and variable: the reconstruction reversed by hand; the cells it
//                 reaches are the line, MLP's transverse pairs and the extreme cell
//   k_adj_visc    per face: the viscous flux reversed by hand
// and k_adj_eos, the interior cells' EOS.
#include "adjoint_flux.cuh"

namespace cfd {

// ------------------------------------------------------------------ inviscid flux
// through the Roe-average velocities, p, T, y1, y2 (gradient ga by pv index) to the states
__device__ __forceinline__ void roe_state_back(const FaceState& L, const FaceState& R, double srl, double srr,
                                               double rd, const double* ravg, const double* ga, double grrho,
                                               FaceGrad& o) {
  o.pl[0] += 0.5 * ga[0]; o.pr[0] += 0.5 * ga[0];
  o.pl[4] += 0.5 * ga[4]; o.pr[4] += 0.5 * ga[4];
  double gl = grrho * srr, gr = grrho * srl;
#pragma unroll
  for (int k = 1; k < NPVM; ++k) {
    if (k == 4) continue;
    const double g = ga[k] * rd;
    o.pl[k] += g * srl;
    o.pr[k] += g * srr;
    gl += g * (L.pv[k] - ravg[k]);
    gr += g * (R.pv[k] - ravg[k]);
  }
  o.rl += gl * 0.5 / srl;
  o.rr += gr * 0.5 / srr;
}

// inviscid_flux_core reversed for Roe (nscheme 1) and AUSM+-up (4): both are
// F = A_L q_L + A_R q_R + (terms along n and the Roe average) with q = (1, u, H, y ...), so
// the cotangent meets the states directly and only the scalars that couple the two sides
// need derivatives of their own, taken by duals over their few inputs.
__device__ __forceinline__ void flux_back(const Par& c, const double* n, const FaceState& L, const FaceState& R,
                                          const EosJac& jc, const double* ravg, const double* lam, FaceGrad& o) {
  const int npv = c.npv;
  const double dl = ::sqrt(n[0] * n[0] + n[1] * n[1] + n[2] * n[2]);
  if (dl == 0.0) return;
  const double idl = 1.0 / dl, nn[3] = {n[0] * idl, n[1] * idl, n[2] * idl};
  const double *pl = L.pv, *pr = R.pv;
  const double srl = ::sqrt(L.rho), srr = ::sqrt(R.rho), rrho = srl * srr, rd = 1.0 / (srl + srr);
  const double hl = L.h + 0.5 * (pl[1] * pl[1] + pl[2] * pl[2] + pl[3] * pl[3]);
  const double hr = R.h + 0.5 * (pr[1] * pr[1] + pr[2] * pr[2] + pr[3] * pr[3]);
  const double ul = nn[0] * pl[1] + nn[1] * pl[2] + nn[2] * pl[3];
  const double ur = nn[0] * pr[1] + nn[1] * pr[2] + nn[2] * pr[3];
  // lam . q of the two sides
  double sl = lam[0] + lam[4] * hl, sr = lam[0] + lam[4] * hr;
#pragma unroll
  for (int k = 1; k < NPVM; ++k)
    if (k != 4) { sl += lam[k] * pl[k]; sr += lam[k] * pr[k]; }
  const double ln = lam[1] * nn[0] + lam[2] * nn[1] + lam[3] * nn[2];
  double ga[NPVM], ml, mr, gul, gur, grrho, grc2;
#pragma unroll
  for (int k = 0; k < NPVM; ++k) ga[k] = 0.0;
  if (c.nscheme == 4) {
    using D = Dual<8>;
    const double un = nn[0] * ravg[1] + nn[1] * ravg[2] + nn[2] * ravg[3];
    const D dul = D::seed(ul, 0), dur = D::seed(ur, 1), dpl = D::seed(pl[0], 2), dpr = D::seed(pr[0], 3);
    const D drr = D::seed(rrho, 4), rc2 = D::seed(jc.c2, 5), am2 = D::seed(un * un, 6);
    const D uref2 = D::seed(c.uref * c.uref, 7);
    const D irc2 = 1.0 / rc2, amid = sqrt(rc2), iamid = amid * irc2;
    const D zmr = dur * iamid, zml = dul * iamid;
    const D s0 = sqrt(sndp2_u<D>(c, rc2, am2, uref2) * irc2);
    const D fmid = s0 * (2.0 - s0);
    D alpha = 3.0 / 16.0 * (-4.0 + 5.0 * fmid * fmid);
    alpha = fmax(fmin(alpha, D(3.0 / 16.0)), D(-3.0 / 4.0));
    const double beta = 0.125;
    D zmmr, pmr, zmpl, ppl;
    if (fabs(zmr) >= 1.0) { zmmr = 0.5 * (zmr - fabs(zmr)); pmr = D(0.5 * (1.0 - ::copysign(1.0, zmr.v))); }
    else {
      const D q1 = zmr * zmr - 1.0, m1 = zmr - 1.0;
      zmmr = -(0.25 * m1 * m1) - beta * (q1 * q1);
      pmr = 0.25 * m1 * m1 * (2.0 + zmr) - alpha * zmr * (q1 * q1);
    }
    if (fabs(zml) >= 1.0) { zmpl = 0.5 * (zml + fabs(zml)); ppl = D(0.5 * (1.0 + ::copysign(1.0, zml.v))); }
    else {
      const D q1 = zml * zml - 1.0, m1 = zml + 1.0;
      zmpl = 0.25 * m1 * m1 + beta * (q1 * q1);
      ppl = 0.25 * m1 * m1 * (2.0 - zml) + alpha * zml * (q1 * q1);
    }
    const D zmid = zmpl + zmmr - 0.25 * fmax(1.0 - am2 * irc2, 0.0) * (dpr - dpl) * irc2 / (drr * fmid);
    const D pmid = ppl * (dpl + c.pref) + pmr * (dpr + c.pref) - 2.0 * ppl * pmr * drr * fmid * amid * (dur - dul);
    // lam . F / dl = z amid rho q + pmid lam . n, z upwind
    const bool up = zmid > 0.0;
    const double rho = up ? L.rho : R.rho, sq_ = up ? sl : sr;
    const D m = zmid * amid;
    double g[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) g[q] = dl * (m.d[q] * rho * sq_ + pmid.d[q] * ln);
    ml = up ? m.v * L.rho * dl : 0.0;
    mr = up ? 0.0 : m.v * R.rho * dl;
    if (up) o.rl += m.v * sl * dl;
    else o.rr += m.v * sr * dl;
    gul = g[0]; gur = g[1]; o.pl[0] += g[2]; o.pr[0] += g[3]; grrho = g[4]; grc2 = g[5];
    const double gun = 2.0 * un * g[6];
#pragma unroll
    for (int e = 0; e < 3; ++e) ga[1 + e] += gun * nn[e];
    o.uref += g[7] * 2.0 * c.uref;
  } else {
    using D = Dual<9>;
    const double u2 = ravg[1] * ravg[1] + ravg[2] * ravg[2] + ravg[3] * ravg[3];
    const double uu = nn[0] * ravg[1] + nn[1] * ravg[2] + nn[2] * ravg[3];
    const double hta = (srl * hl + srr * hr) * rd;
    const D dul = D::seed(ul, 0), dur = D::seed(ur, 1), dpl = D::seed(pl[0], 2), dpr = D::seed(pr[0], 3);
    const D drr = D::seed(rrho, 4), rc2 = D::seed(jc.c2, 5), du2 = D::seed(u2, 6), uuu = D::seed(uu, 7);
    const D uref2 = D::seed(c.uref * c.uref, 8);
    const D sndp2 = sndp2_u<D>(c, rc2, du2, uref2);
    const D q = sndp2 / rc2;
    const D uup = 0.5 * (1.0 + q) * uuu;
    const D ddd = 0.5 * sqrt((1.0 - q) * (1.0 - q) * uuu * uuu + 4.0 * sndp2);
    const D c_star = 0.5 * (fabs(uup + ddd) + fabs(uup - ddd));
    const D m_star = 0.5 * (fabs(uup + ddd) - fabs(uup - ddd)) / ddd;
    const D au = fabs(uuu);
    const D du = m_star * (dur - dul) + (c_star - q * au - 0.5 * (1.0 - q) * uuu * m_star) * (dpr - dpl) / (drr * sndp2);
    const D dp = m_star * (dpr - dpl) + (c_star - au + 0.5 * (1.0 - q) * uuu * m_star) * drr * (dur - dul);
    const D dr = du * drr;
    // lam . F = dl / 2 [rho_l u_l s_l + rho_r u_r s_r + ln (p_l + p_r + 2 pref)
    //   - |u| (rho_r s_r - rho_l s_l - lam4 (p_r - p_l)) - dr lam . q_avg - dp (ln + lam4 u)]
    double sa = lam[0] + lam[4] * hta;
#pragma unroll
    for (int k = 1; k < NPVM; ++k)
      if (k != 4) sa += lam[k] * ravg[k];
    const double hd = 0.5 * dl, jump = R.rho * sr - L.rho * sl - lam[4] * (pr[0] - pl[0]), lu = ln + lam[4] * uu;
    double g[9];
#pragma unroll
    for (int m = 0; m < 9; ++m) g[m] = -hd * (au.d[m] * jump + dr.d[m] * sa + dp.d[m] * lu);
    const double wl = ul + au.v, wr = ur - au.v;   // F carries rho_l (u_l + |u|) q_l + rho_r (u_r - |u|) q_r
    ml = hd * wl * L.rho;
    mr = hd * wr * R.rho;
    o.rl += hd * wl * sl;
    o.rr += hd * wr * sr;
    gul = g[0] + hd * L.rho * sl;
    gur = g[1] + hd * R.rho * sr;
    o.pl[0] += g[2] + hd * (ln - au.v * lam[4]);
    o.pr[0] += g[3] + hd * (ln + au.v * lam[4]);
    grrho = g[4]; grc2 = g[5];
    const double guu = g[7] - hd * dp.v * lam[4];
    const double gq = -hd * dr.v;   // the Roe averages' own share
#pragma unroll
    for (int e = 0; e < 3; ++e) ga[1 + e] += 2.0 * g[6] * ravg[1 + e] + guu * nn[e] + gq * lam[1 + e];
#pragma unroll
    for (int k = 5; k < NPVM; ++k) ga[k] += gq * lam[k];
    // the averaged total enthalpy
    const double gh = gq * lam[4], ghl = gh * srl * rd, ghr = gh * srr * rd;
    o.hl += ghl;
    o.hr += ghr;
#pragma unroll
    for (int e = 1; e < 4; ++e) { o.pl[e] += ghl * pl[e]; o.pr[e] += ghr * pr[e]; }
    o.rl += gh * (hl - hta) * rd * 0.5 / srl;
    o.rr += gh * (hr - hta) * rd * 0.5 / srr;
    o.uref += g[8] * 2.0 * c.uref;
  }
  // the sides' q
  o.hl += ml * lam[4];
  o.hr += mr * lam[4];
#pragma unroll
  for (int k = 1; k < NPVM; ++k) {
    if (k == 4 || k >= npv) continue;
    double a = ml * lam[k], b = mr * lam[k];
    if (k < 4) {
      a += ml * lam[4] * pl[k] + gul * nn[k - 1];
      b += mr * lam[4] * pr[k] + gur * nn[k - 1];
    }
    o.pl[k] += a;
    o.pr[k] += b;
  }
  const int am[4] = {0, 4, 5, 6};
#pragma unroll
  for (int m = 0; m < 4; ++m) ga[am[m]] += grc2 * jc.dc2[m];
  roe_state_back(L, R, srl, srr, rd, ravg, ga, grrho, o);
}

template <>
struct FluxBack<false> {
  static __device__ __forceinline__ void run(const Par& c, const double* nx, const FaceState& L, const FaceState& R,
                                             const EosJac& jc, const double* ravg, const double*, const double* lam,
                                             FaceGrad& o, double*) {
    flux_back(c, nx, L, R, jc, ravg, lam, o);
  }
};

// ------------------------------------------------------------------ reconstruction
// the limiter (physics.cuh) with its derivatives in r, r1, r2 and alp, the branch taken on the
// values as the duals take it: fmin(a, b) keeps a on ties, and so does fmax
struct LimD { double v, r, r1, r2, a; };
__device__ __forceinline__ LimD lmin(const LimD& a, const LimD& b) { return b.v < a.v ? b : a; }
__device__ __forceinline__ LimD lmax(const LimD& a, const LimD& b) { return b.v > a.v ? b : a; }
__device__ __forceinline__ LimD lim_slopes(int nlim, double r, double r1, double r2, double alp) {
  const LimD zero{0.0, 0.0, 0.0, 0.0, 0.0}, one{1.0, 0.0, 0.0, 0.0, 0.0};
  const LimD dr{r, 1.0, 0.0, 0.0, 0.0}, da{alp, 0.0, 0.0, 0.0, 1.0}, dar{alp * r, alp, 0.0, 0.0, r};
  LimD q = zero;
  switch (nlim) {
    case 0: return one;
    case 1: return lmax(zero, lmin(one, dr));
    case 2: return lmax(lmax(zero, lmin(one, dar)), lmin(da, dr));
    case 3: {
      const double s = (r < 0.0) ? -1.0 : 1.0, den = 1.0 + ::fabs(r);
      q.v = (r + ::fabs(r)) / den;
      q.r = (1.0 + s - q.v * s) / den;
      return lmax(zero, lmin(lmin(da, dar), q));
    }
    case 4: q.v = (1.0 + r) / 2.0; q.r = 0.5; return lmax(zero, lmin(lmin(da, dar), q));
    case 5: {
      const double den = nadd(1.0, nmul(r, r));
      q.v = nadd(nmul(r, r), r) / den;
      q.r = (2.0 * r + 1.0 - q.v * 2.0 * r) / den;
      const LimD cr{q.v * r, q.r * r + q.v, 0.0, 0.0, 0.0};
      return lmax(lmax(zero, lmin(cr, one)), lmin(dr, q));
    }
    case 6: {
      const LimD c15{1.5, 0.0, 0.0, 0.0, 0.0};
      q = lmin(c15, da);
      const LimD cr{q.v * r, q.v, 0.0, 0.0, q.a * r};
      return lmax(lmax(zero, lmin(cr, one)), lmin(dr, q));
    }
    case 7: case 9:
      q.v = nadd(1.0, nmul(2.0, r)) / 3.0; q.r = 2.0 / 3.0;
      return nlim == 9 ? q : lmax(zero, lmin(lmin(da, dar), q));
    default:
      q.v = nsub(nadd(nadd(nmul(-2.0, r1), 11.0), nmul(24.0, r)), nmul(3.0, r2)) / 30.0;
      q.r = 24.0 / 30.0; q.r1 = -2.0 / 30.0; q.r2 = -3.0 / 30.0;
      return nlim == 8 ? lmax(zero, lmin(lmin(da, dar), q)) : q;
  }
}

// the first cell, in the stencil's order, of a middle-plane pair (half 0), of one plane
// (half 1 left, 2 right) or of the side plane whose value has key k; -1: none
__device__ __forceinline__ long long extreme_cell(const double* P, long long key, int half, bool side, long long so,
                                                  long long sn, long long s1, long long s2) {
  for (int m = 0; m < 9; ++m) {
    const long long o = (m % 3 - 1) * s1 + (m / 3 - 1) * s2;
    if (side) {
      if (okey(P[so + o]) == key) return so + o;
      continue;
    }
    if (half != 2 && okey(P[o]) == key) return o;
    if (half != 1 && okey(P[sn + o]) == key) return sn + o;
  }
  return -(1ll << 60);
}

__global__ void __launch_bounds__(128) k_adj_recon(DevPtr d, Par c, AdjPtr a, int dir0) {
  const int v = blockIdx.y, slot = blockIdx.z, dir = dir0 + slot, npv = c.npv;
  DirCell f;
  if (!dir_cell<0>(d, dir, blockIdx.x * (long long)blockDim.x + threadIdx.x, f)) return;
  const long long n = d.ncell, g = f.g, sn = f.sn, s1 = f.s1, s2 = f.s2;
  const double gl = fi_planes(d, dir, npv)[v * n + g], gr = fs_plane(d, slot, npv, v, FS_R)[g];
  if (gl == 0.0 && gr == 0.0) return;
  const double* P = d.pv + v * n + g;
  double* G = a.gpv + v * n + g;
  const double cm2 = P[-2 * sn], cm1 = P[-sn], c0 = P[0], c1 = P[sn], c2 = P[2 * sn], c3 = P[3 * sn];
  const double eps = 1.0e-30;
  const double dq = c1 - c0, dqm = c0 - cm1, dqm1 = cm1 - cm2, dqp = c2 - c1, dqp1 = c3 - c2;
  const bool mlp = c.nmuscl == 2;
  double idm, idp;
  if (mlp) {
    const double* ID = fs_plane(d, slot, npv, v, FS_IDQ) + g;
    idm = ID[-sn]; idp = ID[sn];
  } else {
    idm = 1.0 / (dqm + eps); idp = 1.0 / (dqp + eps);
  }
  // gradients of the five differences
  double gdq = 0.0, gdqm = 0.0, gdqm1 = 0.0, gdqp = 0.0, gdqp1 = 0.0;
  double h0 = gl, h1 = gr, hm1 = 0.0, h2 = 0.0;   // and, beyond them, of c0, c1, cm1, c2
#pragma unroll 1
  for (int side = 0; side < 2; ++side) {
    const double go = side ? gr : gl;
    if (go == 0.0) continue;
    const double id = side ? idp : idm;
    // the side's own difference db (dqm or dqp), the far one and the opposite one
    const double db = side ? dqp : dqm, df = side ? dqp1 : dqm1, dx = side ? dqm : dqp;
    const double r = dq * id, r1 = df * id, r2 = dx * id;
    double alp = 2.0, A = 0.0, M = 1.0, N = 1.0, Q = 0.0, cd = 1.0, n1 = 0.0, n2 = 0.0;
    bool on = false, qx = false, inside = false, msel = false;
    int half = 0;
    long long key = 0;
    const double cc = side ? c1 : c0;
    const long long so = side ? 2 * sn : -sn, pl = side ? sn : 0;   // side plane, own plane
    if (mlp) {
      const double *MN = fs_plane(d, slot, npv, v, FS_MN) + g, *MX = fs_plane(d, slot, npv, v, FS_MX) + g;
      const double den = fs_plane(d, slot, npv, v, FS_DEN)[g + pl];
      const long long n0 = __double_as_longlong(MN[0]), n1k = __double_as_longlong(MN[sn]);
      const long long x0 = __double_as_longlong(MX[0]), x1 = __double_as_longlong(MX[sn]);
      const long long ns = __double_as_longlong(MN[so]), xs = __double_as_longlong(MX[so]);
      const long long nA = min(n0, n1k), xA = max(x0, x1);
      const long long no = side ? n1k : n0, xo = side ? x1 : x0;   // the own plane's
      const double cdir = side ? c2 - c0 : c1 - cm1;
      // the middle planes that each extreme spans, and whether the side plane joins
      int hn = 0, hx = 0;
      bool jn = false, jx = false;
      if (den < 0.0) { jn = jx = true; }
      else if ((cdir > 0.0) != (side != 0)) { hn = side ? 2 : 1; jn = true; }
      else { hx = side ? 2 : 1; jx = true; }
      const long long mn = hn ? no : nA, mx = hx ? xo : xA;
      const long long kn = (jn && ns < mn) ? ns : mn, kx = (jx && xs > mx) ? xs : mx;
      const double ax = ::fabs(okey_value(kx) - cc), an = ::fabs(okey_value(kn) - cc);
      qx = !(an < ax);
      Q = qx ? ax : an;
      key = qx ? kx : kn;
      half = qx ? hx : hn;
      msel = qx ? (jx && xs > mx) : (jn && ns < mn);
      inside = true;
      N = ::fabs(den);
      if (!side) {
        M = r > 1.0 ? r : 1.0;
        A = 2.0 * M / (::fabs(dq) + eps) / N * Q;
      } else {
        const double q = (::fabs(dq) <= eps) ? dqp / eps : 1.0 / r;
        M = q > 1.0 ? q : 1.0;
        A = 2.0 * M * ::fabs(id) / N * Q;
      }
      const double m2 = A < 2.0 ? A : 2.0;
      alp = m2 > 1.0 ? m2 : 1.0;
      on = A < 2.0 && A > 1.0;
    }
    const LimD L = lim_slopes(c.nlim, r, r1, r2, alp);
    const double sg = side ? -0.5 : 0.5;
    const double gphi = sg * go * db;
    double gdb = sg * go * L.v, gr0 = gphi * L.r, gid = 0.0;
    const double gA = on ? gphi * L.a : 0.0;
    double gdf = gphi * L.r1 * id, gdx = gphi * L.r2 * id;
    if (gA != 0.0 && inside) {
      if (!side) {
        if (r > 1.0) gr0 += gA * A / M;
        const double gD = -gA * A / (::fabs(dq) + eps);
        gdq += dq < 0.0 ? -gD : gD;
      } else {
        if (M > 1.0) {
          const double gM = gA * A / M;
          if (::fabs(dq) <= eps) gdb += gM / eps;
          else gr0 -= gM * M * M;   // M = 1 / r
        }
        gid += (id < 0.0 ? -1.0 : 1.0) * gA * A / ::fabs(id);
      }
      // N = 1 + |n1 / cd| + |n2 / cd|
      const double gN = -gA * A / N;
      n1 = P[pl + s1] - P[pl - s1];
      n2 = P[pl + s2] - P[pl - s2];
      cd = (side ? c2 - c0 : c1 - cm1) + eps;
      const double icd = 1.0 / cd, t1 = n1 * icd, t2 = n2 * icd;
      const double e1 = (t1 < 0.0 ? -gN : gN), e2 = (t2 < 0.0 ? -gN : gN);
      aadd(G + pl + s1, e1 * icd); aadd(G + pl - s1, -e1 * icd);
      aadd(G + pl + s2, e2 * icd); aadd(G + pl - s2, -e2 * icd);
      const double gcd = -(e1 * t1 + e2 * t2) * icd;
      if (side) { h2 += gcd; h0 -= gcd; } else { h1 += gcd; hm1 -= gcd; }
      // Q = |extreme - cell|
      const double K = (Q != 0.0) ? gA * A / Q
                                  : gA * 2.0 * M / N * (side ? ::fabs(id) : 1.0 / (::fabs(dq) + eps));
      const double gq = (okey_value(key) - cc < 0.0) ? -K : K;
      const long long e = extreme_cell(P, key, half, msel, so, sn, s1, s2);
      if (e > -(1ll << 59)) aadd(G + e, gq);
      if (side) h1 -= gq; else h0 -= gq;
    }
    // r = dq id, r1 = df id, r2 = dx id, id = 1 / (db + eps)
    gdq += gr0 * id;
    gid += gr0 * dq + gphi * L.r1 * df + gphi * L.r2 * dx;
    gdb -= gid * id * id;
    if (side) { gdqp += gdb; gdqp1 += gdf; gdqm += gdx; } else { gdqm += gdb; gdqm1 += gdf; gdqp += gdx; }
  }
  aadd(G, h0 - gdq + gdqm);
  aadd(G + sn, h1 + gdq - gdqp);
  aadd(G - sn, hm1 - gdqm + gdqm1);
  aadd(G - 2 * sn, -gdqm1);
  aadd(G + 2 * sn, h2 + gdqp - gdqp1);
  aadd(G + 3 * sn, gdqp1);
}

// ------------------------------------------------------------------ viscous flux
// vsflux_core reversed: lamV . V with V = sigma n, (sigma n).u + k grad T.n and the diffusion
// of k and omega
__global__ void __launch_bounds__(128) k_adj_visc(DevPtr d, Par c, AdjPtr a, int dir0) {
  const int dir = dir0 + blockIdx.z, npv = c.npv;
  DirCell f;
  if (!dir_cell<0>(d, dir, blockIdx.x * (long long)blockDim.x + threadIdx.x, f)) return;
  const long long n = d.ncell, g = f.g, sn = f.sn, s1 = f.s1, s2 = f.s2, gr = f.g + f.sn;
  double lam[NPVM];
  if (!face_cotangent(a, npv, n, g, gr, lam)) return;
#pragma unroll
  for (int v = 0; v < NPVM; ++v) lam[v] = -lam[v];
  double nx[3];
  face_vec(d, dir == 0 ? GM_CX : (dir == 1 ? GM_EX : GM_TX), g, nx);
  const bool turb = (c.iturb == 0);
  const int ep = (dir == 0) ? GM_EX : (dir == 1 ? GM_TX : GM_CX);
  const int tp = (dir == 0) ? GM_TX : (dir == 1 ? GM_CX : GM_EX);
  double ev[3], tvv[3];
  for (int q = 0; q < 3; ++q) {
    const double* E = d.gm + (ep + q) * n;
    ev[q] = 0.25 * (E[g - s1] + E[g - s1 + sn] + E[g] + E[g + sn]);
    const double* T = d.gm + (tp + q) * n;
    tvv[q] = 0.25 * (T[g - s2] + T[g - s2 + sn] + T[g] + T[g + sn]);
  }
  const double vol = 2.0 / (d.gm[GM_GRD * n + g] + d.gm[GM_GRD * n + gr]);
  double tvl[3] = {0, 0, 0}, tvr[3] = {0, 0, 0};
#pragma unroll
  for (int q = 0; q < 3; ++q)
    if (q < c.ntv) { tvl[q] = d.tv[q * n + g]; tvr[q] = d.tv[q * n + gr]; }
  const double vis = 0.5 * (tvl[0] + tvr[0]), con = 0.5 * (tvl[1] + tvr[1]);
  double emut = 0.0, tcon = 0.0, rho = 0.0, y = 0.0;
  const double cpl = d.dv[11 * n + g], cpr = d.dv[11 * n + gr];
  if (turb) {
    emut = 0.5 * (tvl[2] + tvr[2]);
    tcon = 0.5 * (tvl[2] * cpl + tvr[2] * cpr) / 0.9;
    rho = 0.5 * (d.dv[g] + d.dv[gr]);
    y = 0.5 * (d.gm[(GM_GRD + 4) * n + g] + d.gm[(GM_GRD + 4) * n + gr]);
  }
  const int vars[6] = {1, 2, 3, 4, 7, 8};
  const int nv = turb ? 6 : 4;
  double gd[6][3], cc[6];   // gradients and face averages of u, v, w, T, k, omega
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    gd[q][0] = gd[q][1] = gd[q][2] = cc[q] = 0.0;
    if (q >= nv) continue;
    double x[18];
#pragma unroll
    for (int l = 0; l < 18; ++l) x[l] = d.pv[vars[q] * n + stencil_cell(l, g, sn, s1, s2)];
    face_gradient<double>(x, nx, ev, tvv, vol, gd[q][0], gd[q][1], gd[q][2], cc[q]);
  }
  // ---- reverse: w[q] gradients of gd, wc of cc
  const double c23 = 2.0 / 3.0, mu = vis + emut, kc = con + tcon;
  double w[6][3], wc[6], gvis = 0.0, gmut = 0.0, gcon = 0.0, grho = 0.0;
#pragma unroll
  for (int q = 0; q < 6; ++q) w[q][0] = w[q][1] = w[q][2] = wc[q] = 0.0;
  double ws[3], wn = 0.0;   // lam + lam4 u, and its normal part
#pragma unroll
  for (int i = 0; i < 3; ++i) { ws[i] = lam[1 + i] + lam[4] * cc[i]; wn += ws[i] * nx[i]; }
  const double div = gd[0][0] + gd[1][1] + gd[2][2];
  double gmu = -c23 * div * wn;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    double tn = -c23 * div * nx[i];   // (tau n)_i, sigma = mu tau
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      tn += (gd[i][j] + gd[j][i]) * nx[j];
      w[i][j] = mu * (ws[i] * nx[j] + ws[j] * nx[i]);
      gmu += ws[i] * (gd[i][j] + gd[j][i]) * nx[j];
    }
    w[i][i] -= mu * c23 * wn;
    wc[i] = lam[4] * mu * tn;
  }
  double gtn = 0.0;
#pragma unroll
  for (int j = 0; j < 3; ++j) { w[3][j] = lam[4] * kc * nx[j]; gtn += gd[3][j] * nx[j]; }
  const double gkc = lam[4] * gtn;
  gcon = gkc;
  gvis = gmu;
  if (turb) {
    gmut = gmu;
    const double kf = cc[4], of = cc[5];
    const double gkn = gd[4][0] * nx[0] + gd[4][1] * nx[1] + gd[4][2] * nx[2];
    const double gon = gd[5][0] * nx[0] + gd[5][1] * nx[1] + gd[5][2] * nx[2];
    const double pkw = gd[4][0] * gd[5][0] + gd[4][1] * gd[5][1] + gd[4][2] * gd[5][2];
    const double iof = 1.0 / of, irho = 1.0 / rho, y2 = y * y;
    const double cd0 = 1.712 * rho * iof * pkw;
    const double cdkw = cd0 < 1.0e-10 ? 1.0e-10 : cd0, icd = 1.0 / cdkw, sk = ::sqrt(kf);
    const double t1 = sk * iof / (0.09 * y), t2 = 500.0 * vis * irho * iof / y2, t3 = 3.424 * rho * kf * icd / y2;
    const double m = t2 > t1 ? t2 : t1, arg = t3 < m ? t3 : m;
    const double a2 = arg * arg, bigf = ::tanh(a2 * a2);
    const double tdk = bigf * 0.85 + (1.0 - bigf), tdo = bigf * 0.5 + (1.0 - bigf) * 0.856;
    const double dk = lam[7] * (vis + emut * tdk), dw = lam[8] * (vis + emut * tdo);
    gvis += lam[7] * gkn + lam[8] * gon;
    gmut += lam[7] * tdk * gkn + lam[8] * tdo * gon;
    const double garg = emut * (lam[7] * gkn * -0.15 + lam[8] * gon * -0.356) * (1.0 - bigf * bigf) * 4.0 * arg * a2;
    double gpk = 0.0;
    if (t3 < m) {
      grho += garg * 3.424 * kf * icd / y2;
      wc[4] += garg * 3.424 * rho * icd / y2;
      if (!(cd0 < 1.0e-10)) {
        const double gcd = -garg * t3 * icd;
        grho += gcd * 1.712 * iof * pkw;
        wc[5] -= gcd * cd0 * iof;
        gpk = gcd * 1.712 * rho * iof;
      }
    } else if (t2 > t1) {
      gvis += garg * 500.0 * irho * iof / y2;
      grho -= garg * t2 * irho;
      wc[5] -= garg * t2 * iof;
    } else {
      if (sk > 0.0) wc[4] += garg * 0.5 / sk * iof / (0.09 * y);
      wc[5] -= garg * t1 * iof;
    }
#pragma unroll
    for (int j = 0; j < 3; ++j) {
      w[4][j] = dk * nx[j] + gpk * gd[5][j];
      w[5][j] = dw * nx[j] + gpk * gd[4][j];
    }
  }
  // through the (linear) face gradients and averages to the stencil: the three directions of
  // the gradient as normal, first and second transverse difference
#pragma unroll
  for (int q = 0; q < 6; ++q) {
    if (q >= nv) continue;
    const double wnn = (w[q][0] * nx[0] + w[q][1] * nx[1] + w[q][2] * nx[2]) * vol;
    const double we = (w[q][0] * ev[0] + w[q][1] * ev[1] + w[q][2] * ev[2]) * vol;
    const double wt = (w[q][0] * tvv[0] + w[q][1] * tvv[1] + w[q][2] * tvv[2]) * vol;
    double* G = a.gpv + vars[q] * n + g;
#pragma unroll
    for (int l = 0; l < 18; ++l) {
      double cn, ce, ct, cw;
      grad_coeffs(l, cn, ce, ct, cw);
      aadd(G + (stencil_cell(l, g, sn, s1, s2) - g), cn * wnn + ce * we + ct * wt + cw * wc[q]);
    }
  }
  // face averages of the two cells' transport coefficients, specific heat and density
  const long long cl[2] = {g, gr};
  const double mut[2] = {tvl[2], tvr[2]}, cp[2] = {cpl, cpr};
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const long long q = cl[s];
    aadd(&a.gdt[GD_VIS * n + q], 0.5 * gvis);
    aadd(&a.gdt[GD_CON * n + q], 0.5 * gcon);
    if (turb) {
      aadd(&a.gdt[GD_MUT * n + q], 0.5 * gmut + gkc * 0.5 * cp[s] / 0.9);
      aadd(&a.gdt[GD_CP * n + q], gkc * 0.5 * mut[s] / 0.9);
      aadd(&a.gdt[GD_RHO * n + q], 0.5 * grho);
    }
  }
}

// ------------------------------------------------------------------ cell sources
// Merkle's rates (cavsource_t, ncav = 1) reversed: lam (r_v - r_c) vol
__device__ __forceinline__ void merkle_back(const Par& c, const double* pv, double rho, double vol, double lam,
                                            double* gp, double& grho, double* wp) {
  if (pv[4] >= 647.096) return;
  const Dual<1> ps = h2o_pww<Dual<1>>(Dual<1>::seed(pv[4], 0));
  const double K = 2.0 / (c.rhoref * c.uref * c.uref) * (c.uref / c.l_chord), P = pv[0] + c.pref;
  const double yl = 1.0 - pv[5] - pv[6], s = lam * vol;
  {
    // r_c = min(c_c rho y1 max(P - ps, 0) K, rho clamp)
    const double dp = P - ps.v < 0.0 ? 0.0 : P - ps.v, k = c.c_c * rho * pv[5] * K, X = k * dp;
    const double cl = c.fix_cav_clamp ? pv[5] : pv[4], g = -s;
    if (rho * cl < X) {
      grho += g * cl;
      gp[c.fix_cav_clamp ? 5 : 4] += g * rho;
    } else {
      grho += g * c.c_c * pv[5] * dp * K;
      gp[5] += g * c.c_c * rho * dp * K;
      if (!(P - ps.v < 0.0)) { gp[0] += g * k; gp[4] -= g * k * ps.d[0]; }
      wp[0] -= g * X / c.uref;
      wp[2] += g * rho * pv[5] * dp * K;
    }
  }
  {
    // r_v = min(c_v rho yl max(ps - P, 0) K, rho clamp)
    const double dp = ps.v - P < 0.0 ? 0.0 : ps.v - P, k = c.c_v * rho * yl * K, X = k * dp;
    const double cl = c.fix_cav_clamp ? yl : 1.0 - pv[4] - pv[5], g = s;
    if (rho * cl < X) {
      grho += g * cl;
      gp[5] -= g * rho;
      gp[c.fix_cav_clamp ? 6 : 4] -= g * rho;
    } else {
      grho += g * c.c_v * yl * dp * K;
      gp[5] -= g * c.c_v * rho * dp * K;
      gp[6] -= g * c.c_v * rho * dp * K;
      if (!(ps.v - P < 0.0)) { gp[0] -= g * k; gp[4] += g * k * ps.d[0]; }
      wp[0] -= g * X / c.uref;
      wp[1] += g * rho * yl * dp * K;
    }
  }
}

// sst_source (RANS length) reversed: lam7 r7 + lam8 r8 with respect to the gradients gr
// (u, v, w, k, omega), k, omega, rho, mu, mu_t
struct SstGrad { double gr[5][3], k, o, rho, mu, mut; };
__device__ __forceinline__ void sst_back(const double (*gr)[3], double kk, double oo, double rho, double mu, double mut,
                                         double y, double vol, double lam7, double lam8, SstGrad& G) {
  const double c23 = 2.0 / 3.0, c59 = 5.0 / 9.0, y2 = y * y;
  double strain = 0.0;
#pragma unroll
  for (int i = 0; i < 3; ++i) {
    strain += 2.0 * gr[i][i] * gr[i][i];
#pragma unroll
    for (int j = i + 1; j < 3; ++j) strain += sq(gr[i][j] + gr[j][i]);
  }
  const double div = gr[0][0] + gr[1][1] + gr[2][2];
  const double io = 1.0 / oo, irho = 1.0 / rho, im = 1.0 / mut;
  const double P0 = mut * (strain - c23 * div * div) - c23 * rho * kk * div, lim = 0.9 * rho * kk * oo;
  const bool capped = lim < P0;
  const double prod = capped ? lim : P0;
  const double pkw = gr[3][0] * gr[4][0] + gr[3][1] * gr[4][1] + gr[3][2] * gr[4][2];
  const double cd0 = 1.712 * rho * io * pkw, cdkw = cd0 < 1.0e-10 ? 1.0e-10 : cd0, icd = 1.0 / cdkw;
  const double sk = ::sqrt(kk);
  const double t1 = sk * io / (0.09 * y), t2 = 500.0 * mu * irho * io / y2, t3 = 3.424 * rho * kk * icd / y2;
  const double m = t2 > t1 ? t2 : t1, arg = t3 < m ? t3 : m;
  const double a2 = arg * arg, F = ::tanh(a2 * a2);
  const double ta = F * c59 + (1.0 - F) * 0.44, tb = F * 0.075 + (1.0 - F) * 0.0828;
  const double a = lam7 * vol, b = lam8 * vol;
  const double gprod = a + b * ta * rho * im;
  const double gF = b * ((c59 - 0.44) * rho * im * prod - (0.075 - 0.0828) * rho * oo * oo - 1.712 * rho * io * pkw);
  double gpkw = b * 1.712 * (1.0 - F) * rho * io;
  G.rho = b * (ta * im * prod - tb * oo * oo + 1.712 * (1.0 - F) * io * pkw) - a * 0.09 * kk * oo;
  G.k = -a * 0.09 * rho * oo;   // the destruction is 0.09 rho k omega
  G.o = -a * 0.09 * rho * kk - b * (2.0 * tb * rho * oo + 1.712 * (1.0 - F) * rho * io * io * pkw);
  G.mut = -b * ta * rho * prod * im * im;
  G.mu = 0.0;
  double gs = 0.0, gdiv = 0.0;
  if (capped) {
    G.rho += gprod * 0.9 * kk * oo; G.k += gprod * 0.9 * rho * oo; G.o += gprod * 0.9 * rho * kk;
  } else {
    G.mut += gprod * (strain - c23 * div * div);
    gs = gprod * mut;
    gdiv = -gprod * c23 * (2.0 * mut * div + rho * kk);
    G.rho -= gprod * c23 * kk * div;
    G.k -= gprod * c23 * rho * div;
  }
  const double garg = gF * (1.0 - F * F) * 4.0 * arg * a2;
  if (t3 < m) {
    G.rho += garg * 3.424 * kk * icd / y2;
    G.k += garg * 3.424 * rho * icd / y2;
    if (!(cd0 < 1.0e-10)) {
      const double gcd = -garg * t3 * icd;
      G.rho += gcd * 1.712 * io * pkw;
      G.o -= gcd * cd0 * io;
      gpkw += gcd * 1.712 * rho * io;
    }
  } else if (t2 > t1) {
    G.mu += garg * 500.0 * irho * io / y2;
    G.rho -= garg * t2 * irho;
    G.o -= garg * t2 * io;
  } else {
    if (sk > 0.0) G.k += garg * 0.5 / sk * io / (0.09 * y);
    G.o -= garg * t1 * io;
  }
#pragma unroll
  for (int i = 0; i < 3; ++i) {
#pragma unroll
    for (int j = 0; j < 3; ++j) G.gr[i][j] = (i == j) ? gs * 4.0 * gr[i][i] + gdiv : gs * 2.0 * (gr[i][j] + gr[j][i]);
    G.gr[3][i] = gpkw * gr[4][i];
    G.gr[4][i] = gpkw * gr[3][i];
  }
}

__global__ void __launch_bounds__(128) k_adj_cell_plain(DevPtr d, Par c, AdjPtr a) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  double wp[3] = {0.0, 0.0, 0.0};
  if (t < d.nint) {
    const int b = find_block_interior(d.blk, d.nblk, t);
    int i, j, k;
    const BlockGeom& B = d.blk[b];
    const long long g = interior_cell(B, t - B.int_off, i, j, k);
    const long long n = d.ncell, sj = B.ni, sk = (long long)B.ni * B.nj;
    const int npv = c.npv;
    double lam[NPVM], pv2[NPVM], dv[2] = {d.dv[g], d.dv[n + g]}, gp[NPVM], gd[NGD];
#pragma unroll
    for (int v = 0; v < NPVM; ++v) {
      lam[v] = (v < npv) ? a.lam[v * n + g] : 0.0;
      pv2[v] = (v < npv) ? d.pv[v * n + g] : 0.0;
      gp[v] = 0.0;
    }
#pragma unroll
    for (int m = 0; m < NGD; ++m) gd[m] = 0.0;
    const double vol = d.gm[GM_GRD * n + g];
    if (c.ncav && lam[5] != 0.0) merkle_back(c, pv2, dv[0], vol, lam[5], gp, gd[GD_RHO], wp);
    if (c.iturb == 0 && (lam[7] != 0.0 || lam[8] != 0.0)) {
      const long long nbr[6] = {g - 1, g + 1, g - sj, g + sj, g - sk, g + sk};
      double fa[6][3], grv[5][3];
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        fa[0][q] = d.gm[(GM_CX + q) * n + g - 1]; fa[1][q] = d.gm[(GM_CX + q) * n + g];
        fa[2][q] = d.gm[(GM_EX + q) * n + g - sj]; fa[3][q] = d.gm[(GM_EX + q) * n + g];
        fa[4][q] = d.gm[(GM_TX + q) * n + g - sk]; fa[5][q] = d.gm[(GM_TX + q) * n + g];
      }
      const int gv[5] = {1, 2, 3, 7, 8};
      const double ivol = 1.0 / vol;
#pragma unroll
      for (int q = 0; q < 5; ++q) {
        const double* P = d.pv + gv[q] * n;
        const double c0 = P[g];
        double vv[6];
#pragma unroll
        for (int m = 0; m < 6; ++m) vv[m] = 0.5 * (P[nbr[m]] + c0);
#pragma unroll
        for (int e = 0; e < 3; ++e)
          grv[q][e] = (vv[1] * fa[1][e] + vv[3] * fa[3][e] + vv[5] * fa[5][e] - vv[0] * fa[0][e] - vv[2] * fa[2][e] -
                       vv[4] * fa[4][e]) * ivol;
      }
      SstGrad G;
      sst_back(grv, pv2[7], pv2[8], dv[0], d.tv[g], d.tv[2 * n + g], d.gm[(GM_GRD + 4) * n + g], vol, lam[7], lam[8], G);
      // the cell gradients are linear in the face averages 0.5 (P[nbr] + P[g])
#pragma unroll
      for (int q = 0; q < 5; ++q) {
        double gc = 0.0;
#pragma unroll
        for (int m = 0; m < 6; ++m) {
          const double s = (G.gr[q][0] * fa[m][0] + G.gr[q][1] * fa[m][1] + G.gr[q][2] * fa[m][2]) *
                           ((m & 1) ? 0.5 : -0.5) * ivol;
          gc += s;
          aadd(&a.gpv[gv[q] * n + nbr[m]], s);
        }
        gp[gv[q]] += gc;
      }
      gp[7] += G.k; gp[8] += G.o;
      gd[GD_RHO] += G.rho; gd[GD_VIS] += G.mu; gd[GD_MUT] += G.mut;
    }
    cell_sources_back(d, c, lam, pv2, dv, vol, gp, gd);
#pragma unroll
    for (int v = 0; v < NPVM; ++v)
      if (v < npv) aadd(&a.gpv[v * n + g], gp[v]);
#pragma unroll
    for (int m = 0; m < NGD; ++m) aadd(&a.gdt[m * n + g], gd[m]);
  }
  for (int q = 0; q < 3; ++q) {
    double s = wp[q];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) aadd(&a.gpar[q], s);
  }
}

void launch_adj_cell_plain(const Engine& E, const AdjPtr& a, cudaStream_t s) {
  k_adj_cell_plain<<<(unsigned)((E.nint + 127) / 128), 128, 0, s>>>(E.d, E.par, a);
}

// ------------------------------------------------------------------ interior EOS
// dv and tv(1:2) of an interior cell are its EOS: their gradient goes to (p, T, y1, y2)
__global__ void __launch_bounds__(64) k_adj_eos(DevPtr d, Par c, AdjPtr a) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (t >= d.nint) return;
  const int b = find_block_interior(d.blk, d.nblk, t);
  int i, j, k;
  const long long g = interior_cell(d.blk[b], t - d.blk[b].int_off, i, j, k);
  const long long n = d.ncell;
  double gd[NGD];
  bool any = false;
  for (int m = 0; m < NGD; ++m) {
    gd[m] = (m == GD_MUT) ? 0.0 : a.gdt[m * n + g];
    any = any || gd[m] != 0.0;
  }
  if (!any) return;
  double ge[4];
  eos_chain(c, d.pv[g] + c.pref, d.pv[4 * n + g], d.pv[5 * n + g], d.pv[6 * n + g], gd, ge);
  a.gpv[g] += ge[0];
  a.gpv[4 * n + g] += ge[1];
  a.gpv[5 * n + g] += ge[2];
  a.gpv[6 * n + g] += ge[3];
}

void launch_adj_eos(const Engine& E, const AdjPtr& a, cudaStream_t s) {
  k_adj_eos<<<(unsigned)((E.nint + 63) / 64), 64, 0, s>>>(E.d, E.par, a);
}

void launch_adj_face(const Engine& E, const DevPtr& d, const AdjPtr& a, cudaStream_t s) {
  const Par& c = E.par;
  auto nb = [](long long n, int t) { return (unsigned)((n + t - 1) / t); };
  for (int dir = 0; dir < 3; dir += d.fslots) {
    long long nf = 0;
    for (int q = dir; q < dir + d.fslots; ++q) nf = nf > E.nface[q] ? nf : E.nface[q];
    const unsigned z = (unsigned)d.fslots;
    launch_recon64(E, d, dir, s);
    if (c.nscheme == 2 || c.nscheme == 3) launch_adj_flux_duals(E, d, a, dir, nf, s);
    else k_adj_flux<false><<<dim3(nb(nf, 64), 1, z), 64, 0, s>>>(d, c, a, dir);
    if (c.nmuscl > 0) k_adj_recon<<<dim3(nb(nf, 128), (unsigned)c.npv, z), 128, 0, s>>>(d, c, a, dir);
    if (c.iturb != -3) k_adj_visc<<<dim3(nb(nf, 128), 1, z), 128, 0, s>>>(d, c, a, dir);
  }
}

}  // namespace cfd
