// adjoint_duals.cu -- the parts of the discrete adjoint that stay with duals of eight
// directions: the flux of Roe-M and AUSMPW+, and the cell sources of the cavitation models
// other than Merkle's and of the DES lengths.  The file comment of adjoint.cu describes the
// whole reverse pass.
#include "adjoint_flux.cuh"

namespace cfd {

// ------------------------------------------------------------------ Roe-M, AUSMPW+
// seed layout
enum { S_PL = 0, S_PR = 9, S_RHOL = 18, S_HL, S_C2L, S_RHOR, S_HR, S_C2R, S_UREF = 24, S_SDST = 25, NS_INV = 43 };

static __device__ __noinline__ void flux_back_duals(const Par& c, const double* nx, const FaceState& L,
                                                    const FaceState& R, const EosJac& jc, const double* sdv,
                                                    const double* lam, double* w) {
  const int npv = c.npv;
  for (int k0 = 0; k0 < NS_INV; k0 += DC) {
    FaceStateT<DD> Ld, Rd;
    for (int v = 0; v < NPVM; ++v) { Ld.pv[v] = seed(L.pv[v], S_PL + v, k0); Rd.pv[v] = seed(R.pv[v], S_PR + v, k0); }
    Ld.rho = seed(L.rho, S_RHOL, k0); Ld.h = seed(L.h, S_HL, k0); Ld.c2 = seed(L.c2, S_C2L, k0);
    Rd.rho = seed(R.rho, S_RHOR, k0); Rd.h = seed(R.h, S_HR, k0); Rd.c2 = seed(R.c2, S_C2R, k0);
    DD ravg[NPVM];
    for (int v = 0; v < NPVM; ++v) ravg[v] = DD(0.0);
    roe_state<DD>(npv, Ld, Rd, ravg);
    const int am[4] = {0, 4, 5, 6};
    DD rc2(jc.c2);
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
      for (int q = 0; q < DC; ++q) rc2.d[q] += jc.dc2[m] * ravg[am[m]].d[q];
    const DD uref = seed(c.uref, S_UREF, k0);
    DD sdst[18];
    for (int l = 0; l < 18; ++l) sdst[l] = seed(sdv[l], S_SDST + l, k0);
    DD fx[NPVM];
    inviscid_flux_core<DD>(c, nx, Ld, Rd, sdst, ravg, rc2, uref * uref, fx);
#pragma unroll
    for (int q = 0; q < DC; ++q) {
      if (k0 + q >= NS_INV) break;
      double acc = 0.0;
      for (int v = 0; v < npv; ++v) acc += lam[v] * fx[v].d[q];
      w[k0 + q] = acc;
    }
  }
}

template <>
struct FluxBack<true> {
  static __device__ __forceinline__ void run(const Par& c, const double* nx, const FaceState& L, const FaceState& R,
                                             const EosJac& jc, const double*, const double* sdv, const double* lam,
                                             FaceGrad& o, double* ws) {
    double w[NS_INV];
    flux_back_duals(c, nx, L, R, jc, sdv, lam, w);
    for (int v = 0; v < NPVM; ++v) { o.pl[v] = w[S_PL + v]; o.pr[v] = w[S_PR + v]; }
    o.rl = w[S_RHOL]; o.hl = w[S_HL]; o.c2l = w[S_C2L];
    o.rr = w[S_RHOR]; o.hr = w[S_HR]; o.c2r = w[S_C2R];
    o.uref = w[S_UREF];
    for (int l = 0; l < 18; ++l) ws[l] = w[S_SDST + l];
  }
};

void launch_adj_flux_duals(const Engine& E, const DevPtr& d, const AdjPtr& a, int dir, long long nf, cudaStream_t s) {
  k_adj_flux<true><<<dim3((unsigned)((nf + 63) / 64), 1, (unsigned)d.fslots), 64, 0, s>>>(d, E.par, a, dir);
}

// ------------------------------------------------------------------ cell sources
// Per interior cell: the cavitation source (res(6)), the SST sources (res(8:9)) and the
// dual-time source, as k_rhs adds them (src/rhs_module.f90:540-642).
// Merkle's rates and the RANS SST source are reversed by hand (k_adj_cell_plain, adjoint_face.cu);
// the other cavitation models and the DES lengths by duals here.
__global__ void __launch_bounds__(64) k_adj_cell(DevPtr d, Par c, AdjPtr a) {
  const long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  double wp[3] = {0.0, 0.0, 0.0};
  if (t < d.nint) {
    const int b = find_block_interior(d.blk, d.nblk, t);
    int i, j, k;
    const BlockGeom& B = d.blk[b];
    const long long g = interior_cell(B, t - B.int_off, i, j, k);
    const long long n = d.ncell, sj = B.ni, sk = (long long)B.ni * B.nj;
    const int npv = c.npv;
    double lam[NPVM], pv2[NPVM], dv[NDV];
    for (int v = 0; v < NPVM; ++v) {
      lam[v] = (v < npv) ? a.lam[v * n + g] : 0.0;
      pv2[v] = (v < npv) ? d.pv[v * n + g] : 0.0;
    }
    for (int v = 0; v < NDV; ++v) dv[v] = d.dv[v * n + g];
    const double vol = d.gm[GM_GRD * n + g];
    double gp[NPVM], gd[NGD];
    for (int v = 0; v < NPVM; ++v) gp[v] = 0.0;
    for (int m = 0; m < NGD; ++m) gd[m] = 0.0;
    // ---- cavitation: res(6) += r_v - r_c; seeds p, T, y1, y2, rho, rho_l, rho_v, rho_g (Kunz's
    // gas volume fraction), uref, c_v, c_c
    if (c.ncav && lam[5] != 0.0) {
      const int pvs[4] = {0, 4, 5, 6};
      const int dvs[4] = {0, 2, 3, 4};
      double w[11];
      for (int k0 = 0; k0 < 11; k0 += DC) {
        DD p2[NPVM], dd[NDV];
        for (int v = 0; v < NPVM; ++v) p2[v] = DD(pv2[v]);
        for (int q = 0; q < NDV; ++q) dd[q] = DD(dv[q]);
        for (int m = 0; m < 4; ++m) p2[pvs[m]] = seed(pv2[pvs[m]], m, k0);
        for (int m = 0; m < 4; ++m) dd[dvs[m]] = seed(dv[dvs[m]], 4 + m, k0);
        const CavOutT<DD> o = cavsource_t<DD>(c, p2, dd, vol, seed(c.uref, 8, k0), seed(c.c_v, 9, k0),
                                              seed(c.c_c, 10, k0));
#pragma unroll
        for (int q = 0; q < DC; ++q)
          if (k0 + q < 11) w[k0 + q] = lam[5] * (o.r_v.d[q] - o.r_c.d[q]);
      }
      for (int m = 0; m < 4; ++m) gp[pvs[m]] += w[m];
      gd[GD_RHO] += w[4]; gd[GD_RL] += w[5]; gd[GD_RV] += w[6]; gd[GD_RG] += w[7];
      wp[0] += w[8]; wp[1] += w[9]; wp[2] += w[10];
    }
    // ---- SST: res(8) += r7, res(9) += r8; seeds the 15 cell gradients, k, omega, rho, mu, mu_t
    if (c.iturb == 0 && (lam[7] != 0.0 || lam[8] != 0.0)) {
      const long long nbr[6] = {g - 1, g + 1, g - sj, g + sj, g - sk, g + sk};
      double fa[6][3];
      for (int q = 0; q < 3; ++q) {
        fa[0][q] = d.gm[(GM_CX + q) * n + g - 1]; fa[1][q] = d.gm[(GM_CX + q) * n + g];
        fa[2][q] = d.gm[(GM_EX + q) * n + g - sj]; fa[3][q] = d.gm[(GM_EX + q) * n + g];
        fa[4][q] = d.gm[(GM_TX + q) * n + g - sk]; fa[5][q] = d.gm[(GM_TX + q) * n + g];
      }
      const int gv[5] = {1, 2, 3, 7, 8};
      double grv[5][3];
      const double ivol = 1.0 / vol;
      for (int q = 0; q < 5; ++q) {
        const double* P = d.pv + gv[q] * n;
        const double c0 = P[g];
        const double v1 = 0.5 * (P[nbr[0]] + c0), v2 = 0.5 * (P[nbr[1]] + c0), v3 = 0.5 * (P[nbr[2]] + c0);
        const double v4 = 0.5 * (P[nbr[3]] + c0), v5 = 0.5 * (P[nbr[4]] + c0), v6 = 0.5 * (P[nbr[5]] + c0);
        for (int e = 0; e < 3; ++e)
          grv[q][e] = (v2 * fa[1][e] + v4 * fa[3][e] + v6 * fa[5][e] - v1 * fa[0][e] - v3 * fa[2][e] - v5 * fa[4][e]) * ivol;
      }
      const double mu = d.tv[g], mut = d.tv[2 * n + g];
      const double y5 = d.gm[(GM_GRD + 4) * n + g];
      double w[20];
      const double hmax = c.ides ? grid_hmax<double>(fa, vol) : 0.0;
      for (int k0 = 0; k0 < 20; k0 += DC) {
        DD gr[5][3];
        for (int q = 0; q < 5; ++q)
          for (int e = 0; e < 3; ++e) gr[q][e] = seed(grv[q][e], 3 * q + e, k0);
        const SstOut<DD> so = sst_source<DD>(gr, seed(pv2[7], 15, k0), seed(pv2[8], 16, k0), seed(dv[0], 17, k0),
                                             seed(mu, 18, k0), seed(mut, 19, k0), y5, vol, c.ides, hmax);
#pragma unroll
        for (int q = 0; q < DC; ++q)
          if (k0 + q < 20) w[k0 + q] = lam[7] * so.r7.d[q] + lam[8] * so.r8.d[q];
      }
      // the cell gradients are linear in the face averages 0.5 (P[nbr] + P[g])
      const double sgn[6] = {-1.0, 1.0, -1.0, 1.0, -1.0, 1.0};
      for (int q = 0; q < 5; ++q) {
        double gc = 0.0;
        for (int m = 0; m < 6; ++m) {
          double s = 0.0;
          for (int e = 0; e < 3; ++e) s += w[3 * q + e] * fa[m][e];
          s *= 0.5 * sgn[m] * ivol;
          gc += s;
          aadd(&a.gpv[gv[q] * n + nbr[m]], s);
        }
        gp[gv[q]] += gc;
      }
      gp[7] += w[15]; gp[8] += w[16];
      gd[GD_RHO] += w[17]; gd[GD_VIS] += w[18]; gd[GD_MUT] += w[19];
    }
    cell_sources_back(d, c, lam, pv2, dv, vol, gp, gd);
    for (int v = 0; v < npv; ++v) aadd(&a.gpv[v * n + g], gp[v]);
    for (int m = 0; m < NGD; ++m) aadd(&a.gdt[m * n + g], gd[m]);
  }
  for (int q = 0; q < 3; ++q) {
    double s = wp[q];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) aadd(&a.gpar[q], s);
  }
}

void launch_adj_cell(const Engine& E, const AdjPtr& a, cudaStream_t s) {
  k_adj_cell<<<(unsigned)((E.nint + 63) / 64), 64, 0, s>>>(E.d, E.par, a);
}

}  // namespace cfd
