// eos_mixed.cu -- the mixed form's cell EOS: dv and tv(1:2) of the interior cells from their pv
// (eos%deteos as the update calls it, src/update_module.f90:689), deteos_split's arithmetic
// in passes.
//
// What bounds it: the FP64 pipe (conversions and the mixture's sums, about 60 issue slots a
// cell) and the FP32 issue slots (about 3000 instructions a cell).  As one kernel, with the
// update, it was bound by neither: some 8000 instructions of straight code, which each warp
// walks at its own pace, do not stay in the instruction cache (8.9 of 13 stall cycles per
// issue were waits for an instruction; 2.9 ms on the 3.0 M-cell batched case, 6.1 ms on the
// 14.2 M-cell one), and a warp with some vapour ran the liquid's sums twice.  Now
//   k_eos_liq         the liquid's df64 sums and the gas, every cell; cells with vapour are
//                     listed by the vapour sums they need
//   k_eos_vap         the vapour's df64 sums of the listed cells, full warps, a grid row per
//                     list
//   k_eos_mix         FP32 derivatives and transport properties, the mixture
// with the five phase values between them in the face records' planes (idle then).
#include <algorithm>
#include "engine.cuh"

namespace cfd {

enum { ES_IL = 0, ES_HL, ES_IG, ES_IV, ES_HV, NES };
static_assert(NES * 2 <= 24, "the phase values fit the face records' planes");

// the padded cell of interior cell q
__device__ __forceinline__ long long eos_cell(const DevPtr& d, long long q) {
  const int b = find_block_interior(d.blk, d.nblk, q);
  int i, j, k;
  return interior_cell(d.blk[b], q - d.blk[b].int_off, i, j, k);
}

__global__ void __launch_bounds__(256) k_eos_liq(DevPtr d, Par c, int* cnt) {
  const long long n = d.ncell;
  double* S = reinterpret_cast<double*>(d.frec);
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < d.nint; q += (long long)gridDim.x * blockDim.x) {
    const long long g = eos_cell(d, q);
    const double p = d.pv[g] + c.pref, t = d.pv[4 * n + g], y1 = d.pv[5 * n + g];
    double il, hl, ig;
    liquid_inv_df64(df64(p), df64(t), &il, &hl, &ig);
    S[ES_IL * n + g] = il;
    S[ES_HL * n + g] = hl;
    S[ES_IG * n + g] = ig;
    if (y1 != 0.0) {
      list_add(d, cnt, above_psat(p, t) ? MX_META : MX_STABLE, (int)g);
    }
  }
}

template <bool META>
__device__ __forceinline__ void eos_vap(const DevPtr& d, const Par& c, const int* cnt) {
  const int* L;
  const int m = list_of(d, cnt, META ? MX_META : MX_STABLE, L);
  const long long n = d.ncell;
  double* S = reinterpret_cast<double*>(d.frec);
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < m; q += gridDim.x * blockDim.x) {
    const long long g = L[q];
    double iv, hv;
    vapour_inv_df64(df64(d.pv[g] + c.pref), df64(d.pv[4 * n + g]), META, &iv, &hv);
    S[ES_IV * n + g] = iv;
    S[ES_HV * n + g] = hv;
  }
}

__global__ void __launch_bounds__(256) k_eos_vap(DevPtr d, Par c, const int* cnt) {
  if (blockIdx.y == 0) eos_vap<true>(d, c, cnt);
  else eos_vap<false>(d, c, cnt);
}

__global__ void __launch_bounds__(256) k_eos_mix(DevPtr d, Par c) {
  const long long n = d.ncell;
  const double* S = reinterpret_cast<const double*>(d.frec);
  int bad = 0;
  for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < d.nint; q += (long long)gridDim.x * blockDim.x) {
    const long long g = eos_cell(d, q);
    const double p = d.pv[g] + c.pref, t = d.pv[4 * n + g], y1 = d.pv[5 * n + g], y2 = d.pv[6 * n + g];
    double dv[NDV], tv[2];
    if (c.fluid == 1) {
      deteos_split_stiffened(c.with_prop, p, t, y1, y2, dv, tv, &d.sc->snd2_fallbacks);
    } else {
      double iv = 0.0, hv = 0.0;
      if (y1 != 0.0) { iv = S[ES_IV * n + g]; hv = S[ES_HV * n + g]; }
      deteos_split_mix(c.with_prop, p, t, y1, y2, above_psat(p, t), S[ES_IL * n + g], S[ES_HL * n + g], iv, hv,
                       S[ES_IG * n + g], dv, tv, &d.sc->snd2_fallbacks);
    }
#pragma unroll
    for (int v = 0; v < NDV; ++v) {
      d.dv[v * n + g] = dv[v];
      if (!finite_bits(dv[v])) bad = 1;
    }
    if (c.with_prop)
#pragma unroll
      for (int v = 0; v < 2; ++v)
        if (v < c.ntv) d.tv[v * n + g] = tv[v];
  }
  if (bad) atomicExch(&d.sc->nonfinite, 1);
}

void launch_eos_cells(const Engine& E, cudaStream_t s) {
  const DevPtr& d = E.d;
  const Par& c = E.par;
  int dev = 0, nsm = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
  auto grid = [&](int per) {
    return (unsigned)std::max<long long>(1, std::min<long long>((E.nint + 255) / 256, (long long)per * nsm));
  };
  if (c.fluid != 1) {
    int* cnt = d.mxn + MXN_FACE;
    cudaMemsetAsync(cnt, 0, MX_KINDS * sizeof(int), s);
    k_eos_liq<<<grid(32), 256, 0, s>>>(d, c, cnt);
    k_eos_vap<<<dim3(grid(4), 2), 256, 0, s>>>(d, c, cnt);
  }
  k_eos_mix<<<grid(32), 256, 0, s>>>(d, c);
}

int eos_cells_launches(const Engine& E) { return E.par.fluid != 1 ? 3 : 1; }

}  // namespace cfd
