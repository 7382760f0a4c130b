// faces64.cuh -- what the FP64 form's face kernels (flux.cu) and their reverse
// (adjoint_face.cu) share: the numbering of faces and of the cells around them, the
// integer-pipe order of doubles, and the reconstruction's scratch planes.
#pragma once
#include "engine.cuh"

namespace cfd {

// the faces (EXT = 0) or the cells -1 .. +1 around them along the normal (EXT = 3) of direction
// dir: the cell of flat index t, block-major, then (k, j, i) of the (left) cell
struct DirCell {
  long long g, sn, s1, s2;   // cell, normal and transverse strides
  int b;
};
template <int EXT>
__device__ __forceinline__ bool dir_cell(const DevPtr& d, int dir, long long t, DirCell& o) {
  const BlockGeom* blk = d.blk;
  int b = 0;
  while (b + 1 < d.nblk && t >= (EXT ? blk[b + 1].plane_off[dir] : blk[b + 1].face_off[dir])) ++b;
  const BlockGeom& B = blk[b];
  const long long loc = t - (EXT ? B.plane_off[dir] : B.face_off[dir]);
  const int fi = B.imax - 1 + (dir == 0 ? 1 + EXT : 0), fj = B.jmax - 1 + (dir == 1 ? 1 + EXT : 0);
  const int fk = B.kmax - 1 + (dir == 2 ? 1 + EXT : 0);
  if (loc >= (long long)fi * fj * fk) return false;
  const int first = EXT ? 0 : 1;   // the first left cell, less one with EXT
  const int i = (int)(loc % fi) + (dir == 0 ? first : 2);
  const long long r = loc / fi;
  const int j = (int)(r % fj) + (dir == 1 ? first : 2);
  const int k = (int)(r / fj) + (dir == 2 ? first : 2);
  const long long sj = B.ni, sk = (long long)B.ni * B.nj;
  o.b = b;
  o.g = B.off + (i + 1) + sj * (j + 1) + sk * (k + 1);
  if (dir == 0) { o.sn = 1; o.s1 = sj; o.s2 = sk; }
  else if (dir == 1) { o.sn = sj; o.s1 = sk; o.s2 = 1; }
  else { o.sn = sk; o.s1 = 1; o.s2 = sj; }
  return true;
}

__device__ __forceinline__ bool is_zero(double x) { return (__double_as_longlong(x) << 1) == 0; }

// the left face states, then the fluxes, of a direction (npv planes; fi1: one direction's at a time)
__device__ __forceinline__ double* fi_planes(const DevPtr& d, int dir, int npv) {
  return d.fi + (long long)(d.fi1 ? 0 : dir) * npv * d.ncell;
}

// scratch planes of one direction slot and variable
enum { FS_MN = 0, FS_MX, FS_DEN, FS_IDQ, FS_R, NFS };
__device__ __forceinline__ double* fs_plane(const DevPtr& d, int slot, int npv, int v, int q) {
  return d.fsc + ((long long)(slot * npv + v) * d.nfs + (d.nfs == 1 ? 0 : q)) * d.ncell;
}

// per-cell planes and face states of directions dir .. dir + d.fslots - 1 (flux.cu)
void launch_recon64(const Engine& E, const DevPtr& d, int dir, cudaStream_t s);

}  // namespace cfd
