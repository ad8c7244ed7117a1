// ipg_snap_geom.cuh — switching function and per-pair geometry of the SNAP kernels.
#pragma once

#include "ipg_snap.cuh"

namespace {

// Species ids are validated by the neighbor build (status word); clamping here keeps a
// bad id from indexing the per-species tables.
__device__ __forceinline__ int clamp_sp(int s, int nsp) { return s < 0 ? 0 : (s >= nsp ? nsp - 1 : s); }

__device__ __forceinline__ double sfac_of(const SnapDev& S, double r, double rcut) {  // compute_ui.jl:350-364
  if (!S.switch_flag) return 1.0;
  if (r <= S.rmin0) return 1.0;
  if (r > rcut) return 0.0;
  return 0.5 * (cos((r - S.rmin0) * (M_PI / (rcut - S.rmin0))) + 1.0);
}
__device__ __forceinline__ double dsfac_of(const SnapDev& S, double r, double rcut) {  // compute_ui.jl:366-380
  if (!S.switch_flag) return 0.0;
  if (r <= S.rmin0) return 0.0;
  double rcutfac = M_PI / (rcut - S.rmin0);
  return -0.5 * (sin((r - S.rmin0) * rcutfac) * rcutfac);
}

// Per-pair geometry for the derivative recursion (compute_duidrj, compute_ui.jl:328-347
// and the prologue of compute_duarray, :191-216).
struct PairGeom {
  double2 a, b;
  double2 da[3], db[3];
  double u[3];
  double sfac, dsfac;
};

__device__ __forceinline__ void geom_du(const SnapDev& S, double x, double y, double z, double rcut, double wj,
                                        PairGeom& G) {
  double rsq = x * x + y * y + z * z;
  double r = sqrt(rsq);
  double rscale0 = S.rfac0 * M_PI / (rcut - S.rmin0);
  double theta0 = (r - S.rmin0) * rscale0;
  double sn, cs;
  sincos(theta0, &sn, &cs);
  double z0 = r * cs / sn;
  double dz0dr = z0 / r - (r * rscale0) * (rsq + z0 * z0) / rsq;
  double rinv = 1.0 / r;
  G.u[0] = x * rinv;
  G.u[1] = y * rinv;
  G.u[2] = z * rinv;
  double r0inv = 1.0 / sqrt(r * r + z0 * z0);
  G.a = make_double2(z0 * r0inv, -z * r0inv);
  G.b = make_double2(y * r0inv, -x * r0inv);
  double dr0invdr = -r0inv * r0inv * r0inv * (r + z0 * dz0dr);
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double dr0 = dr0invdr * G.u[k];
    double dz0 = dz0dr * G.u[k];
    G.da[k] = make_double2(dz0 * r0inv + z0 * dr0, -z * dr0);
    G.db[k] = make_double2(y * dr0, -x * dr0);
  }
  G.da[2].y += -r0inv;
  G.db[0].y += -r0inv;
  G.db[1].x += r0inv;
  G.sfac = sfac_of(S, r, rcut) * wj;
  G.dsfac = dsfac_of(S, r, rcut) * wj;
}

}  // namespace
