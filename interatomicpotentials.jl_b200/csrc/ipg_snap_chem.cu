// ipg_snap_chem.cu — explicit multi-element SNAP (chem_flag) and quadratic SNAP by the adjoint
// route: Y = dE/dU of every element from the Z of every element pair, instead of the dB/dr of
// every pair and element triple (compute_b.jl:104-400).
//
// E = sum over element triples (p, q, e) and components b = (j1, j2, j) of beta B, with
// B = sum conj(U_e^j) Z^{pq}(j1, j2, j) trilinear in U.  A Z triple of the element pair (p, q)
// belongs to one component and serves one to three terms of its derivative; in the Y of element e
// it carries the factor of those terms times beta of the triples (p, q, e), (e, q, p), (q, e, p)
// (the triples of the three terms in compute_b.jl:196, 250, 305).  Quadratic SNAP is the same with
// each atom's effective linear coefficients beta_k + sum_l a_kl B_l.
//
// Forces then cost one pass of the pair kernel on U instead of nelem^2 contractions of every
// pair's dU with the owner's Z.  1,999 atoms, two species, twojmax 6: 3251 -> 364 us per call.
#include <algorithm>

#include "ipg_snap.cuh"

namespace {

__device__ __forceinline__ int sp_of(const int32_t* __restrict__ species, int64_t i, int nsp) {
  const int s = species[i];
  return s < 0 ? 0 : (s >= nsp ? nsp - 1 : s);
}

// coef[((e ne^2 + p ne + q) ntrip + t)][nc], atoms in lanes.
__global__ void __launch_bounds__(128) k_chem_coef(const __grid_constant__ SnapDev S, int64_t a0, int64_t nc,
                                                   const int32_t* __restrict__ species, double* __restrict__ coef) {
  const int64_t l = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= nc) return;
  const int ne = S.nelem, nt = S.n_ytrip, KB = S.klin / (ne * ne * ne);
  const double* bt = S.beta + (size_t)sp_of(species, a0 + l, S.nsp) * S.K;
  for (int x = blockIdx.y; x < ne * ne * ne * nt; x += gridDim.y) {
    const int t = x % nt, y = x / nt, q = y % ne, p = (y / ne) % ne, e = y / (ne * ne);
    const int pk = S.ytrip_b[t], b = pk & 0xffff;
    double c = 0.0;
    if ((pk >> 16) & 1) c += bt[((p * ne + q) * ne + e) * KB + b];
    if ((pk >> 17) & 1) c += bt[((e * ne + q) * ne + p) * KB + b];
    if ((pk >> 18) & 1) c += bt[((q * ne + e) * ne + p) * KB + b];
    coef[(size_t)x * nc + l] = S.ytrip_fac[t] * c;
  }
}

// One warp per atom, lanes over the linear components k: beff_k = beta_k + sum_l a_kl B_l, and
// E_i = beta . B_ext (the linear components, then 0.5 B_k^2 and B_k B_l, l > k, k outer).
constexpr int QC_WARPS = 4;
__global__ void __launch_bounds__(QC_WARPS * 32) k_quad_coef(const __grid_constant__ SnapDev S, int64_t a0,
                                                             int64_t nc, const int32_t* __restrict__ species,
                                                             const double* __restrict__ B, double* __restrict__ Ei,
                                                             double* __restrict__ coef) {
  extern __shared__ double qsm[];  // [QC_WARPS][2][klin]: B and beff of the warp's atom
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, KL = S.klin;
  const int64_t l = (int64_t)blockIdx.x * QC_WARPS + w;
  if (l >= nc) return;  // warp-uniform; the kernel synchronises only within a warp
  const int64_t i = a0 + l;
  double* bs = qsm + (size_t)w * 2 * KL;
  double* be = bs + KL;
  const double* bt = S.beta + (size_t)sp_of(species, i, S.nsp) * S.K;
  for (int k = lane; k < KL; k += 32) bs[k] = B[(size_t)i * KL + k];
  __syncwarp();
  double e = 0.0;
  for (int k = lane; k < KL; k += 32) {
    const double bk = bs[k];
    const double* row = bt + KL + (size_t)k * KL - (size_t)k * (k - 1) / 2;  // 0.5 B_k^2, then B_k B_l
    double g = fma(row[0], bk, bt[k]);
    double t = fma(row[0], 0.5 * bk * bk, bt[k] * bk);
    for (int m = k + 1; m < KL; m++) {
      t = fma(row[m - k], bk * bs[m], t);
      g = fma(row[m - k], bs[m], g);
    }
    for (int m = 0; m < k; m++) g = fma(bt[KL + (size_t)m * KL - (size_t)m * (m - 1) / 2 + k - m], bs[m], g);
    be[k] = g;
    e += t;
  }
  e = warp_sum(e);
  if (lane == 0) Ei[i] = e;
  __syncwarp();
  for (int t = lane; t < S.n_ytrip; t += 32) {
    const int pk = S.ytrip_b[t];
    coef[(size_t)t * nc + l] = S.ytrip_fac[t] * __popc(pk >> 16) * be[pk & 0xffff];
  }
}

// Y' of one tile (level j, row mb, CY_MA elements) of 32 atoms per warp, every element at once: per
// element pair and triple of the level, the tile's Z against nelem coefficients.  Bound by the latency
// of the reads of Z (each element once): with a warp a row 88 us at 1,999 atoms, two elements, twojmax 6,
// with a warp a tile 52.
// The tiles' energies go to epart [tiles][nc].
constexpr int CY_MA = 3, CY_WARPS = 4;
__host__ __device__ inline int cy_tiles(int j) { return (j + CY_MA) / CY_MA; }  // of a row of level j
template <int NE>
__global__ void __launch_bounds__(CY_WARPS * 32) k_chem_y(const __grid_constant__ SnapDev S, int64_t n, int64_t a0,
                                                          int64_t nc, const double* __restrict__ coef,
                                                          const double2* __restrict__ Z,
                                                          const double2* __restrict__ utot, double2* __restrict__ yout,
                                                          double* __restrict__ epart, int ntile, int e0) {
  const int lane = threadIdx.x & 31, r = blockIdx.y * CY_WARPS + (threadIdx.x >> 5);
  if (r >= ntile) return;
  int j = S.J, x0 = r;  // the largest level first: its tiles take the longest
  while (x0 >= (j / 2 + 1) * cy_tiles(j)) x0 -= (j / 2 + 1) * cy_tiles(j), j--;
  const int mb = x0 / cy_tiles(j), m0 = x0 % cy_tiles(j) * CY_MA;
  const int64_t l = (int64_t)blockIdx.x * 32 + lane;
  const bool valid = l < nc;
  const int64_t la = valid ? l : nc - 1;
  const int ne = S.nelem, nt = S.n_ytrip, M = S.idxz_max;
  const int32_t* lev = S.ylev;
  const int t0 = lev[j], t1 = lev[j + 1];
  const int32_t* trips = lev + S.J + 2;
  const int nma = 2 * mb == j ? mb + 1 : j + 1, h0 = S.half_block[j] + mb * (j + 1);
  double en = 0.0;
  if (m0 < nma) {  // the row of a level's middle ends there
    double2 acc[NE][CY_MA];
#pragma unroll
    for (int e = 0; e < NE; e++)
#pragma unroll
      for (int m = 0; m < CY_MA; m++) acc[e][m] = make_double2(0.0, 0.0);
    for (int pq = 0; pq < ne * ne; pq++)
#pragma unroll 4
      for (int x = t0; x < t1; x++) {
        const int t = trips[x];
        const double2* z = Z + ((size_t)pq * M + S.ytrip_jjz[t] + mb * (j + 1) + m0) * nc + la;
        double2 zv[CY_MA];
#pragma unroll
        for (int m = 0; m < CY_MA; m++) zv[m] = m0 + m < nma ? z[(size_t)m * nc] : make_double2(0.0, 0.0);
#pragma unroll
        for (int e = 0; e < NE; e++) {
          const double c = e0 + e < ne ? coef[((size_t)((e0 + e) * ne * ne + pq) * nt + t) * nc + la] : 0.0;
#pragma unroll
          for (int m = 0; m < CY_MA; m++) {
            acc[e][m].x = fma(c, zv[m].x, acc[e][m].x);
            acc[e][m].y = fma(c, zv[m].y, acc[e][m].y);
          }
        }
      }
#pragma unroll
    for (int e = 0; e < NE; e++) {
      if (e0 + e >= ne) break;
#pragma unroll
      for (int m = 0; m < CY_MA; m++) {
        if (m0 + m >= nma) break;
        const int h = h0 + m0 + m;
        const double w = 2 * mb == j && m0 + m == mb ? 0.5 : 1.0;
        const double2 y = make_double2(w * acc[e][m].x, w * acc[e][m].y);
        if (valid) yout[((size_t)h * n + a0 + l) * ne + e0 + e] = y;
        if (epart) {
          const double2 u = utot[((size_t)(e0 + e) * n + a0 + la) * S.idxu_max + S.u_of_h[h]];
          en += u.x * y.x + u.y * y.y;
        }
      }
    }
  }
  if (epart && valid) epart[(size_t)r * nc + l] = (e0 ? epart[(size_t)r * nc + l] : 0.0) + en;
}

// E_i = (2/3) sum of the tiles' energies, shifted by beta of the triples that carry bzero.
__global__ void k_chem_energy(const __grid_constant__ SnapDev S, int64_t a0, int64_t nc, int ntile,
                              const int32_t* __restrict__ species, const double* __restrict__ epart,
                              double* __restrict__ Ei) {
  const int64_t l = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= nc) return;
  double t = 0.0;
#pragma unroll 5
  for (int r = 0; r < ntile; r++) t += epart[(size_t)r * nc + l];
  t *= 2.0 / 3.0;
  if (S.bzero_flag) {
    const int ne = S.nelem, KB = S.klin / (ne * ne * ne), si = sp_of(species, a0 + l, S.nsp);
    const double* bt = S.beta + (size_t)si * S.K;
    for (int tri = 0; tri < ne * ne * ne; tri++) {
      if (!S.wselfall && tri != (si * ne + si) * ne + si) continue;
      for (int b = 0; b < KB; b++) t -= bt[tri * KB + b] * S.bzero[S.db[b].l[0]];
    }
  }
  Ei[a0 + l] = t;
}

}  // namespace

int launch_chem_coef(ipg_ctx* ctx, const SnapDev& S, int64_t a0, int64_t nc, const int32_t* species, double* coef) {
  if (nc <= 0) return IPG_OK;
  const int rows = S.nelem * S.nelem * S.nelem * S.n_ytrip;
  const dim3 grid((unsigned)((nc + 127) / 128), (unsigned)std::min(rows, 256));
  IPG_LAUNCH(ctx, k_chem_coef, grid, 128, 0, S, a0, nc, species, coef);
  return IPG_OK;
}

int launch_quad_coef(ipg_ctx* ctx, const SnapDev& S, int64_t a0, int64_t nc, const int32_t* species, const double* B,
                     double* Ei, double* coef) {
  if (nc <= 0) return IPG_OK;
  IPG_LAUNCH(ctx, k_quad_coef, (unsigned)((nc + QC_WARPS - 1) / QC_WARPS), QC_WARPS * 32,
             (size_t)QC_WARPS * 2 * S.klin * sizeof(double), S, a0, nc, species, B, Ei, coef);
  return IPG_OK;
}

int launch_chem_y(ipg_ctx* ctx, const SnapDev& S, int64_t n, int64_t a0, int64_t nc, const int32_t* species,
                  const double* coef, const double2* Z, const double2* utot, double2* yout, double* Ei) {
  if (nc <= 0) return IPG_OK;
  int ntile = 0;
  for (int j = 0; j <= S.J; j++) ntile += (j / 2 + 1) * cy_tiles(j);
  double* epart = nullptr;
  if (Ei) IPG_RET(scratch(ctx, "chem_epart", (size_t)ntile * nc, &epart));
  const dim3 grid((unsigned)((nc + 31) / 32), (unsigned)((ntile + CY_WARPS - 1) / CY_WARPS));
  for (int e0 = 0; e0 < S.nelem; e0 += 3) {  // three elements per pass over Z
    const int k = std::min(3, S.nelem - e0);
    if (k == 1)
      IPG_TIMED_LAUNCH(ctx, "snap_atom", k_chem_y<1>, grid, CY_WARPS * 32, 0, S, n, a0, nc, coef, Z, utot, yout,
                       epart, ntile, e0);
    else if (k == 2)
      IPG_TIMED_LAUNCH(ctx, "snap_atom", k_chem_y<2>, grid, CY_WARPS * 32, 0, S, n, a0, nc, coef, Z, utot, yout,
                       epart, ntile, e0);
    else
      IPG_TIMED_LAUNCH(ctx, "snap_atom", k_chem_y<3>, grid, CY_WARPS * 32, 0, S, n, a0, nc, coef, Z, utot, yout,
                       epart, ntile, e0);
  }
  if (Ei)
    IPG_LAUNCH(ctx, k_chem_energy, (unsigned)((nc + 127) / 128), 128, 0, S, a0, nc, ntile, species, epart, Ei);
  return IPG_OK;
}
