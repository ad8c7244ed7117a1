// ipg_snap_db.cu — dB/dr of every pair from the register chains (twojmax <= YR_MAX_J), and its
// contraction with beta (compute_dbidrj, compute_b.jl:104-400; linear_potential.jl:20-49).
//
//   dB_i/dr_ij [b][k] = 2 sum_t fac_t sum_half w Re(conj(dU_ij,k) Z_i(t)).
//
// Every Z triple z belongs to one component jjb(z) with one multiplier m(z) (its coincidence
// count and, unnormalised, (j1+1)/(j+1)), the same pair the Y coefficients use, so
// dB[b][k] = 2 sum_{z: jjb(z) = b} m(z) sum_half w Re(conj(dU_k) Z_z).
//
// One block per owner atom, three warps, one lane per pair.  Warp k runs the chains of U alone and
// forms dU_k of each row by the generator identity (dU/dr = U times an su(2) generator,
// ipg_snap_chain.cuh); the rows of the three directions meet in shared memory (two buffers, one
// barrier per row), and warp g contracts all three with the owner's Z of the components
// b % 3 == g: a Z element, scaled by 2 m(z) w, is loaded once for six FMAs into 3 K / 3 register
// accumulators.  One loop over a row's elements holds the level's Z triples: unrolled over the
// elements too, the code would not fit the instruction cache.
//
// Bound by FP64 latency at six to nine warps per SM (FP64 pipe 37%, shared memory 47% at twojmax 8;
// the accumulators fill the registers).  16,000 atoms, twojmax 8: 1.90 ms, contraction with beta
// included, against 2.33 + 0.14 ms of a producer warp on the forward tangent chains with a consumer
// warp per direction and a separate contraction; a direction per warp with all K accumulators took
// 3.11 ms (each Z element loaded for two FMAs), a copy of the chains' code per warp 2.60 ms
// (instruction cache).  48 configurations, twojmax 6: 0.45 -> 0.29 ms.
#include "ipg_snap_chain.cuh"
#include "ipg_snap_geom.cuh"

namespace {

namespace plaintab {
constexpr int zrow_count(int j) { return (j / 2 + 1) * (j + 1); }
constexpr int imin(int a, int b) { return a < b ? a : b; }
constexpr int idxb_of(int J, int a, int b, int c) {
  int k = 0;
  for (int j1 = 0; j1 <= J; j1++)
    for (int j2 = 0; j2 <= j1; j2++)
      for (int j = j1 - j2; j <= imin(J, j1 + j2); j += 2)
        if (j >= j1) {
          if (j1 == a && j2 == b && j == c) return k;
          k++;
        }
  return -1;
}
constexpr int nb_of(int J) {
  int k = 0;
  for (int j1 = 0; j1 <= J; j1++)
    for (int j2 = 0; j2 <= j1; j2++)
      for (int j = j1 - j2; j <= imin(J, j1 + j2); j += 2)
        if (j >= j1) k++;
  return k;
}
constexpr int LMAX = 64;
struct Level {  // the Z triples (j1, j2, L) of level L
  int n = 0;
  int z0[LMAX] = {};   // first Z entry
  int jjb[LMAX] = {};  // component
};
constexpr Level level_of(int J, int L) {
  Level T;
  int z = 0;
  for (int j1 = 0; j1 <= J; j1++)
    for (int j2 = 0; j2 <= j1; j2++)
      for (int j = j1 - j2; j <= imin(J, j1 + j2); j += 2) {
        if (j == L && T.n < LMAX) {
          T.z0[T.n] = z;
          T.jjb[T.n] = j >= j1 ? idxb_of(J, j1, j2, j) : (j >= j2 ? idxb_of(J, j, j2, j1) : idxb_of(J, j2, j, j1));
          T.n++;
        }
        z += zrow_count(j);
      }
  return T;
}
}  // namespace plaintab


constexpr int DB_T = 96;  // three warps
// Resident blocks per SM that the registers are bounded for: at twojmax 8 the bound of three (168
// registers) spills and takes 2.56 ms at 16,000 atoms against 1.90; at 6 it does not.
constexpr int db_minb(int J) { return J > 6 ? 2 : 3; }
constexpr int DB_ROW = 3 * 32;  // elements of a row buffer per ma: [direction][lane]

// The three directions' element against the triples of level L whose component belongs to group G.
template <int J, int L, int G, int Q, int NQ, int NA>
__device__ __forceinline__ void db_dot(double (&acc)[NA][3], double2 d0, double2 d1, double2 d2,
                                       const double2* __restrict__ zr) {
  if constexpr (Q < NQ) {
    constexpr int z0 = plaintab::level_of(J, L).z0[Q], b = plaintab::level_of(J, L).jjb[Q];
    if constexpr (b % 3 == G) {
      const double2 z = zr[z0];
      acc[b / 3][0] = fma(d0.x, z.x, fma(d0.y, z.y, acc[b / 3][0]));
      acc[b / 3][1] = fma(d1.x, z.x, fma(d1.y, z.y, acc[b / 3][1]));
      acc[b / 3][2] = fma(d2.x, z.x, fma(d2.y, z.y, acc[b / 3][2]));
    }
    db_dot<J, L, G, Q + 1, NQ, NA>(acc, d0, d1, d2, zr);
  }
}

// The pair's side of a row: dU_k = A U + U (g1 D1 + g2 D2 + g3 D3) (as stage_vlie).
struct DbPair {
  double A, g1, g2, g3;
};

// Row mb of level j: this warp's direction into buffer vb, then the contraction of all three.
template <int J, int j, int NA>
__device__ __forceinline__ void db_row(const snapchain::ChainU<J>& s, const DbPair& P, int mb, double2* rows,
                                       int& parity, const double2* zo, double (&acc)[NA][3]) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double2* buf = rows + parity * (J + 1) * DB_ROW;
  double2* vb = buf + threadIdx.x;
  parity ^= 1;
  const int last = (2 * mb == j) ? mb : j;
#pragma unroll
  for (int ma = 0; ma <= j; ma++) {
    if (ma > last) break;
    const double2 u = s.u[ma];
    const double c1 = P.g1 * (double)(j - 2 * ma);  // i u = (-u.y, u.x)
    double vx = fma(P.A, u.x, -(c1 * u.y)), vy = fma(P.A, u.y, c1 * u.x);
    if (ma > 0) {  // s_{ma-1} (g2 + i g3) u[ma-1]
      const double sg = snapchain::c_sgen[(j * snapchain::SGEN_ROWS + mb) * snapchain::RPQ_STRIDE + ma - 1];
      const double2 w = s.u[ma - 1];
      const double px = sg * P.g2, py = sg * P.g3;
      vx = fma(px, w.x, fma(-py, w.y, vx));
      vy = fma(px, w.y, fma(py, w.x, vy));
    }
    if (ma < j) {  // s_ma (-g2 + i g3) u[ma+1]
      const double sg = snapchain::c_sgen[(j * snapchain::SGEN_ROWS + mb) * snapchain::RPQ_STRIDE + ma];
      const double2 w = s.u[ma + 1];
      const double px = -sg * P.g2, py = sg * P.g3;
      vx = fma(px, w.x, fma(-py, w.y, vx));
      vy = fma(px, w.y, fma(py, w.x, vy));
    }
    vb[ma * DB_ROW] = make_double2(vx, vy);
  }
  // a buffer is written again two rows later, after the barrier of the row between, which every
  // warp reaches only when it is done with this one
  __syncthreads();
  constexpr int NQ = plaintab::level_of(J, j).n;
  const double2* zr = zo + mb * (j + 1);
  const double2* r = buf + lane;
  if (warp == 0) {
#pragma unroll 1
    for (int ma = 0; ma <= last; ma++, r += DB_ROW) db_dot<J, j, 0, 0, NQ, NA>(acc, r[0], r[32], r[64], zr + ma);
  } else if (warp == 1) {
#pragma unroll 1
    for (int ma = 0; ma <= last; ma++, r += DB_ROW) db_dot<J, j, 1, 0, NQ, NA>(acc, r[0], r[32], r[64], zr + ma);
  } else {
#pragma unroll 1
    for (int ma = 0; ma <= last; ma++, r += DB_ROW) db_dot<J, j, 2, 0, NQ, NA>(acc, r[0], r[32], r[64], zr + ma);
  }
}

template <int J, int j, int NA>
__device__ __forceinline__ void db_level(snapchain::ChainU<J>& s, double2 a, double2 b, const DbPair& P, int mb,
                                         double2* rows, int& parity, double2 (&sv)[J + 1], const double2* zo,
                                         double (&acc)[NA][3]) {
  if constexpr (j <= J) {
    snapchain::advance_u_rt<J, j>(s, a, b, mb);
    db_row<J, j, NA>(s, P, mb, rows, parity, zo, acc);
    if constexpr (j % 2 == 1 && (j + 1) / 2 <= J / 2) {
      if (j == 2 * mb + 1) {  // start row of chain mb+1: the mirror of this row
        constexpr int R = (j + 1) / 2;
#pragma unroll
        for (int c = 0; c <= j; c++) {
          const double sg = ((c + R) & 1) ? -1.0 : 1.0;
          sv[c] = make_double2(sg * s.u[j - c].x, -sg * s.u[j - c].y);
        }
      }
    }
  }
}

// A warp's part of a pass over 32 pairs: every row, then (bt) its share of beta . dbl into
// fp [group][direction][lane], and its components of pairs 16 h .. 16 h + 15 into the tile ob.
// Every warp meets the same barriers: one per row, two per output tile.
template <int J>
__device__ __forceinline__ void db_pass(double2 a, double2 b, const DbPair& P, double2* rows, const double2* zo,
                                        const double* __restrict__ bt, double* fp, double* ob, int64_t p0, int64_t pe,
                                        double* __restrict__ dbl, double* __restrict__ fvec) {
  constexpr int NB = plaintab::nb_of(J), NA = (NB + 2) / 3;
  const int lane = threadIdx.x & 31, G = threadIdx.x >> 5;
  double acc[NA][3];
#pragma unroll
  for (int q = 0; q < NA; q++) acc[q][0] = acc[q][1] = acc[q][2] = 0.0;
  snapchain::ChainU<J> s;
  double2 sv[J + 1];
#pragma unroll
  for (int c = 0; c <= J; c++) s.u[c] = sv[c] = make_double2(0.0, 0.0);
  s.u[0] = make_double2(1.0, 0.0);
  int parity = 0;
  db_row<J, 0, NA>(s, P, 0, rows, parity, zo, acc);
#pragma unroll 1
  for (int mb = 0; mb <= J / 2; mb++) {
    if (mb > 0) {
#pragma unroll
      for (int c = 0; c <= J; c++)
        if (c < 2 * mb) s.u[c] = sv[c];
    }
    switch (mb == 0 ? 1 : 2 * mb) {  // chain mb runs levels 2mb (1 for chain 0) .. J
#define IPG_LEVEL(JJ) \
  case JJ:            \
    db_level<J, JJ, NA>(s, a, b, P, mb, rows, parity, sv, zo, acc);
      IPG_LEVEL(1) IPG_LEVEL(2) IPG_LEVEL(3) IPG_LEVEL(4) IPG_LEVEL(5) IPG_LEVEL(6) IPG_LEVEL(7) IPG_LEVEL(8)
#undef IPG_LEVEL
      default:
        break;
    }
  }
  if (bt) {
    double f[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int q = 0; q < NA; q++)
      if (3 * q + G < NB)
#pragma unroll
        for (int k = 0; k < 3; k++) f[k] = fma(bt[3 * q + G], acc[q][k], f[k]);
#pragma unroll
    for (int k = 0; k < 3; k++) fp[(G * 3 + k) * 32 + lane] = f[k];
  }
  for (int h = 0; h < 2; h++) {
    __syncthreads();
    if (h == 0 && bt && p0 + lane < pe)  // direction G of the pair: the groups in order
      fvec[3 * (p0 + lane) + G] = (fp[G * 32 + lane] + fp[(3 + G) * 32 + lane]) + fp[(6 + G) * 32 + lane];
    if ((lane >> 4) == h) {
#pragma unroll
      for (int q = 0; q < NA; q++)
        if (3 * q + G < NB)
#pragma unroll
          for (int k = 0; k < 3; k++) ob[(lane & 15) * (3 * NB) + 3 * (3 * q + G) + k] = acc[q][k];
    }
    __syncthreads();
    const int64_t q0 = p0 + 16 * h, left = pe - q0;
    const int m = left <= 0 ? 0 : (int)(left < 16 ? left : 16) * 3 * NB;
    for (int x = threadIdx.x; x < m; x += DB_T) dbl[(size_t)q0 * 3 * NB + x] = ob[x];
  }
}

// dbl[p][b][k] of the pairs of owners b0 .. b0 + gridDim.x - 1, their Z in the chunk of atoms
// a0.. (stride zs); fvec (optional): [p][k] = beta of the owner . dbl[p].
template <int J>
__global__ void __launch_bounds__(DB_T, db_minb(J)) k_snap_db(const __grid_constant__ SnapDev S, int64_t b0,
                                                     const int64_t* __restrict__ off,
                                                     const int32_t* __restrict__ nbr,
                                                     const double* __restrict__ rij,
                                                     const int32_t* __restrict__ species, int64_t a0, int64_t zs,
                                                     const double2* __restrict__ Z, double* __restrict__ dbl,
                                                     double* __restrict__ fvec) {
  static_assert(J <= YR_MAX_J, "twojmax <= 8");
  constexpr int NB = plaintab::nb_of(J);
  // the transposed output of 16 pairs shares the row buffers' space
  static_assert(16 * 3 * NB * 8 <= 2 * (J + 1) * DB_ROW * 16, "the output tile fits the row buffers");
  extern __shared__ __align__(16) unsigned char fsm[];
  double2* rows = reinterpret_cast<double2*>(fsm);  // [2][J+1][DB_ROW]
  double2* zo = rows + 2 * (J + 1) * DB_ROW;        // [idxz_max] the owner's Z, scaled
  __shared__ double fp[3 * 3 * 32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t o = b0 + blockIdx.x;
  const int64_t pb = off[o], pe = off[o + 1];
  if (pb == pe) return;  // block-uniform
  for (int z = threadIdx.x; z < S.idxz_max; z += DB_T) {
    const double2* src = Z + (size_t)z * zs + (o - a0);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(zo + z)),
                 "l"(src));
  }
  asm volatile("cp.async.commit_group;");
  const int si = clamp_sp(species[o], S.nsp);
  const double* bt = fvec ? S.beta + (size_t)si * S.K : nullptr;
  for (int64_t p0 = pb; p0 < pe; p0 += 32) {
    const int64_t p = p0 + lane;
    double2 a = make_double2(1.0, 0.0), b = make_double2(0.0, 0.0);  // idle lanes: zero weights
    DbPair P = {0.0, 0.0, 0.0, 0.0};
    if (p < pe) {
      const int sj = clamp_sp(species[nbr[p]], S.nsp);
      const double rcut = (S.radii[si] + S.radii[sj]) * S.rcutfac;
      PairGeom G;
      geom_du(S, rij[3 * p], rij[3 * p + 1], rij[3 * p + 2], rcut, S.weight[sj], G);
      a = G.a;
      b = G.b;
      const double2 da = warp == 0 ? G.da[0] : (warp == 1 ? G.da[1] : G.da[2]);
      const double2 db = warp == 0 ? G.db[0] : (warp == 1 ? G.db[1] : G.db[2]);
      P.A = G.dsfac * (warp == 0 ? G.u[0] : (warp == 1 ? G.u[1] : G.u[2]));
      P.g1 = G.sfac * (a.y * da.x - a.x * da.y + b.x * db.y - b.y * db.x);  // Im(a conj(da) + conj(b) db)
      P.g2 = G.sfac * (b.x * da.x + b.y * da.y - a.x * db.x - a.y * db.y);  // Re(conj(b) da - a conj(db))
      P.g3 = G.sfac * (b.x * da.y - b.y * da.x - a.y * db.x + a.x * db.y);  // Im(conj(b) da - a conj(db))
    }
    if (p0 == pb) {  // the owner's Z is here: scale what this thread copied
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      for (int z = threadIdx.x; z < S.idxz_max; z += DB_T) {
        const double f = S.zfac[z];
        const double2 v = zo[z];
        zo[z] = make_double2(f * v.x, f * v.y);
      }
    }
    __syncthreads();  // Z is scaled; the last pass's output tile is read
    double* ob = reinterpret_cast<double*>(fsm);
    db_pass<J>(a, b, P, rows, zo, bt, fp, ob, p0, pe, dbl, fvec);
  }
}

template <int J>
int launch_db_j(ipg_ctx* ctx, const SnapDev& S, int64_t b0, int64_t b1, const PairList& pl, const int32_t* species,
                int64_t a0, int64_t zs, const double2* Z, double* dbl, double* fvec) {
  if (plaintab::nb_of(J) != S.K) return ipg_fail(ctx, IPG_ERR_UNSUPPORTED, "plain chain tables disagree");
  const int sm = (int)((2 * (J + 1) * DB_ROW + (size_t)S.idxz_max) * sizeof(double2));
  IPG_RET(ipg_smem_limit(ctx, k_snap_db<J>, sm));
  IPG_TIMED_LAUNCH(ctx, "snap_dbfused", k_snap_db<J>, (unsigned)(b1 - b0), DB_T, sm, S, b0, pl.d_off, pl.d_j, pl.d_r,
                   species, a0, zs, Z, dbl, fvec);
  return IPG_OK;
}

}  // namespace

cudaError_t snapdb_upload_constants() { return snapchain::upload_constants(); }

int launch_db(ipg_ctx* ctx, const SnapDev& S, int64_t b0, int64_t b1, const PairList& pl, const int32_t* species,
              int64_t a0, int64_t zs, const double2* Z, double* dbl, double* fvec) {
  if (b1 <= b0) return IPG_OK;
  switch (S.J) {
#define IPG_J(JJ) \
  case JJ:        \
    return launch_db_j<JJ>(ctx, S, b0, b1, pl, species, a0, zs, Z, dbl, fvec);
    IPG_J(0) IPG_J(1) IPG_J(2) IPG_J(3) IPG_J(4) IPG_J(5) IPG_J(6) IPG_J(7) IPG_J(8)
#undef IPG_J
    default:
      return IPG_ERR_UNSUPPORTED;
  }
}
