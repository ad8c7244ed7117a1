// ipg_snap.cuh — SNAP tables and device-side descriptor of a SNAP basis.
#pragma once

#include "ipg_internal.cuh"

// One Z entry (one (j1, j2, j, ma, mb) of the idxz list, prebuilt_arrays.jl:183-216),
// with the start offsets of its CG double sum precomputed.
struct ZDev {
  int8_t j1, j2, j, na, nb, pad0, pad1, pad2;  // twojmax <= 12 bounds every index
  int8_t ma1min, ma2max, mb1min, mb2max;       // row/column starts of the two U factors
  int32_t u1base;  // idxu_block[j1] + (j1+1)*mb1min + ma1min
  int32_t u2base;  // idxu_block[j2] + (j2+1)*mb2max + ma2max
  int32_t icga0;   // ma1min*(j2+1) + ma2max
  int32_t icgb0;   // mb1min*(j2+1) + mb2max
  int32_t cgoff;   // idxcg_block[j1][j2][j]
};
static_assert(sizeof(ZDev) == 32, "ZDev is read as two 16-byte words");

// One bispectrum component (j1, j2, j) and the three half-plane sums of its
// derivative (compute_b.jl:207-400): level l[t], first Z index z0[t], factor fac[t].
struct DBDev {
  int32_t l[3];
  int32_t z0[3];
  double fac[3];
};

constexpr int SNAP_MAX_J = 12;
constexpr int YS_WARPS = 8;     // warps of the atoms-in-lanes Y kernels
constexpr int YS_ATOMS = 32;    // atoms per block of those kernels (one per lane)
constexpr int YR_MAX_J = 8;     // largest twojmax of the streamed Y / Z kernel

// Streamed Y / Z contraction (ipg_snap_y.cu): an item is the entries (k = -(2 mb - j), YT adjacent
// columns c = 2 ma - j) of every level j, jmin <= j <= J of its parity.  Its weights [row pair]
// [step][level][YT] follow one another in a stream of 16-byte units; a record is a run of row
// pairs of one (j1, j2), as many as fit YREC units.  Items, records and row pairs travel as a
// kernel parameter (constant bank), so that everything but the products runs on uniform registers.
constexpr int YT = 2;                  // columns per item
constexpr int YNJ = YR_MAX_J / 2 + 1;  // levels per item, at most
constexpr int YGUARD = 2;              // a row walk reads at most two entries past either end of a row
constexpr int YREC = 48;               // 16-byte units per record, at most
// record: row pairs (4 bits) | steps of each << 4 | levels << 8 | first of them << 11 | first, last
// record of its (j1, j2) << 14, 15 | size in units << 16 | first triple << 24
constexpr int YF_STEPS = 4, YF_N = 8, YF_LO = 11, YF_SIZE = 16, YF_TRIP = 24;
constexpr uint32_t YF_FIRST = 1u << 14, YF_LAST = 1u << 15;
// row pair: byte offsets, in the block's half plane, of the first element of row 1 and of the
// element of row 2 for column t = 0 (signed: it may lie before the row); bit 0: that row lies
// beyond the half plane
struct YkItem {
  int32_t unit;            // first unit of its weights
  int16_t rec, nrec, pair; // first record, records, first row pair
  int16_t k, c0, nt, jmin; // nt: columns in use
  int16_t pad;
};
constexpr int YK_ITEMS = 40, YK_RECS = 1200, YK_PAIRS = 2400;
struct YkTab {
  YkItem item[YK_ITEMS];  // longest first
  uint32_t rec[YK_RECS + 4];  // zero past the last: the walk looks two records ahead
  int2 pair[YK_PAIRS];
  int32_t nitem, pad;
};
constexpr int YM_Y = 0, YM_Z = 1, YM_YZ = 2;  // what launch_ystream writes

struct SnapDev {
  int J, nsp, K, idxu_max, idxz_max, u_half, ext_max, idxcg_max;
  int switch_flag, bzero_flag, bnorm_flag;
  int n_ytrip;  // streamed Y / Z: triples
  double rcutfac, rmin0, rfac0, wself;
  double radii[IPG_MAX_SNAP_SPECIES], weight[IPG_MAX_SNAP_SPECIES];
  int idxu_block[SNAP_MAX_J + 2];
  int half_block[SNAP_MAX_J + 2];
  double bzero[SNAP_MAX_J + 1];
  const double* rootpq;  // [(J+2)*(J+2)]
  const double* cglist;  // [idxcg_max]
  const ZDev* idxz;      // [idxz_max]
  const DBDev* db;       // [K]
  const int32_t* y_off;  // [u_half+1]  CSR: Z entries feeding each half-plane Y entry
  const int32_t* y_jjz;  // [idxz_max]
  const double* ycoef;   // [nsp][idxz_max] multiplicity * factor * beta (set per beta)
  const double* beta;    // [nsp][K]
  const int32_t* zperm;  // [idxz_max] Z entries ordered by loop shape (nb, na)
  // Y schedule of the atoms-in-lanes kernel: warp w owns half-plane entries
  // ysched_h[ysched_off[w] .. ysched_off[w+1]) (cost-balanced), ysched_w their weights
  const int32_t* ysched_off;  // [YS_WARPS+1]
  const int32_t* ysched_h;
  const double* ysched_w;
  const int32_t* u_of_h;      // [u_half] index of half-plane entry h in the full Utot
  const int32_t* h_info;      // [u_half] m | j << 8 | (m within the row's weighted entries) << 16, m = column ma
  const double2* h_sgen;      // [u_half] the generator factors (s_m, s_{m-1}), s_m = sqrt((m+1)(j-m)), 0 off the row
  const double2* ykstream;    // streamed Y / Z (twojmax <= YR_MAX_J): the weights
  const double* zfac;         // [idxz_max] 2 m(z) w of the dB/dr contraction
  const int32_t* ytrip_jjz;  // [n_ytrip] first Z entry of each triple
  const int32_t* ytrip_b;    // [n_ytrip] its component | the derivative terms it serves (bits 0-2) << 16
  const double* ytrip_fac;   // [n_ytrip] factor of each of those terms
  const int32_t* ylev;       // [J+2] offsets, then the triples of every level in order
  // explicit multi-element SNAP (chem_flag) and quadratic SNAP: K is then the number of
  // components per species block, klin of them linear (idxb_max per element triple), the rest
  // the products B_k B_l (k <= l) of quadratic_flag
  int chem, nelem, wselfall, literal_chem_z, quadratic, klin;
  const double* beta0;  // [1] energy offset of LBasisPotential (device, like ebias)
  const double* ebias;  // [nsp] -beta[s] . bzero (energy shift of bzero_flag), device memory so that
                        // a captured graph sees the beta of each replay
};

struct SnapHost {
  int J = 0, idxu_max = 0, idxz_max = 0, idxb_max = 0, idxcg_max = 0, u_half = 0, ext_max = 0;
  std::vector<int> idxu_block, half_block, idxcg_block, idxz_block, idxb_block;
  std::vector<int> idxb;  // 3 per component
  std::vector<ZDev> idxz;
  std::vector<int> zjju_half;  // half-plane index of each Z entry
  std::vector<DBDev> db;
  std::vector<double> cglist, rootpq, bzero;
  std::vector<int32_t> y_off, y_jjz;
  std::vector<int32_t> y_jjb;     // component whose beta scales each Z entry in Y
  std::vector<double> zfac;       // 2 y_mult, halved on the middle element of an even level
  std::vector<double> y_mult;     // multiplicity * (j1+1)/(j+1) factor of each Z entry
  std::vector<int32_t> zperm;     // Z entries sorted by (nb, na): equal trip counts per warp
  std::vector<int32_t> ysched_off, ysched_h, u_of_h, h_info;
  std::vector<double> h_sgen;  // 2 per half-plane entry
  std::vector<double> ysched_w;
  YkTab yktab;
  std::vector<double> ykstream;  // 2 per 16-byte unit
  std::vector<int32_t> ytrip_jjz, ytrip_b, ylev;
  std::vector<double> ytrip_fac;
};

int snap_build_tables(const ipg_snap_params& p, SnapHost& h);

struct ipg_ctx;
// Y' and E_i (YM_Y), Z (YM_Z) or both (YM_YZ) of n atoms from their Utot (ipg_snap_y.cu).
int launch_ystream(ipg_ctx* ctx, const SnapDev& dev, const YkTab& tab, int ym, const char* tname, int64_t n,
                   const int32_t* species, const double2* utot, double2* yout, double* Ei, double2* zout);
// Tangent of Y' along Udot = -V (V [u_half][n] as written by k_snap_vlie): ydot [u_half][n].
int launch_ytangent(ipg_ctx* ctx, const SnapDev& dev, const YkTab& tab, int64_t n, const int32_t* species,
                    const double2* utot, const double2* V, double2* ydot);
// Z of every ordered pair (p, q) of ne elements, zstride apart: the first factor of every product from
// element p's Utot, the second from q's (ustride apart).
int launch_zpairs(ipg_ctx* ctx, const SnapDev& dev, const YkTab& tab, int64_t n, const int32_t* species, int ne,
                  const double2* utot, int64_t ustride, double2* zout, int64_t zstride);
// Descriptor outputs from dbl [pair][K][3], the dB/dr of every pair (ipg_snap_desc.cu): dB
// [n][K nsp][3], or [3 n][K nsp] with rows; Wd [K nsp][6] of one configuration; the fitting rows
// Aw [nconf][6][K nsp] and Ae [nconf][K nsp] (from B [n][K]).  Any output may be null; the list
// transpose is read for dB only.
int launch_descriptors(ipg_ctx* ctx, int K, int nsp, int nconf, const int64_t* h_off, const PairList& pl,
                       const int32_t* species, const double* pos, const double* dbl, const double* B,
                       double* dB, bool rows, double* Wd, double* Aw, double* Ae);
// dB/dr of the pairs of owners b0 .. b1-1 (dbl [pair][K][3]) from their Z (atoms a0.., stride zs),
// and, with fvec, its contraction with the owner's beta (ipg_snap_db.cu).
int launch_db(ipg_ctx* ctx, const SnapDev& S, int64_t b0, int64_t b1, const PairList& pl, const int32_t* species,
              int64_t a0, int64_t zs, const double2* Z, double* dbl, double* fvec);
cudaError_t snapdb_upload_constants();
// Element-resolved and quadratic SNAP by the adjoint route (ipg_snap_chem.cu), twojmax <= YR_MAX_J.
// All of atoms a0 .. a0+nc-1: coef [nelem][nelem^2][n_ytrip][nc] is the weight of every Z triple of
// every element pair in the Y of every element.
int launch_chem_coef(ipg_ctx* ctx, const SnapDev& S, int64_t a0, int64_t nc, const int32_t* species, double* coef);
// Quadratic SNAP (one element): E_i and the coefficients from the linear B [n][klin].
int launch_quad_coef(ipg_ctx* ctx, const SnapDev& S, int64_t a0, int64_t nc, const int32_t* species, const double* B,
                     double* Ei, double* coef);
// Weighted Y' [u_half][n nelem] (atom-major elements) from Z [nelem^2][idxz_max][nc], and with
// Ei (element-resolved linear SNAP) the energies, from utot [nelem][n][idxu_max].
int launch_chem_y(ipg_ctx* ctx, const SnapDev& S, int64_t n, int64_t a0, int64_t nc, const int32_t* species,
                  const double* coef, const double2* Z, const double2* utot, double2* yout, double* Ei);
