// ipg_pair.cu — fused multi-term empirical pair potentials.
//
// Replaces, for every term of a LinearCombinationPotential at once, the per-term
// neighbor build + pair loop of src/types/empirical_potential.jl:20-67 with one pass over
// the cell list at the largest cutoff, each term keeping its own cutoff (PeriodicEuclidean
// distance <= rcut_t, as the term's own neighbor list would) and species filter (both
// species in the term's set, empirical_potential.jl:26-43).
//
// Half-stencil tiles (k_pair_half).  Like the reference's half list (nnlist.jl:39-40, m > n),
// every unordered pair is evaluated once.  A work item is a (home cell A, offset k) pair,
// one warp each: k = 0 is A itself (pairs of slots s < s'), k = 1..13 the 13 neighbor cells
// of the forward half of the 27-cell stencil.  Lanes own the atoms of the target cell, the warp
// walks the home cell's atoms one row at a time, the pairs that can be within the largest cutoff
// are queued in (row, lane) order, and every 32 of them are evaluated by the whole warp.  The
// force of each pair goes to its two atoms' owner lanes, which add the pairs of a batch in queue
// order, so every sum runs in a fixed order (no atomics).  A warp writes its row sums and column
// sums to its own slots of a partial-force buffer, [14 home offsets + 13 target offsets][slot][3],
// which k_pair_finish sums per atom in a fixed order.  Each pair's force term is the reference's:
// with lo < hi the atom ids, r = get_displacement(x_lo, x_hi) (nnlist.jl:18-21), f = g(R) r,
// F_lo += f, F_hi -= f; only the order of summation differs.
//
// Only one candidate in eight is within the cutoff, so the row walk tests them in 32 bits on
// cell-relative positions: with at least 3 cells on every periodic axis a pair within the cutoff
// is at the image that its two cells define, so no minimum image is needed, and the test's
// threshold covers the rounding of the 32-bit coordinates (prefilter_threshold).  It only
// proposes; the reference's own test and all arithmetic of the pairs it proposes are 64-bit.
//
// The half stencil visits each pair of neighboring cells once only when every periodic axis
// has at least 3 cells; otherwise the full-stencil walk (ipg_pair.cuh) runs instead.
#include "ipg_pair.cuh"

namespace {

constexpr int PAIR_T = 128;
constexpr int PAIR_WARPS = PAIR_T / 32;

// The full-stencil walk, one warp per atom (the fallback for grids with fewer than 3 cells
// on a periodic axis).
__global__ void __launch_bounds__(PAIR_T) k_pair_eval(const __grid_constant__ PairTerms TT, int64_t n,
                                                      const ConfGrid* __restrict__ grid,
                                                      const int64_t* __restrict__ cell_start,
                                                      const int32_t* __restrict__ cell_atoms,
                                                      const double4* __restrict__ spos, double* __restrict__ F,
                                                      double* __restrict__ partial) {
  __shared__ PairHit hits[PAIR_WARPS][64];
  __shared__ double red[PAIR_WARPS][7];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t s = (int64_t)blockIdx.x * PAIR_WARPS + w;
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};  // E, W[6]
  if (s < n) pair_walk_atom(TT, grid[0], cell_start, cell_atoms, spos, s, hits[w], lane, acc, F);  // warp-uniform
#pragma unroll
  for (int k = 0; k < 7; k++) {
    const double v = warp_sum(acc[k]);
    if (lane == 0) red[w][k] = v;
  }
  __syncthreads();
  if (threadIdx.x < 7) {
    double v = 0.0;
    for (int q = 0; q < PAIR_WARPS; q++) v += red[q][threadIdx.x];
    partial[(int64_t)blockIdx.x * 7 + threadIdx.x] = v;
  }
}

// ---------------------------------------------------------------------------------
// Half-stencil tiles.
constexpr int HALF_OFFSETS = 14;  // self + 13 forward neighbors
constexpr int PBUF_SLOTS = 27;    // partial forces per atom: 14 as a home atom, 13 as a target

// Offset k of the half stencil: 0 = (0,0,0); 1..13 = the (dx,dy,dz) with dz > 0, or dz = 0
// and dy > 0, or dz = dy = 0 and dx > 0.
__device__ __forceinline__ void half_offset(int k, int& dx, int& dy, int& dz) {
  if (k == 0) {
    dx = dy = dz = 0;
  } else if (k == 1) {
    dx = 1, dy = 0, dz = 0;
  } else if (k <= 4) {
    dx = k - 3, dy = 1, dz = 0;  // k = 2, 3, 4 -> dx = -1, 0, 1
  } else {
    const int q = k - 5;  // 0..8
    dx = q % 3 - 1, dy = q / 3 - 1, dz = 1;
  }
}

// Cell coordinate c + d along an axis of nc cells: wrapped on a periodic axis (nc >= 3 there,
// so c + d stays a distinct cell), -1 when it leaves an open axis.
__device__ __forceinline__ int shift_axis(int c, int d, int nc, bool periodic) {
  int t = c + d;
  if (periodic) return t < 0 ? t + nc : (t >= nc ? t - nc : t);
  return (t < 0 || t >= nc) ? -1 : t;
}

struct PairBox {
  double L[3];  // box lengths, by value: the constant bank instead of registers
};

// Per-warp shared memory of the half-stencil walk.
struct HalfWarp {
  double f[3][32];     // the forces of a batch
  double col[3][32];   // column sums of the tile
  float4 home[32];     // the rows' cell-relative positions
  int rows[32];        // per row: first pair of the batch that belongs to it | their count << 8
  uint16_t q[96];      // queued pairs, row | column << 8
};

// get_displacement (nnlist.jl:18-21) along an axis when |dx| < L (disp_axis_dev's result).
__device__ __forceinline__ double disp_near(double L, double dx) {
  if (isinf(L)) return dx;
  const double d = dx < 0.0 ? __dadd_rn(dx, L) : (dx == 0.0 ? 0.0 : dx);
  return __dmul_rn(2.0, d) < L ? d : __dsub_rn(d, L);
}

// Evaluates the first nh queued pairs (one per lane) and hands each pair's force to its row
// owner (fa += f) and its column's sum (-= f).  E and W accumulate lane-wise.
//
// The hand-off, in queue order: a row's pairs are contiguous, so its owner lane adds a run of the
// batch's forces; a column's pairs take turns by their rank among the pairs of that column (a match
// over the lanes), each turn touching a column at most once.  About nine and four short steps a
// batch, all with warp-uniform trip counts.
__device__ __forceinline__ void half_eval(const PairTerms& TT, const PairBox& B, int nh, int lane, int row0, int col0,
                                          const int32_t* __restrict__ cell_atoms, const double4* __restrict__ spos,
                                          HalfWarp& st, double* acc, double* fa) {
  constexpr unsigned FULL = 0xffffffffu;
  const bool act = lane < nh;
  const int e = act ? st.q[lane] : 0;  // idle lanes: the first row and column, and no force
  const int row = e & 0xff, col = e >> 8;
  const double4 xa = spos[row0 + row], xt = spos[col0 + col];
  // r = get_displacement(x_lo, x_hi) seen from the row atom
  const bool lo = cell_atoms[row0 + row] < cell_atoms[col0 + col];
  const double x0 = __dsub_rn(xa.x, xt.x), x1 = __dsub_rn(xa.y, xt.y), x2 = __dsub_rn(xa.z, xt.z);
  double d2, r0, r1, r2;
  if (__all_sync(FULL, fabs(x0) < B.L[0] && fabs(x1) < B.L[1] && fabs(x2) < B.L[2])) {
    const double a0 = fabs(x0), a1 = fabs(x1), a2 = fabs(x2);  // PeriodicEuclidean (an open axis has L = inf)
    d2 = sumsq3_dev(fmin(a0, __dsub_rn(B.L[0], a0)), fmin(a1, __dsub_rn(B.L[1], a1)), fmin(a2, __dsub_rn(B.L[2], a2)));
    r0 = disp_near(B.L[0], lo ? x0 : -x0);
    r1 = disp_near(B.L[1], lo ? x1 : -x1);
    r2 = disp_near(B.L[2], lo ? x2 : -x2);
  } else {  // a separation of a box length or more
    d2 = sumsq3_dev(pe_axis_dev(B.L[0], xa.x, xt.x), pe_axis_dev(B.L[1], xa.y, xt.y), pe_axis_dev(B.L[2], xa.z, xt.z));
    r0 = disp_axis_dev(B.L[0], lo ? xa.x : xt.x, lo ? xt.x : xa.x);
    r1 = disp_axis_dev(B.L[1], lo ? xa.y : xt.y, lo ? xt.y : xa.y);
    r2 = disp_axis_dev(B.L[2], lo ? xa.z : xt.z, lo ? xt.z : xa.z);
  }
  double V, g;
  pair_terms_sum_warp(TT, act, r0 * r0 + r1 * r1 + r2 * r2, d2, (int)xa.w, (int)xt.w, V, g);
  if (!act) r0 = r1 = r2 = 0.0;
  const double gs = lo ? g : -g;  // the row atom's force is along r for lo, against it otherwise
  const double fx = gs * r0, fy = gs * r1, fz = gs * r2;
  acc[0] += V;
  // empirical_potential.jl:63-64: r * f' -> [xx, yy, zz, zy, zx, yx]
  const double hx = g * r0, hy = g * r1, hz = g * r2;
  acc[1] += r0 * hx;
  acc[2] += r1 * hy;
  acc[3] += r2 * hz;
  acc[4] += r2 * hy;
  acc[5] += r2 * hx;
  acc[6] += r1 * hx;
  st.f[0][lane] = fx;
  st.f[1][lane] = fy;
  st.f[2][lane] = fz;
  st.rows[lane] = 0;
  const int key = act ? row : 64;
  const int prev = __shfl_up_sync(FULL, key, 1);
  const unsigned heads = __ballot_sync(FULL, lane == 0 || key != prev);  // first pair of each row, first idle lane
  const unsigned same = __match_any_sync(FULL, act ? col : 32 + lane);
  const int rank = __popc(same & ((1u << lane) - 1u));
  __syncwarp();
  int len = 0;
  if (act && ((heads >> lane) & 1u)) {
    const unsigned above = heads & (0xfffffffeu << lane);  // later heads
    len = (above ? __ffs(above) - 1 : 32) - lane;          // idle lanes start a run of their own
    st.rows[row] = lane | len << 8;
  }
  const int turns = (int)__reduce_max_sync(FULL, (unsigned)rank) + 1;
  const int longest = (int)__reduce_max_sync(FULL, (unsigned)len);
  for (int k = 0; k < turns; k++) {
    if (act && rank == k) {
      st.col[0][col] -= fx;
      st.col[1][col] -= fy;
      st.col[2][col] -= fz;
    }
    __syncwarp();
  }
  const int run = st.rows[lane], n = run >> 8;
  const double* f = &st.f[0][run & 0xff];
  for (int k = 0; k < longest; k++, f++) {
    if (k < n) {
      fa[0] += f[0];
      fa[1] += f[32];
      fa[2] += f[64];
    }
  }
  __syncwarp();
}

__device__ __forceinline__ void pbuf_put(double* __restrict__ P, int64_t n, int slot_kind, int64_t s, const double* f,
                                         bool accumulate) {
  double* q = P + 3 * ((int64_t)slot_kind * n + s);
  if (accumulate) {
    q[0] += f[0];
    q[1] += f[1];
    q[2] += f[2];
  } else {
    q[0] = f[0];
    q[1] = f[1];
    q[2] = f[2];
  }
}

// Bound by issue slots (61% at a million atoms, the FP64 pipe 25%, DRAM 2%) and the latency of dependent
// instructions (2.9 cycles an issue waiting); at 32,000 atoms also by the wait for the last warps (issue 50%
// of the active cycles).  Full 64-bit tests of every candidate, rows
// loaded one by one and a hand-off between two warp barriers a row took 35.8 ms a call at 4.1 M atoms
// with five terms; 32-bit tests and masked hand-offs 17.7 ms; warp-uniform control flow in
// half_eval (terms, cutoffs, distances, hand-off: lane-wise branches cost reconvergence around
// each) 15.2 ms.  32,000 atoms: 540, 309, 273 us; 1,000 atoms, one term: 92, 70, 67 us.
// PAIR_MINB: resident blocks per SM the register allocation is bounded for; 3, 4, 5, 6 (164, 128,
// 96, 80 registers) took 18.9, 15.7, 15.2, 15.2 ms at 4.1 M atoms, 323, 275, 273, 281 us at 32,000
// and 66.8, 66.1, 67.1, 69.0 us at 1,000.
constexpr int PAIR_MINB = 5;
__global__ void __launch_bounds__(PAIR_T, PAIR_MINB) k_pair_half(const __grid_constant__ PairTerms TT,
                                                                 const __grid_constant__ PairBox B, int64_t n,
                                                                 const ConfGrid* __restrict__ grid, int64_t ncells,
                                                                 const int64_t* __restrict__ cell_start,
                                                                 const int32_t* __restrict__ cell_atoms,
                                                                 const double4* __restrict__ spos,
                                                                 const float4* __restrict__ srel, float thr,
                                                                 double* __restrict__ P,
                                                                 double* __restrict__ partial) {
  __shared__ HalfWarp stage[PAIR_WARPS];
  __shared__ double red[PAIR_WARPS][7];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  HalfWarp& st = stage[w];
  double acc[7] = {0, 0, 0, 0, 0, 0, 0};  // E, W[6] of every item this warp takes
  // grid-stride over the items (a fixed assignment, so E and W sum in a fixed order); the
  // block's warps meet at a barrier only once, at the end
  const int64_t nitems = ncells * HALF_OFFSETS;
  const int64_t wstride = (int64_t)gridDim.x * PAIR_WARPS;
  for (int64_t item = (int64_t)blockIdx.x * PAIR_WARPS + w; item < nitems; item += wstride) {  // warp-uniform
    const ConfGrid& g = grid[0];
    // cells and atoms number below 2^31: 32-bit index arithmetic
    const int A = (int)(item / HALF_OFFSETS);
    const int k = (int)(item - (int64_t)A * HALF_OFFSETS);
    const int nxy = g.nc[0] * g.nc[1];
    const int cz = A / nxy, rem = A - cz * nxy;
    const int cy = rem / g.nc[0], cx = rem - cy * g.nc[0];
    int dx, dy, dz;
    half_offset(k, dx, dy, dz);
    const int tx = shift_axis(cx, dx, g.nc[0], !isinf(B.L[0]));
    const int ty = shift_axis(cy, dy, g.nc[1], !isinf(B.L[1]));
    const int tz = shift_axis(cz, dz, g.nc[2], !isinf(B.L[2]));
    if (tx < 0 || ty < 0 || tz < 0) continue;
    const int T = (tz * g.nc[1] + ty) * g.nc[0] + tx;
    const int a0 = (int)cell_start[A], a1 = (int)cell_start[A + 1], t0 = (int)cell_start[T],
              t1 = (int)cell_start[T + 1];
    // the target cell's corner relative to the home cell's, at the image these two cells define
    const float sx = dx * g.edge[0], sy = dy * g.edge[1], sz = dz * g.edge[2];
    const int home_kind = k, tgt_kind = k == 0 ? 0 : HALF_OFFSETS - 1 + k;
    // cells of at most 32 atoms are one tile and its sums are stored; larger cells take
    // several tiles, whose sums accumulate into zeroed slots, as do the row and column sums
    // of the home cell with itself (each slot is always written by the same lane, in tile
    // order)
    const bool multi = (a1 - a0 > 32) || (t1 - t0 > 32) || k == 0;
    if (multi) {
      const double z[3] = {0.0, 0.0, 0.0};
      for (int s = a0 + lane; s < a1; s += 32) pbuf_put(P, n, home_kind, s, z, false);
      if (k != 0)
        for (int s = t0 + lane; s < t1; s += 32) pbuf_put(P, n, tgt_kind, s, z, false);
      __syncwarp();
    }
    if (a0 == a1 && k != 0)  // no home atoms: the target atoms still get their (zero) slot
      for (int s = t0 + lane; s < t1; s += 32) {
        const double z[3] = {0.0, 0.0, 0.0};
        pbuf_put(P, n, tgt_kind, s, z, false);
      }
    const unsigned lt = (1u << lane) - 1u;
    for (int rc = a0; rc < a1; rc += 32) {
      const int ra = a1 - rc < 32 ? a1 - rc : 32;
      double fa[3] = {0.0, 0.0, 0.0};  // row sums of row rc + lane
      __syncwarp();
      if (lane < ra) st.home[lane] = srel[rc + lane];
      for (int cc = t0; cc < t1; cc += 32) {
        const int ts = cc + lane;
        const bool tv = ts < t1;
        const float4 b = tv ? srel[ts] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        const float bx = b.x + sx, by = b.y + sy, bz = b.z + sz;
        // a cell with itself: the rows before the lane's own slot; another cell: every row
        const int lim = !tv ? 0 : (k == 0 && ts - rc < ra ? ts - rc : ra);
        st.col[0][lane] = st.col[1][lane] = st.col[2][lane] = 0.0;
        int nh = 0;
        __syncwarp();
        for (int q = 0; q < ra + 2; q += 2) {  // the last step evaluates what is left
          if (q < ra) {
#pragma unroll
            for (int u = 0; u < 2; u++) {
              const float4 a = st.home[(q + u) & 31];  // past the last row: any value, lim excludes it
              const float x = a.x - bx, y = a.y - by, z = a.z - bz;
              const bool ok = fmaf(x, x, fmaf(y, y, z * z)) <= thr && q + u < lim;
              const unsigned bal = __ballot_sync(0xffffffffu, ok);
              if (ok) st.q[nh + __popc(bal & lt)] = (uint16_t)((q + u) | (lane << 8));
              nh += __popc(bal);
            }
            __syncwarp();
          }
          // one call site of the term code: full batches, then the rest after the last row
          while (nh >= 32 || (q >= ra && nh > 0)) {
            const int m = nh < 32 ? nh : 32;
            half_eval(TT, B, m, lane, rc, cc, cell_atoms, spos, st, acc, fa);
            uint16_t e0 = 0, e1 = 0;  // the rest of the queue (fewer than 64 pairs) moves up
            if (lane < nh - m) e0 = st.q[m + lane];
            if (lane + 32 < nh - m) e1 = st.q[m + lane + 32];
            __syncwarp();
            if (lane < nh - m) st.q[lane] = e0;
            if (lane + 32 < nh - m) st.q[lane + 32] = e1;
            nh -= m;
            __syncwarp();
          }
        }
        if (tv) {
          const double ft[3] = {st.col[0][lane], st.col[1][lane], st.col[2][lane]};
          pbuf_put(P, n, tgt_kind, ts, ft, multi);
        }
        __syncwarp();
      }
      if (lane < ra) pbuf_put(P, n, home_kind, rc + lane, fa, multi);
      __syncwarp();
    }
  }
#pragma unroll
  for (int q = 0; q < 7; q++) {
    const double v = warp_sum(acc[q]);
    if (lane == 0) red[w][q] = v;
  }
  __syncthreads();
  if (threadIdx.x < 7) {
    double v = 0.0;
    for (int q = 0; q < PAIR_WARPS; q++) v += red[q][threadIdx.x];
    partial[(int64_t)blockIdx.x * 7 + threadIdx.x] = v;
  }
}

// E and W6 from the per-block partials of nblocks blocks in a fixed order (one block of
// FINISH_T threads); component 0 goes to E, 1..6 to W6 (either may be null).
constexpr int FINISH_T = 256;
__device__ __forceinline__ void reduce_partials(int64_t nblocks, const double* __restrict__ partial,
                                                double* __restrict__ E, double* __restrict__ W6) {
  __shared__ double sm[FINISH_T / 32][7];
  double v[7] = {0, 0, 0, 0, 0, 0, 0};
  for (int64_t b = threadIdx.x; b < nblocks; b += FINISH_T)
#pragma unroll
    for (int k = 0; k < 7; k++) v[k] += partial[b * 7 + k];
#pragma unroll
  for (int k = 0; k < 7; k++) {
    v[k] = warp_sum(v[k]);
    if ((threadIdx.x & 31) == 0) sm[threadIdx.x >> 5][k] = v[k];
  }
  __syncthreads();
  if (threadIdx.x < 7) {
    double s = 0.0;
    for (int q = 0; q < FINISH_T / 32; q++) s += sm[q][threadIdx.x];
    if (threadIdx.x == 0 && E) *E = s;
    if (threadIdx.x > 0 && W6) W6[threadIdx.x - 1] = s;
  }
}

__global__ void __launch_bounds__(FINISH_T) k_reduce_partials(int64_t nblocks, const double* __restrict__ partial,
                                                              double* __restrict__ E, double* __restrict__ W6) {
  reduce_partials(nblocks, partial, E, W6);
}

// F of every atom: its 14 partial sums as a home atom (offsets k whose target cell exists)
// and its 13 as a target (offsets k whose home cell, its own cell - offset k, exists), in
// that fixed order; the loads are independent of one another, so they are in flight together.
// The last block reduces E and W6 instead, beside the gather.
__global__ void __launch_bounds__(FINISH_T) k_pair_finish(int64_t n, const ConfGrid* __restrict__ grid,
                                                          const int32_t* __restrict__ cell_atoms,
                                                          const double4* __restrict__ spos,
                                                          const double* __restrict__ P, double* __restrict__ F,
                                                          int64_t nblocks, const double* __restrict__ partial,
                                                          double* __restrict__ E, double* __restrict__ W6) {
  if (blockIdx.x == gridDim.x - 1) {
    reduce_partials(nblocks, partial, E, W6);
    return;
  }
  const int64_t s = (int64_t)blockIdx.x * FINISH_T + threadIdx.x;
  if (s >= n) return;
  const ConfGrid& g = grid[0];
  const double4 x = spos[s];
  int c[3];
  cell_coords(g, x.x, x.y, x.z, c);
  unsigned in[3];  // bit d + 1: the cell at offset d along the axis exists
#pragma unroll
  for (int a = 0; a < 3; a++) {
    const bool per = !isinf(g.L[a]);
    in[a] = 2u | (per || c[a] > 0 ? 1u : 0u) | (per || c[a] + 1 < g.nc[a] ? 4u : 0u);
  }
  double f0 = 0.0, f1 = 0.0, f2 = 0.0;
#pragma unroll
  for (int kind = 0; kind < PBUF_SLOTS; kind++) {
    const int k = kind < HALF_OFFSETS ? kind : kind - (HALF_OFFSETS - 1);
    const int sg = kind < HALF_OFFSETS ? 1 : -1;
    int d[3];
    half_offset(k, d[0], d[1], d[2]);
    const bool ok = (in[0] >> (1 + sg * d[0])) & (in[1] >> (1 + sg * d[1])) & (in[2] >> (1 + sg * d[2])) & 1u;
    const double* q = P + 3 * ((int64_t)kind * n + s);
    if (ok) {
      f0 += q[0];
      f1 += q[1];
      f2 += q[2];
    }
  }
  const int64_t i = cell_atoms[s];
  F[3 * i] = f0;
  F[3 * i + 1] = f1;
  F[3 * i + 2] = f2;
}

int prepare_terms(ipg_ctx* ctx, const ipg_pair_term* terms, int nterms, PairTerms& pt) {
  char err[256];
  const int st = pair_prepare_terms(terms, nterms, pt, err, sizeof(err));
  return st == IPG_OK ? IPG_OK : ipg_fail(ctx, st, "%s", err);
}

int pair_eval_device(ipg_ctx* ctx, int64_t n, const double* d_pos, const int32_t* d_species, const double L[3],
                     const ipg_pair_term* terms, int32_t nterms, double* d_E, double* d_F, double* d_W6,
                     uint32_t flags, std::vector<ConfGrid>* grid_out = nullptr) {
  PairTerms pt;
  IPG_RET(prepare_terms(ctx, terms, nterms, pt));
  IPG_RET(ipg_status_reset(ctx));
  int64_t aoff[2] = {0, n};
  CellList cl;
  IPG_RET(ipg_build_cells(ctx, "pair_", n, d_pos, d_species, 64, 1, aoff, L, pt.rcut_max, cl));
  if (grid_out) *grid_out = cl.h_grid;
  const ConfGrid& g = cl.h_grid[0];
  bool half = n > 0 && !ctx->pair_full_stencil;
  for (int a = 0; a < 3; a++) half &= std::isinf(g.L[a]) || g.nc[a] >= 3;
  double* partial;
  int64_t nb;
  double* Eo = (flags & IPG_WANT_E) ? d_E : nullptr;
  double* Wo = (flags & IPG_WANT_W) ? d_W6 : nullptr;
  const bool want_f = (flags & IPG_WANT_F) && d_F;
  IPG_RET(ipg_timing_mark(ctx, "pair_eval", true));
  if (half) {
    const int64_t items = cl.ncells * HALF_OFFSETS;
    // Grid-stride over the items: a block costs its start, its reduction and the wait for its slowest
    // warp, so it takes several items a warp, but no fewer blocks than fill the GPU once; large systems
    // take up to 16 waves, which even out the cells.  Against four waves at most: 32,000 atoms (18,000
    // items) 274 -> 241 us with six items a warp, 261 with three; 4.1 M atoms 15.2 -> 14.8 ms.
    const int64_t one = (items + PAIR_WARPS - 1) / PAIR_WARPS, wave = (int64_t)ctx->num_sms * PAIR_MINB;
    nb = std::max<int64_t>(1, std::min(one, std::max(wave, std::min(one / 6, 16 * wave))));
    const PairBox box = {{g.L[0], g.L[1], g.L[2]}};
    double* P;
    IPG_RET(scratch(ctx, "pair_partial", (size_t)nb * 7, &partial));
    IPG_RET(scratch(ctx, "pair_pbuf", (size_t)PBUF_SLOTS * 3 * n, &P));
    IPG_LAUNCH(ctx, k_pair_half, (unsigned)nb, PAIR_T, 0, pt, box, n, cl.d_grid, cl.ncells, cl.d_cell_start,
               cl.d_cell_atoms, cl.d_spos, cl.d_srel, prefilter_threshold(g, pt.rcut_max), P, partial);
    if (want_f)
      IPG_LAUNCH(ctx, k_pair_finish, (unsigned)((n + FINISH_T - 1) / FINISH_T + 1), FINISH_T, 0, n, cl.d_grid,
                 cl.d_cell_atoms, cl.d_spos, P, d_F, nb, partial, Eo, Wo);
  } else {
    nb = std::max<int64_t>(1, (n + PAIR_WARPS - 1) / PAIR_WARPS);
    IPG_RET(scratch(ctx, "pair_partial", (size_t)nb * 7, &partial));
    IPG_LAUNCH(ctx, k_pair_eval, (unsigned)nb, PAIR_T, 0, pt, n, cl.d_grid, cl.d_cell_start, cl.d_cell_atoms,
               cl.d_spos, want_f ? d_F : nullptr, partial);
  }
  IPG_RET(ipg_timing_mark(ctx, "pair_eval", false));
  if (!half || !want_f) IPG_LAUNCH(ctx, k_reduce_partials, 1, FINISH_T, 0, nb, partial, Eo, Wo);
  return IPG_OK;
}

// ---- CUDA graphs of the device evaluation (IPG_PAIR_GRAPH) --------------------------------
ipg_ctx::PairGraph* pair_graph_find(ipg_ctx* ctx, int64_t n, const double* d_pos, const int32_t* d_species,
                                    const double L[3], const ipg_pair_term* terms, int32_t nterms,
                                    const double* d_E, const double* d_F, const double* d_W6, uint32_t flags) {
  const size_t tb = sizeof(ipg_pair_term) * (size_t)nterms;
  for (auto& g : ctx->pair_graphs)
    if (g.n == n && g.L[0] == L[0] && g.L[1] == L[1] && g.L[2] == L[2] && g.pos == d_pos && g.sp == d_species &&
        g.E == d_E && g.F == d_F && g.W6 == d_W6 && g.flags == flags && g.terms.size() == tb &&
        memcmp(g.terms.data(), terms, tb) == 0 && g.full_stencil == (int)ctx->pair_full_stencil)
      return &g;
  return nullptr;
}

// Uploads the cell grid the graph reads and launches it; IPG_ERR_NOT_CAPTURED when there is
// no usable graph (none for this key, or a scratch buffer moved since the capture).
int pair_graph_replay(ipg_ctx* ctx, int64_t n, const double* d_pos, const int32_t* d_species, const double L[3],
                      const ipg_pair_term* terms, int32_t nterms, double* d_E, double* d_F, double* d_W6,
                      uint32_t flags) {
  ipg_ctx::PairGraph* g = pair_graph_find(ctx, n, d_pos, d_species, L, terms, nterms, d_E, d_F, d_W6, flags);
  if (!g) return IPG_ERR_NOT_CAPTURED;
  ConfGrid* d_grid = nullptr;
  if (g->gen == ctx->scratch_gen) IPG_RET(scratch(ctx, "pair_grid", 1, &d_grid));
  if (g->gen != ctx->scratch_gen) {
    cudaGraphExecDestroy(g->exec);
    ctx->pair_graphs.erase(ctx->pair_graphs.begin() + (g - ctx->pair_graphs.data()));
    return IPG_ERR_NOT_CAPTURED;
  }
  CUDA_RET(ctx, cudaMemcpyAsync(d_grid, g->grid.data(), g->grid.size(), cudaMemcpyHostToDevice, ctx->stream));
  IPG_RET(ipg_status_reset(ctx));
  CUDA_RET(ctx, cudaGraphLaunch(g->exec, ctx->stream));
  ctx->pair_graph_replays++;
  return ipg_status_check(ctx, "ipg_pair_eval_dev (graph)");
}

// Captures the evaluation just run eagerly with the same inputs (every scratch buffer already
// has its size).  A failure only means that later calls run eagerly.
void pair_graph_capture(ipg_ctx* ctx, int64_t n, const double* d_pos, const int32_t* d_species, const double L[3],
                        const ipg_pair_term* terms, int32_t nterms, double* d_E, double* d_F, double* d_W6,
                        uint32_t flags) {
  if (ctx->pair_graphs.size() >= 8) {
    cudaGraphExecDestroy(ctx->pair_graphs.front().exec);
    ctx->pair_graphs.erase(ctx->pair_graphs.begin());
  }
  ipg_ctx::PairGraph g;
  g.n = n;
  for (int a = 0; a < 3; a++) g.L[a] = L[a];
  g.pos = d_pos;
  g.sp = d_species;
  g.E = d_E;
  g.F = d_F;
  g.W6 = d_W6;
  g.flags = flags;
  g.terms.assign(reinterpret_cast<const char*>(terms), reinterpret_cast<const char*>(terms) + sizeof(ipg_pair_term) * nterms);
  g.full_stencil = ctx->pair_full_stencil;
  const uint64_t gen0 = ctx->scratch_gen;
  std::vector<ConfGrid> grid;
  const bool timing = ctx->timing;
  ctx->timing = false;
  ctx->capturing = true;
  cudaGraph_t graph = nullptr;
  int st = IPG_OK;
  if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeRelaxed) != cudaSuccess) {
    st = IPG_ERR_CUDA;
  } else {
    st = pair_eval_device(ctx, n, d_pos, d_species, L, terms, nterms, d_E, d_F, d_W6, flags, &grid);
    cudaError_t e = cudaStreamEndCapture(ctx->stream, &graph);
    if (st == IPG_OK && e != cudaSuccess) st = IPG_ERR_CUDA;
  }
  ctx->capturing = false;
  ctx->timing = timing;
  if (st == IPG_OK && graph && ctx->scratch_gen == gen0 && grid.size() == 1 &&
      cudaGraphInstantiate(&g.exec, graph, 0) == cudaSuccess) {
    g.grid.assign(reinterpret_cast<const char*>(grid.data()), reinterpret_cast<const char*>(grid.data() + 1));
    g.gen = ctx->scratch_gen;
    ctx->pair_graphs.push_back(std::move(g));
  }
  if (graph) cudaGraphDestroy(graph);
  cudaGetLastError();  // a failed capture leaves no sticky error behind
}

int check_pair_args(ipg_ctx* ctx, int64_t n, const void* pos, const void* species, const double* L,
                    const ipg_pair_term* terms, int32_t nterms, const void* E, const void* F, const void* W6,
                    uint32_t flags) {
  if (!ctx) return IPG_ERR_ARG;
  if (n < 0 || n >= INT32_MAX) return ipg_fail(ctx, IPG_ERR_ARG, "n out of range");
  if ((n > 0 && (!pos || !species)) || !L || (nterms > 0 && !terms))
    return ipg_fail(ctx, IPG_ERR_ARG, "null input pointer");
  if ((flags & IPG_WANT_E) && !E) return ipg_fail(ctx, IPG_ERR_ARG, "E requested but NULL");
  if ((flags & IPG_WANT_F) && !F && n > 0) return ipg_fail(ctx, IPG_ERR_ARG, "F requested but NULL");
  if ((flags & IPG_WANT_W) && !W6) return ipg_fail(ctx, IPG_ERR_ARG, "W6 requested but NULL");
  return IPG_OK;
}

}  // namespace

extern "C" {

int ipg_pair_eval(ipg_ctx* ctx, int64_t n, const double* pos, const int32_t* species, const double L[3],
                  const ipg_pair_term* terms, int32_t nterms, double* E, double* F, double* W6, uint32_t flags) {
  IPG_RET(check_pair_args(ctx, n, pos, species, L, terms, nterms, E, F, W6, flags));
  CUDA_RET(ctx, cudaSetDevice(ctx->device));
  if (!host_all_finite(pos, 3 * n)) return ipg_fail(ctx, IPG_ERR_NONFINITE, "non-finite position");
  if (!host_species_ok(species, n, 64)) return ipg_fail(ctx, IPG_ERR_SPECIES, "species id out of range 0..63");
  double *d_pos, *d_out;
  int32_t* d_sp;
  IPG_RET(scratch(ctx, "pair_in_pos", 3 * (size_t)n + 3, &d_pos));
  IPG_RET(scratch(ctx, "pair_in_sp", (size_t)n + 1, &d_sp));
  IPG_RET(scratch(ctx, "pair_out", 3 * (size_t)n + 8, &d_out));
  if (n) {
    IPG_RET(ipg_copy_h2d(ctx, d_pos, pos, sizeof(double) * 3 * n));
    IPG_RET(ipg_copy_h2d(ctx, d_sp, species, sizeof(int32_t) * n));
  }
  // d_out layout: [E, W6 (6), pad, F (3n)]
  IPG_RET(pair_eval_device(ctx, n, d_pos, d_sp, L, terms, nterms, d_out, d_out + 8, d_out + 1,
                           flags | IPG_WANT_E | IPG_WANT_W));
  std::vector<double> head(8);
  CUDA_RET(ctx, cudaMemcpyAsync(head.data(), d_out, sizeof(double) * 8, cudaMemcpyDeviceToHost, ctx->stream));
  if ((flags & IPG_WANT_F) && n) IPG_RET(ipg_copy_d2h(ctx, F, d_out + 8, sizeof(double) * 3 * n));
  IPG_RET(ipg_status_check(ctx, "ipg_pair_eval"));
  if (flags & IPG_WANT_E) *E = head[0];
  if (flags & IPG_WANT_W) memcpy(W6, head.data() + 1, 6 * sizeof(double));
  return IPG_OK;
}

int ipg_pair_eval_dev(ipg_ctx* ctx, int64_t n, const double* d_pos, const int32_t* d_species, const double L[3],
                      const ipg_pair_term* terms, int32_t nterms, double* d_E, double* d_F, double* d_W6,
                      uint32_t flags) {
  IPG_RET(check_pair_args(ctx, n, d_pos, d_species, L, terms, nterms, d_E, d_F, d_W6, flags));
  CUDA_RET(ctx, cudaSetDevice(ctx->device));
  const bool want_graph = (flags & IPG_PAIR_GRAPH) && n > 0 && !std::isinf(L[0]) && !std::isinf(L[1]) &&
                          !std::isinf(L[2]);
  flags &= IPG_WANT_E | IPG_WANT_F | IPG_WANT_W;
  if (want_graph) {
    const int st = pair_graph_replay(ctx, n, d_pos, d_species, L, terms, nterms, d_E, d_F, d_W6, flags);
    if (st != IPG_ERR_NOT_CAPTURED) return st;
  }
  IPG_RET(pair_eval_device(ctx, n, d_pos, d_species, L, terms, nterms, d_E, d_F, d_W6, flags));
  IPG_RET(ipg_status_check(ctx, "ipg_pair_eval_dev"));
  if (want_graph) pair_graph_capture(ctx, n, d_pos, d_species, L, terms, nterms, d_E, d_F, d_W6, flags);
  return IPG_OK;
}

}  // extern "C"
