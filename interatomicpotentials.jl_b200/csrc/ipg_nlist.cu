// ipg_nlist.cu — cell-list neighbor build (replaces the BallTree + PeriodicEuclidean
// search of src/nnlist.jl:23-46 and src/BasisSystems/SNAP/utilities/utl.jl:38-101).
//
// Pipeline (all on the context's stream):
//   k_extent       per-configuration min/max of open axes (only when an axis is open)
//   k_cell_count   cell id per atom + histogram; the histogram's old value is the atom's arrival
//   scan           cell_start
//   k_cell_fill    atom ids into their cells, in arrival order
//   k_cell_place   each atom's rank among its cell's ids (deterministic slot order): cell_atoms,
//                  spos
//   k_cells_small  all of these in one block, for few atoms and cells
// and, for a materialised list:
//   k_pair_count / scan / k_pair_emit / k_pair_sort, optionally the transpose.
// Membership is decided per candidate with the reference's own arithmetic
// (PeriodicEuclidean distance, get_displacement), so any cell edge >= the search radius
// proposes every pair exactly once.
#include <algorithm>

#include "ipg_internal.cuh"

namespace {

__global__ void k_extent(const double* __restrict__ pos, const ConfGrid* __restrict__ grid, double* __restrict__ ext) {
  // one block per configuration; ext[c*6 + a] = min, ext[c*6 + 3 + a] = max
  const ConfGrid g = grid[blockIdx.x];
  __shared__ double smin[3][32], smax[3][32];
  double mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
  for (int64_t i = threadIdx.x; i < g.natoms; i += blockDim.x) {
    const double* p = pos + 3 * (g.atom_off + i);
#pragma unroll
    for (int a = 0; a < 3; a++) {
      mn[a] = fmin(mn[a], p[a]);
      mx[a] = fmax(mx[a], p[a]);
    }
  }
#pragma unroll
  for (int a = 0; a < 3; a++)
    for (int o = 16; o > 0; o >>= 1) {
      mn[a] = fmin(mn[a], __shfl_xor_sync(0xffffffffu, mn[a], o));
      mx[a] = fmax(mx[a], __shfl_xor_sync(0xffffffffu, mx[a], o));
    }
  int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0)
    for (int a = 0; a < 3; a++) {
      smin[a][w] = mn[a];
      smax[a][w] = mx[a];
    }
  __syncthreads();
  if (threadIdx.x < 3) {
    int a = threadIdx.x;
    double m = INFINITY, M = -INFINITY;
    for (int q = 0; q < (int)(blockDim.x >> 5); q++) {
      m = fmin(m, smin[a][q]);
      M = fmax(M, smax[a][q]);
    }
    ext[blockIdx.x * 6 + a] = m;
    ext[blockIdx.x * 6 + 3 + a] = M;
  }
}

// The configuration and cell of atom i (out of range or non-finite inputs are reported and
// placed in some cell).
__device__ __forceinline__ int64_t cell_of_atom(int64_t i, const double* __restrict__ pos,
                                                const int32_t* __restrict__ species, int nsp,
                                                const ConfGrid* __restrict__ grid, int nconf, int* conf,
                                                int* status) {
  // configuration by binary search over atom offsets
  int lo = 0, hi = nconf - 1;
  while (lo < hi) {
    int mid = (lo + hi + 1) >> 1;
    if (grid[mid].atom_off <= i) lo = mid;
    else hi = mid - 1;
  }
  const ConfGrid& g = grid[lo];
  double x = pos[3 * i], y = pos[3 * i + 1], z = pos[3 * i + 2];
  if (!isfinite(x) || !isfinite(y) || !isfinite(z)) {
    dev_raise(status, IPG_ERR_NONFINITE);
    x = y = z = 0.0;
  }
  if (species && (species[i] < 0 || species[i] >= nsp)) dev_raise(status, IPG_ERR_SPECIES);
  int c[3];
  cell_coords(g, x, y, z, c);
  *conf = lo;
  return g.cell_off + ((int64_t)c[2] * g.nc[1] + c[1]) * g.nc[0] + c[0];
}

// Atom i of cell c (of grid g) into slot s of the cell order; srel receives its position
// relative to the cell's lower corner (in units of g.rel), and its id in w.
__device__ __forceinline__ void place_atom(int32_t i, int64_t s, const ConfGrid& g, int64_t c,
                                           const double* __restrict__ pos, const int32_t* __restrict__ species,
                                           int nsp, int32_t* __restrict__ cell_atoms,
                                           double4* __restrict__ spos, float4* __restrict__ srel) {
  cell_atoms[s] = i;
  int sp = species ? species[i] : 0;
  sp = sp < 0 ? 0 : (sp > nsp - 1 ? nsp - 1 : sp);  // bad ids were reported with the cell
  const double x = pos[3 * (int64_t)i], y = pos[3 * (int64_t)i + 1], z = pos[3 * (int64_t)i + 2];
  spos[s] = make_double4(x, y, z, (double)sp);
  const int k = (int)(c - g.cell_off), nxy = g.nc[0] * g.nc[1];
  const int cz = k / nxy, cy = (k - cz * nxy) / g.nc[0], cx = k - cz * nxy - cy * g.nc[0];
  srel[s] = make_float4((float)((cell_wrap(g, 0, x) - cx * g.cs[0]) * g.rel),
                        (float)((cell_wrap(g, 1, y) - cy * g.cs[1]) * g.rel),
                        (float)((cell_wrap(g, 2, z) - cz * g.cs[2]) * g.rel), __int_as_float(i));
}

__global__ void k_cell_count(int64_t n, const double* __restrict__ pos, const int32_t* __restrict__ species, int nsp,
                             const ConfGrid* __restrict__ grid, int nconf, int32_t* __restrict__ conf,
                             int32_t* __restrict__ cell_of, int32_t* __restrict__ arrival,
                             int64_t* __restrict__ count, int* status) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int c;
  const int64_t cell = cell_of_atom(i, pos, species, nsp, grid, nconf, &c, status);
  conf[i] = c;
  cell_of[i] = (int32_t)cell;
  arrival[i] = (int32_t)atomicAdd((unsigned long long*)&count[cell], 1ull);
}

__global__ void k_cell_fill(int64_t n, const int32_t* __restrict__ cell_of, const int32_t* __restrict__ arrival,
                            const int64_t* __restrict__ cell_start, int32_t* __restrict__ unsorted) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  unsorted[cell_start[cell_of[i]] + arrival[i]] = (int32_t)i;
}

// One thread per atom: its slot is its cell's start plus its rank among the cell's ids, so the
// slots are ascending inside a cell whatever the arrival order.  A sort by one thread per cell
// was a serial chain of loads: 58 us at 32,000 atoms (about 25 per cell), 13 us at 8,192 in cells of
// 14; this kernel, which also writes what a separate gather wrote, takes 5.4 and 5.0 us.
__global__ void __launch_bounds__(128) k_cell_place(int64_t n, const int32_t* __restrict__ unsorted,
                                                    const int32_t* __restrict__ cell_of,
                                                    const int64_t* __restrict__ cell_start,
                                                    const ConfGrid* __restrict__ grid,
                                                    const int32_t* __restrict__ conf,
                                                    const double* __restrict__ pos,
                                                    const int32_t* __restrict__ species, int nsp,
                                                    int32_t* __restrict__ cell_atoms,
                                                    double4* __restrict__ spos, float4* __restrict__ srel) {
  const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  const int32_t i = unsorted[t];
  const int64_t c = cell_of[i], s0 = cell_start[c], s1 = cell_start[c + 1];
  int64_t rank = 0;
#pragma unroll 8
  for (int64_t q = s0; q < s1; q++) rank += unsorted[q] < i;
  place_atom(i, s0 + rank, grid[conf[i]], c, pos, species, nsp, cell_atoms, spos, srel);
}

// The whole cell list in one block (count, scan, fill, rank, place through shared memory), for
// at most SMALL_ATOMS atoms and SMALL_CELLS cells: there the five launches it replaces cost more
// than one SM's work: 6.3 us against 39 us of kernels and two clears at 1,000 atoms.
constexpr int SMALL_T = 1024;
constexpr int SMALL_ATOMS = 4 * SMALL_T, SMALL_CELLS = 4 * SMALL_T;
__global__ void __launch_bounds__(SMALL_T) k_cells_small(int n, int ncells, const double* __restrict__ pos,
                                                         const int32_t* __restrict__ species, int nsp,
                                                         const ConfGrid* __restrict__ grid, int nconf,
                                                         int32_t* conf, int64_t* __restrict__ cell_start,
                                                         int32_t* __restrict__ cell_atoms,
                                                         double4* __restrict__ spos,
                                                         float4* __restrict__ srel, int* status) {
  __shared__ int start[SMALL_CELLS + 1];
  __shared__ int32_t unsorted[SMALL_ATOMS];
  __shared__ int wsum[SMALL_T / 32];
  constexpr int PER = SMALL_ATOMS / SMALL_T, CPER = SMALL_CELLS / SMALL_T;
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  for (int c = t; c <= ncells; c += SMALL_T) start[c] = 0;
  __syncthreads();
  int cell[PER], arr[PER];
#pragma unroll
  for (int q = 0; q < PER; q++) {
    const int i = q * SMALL_T + t;
    cell[q] = 0;
    arr[q] = 0;
    if (i < n) {
      int cf;
      cell[q] = (int)cell_of_atom(i, pos, species, nsp, grid, nconf, &cf, status);
      conf[i] = cf;
      arr[q] = atomicAdd(&start[cell[q]], 1);
    }
  }
  __syncthreads();
  // exclusive scan of the counts, CPER consecutive cells per thread
  int v[CPER], run = 0;
#pragma unroll
  for (int q = 0; q < CPER; q++) {
    const int c = CPER * t + q;
    v[q] = run;
    run += c < ncells ? start[c] : 0;
  }
  int incl = run;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += u;
  }
  if (lane == 31) wsum[w] = incl;
  __syncthreads();
  if (w == 0) {
    int u = wsum[lane];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, u, o);
      if (lane >= o) u += x;
    }
    wsum[lane] = u;
  }
  __syncthreads();
  const int excl = incl - run + (w > 0 ? wsum[w - 1] : 0);
#pragma unroll
  for (int q = 0; q < CPER; q++) {
    const int c = CPER * t + q;
    if (c < ncells) {
      start[c] = excl + v[q];
      cell_start[c] = excl + v[q];
    }
  }
  if (t == 0) {
    start[ncells] = n;
    cell_start[ncells] = n;
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < PER; q++)
    if (q * SMALL_T + t < n) unsorted[start[cell[q]] + arr[q]] = q * SMALL_T + t;
  __syncthreads();
#pragma unroll
  for (int q = 0; q < PER; q++) {
    const int i = q * SMALL_T + t;
    if (i >= n) continue;
    const int s0 = start[cell[q]], s1 = start[cell[q] + 1];
    int rank = 0;
    for (int k = s0; k < s1; k++) rank += unsorted[k] < i;
    place_atom(i, s0 + rank, grid[conf[i]], cell[q], pos, species, nsp, cell_atoms, spos, srel);
  }
}

// ---------------------------------------------------------------------------------
// Pair tests.  HALF: nnlist.jl:39-44.  FULL: utl.jl:81-93.
struct PairTest {
  int mode;          // IPG_NLIST_HALF / IPG_NLIST_FULL
  int literal;       // utl.jl:81 literal search radius
  int nsp;
  double rcut;       // HALF: cutoff; FULL: candidate radius (cutmax or sqrt(cutmax))
  double rcut2_lo, rcut2_hi;  // rcut^2 (1 -/+ 1e-12)
  double cutsq[64];  // FULL: [nsp][nsp], nsp <= 8
};

// Returns true when (i, j) belongs to the list; r receives the stored displacement.
__device__ __forceinline__ bool pair_ok(const PairTest& t, const double* L, int32_t i, double4 xi, int32_t j,
                                        double4 xj, double* r) {
  if (t.mode == IPG_NLIST_HALF) {
    if (j <= i) return false;
  } else if (j == i) {
    return false;
  }
  double s0 = pe_axis_dev(L[0], xi.x, xj.x);
  double s1 = pe_axis_dev(L[1], xi.y, xj.y);
  double s2 = pe_axis_dev(L[2], xi.z, xj.z);
  // sqrt(d2) <= rcut decided exactly; the squared bounds (1e-12 relative margin, far
  // above the rounding of sqrt and of rcut^2) settle all but the boundary cases
  const double d2 = sumsq3_dev(s0, s1, s2);
  if (d2 > t.rcut2_hi) return false;
  if (d2 >= t.rcut2_lo && sqrt(d2) > t.rcut) return false;
  r[0] = disp_axis_dev(L[0], xi.x, xj.x);
  r[1] = disp_axis_dev(L[1], xi.y, xj.y);
  r[2] = disp_axis_dev(L[2], xi.z, xj.z);
  if (t.mode == IPG_NLIST_HALF) return true;
  r[0] = -r[0];
  r[1] = -r[1];
  r[2] = -r[2];
  double rsq = sumsq3_dev(r[0], r[1], r[2]);
  return rsq <= t.cutsq[(int)xi.w * t.nsp + (int)xj.w];
}

// One warp per atom (cell-sorted order): lanes take consecutive candidates of each
// stencil range (coalesced), ballots count the members, and the emit pass writes them
// in candidate order (ballot prefix), so the list is deterministic.
template <bool EMIT>
__global__ void __launch_bounds__(128) k_pair_walk(int64_t n, PairTest t, const ConfGrid* __restrict__ grid,
                                                   const int32_t* __restrict__ conf,
                                                   const int64_t* __restrict__ cell_start,
                                                   const int32_t* __restrict__ cell_atoms,
                                                   const double4* __restrict__ spos, int64_t* __restrict__ cnt,
                                                   const int64_t* __restrict__ off, int32_t* __restrict__ outj,
                                                   double* __restrict__ outr) {
  const int lane = threadIdx.x & 31;
  const int64_t s = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (s >= n) return;  // warp-uniform
  const int32_t i = cell_atoms[s];
  const double4 xi = spos[s];
  const ConfGrid g = grid[conf[i]];
  int c[3];
  cell_coords(g, xi.x, xi.y, xi.z, c);
  StencilRanges R;
  stencil_ranges(g, c, cell_start, R);
  int64_t k = 0;
  const int64_t base = EMIT ? off[i] : 0;
  const int64_t end = EMIT ? off[i + 1] : 0;
  const unsigned lt = (1u << lane) - 1u;
  for (int r = 0; r < R.n; r++)
    for (int64_t q0 = R.beg[r]; q0 < R.end[r]; q0 += 32) {
      const int64_t q = q0 + lane;
      double rr[3];
      bool ok = false;
      if (q < R.end[r]) ok = pair_ok(t, g.L, i, xi, cell_atoms[q], spos[q], rr);
      const unsigned bal = __ballot_sync(0xffffffffu, ok);
      if (EMIT && ok) {
        const int64_t o = base + k + __popc(bal & lt);
        if (o < end) {  // a list cut at the capacity (capacity mode) drops its tail
          outj[o] = cell_atoms[q];
          outr[3 * o] = rr[0];
          outr[3 * o + 1] = rr[1];
          outr[3 * o + 2] = rr[2];
        }
      }
      k += __popc(bal);
    }
  if (!EMIT && lane == 0) cnt[i] = k;
}

// Verlet-skin reuse: the pairs of a list built with enlarged cutoffs that satisfy the true
// test (pair_ok, the same arithmetic as a fresh build) at the current positions.  One warp
// per atom, lanes over its cached candidates, emission in the cached order.
template <bool EMIT>
__global__ void __launch_bounds__(128) k_filter_walk(int64_t n, PairTest t, const ConfGrid* __restrict__ grid,
                                                     const int32_t* __restrict__ conf,
                                                     const int64_t* __restrict__ coff,
                                                     const int32_t* __restrict__ cj, const double* __restrict__ pos,
                                                     const int32_t* __restrict__ species, int nsp,
                                                     int64_t* __restrict__ cnt, const int64_t* __restrict__ off,
                                                     int32_t* __restrict__ outj, double* __restrict__ outr,
                                                     int* __restrict__ status) {
  const int lane = threadIdx.x & 31;
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= n) return;  // warp-uniform
  // ids are clamped so every table read stays in bounds; an id out of range is an error
  if (!EMIT && lane == 0 && species && (species[i] < 0 || species[i] >= nsp)) dev_raise(status, IPG_ERR_SPECIES);
  const int si = species ? (species[i] < 0 ? 0 : (species[i] >= nsp ? nsp - 1 : species[i])) : 0;
  const double4 xi = make_double4(pos[3 * i], pos[3 * i + 1], pos[3 * i + 2], (double)si);
  const double* L = grid[conf[i]].L;
  int64_t k = 0;
  const int64_t base = EMIT ? off[i] : 0;
  const unsigned lt = (1u << lane) - 1u;
  for (int64_t q0 = coff[i]; q0 < coff[i + 1]; q0 += 32) {
    const int64_t q = q0 + lane;
    double rr[3];
    bool ok = false;
    int32_t j = 0;
    if (q < coff[i + 1]) {
      j = cj[q];
      const int sj = species ? (species[j] < 0 ? 0 : (species[j] >= nsp ? nsp - 1 : species[j])) : 0;
      ok = pair_ok(t, L, (int32_t)i, xi, j, make_double4(pos[3 * j], pos[3 * j + 1], pos[3 * j + 2], (double)sj), rr);
    }
    const unsigned bal = __ballot_sync(0xffffffffu, ok);
    if (EMIT && ok) {
      const int64_t o = base + k + __popc(bal & lt);
      outj[o] = j;
      outr[3 * o] = rr[0];
      outr[3 * o + 1] = rr[1];
      outr[3 * o + 2] = rr[2];
    }
    k += __popc(bal);
  }
  if (!EMIT && lane == 0) cnt[i] = k;
}

// Largest squared minimum-image displacement since the reference positions, as the bit
// pattern of a non-negative double (ordered like the integers).  A non-finite position, or a
// species id that differs from the one at the build, counts as an infinite move, so the
// caller rebuilds the list (and the fresh build reports the bad input).
__global__ void k_max_disp2(int64_t n, const ConfGrid* __restrict__ grid, const int32_t* __restrict__ conf,
                            const double* __restrict__ pos, const double* __restrict__ ref,
                            const int32_t* __restrict__ species, const int32_t* __restrict__ ref_species,
                            unsigned long long* __restrict__ out) {
  __shared__ unsigned long long sm[256];
  double m = 0.0;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const double* L = grid[conf[i]].L;
    double d2 = 0.0;
    for (int a = 0; a < 3; a++) {
      const double s = pe_axis_dev(L[a], pos[3 * i + a], ref[3 * i + a]);
      d2 += s * s;
    }
    if (!(d2 <= 1.7976931348623157e308)) d2 = INFINITY;  // NaN or Inf: never reuse
    if (species && ref_species && species[i] != ref_species[i]) d2 = INFINITY;
    m = fmax(m, d2);
  }
  sm[threadIdx.x] = (unsigned long long)__double_as_longlong(m);
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if ((int)threadIdx.x < o) sm[threadIdx.x] = sm[threadIdx.x] > sm[threadIdx.x + o] ? sm[threadIdx.x] : sm[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicMax(out, sm[0]);
}

// Capacity mode: a total above cap is an error (status), and every offset is cut at cap
// so that all later kernels stay inside the buffers.
// (Offsets are non-decreasing, so cutting each one at cap on its own is the same as
// cutting the lists; no thread reads another's offset.)  So is, in the padded walk (kcap > 0), an
// atom with more hits than slots.
__global__ void k_clamp_offsets(int64_t n, int64_t* __restrict__ off, int64_t cap, const int* __restrict__ maxcnt,
                                int kcap, int* __restrict__ status) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0 && kcap > 0 && *maxcnt > kcap) atomicExch(status, IPG_ERR_CAPACITY);
  if (i > n) return;
  if (off[i] > cap) {
    if (i == n) atomicExch(status, IPG_ERR_CAPACITY);
    off[i] = cap;
  }
}

// The same walk by cells: every atom of a cell has the same stencil, so a warp takes a group of
// 32 >> split atoms of a cell, loads each chunk of 32 candidates once and tests it against every
// atom of the group, in two phases.  Phase 1 applies a test that is false only when pair_ok is,
// WALK_ILP atoms at a time so that their chains overlap, and queues the (atom, candidate) pairs
// that pass in (atom, lane) order in a per-warp ring.  Phase 2 runs the full pair_ok on 32 queued
// pairs at a time, one per lane, and emits the members after each atom's running count (shared
// memory).  One test in eight passes: with the member path inside the chunk loop, the few members
// of a chunk made every lane run it.  Each atom's hits come out in candidate order, as from
// k_pair_walk: lane k of the warp holds the k-th cell of the stencil in that order, and the chunks
// run through the cells' atoms end to end (walk_chunk), the next one loading while the present
// one is tested.
//
// Phase 1 tests in 32 bits on cell-relative positions where the grid allows it (REL: the walk's
// radius within the cells', at least 3 cells on every periodic axis, so that a pair within the
// radius is at the image that its two cells define; the threshold covers the rounding,
// prefilter_threshold), and otherwise as pair_ok does: the periodic distance against the radius,
// with the same arithmetic; a separation of a box length or more is left to the full test.
//
// Bound by latency (a cell is a serial chain of chunks) and, in the 64-bit test, FP64 issue.  Against
// one warp a cell, ranges listed serially, no loads ahead and the 64-bit test only: 345 -> 315 us a
// call at 8,192 atoms in 14s, 2,580 -> 2,525 at 54,000 in 31s, 519 -> 477 at 1,999, 206 -> 182 at 249
// (the whole energy and forces; REL alone 18, 60, 5 and 4 us of these).
// The split: a cell's atoms go to 8 warps where there are no more cells than SMs (249 atoms in 8
// cells: 182 against 193 us; 1,999 in 64: 477 against 488).  Beyond that every warp's start (the
// stencil's cells, the first chunk) costs more than the shorter chains give: 512 cells 3,146
// against 3,125 us a pullback, 1,728 cells 2,607 against 2,525.
constexpr int WALKC_WARPS = 4;
constexpr int WALK_ILP = 4;    // atoms per phase-1 step
constexpr int WALK_RING = 256;  // queue entries per warp (a step adds at most 32 * WALK_ILP to fewer than 32)
struct WalkAtom {
  double4 x;
  int64_t base, end;
  int32_t i, cnt;  // atom id, hits so far
};
struct WalkQ {
  int32_t slot, ii;  // candidate slot, group atom
};
struct WalkShared {
  WalkAtom a[32];
  float4 rel[32];  // the atoms' cell-relative positions, w = id
  WalkQ q[WALK_RING];
};
// Lane k: the k-th non-empty cell of the stencil.
struct WalkStencil {
  int start, base;  // its first candidate's place in the walk (INT_MAX: no cell), slot minus place
  float sx, sy, sz;  // its corner relative to the home cell's at the image of the stencil
  int total;         // candidates
};

// The first test of pair_ok: false only when pair_ok is false.  Branch-free: every term is
// formed, and the flags are combined bitwise.
__device__ __forceinline__ bool walk_prefilter(const PairTest& t, const double* L, int32_t i, double4 xi, int32_t j,
                                               double4 xj) {
  const bool other = t.mode == IPG_NLIST_HALF ? j > i : j != i;
  // pe_axis_dev for |a - b| < L (an open axis has L = inf, where min(s1, inf) = s1)
  const double s0 = fabs(__dsub_rn(xi.x, xj.x)), s1 = fabs(__dsub_rn(xi.y, xj.y)), s2 = fabs(__dsub_rn(xi.z, xj.z));
  const bool far = !(s0 < L[0]) | !(s1 < L[1]) | !(s2 < L[2]);  // fmod case or NaN: full test
  const double m0 = fmin(s0, __dsub_rn(L[0], s0)), m1 = fmin(s1, __dsub_rn(L[1], s1)),
               m2 = fmin(s2, __dsub_rn(L[2], s2));
  return other & (far | (sumsq3_dev(m0, m1, m2) <= t.rcut2_hi));
}

// Stencil of cell cc, in stencil_ranges' order (z, y in the order of stencil_axis, x ascending).
__device__ __forceinline__ void walk_stencil(const ConfGrid& g, const int* cc, const int64_t* __restrict__ cell_start,
                                             int lane, WalkShared& sh, WalkStencil& st) {
  constexpr unsigned FULL = 0xffffffffu;
  int ax[3][3], na[3];
#pragma unroll
  for (int a = 0; a < 3; a++) na[a] = stencil_axis(cc[a], g.nc[a], !isinf(g.L[a]), ax[a]);
  int beg = 0, len = 0;
  float s[3] = {0.0f, 0.0f, 0.0f};
  if (lane < na[0] * na[1] * na[2]) {
    const int k[3] = {lane % na[0], lane / na[0] % na[1], lane / (na[0] * na[1])};
    int c[3];
#pragma unroll
    for (int a = 0; a < 3; a++) {
      if (a == 0) {  // the k-th smallest of the distinct cells
        c[0] = 0;
        for (int q = 0; q < na[0]; q++) {
          int below = 0;
          for (int u = 0; u < na[0]; u++) below += ax[0][u] < ax[0][q];
          if (below == k[0]) c[0] = ax[0][q];
        }
      } else {
        c[a] = ax[a][k[a]];
      }
      int d = c[a] - cc[a];  // in -1..1 but for the wrap
      d = d > 1 ? d - g.nc[a] : (d < -1 ? d + g.nc[a] : d);
      s[a] = d * g.edge[a];
    }
    const int64_t cell = g.cell_off + ((int64_t)c[2] * g.nc[1] + c[1]) * g.nc[0] + c[0];
    beg = (int)cell_start[cell];
    len = (int)cell_start[cell + 1] - beg;
  }
  int incl = len;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int v = __shfl_up_sync(FULL, incl, o);
    if (lane >= o) incl += v;
  }
  st.total = __shfl_sync(FULL, incl, 31);
  // the empty cells drop out (through the warp's shared memory)
  const unsigned some = __ballot_sync(FULL, len > 0);
  if (len > 0) {
    const int at = __popc(some & ((1u << lane) - 1u));
    sh.q[at] = WalkQ{incl - len, beg - (incl - len)};
    sh.rel[at] = make_float4(s[0], s[1], s[2], 0.0f);
  }
  __syncwarp();
  const bool have = lane < __popc(some);
  st.start = have ? sh.q[lane].slot : INT_MAX;
  st.base = have ? sh.q[lane].ii : 0;
  st.sx = have ? sh.rel[lane].x : 0.0f;
  st.sy = have ? sh.rel[lane].y : 0.0f;
  st.sz = have ? sh.rel[lane].z : 0.0f;
  __syncwarp();
}

// A chunk of candidates: lane l holds the one at place P + l.
struct WalkChunk {
  int slot;  // -1: past the last candidate
  int32_t j;
  float4 r;   // REL: relative to the home cell's corner
  double4 x;  // otherwise
};
template <bool REL>
__device__ __forceinline__ void walk_chunk(const WalkStencil& st, int P, int lane,
                                           const int32_t* __restrict__ cell_atoms, const double4* __restrict__ spos,
                                           const float4* __restrict__ srel, WalkChunk& ch) {
  constexpr unsigned FULL = 0xffffffffu;
  // the cell of place P + l is the last that starts at or before it
  const int d = st.start - P;
  const int before = __popc(__ballot_sync(FULL, d <= 0));
  const unsigned marks = __reduce_or_sync(FULL, d > 0 && d < 32 ? 1u << d : 0u);
  const int k = before - 1 + __popc(marks & ((2u << lane) - 1u));
  const int base = __shfl_sync(FULL, st.base, k);
  const bool in = P + lane < st.total;
  ch.slot = in ? base + P + lane : -1;
  if (REL) {
    const float sx = __shfl_sync(FULL, st.sx, k), sy = __shfl_sync(FULL, st.sy, k), sz = __shfl_sync(FULL, st.sz, k);
    if (in) {
      ch.r = srel[ch.slot];
      ch.r.x += sx;
      ch.r.y += sy;
      ch.r.z += sz;
      ch.j = __float_as_int(ch.r.w);
    }
  } else if (in) {
    ch.j = cell_atoms[ch.slot];
    ch.x = spos[ch.slot];
  }
}

// The group of G atoms in sh against every candidate (WM as for k_pair_walk_cells).
template <int WM, bool REL>
__device__ __forceinline__ void walk_group(const PairTest& t, const ConfGrid& g, const WalkStencil& st, int G,
                                           int lane, float thr, const int32_t* __restrict__ cell_atoms,
                                           const double4* __restrict__ spos, const float4* __restrict__ srel,
                                           WalkShared& sh, int32_t* __restrict__ outj, double* __restrict__ outr) {
  constexpr unsigned FULL = 0xffffffffu;
  const unsigned lt = (1u << lane) - 1u;
  WalkAtom* A = sh.a;
  const bool half = t.mode == IPG_NLIST_HALF;
  int P = 0, ii = 0;
  unsigned head = 0, tail = 0;  // ring positions (mod WALK_RING) of the first and next entries
  WalkChunk cur, nxt;
  walk_chunk<REL>(st, 0, lane, cell_atoms, spos, srel, nxt);
  // the (chunk, atoms) sequence flattened, so that phase 2 has one call site: each pass takes one
  // step of phase 1, then drains full batches, and the remainder after the last step
  for (;;) {
    const bool more = P < st.total;  // warp-uniform
    if (more) {
      if (ii == 0) {
        cur = nxt;
        if (P + 32 < st.total) walk_chunk<REL>(st, P + 32, lane, cell_atoms, spos, srel, nxt);
      }
      bool cand[WALK_ILP];
#pragma unroll
      for (int k = 0; k < WALK_ILP; k++) {
        const int a = ii + k < G ? ii + k : ii;
        const bool in = (cur.slot >= 0) & (ii + k < G);
        if (REL) {
          const float4 h = sh.rel[a];
          const int32_t i = __float_as_int(h.w);
          const float x = h.x - cur.r.x, y = h.y - cur.r.y, z = h.z - cur.r.z;
          cand[k] = in & (half ? cur.j > i : cur.j != i) & (fmaf(x, x, fmaf(y, y, z * z)) <= thr);
        } else {
          cand[k] = in & walk_prefilter(t, g.L, A[a].i, A[a].x, cur.j, cur.x);
        }
      }
#pragma unroll
      for (int k = 0; k < WALK_ILP; k++) {
        const unsigned bal = __ballot_sync(FULL, cand[k]);
        if (cand[k]) sh.q[(tail + __popc(bal & lt)) % WALK_RING] = WalkQ{cur.slot, ii + k};
        tail += __popc(bal);
      }
      ii += WALK_ILP;
      if (ii >= G) {
        ii = 0;
        P += 32;
      }
    }
    while (tail - head >= 32u || (!more && tail != head)) {  // phase 2 on the next m queued pairs
      __syncwarp();
      const int m = tail - head < 32u ? (int)(tail - head) : 32;
      bool ok = false;
      int e_ii = 0;
      int32_t e_j = 0;
      double rr[3];
      if (lane < m) {
        const WalkQ e = sh.q[(head + lane) % WALK_RING];
        e_ii = e.ii;
        e_j = cell_atoms[e.slot];
        ok = pair_ok(t, g.L, A[e_ii].i, A[e_ii].x, e_j, spos[e.slot], rr);
      }
      const unsigned bal = __ballot_sync(FULL, ok);
      // lanes of the same atom: its members rank after the atom's running count
      const unsigned grp = __match_any_sync(FULL, lane < m ? e_ii : 32 + lane);
      if (WM != 0 && ok) {
        const int64_t o = A[e_ii].base + A[e_ii].cnt + __popc(bal & grp & lt);
        if (o < A[e_ii].end) {  // a list cut at the capacity (capacity mode) drops its tail
          outj[o] = e_j;
          outr[3 * o] = rr[0];
          outr[3 * o + 1] = rr[1];
          outr[3 * o + 2] = rr[2];
        }
      }
      __syncwarp();
      if (lane < m && (grp >> lane) == 1u) A[e_ii].cnt += __popc(bal & grp);  // the group's last lane
      head += m;
      __syncwarp();
    }
    if (!more) break;
  }
}

// WM 0: count each atom's hits into cnt (and their maximum into *maxcnt); 1: emit them at
// off[i]..off[i+1]; 2: both at once, emitting into kcap padded slots per atom (i * kcap ..),
// hits beyond kcap dropped (the count and *maxcnt still see them).
template <int WM>
__global__ void __launch_bounds__(WALKC_WARPS * 32) k_pair_walk_cells(
    int64_t ncells, int split, bool rel_ok, PairTest t, const ConfGrid* __restrict__ grid,
    const int32_t* __restrict__ conf, const int64_t* __restrict__ cell_start, const int32_t* __restrict__ cell_atoms,
    const double4* __restrict__ spos, const float4* __restrict__ srel, int64_t* __restrict__ cnt,
    const int64_t* __restrict__ off, int32_t* __restrict__ outj, double* __restrict__ outr, int kcap,
    int* __restrict__ maxcnt) {
  __shared__ WalkShared shw[WALKC_WARPS];
  const int lane = threadIdx.x & 31;
  WalkShared& sh = shw[threadIdx.x >> 5];
  const int64_t u = (int64_t)blockIdx.x * WALKC_WARPS + (threadIdx.x >> 5);
  const int64_t c = u >> split;
  if (c >= ncells) return;  // warp-uniform; the kernel synchronises only within a warp
  const int gw = 32 >> split;  // atoms of a group; a cell's groups go to its 2^split warps in turn
  const int64_t s0 = cell_start[c] + gw * (u & ((1 << split) - 1)), s1 = cell_start[c + 1];
  if (s0 >= s1) return;
  const ConfGrid g = grid[conf[cell_atoms[s0]]];
  int cc[3];
  {
    const int64_t k = c - g.cell_off;
    const int nxy = g.nc[0] * g.nc[1];
    cc[2] = (int)(k / nxy);
    const int rem = (int)(k - (int64_t)cc[2] * nxy);
    cc[1] = rem / g.nc[0];
    cc[0] = rem - cc[1] * g.nc[0];
  }
  WalkStencil st;
  walk_stencil(g, cc, cell_start, lane, sh, st);
  bool rel = rel_ok;
#pragma unroll
  for (int a = 0; a < 3; a++) rel &= isinf(g.L[a]) || g.nc[a] >= 3;
  const float thr = prefilter_threshold(g, t.rcut);
  for (int64_t g0 = s0; g0 < s1; g0 += 32) {
    const int G = (int)((s1 - g0) < gw ? (s1 - g0) : gw);
    __syncwarp();
    if (lane < G) {
      const int32_t i = cell_atoms[g0 + lane];
      sh.rel[lane] = srel[g0 + lane];
      sh.a[lane].i = i;
      sh.a[lane].cnt = 0;
      sh.a[lane].x = spos[g0 + lane];
      if (WM == 1) {
        sh.a[lane].base = off[i];
        sh.a[lane].end = off[i + 1];
      } else {
        sh.a[lane].base = (int64_t)i * kcap;
        sh.a[lane].end = (int64_t)i * kcap + kcap;
      }
    }
    __syncwarp();
    if (rel)
      walk_group<WM, true>(t, g, st, G, lane, thr, cell_atoms, spos, srel, sh, outj, outr);
    else
      walk_group<WM, false>(t, g, st, G, lane, thr, cell_atoms, spos, srel, sh, outj, outr);
    if (WM != 1) {
      int km = 0;
      if (lane < G) {
        km = sh.a[lane].cnt;
        cnt[sh.a[lane].i] = km;
      }
      km = __reduce_max_sync(0xffffffffu, km);
      if (lane == 0) atomicMax(maxcnt, km);
    }
  }
}

// Padded emission (k_pair_walk_cells<2>) to the CSR list: slot t of atom i goes to off[i] + t.  In
// capacity mode an atom may have more hits than its kcap slots: the list is then thrown away
// (k_clamp_offsets reports it), but the kernels that follow still read it, so the entries without a slot
// become pairs of the atom with itself (at the last slot's distance).  They held what the buffer had: the
// atoms of another, possibly larger system, or nothing yet.
__global__ void k_pad_compact(int64_t n, int kcap, const int64_t* __restrict__ off, const int32_t* __restrict__ pj,
                              const double* __restrict__ pr, int32_t* __restrict__ j, double* __restrict__ r) {
  const int64_t s = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= n * kcap) return;
  const int64_t i = s / kcap, t = s - i * kcap, e = off[i + 1];
  for (int64_t b = off[i] + t, o = b; o < e; o++) {
    j[o] = o == b ? pj[s] : (int32_t)i;
    r[3 * o] = pr[3 * s];
    r[3 * o + 1] = pr[3 * s + 1];
    r[3 * o + 2] = pr[3 * s + 2];
    if (t + 1 < kcap) break;
  }
}

// Sorts each atom's list by neighbor index (insertion sort; lists are short).
__global__ void k_pair_sort(int64_t n, const int64_t* __restrict__ off, int32_t* __restrict__ j,
                            double* __restrict__ r) {
  int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int64_t s = off[i], e = off[i + 1];
  for (int64_t a = s + 1; a < e; a++) {
    int32_t v = j[a];
    double r0 = r[3 * a], r1 = r[3 * a + 1], r2 = r[3 * a + 2];
    int64_t b = a - 1;
    while (b >= s && j[b] > v) {
      j[b + 1] = j[b];
      r[3 * (b + 1)] = r[3 * b];
      r[3 * (b + 1) + 1] = r[3 * b + 1];
      r[3 * (b + 1) + 2] = r[3 * b + 2];
      b--;
    }
    j[b + 1] = v;
    r[3 * (b + 1)] = r0;
    r[3 * (b + 1) + 1] = r1;
    r[3 * (b + 1) + 2] = r2;
  }
}

// Transpose: rev[p] of pair p = (i -> k) is the pair (k -> i).  The lists it serves (the full SNAP
// lists) have one image per pair and are symmetric but for pairs at the cutoff to the last bit, which
// the rounding of the two minimum images can put on one list only (and lists cut at a capacity, whose
// result the capacity error discards).  So the pairs that end at i are the reverses of those that i
// owns, and the chain of the pairs without a reverse: one[i] - 1, then rev[p] = -2 - the next (-1: none).
//
// One warp per owner i, one lane per pair (32 at a time); each lane looks through the neighbors of k
// on its own, so the lanes' loads overlap: 48 us at 54,000 atoms, 6 at 249.  Lists of their own for the
// pairs that end at each atom took counts, their scan and a clear besides, 10 us at 249 atoms.
__global__ void k_rev_pair(int64_t n, const int64_t* __restrict__ off, const int32_t* __restrict__ j,
                           int64_t* __restrict__ rev, int64_t* __restrict__ one) {
  const int lane = threadIdx.x & 31;
  const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  if (i >= n) return;  // warp-uniform
  const int64_t p1 = off[i + 1];
  for (int64_t p = off[i] + lane; p < p1; p += 32) {
    const int32_t k = j[p];
    const int64_t q0 = off[k], q1 = off[k + 1];
    int64_t r = -1;
#pragma unroll 4
    for (int64_t q = q0; q < q1; q++)
      if (j[q] == i) r = q;
    if (r < 0) r = -1 - (int64_t)atomicExch((unsigned long long*)&one[k], (unsigned long long)(p + 1));
    rev[p] = r;
  }
}

inline unsigned nblk(int64_t n, int t) { return (unsigned)std::max<int64_t>(1, (n + t - 1) / t); }

}  // namespace

int ipg_build_cells(ipg_ctx* ctx, const char* prefix, int64_t n, const double* d_pos, const int32_t* d_species,
                    int nsp, int nconf, const int64_t* h_atom_off, const double* h_L, double radius, CellList& cl) {
  std::string pre(prefix);
  cl.nconf = nconf;
  cl.n = n;
  cl.radius = radius;
  cl.h_grid.assign(nconf, ConfGrid());
  bool any_open = false;
  for (int c = 0; c < nconf; c++) {
    ConfGrid& g = cl.h_grid[c];
    g.atom_off = h_atom_off[c];
    g.natoms = h_atom_off[c + 1] - h_atom_off[c];
    for (int a = 0; a < 3; a++) {
      double L = h_L[3 * c + a];
      if (!(L > 0.0)) return ipg_fail(ctx, IPG_ERR_ARG, "box length L[%d] of configuration %d must be > 0", a, c);
      g.L[a] = std::isinf(L) ? INFINITY : L;
      any_open |= std::isinf(L);
    }
  }
  IPG_RET(scratch(ctx, (pre + "grid").c_str(), nconf, &cl.d_grid));
  std::vector<double> ext(6 * (size_t)nconf, 0.0);
  if (any_open && n > 0 && ctx->capturing)
    return ipg_fail(ctx, IPG_ERR_UNSUPPORTED, "open boundaries cannot be captured in a graph");
  if (any_open && n > 0) {
    CUDA_RET(ctx, cudaMemcpyAsync(cl.d_grid, cl.h_grid.data(), sizeof(ConfGrid) * nconf, cudaMemcpyHostToDevice,
                                  ctx->stream));
    double* d_ext;
    IPG_RET(scratch(ctx, (pre + "ext").c_str(), 6 * (size_t)nconf, &d_ext));
    IPG_LAUNCH(ctx, k_extent, nconf, 256, 0, d_pos, cl.d_grid, d_ext);
    CUDA_RET(ctx, cudaMemcpyAsync(ext.data(), d_ext, sizeof(double) * 6 * nconf, cudaMemcpyDeviceToHost, ctx->stream));
    CUDA_RET(ctx, cudaStreamSynchronize(ctx->stream));
  }
  const double rc = radius * (1.0 + 1e-9);
  int64_t cell_total = 0;
  for (int c = 0; c < nconf; c++) {
    ConfGrid& g = cl.h_grid[c];
    int64_t tot = 1;
    double e3[3];
    for (int a = 0; a < 3; a++) {
      double lo = 0.0, e = g.L[a];
      if (std::isinf(g.L[a])) {
        lo = ext[6 * c + a];
        e = ext[6 * c + 3 + a] - lo;
        if (!(e >= 0.0) || !std::isfinite(e)) {  // empty config or non-finite input
          lo = 0.0;
          e = 0.0;
        }
      }
      g.lo[a] = lo;
      e3[a] = e;
      int nc = 1;
      if (rc > 0.0 && std::isfinite(rc) && e > 0.0) nc = (int)std::max(1.0, std::min(std::floor(e / rc), 1024.0));
      g.nc[a] = nc;
      tot *= nc;
    }
    while (tot > std::max<int64_t>(64, 8 * g.natoms)) {  // keep the grid proportional to the atoms
      int a = (g.nc[0] >= g.nc[1] && g.nc[0] >= g.nc[2]) ? 0 : (g.nc[1] >= g.nc[2] ? 1 : 2);
      tot /= g.nc[a];
      g.nc[a] = std::max(1, g.nc[a] / 2);
      tot *= g.nc[a];
    }
    for (int a = 0; a < 3; a++) g.cs[a] = e3[a] > 0.0 ? e3[a] / g.nc[a] : 1.0;
    const int e2 = std::ilogb(std::max(g.cs[0], std::max(g.cs[1], g.cs[2])));
    g.rel = std::ldexp(1.0, -std::max(-1000, std::min(1000, e2)));
    for (int a = 0; a < 3; a++) g.edge[a] = (float)(g.cs[a] * g.rel);
    g.cell_off = cell_total;
    cell_total += tot;
  }
  if (cell_total >= (int64_t)INT32_MAX) return ipg_fail(ctx, IPG_ERR_CAPACITY, "too many cells");
  cl.ncells = cell_total;
  if (!ctx->capturing)  // a captured graph's grid table is uploaded before each replay
    CUDA_RET(ctx, cudaMemcpyAsync(cl.d_grid, cl.h_grid.data(), sizeof(ConfGrid) * nconf, cudaMemcpyHostToDevice,
                                  ctx->stream));
  int64_t* count;
  int32_t *cell_of, *arrival, *unsorted;
  IPG_RET(scratch(ctx, (pre + "conf").c_str(), n, &cl.d_conf));
  IPG_RET(scratch(ctx, (pre + "cell_of").c_str(), n, &cell_of));
  IPG_RET(scratch(ctx, (pre + "cell_start").c_str(), cell_total + 1, &cl.d_cell_start));
  IPG_RET(scratch(ctx, (pre + "cell_arrival").c_str(), n, &arrival));
  IPG_RET(scratch(ctx, (pre + "cell_unsorted").c_str(), n, &unsorted));
  IPG_RET(scratch(ctx, (pre + "cell_atoms").c_str(), n, &cl.d_cell_atoms));
  IPG_RET(scratch(ctx, (pre + "spos").c_str(), n, &cl.d_spos));
  IPG_RET(scratch(ctx, (pre + "srel").c_str(), n, &cl.d_srel));
  count = cl.d_cell_start;
  if (n > 0 && n <= SMALL_ATOMS && cell_total <= SMALL_CELLS) {
    IPG_LAUNCH(ctx, k_cells_small, 1, SMALL_T, 0, (int)n, (int)cell_total, d_pos, d_species, nsp, cl.d_grid, nconf,
               cl.d_conf, cl.d_cell_start, cl.d_cell_atoms, cl.d_spos, cl.d_srel,
               ctx->d_status);
    return IPG_OK;
  }
  CUDA_RET(ctx, cudaMemsetAsync(count, 0, sizeof(int64_t) * (cell_total + 1), ctx->stream));
  if (n == 0) return IPG_OK;
  IPG_LAUNCH(ctx, k_cell_count, nblk(n, 256), 256, 0, n, d_pos, d_species, nsp, cl.d_grid, nconf, cl.d_conf, cell_of,
             arrival, count, ctx->d_status);
  IPG_RET(ipg_scan_i64(ctx, count, cl.d_cell_start, cell_total + 1));
  IPG_LAUNCH(ctx, k_cell_fill, nblk(n, 256), 256, 0, n, cell_of, arrival, cl.d_cell_start, unsorted);
  IPG_LAUNCH(ctx, k_cell_place, nblk(n, 128), 128, 0, n, unsorted, cell_of, cl.d_cell_start, cl.d_grid,
             cl.d_conf, d_pos, d_species, nsp, cl.d_cell_atoms, cl.d_spos, cl.d_srel);
  return IPG_OK;
}

namespace {
int build_transpose(ipg_ctx* ctx, const std::string& pre, int64_t n, PairList& pl) {
  IPG_RET(scratch(ctx, (pre + "rev").c_str(), pl.npairs + 1, &pl.d_rev));
  if (pl.npairs > 0)
    IPG_LAUNCH(ctx, k_rev_pair, nblk(32 * n, 128), 128, 0, n, pl.d_off, pl.d_j, pl.d_rev, pl.d_one);
  return IPG_OK;
}
}  // namespace

int ipg_build_pairs(ipg_ctx* ctx, const char* prefix, const CellList& cl, const int32_t* d_species, int nsp,
                    const double* h_cut, int mode, bool want_transpose, PairList& pl, bool sorted, int64_t cap,
                    int walk_warps, bool count_only) {
  const int wt = 32 * std::max(1, std::min(4, walk_warps));
  (void)d_species;
  IPG_RET(ipg_side_join(ctx));
  std::string pre(prefix);
  PairTest t;
  memset(&t, 0, sizeof(t));
  t.mode = mode & 0xff;
  t.literal = (mode & IPG_NLIST_LITERAL_SQRT) ? 1 : 0;
  t.nsp = nsp;
  if (t.mode == IPG_NLIST_HALF) {
    t.rcut = h_cut[0];
  } else {
    if (nsp < 1 || nsp > 8) return ipg_fail(ctx, IPG_ERR_ARG, "nspecies must be in 1..8 for a full list");
    double cutmax2 = 0.0;
    for (int q = 0; q < nsp * nsp; q++) {
      t.cutsq[q] = h_cut[q];
      cutmax2 = std::max(cutmax2, h_cut[q]);
    }
    double cutmax = std::sqrt(cutmax2);
    t.rcut = t.literal ? std::sqrt(cutmax) : cutmax;
  }
  t.rcut2_lo = t.rcut * t.rcut * (1.0 - 1e-12);
  t.rcut2_hi = t.rcut * t.rcut * (1.0 + 1e-12);
  int64_t n = cl.n;
  pl.n = n;
  int64_t* cnt;
  IPG_RET(scratch(ctx, (pre + "off").c_str(), 2 * n + 1, &pl.d_off));
  pl.d_one = pl.d_off + n + 1;
  cnt = pl.d_off;
  CUDA_RET(ctx, cudaMemsetAsync(cnt, 0, sizeof(int64_t) * (want_transpose ? 2 * n + 1 : n + 1), ctx->stream));
  const bool by_cell = ctx->walk_by_cell;
  // One walk instead of two when a previous build of this list gave the per-atom maximum:
  // emit into padded slots while counting, then compact (or, if an atom overflowed its
  // slots, emit again at the counted offsets).  In capacity mode (graph capture) there is no
  // read-back: an overflow sets IPG_ERR_CAPACITY in the device status word instead.
  int* maxcnt;
  IPG_RET(scratch(ctx, (pre + "maxcnt").c_str(), 1, &maxcnt));
  CUDA_RET(ctx, cudaMemsetAsync(maxcnt, 0, sizeof(int), ctx->stream));
  int kcap = (by_cell && !count_only && ctx->walk_single) ? ctx->walk_kcap[pre] : 0;
  if ((double)n * kcap * 28.0 > 2.0 * (1 << 30)) kcap = 0;  // padded slots within 2 GiB
  int32_t* pad_j = nullptr;
  double* pad_r = nullptr;
  if (kcap > 0 && n > 0) {
    IPG_RET(scratch(ctx, (pre + "pad_j").c_str(), (size_t)n * kcap + 1, &pad_j));
    IPG_RET(scratch(ctx, (pre + "pad_r").c_str(), 3 * (size_t)n * kcap + 3, &pad_r));
  }
  const int split = cl.ncells <= ctx->num_sms ? 3 : 0;
  const bool rel_ok = t.rcut <= cl.radius;
  if (n > 0) {
    if (by_cell && kcap > 0)
      IPG_LAUNCH(ctx, k_pair_walk_cells<2>, nblk(cl.ncells << split, WALKC_WARPS), WALKC_WARPS * 32, 0, cl.ncells, split,
                 rel_ok, t, cl.d_grid, cl.d_conf, cl.d_cell_start, cl.d_cell_atoms, cl.d_spos, cl.d_srel, cnt, nullptr, pad_j,
                 pad_r, kcap, maxcnt);
    else if (by_cell)
      IPG_LAUNCH(ctx, k_pair_walk_cells<0>, nblk(cl.ncells << split, WALKC_WARPS), WALKC_WARPS * 32, 0, cl.ncells, split,
                 rel_ok, t, cl.d_grid, cl.d_conf, cl.d_cell_start, cl.d_cell_atoms, cl.d_spos, cl.d_srel, cnt, nullptr, nullptr,
                 nullptr, 0, maxcnt);
    else
      IPG_LAUNCH(ctx, k_pair_walk<false>, nblk(32 * n, wt), wt, 0, n, t, cl.d_grid, cl.d_conf, cl.d_cell_start,
                 cl.d_cell_atoms, cl.d_spos, cnt, nullptr, nullptr, nullptr);
  }
  IPG_RET(ipg_scan_i64(ctx, cnt, pl.d_off, n + 1));
  pl.d_np = pl.d_off + n;
  int hmax = 0;
  if (cap > 0) {  // capacity mode: no read-back
    pl.npairs = cap;
    IPG_LAUNCH(ctx, k_clamp_offsets, nblk(n + 1, 256), 256, 0, n, pl.d_off, cap, maxcnt, n > 0 ? kcap : 0,
               ctx->d_status);
  } else {
    CUDA_RET(ctx, cudaMemcpyAsync(&pl.npairs, pl.d_off + n, sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream));
    CUDA_RET(ctx, cudaMemcpyAsync(&hmax, maxcnt, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
    CUDA_RET(ctx, cudaStreamSynchronize(ctx->stream));
    if (by_cell && !count_only) ctx->walk_kcap[pre] = ((hmax + hmax / 8 + 4 + 7) / 8) * 8;  // next build
  }
  if (pl.npairs >= (int64_t)1 << 40) return ipg_fail(ctx, IPG_ERR_CAPACITY, "pair count overflow");
  if (count_only) return IPG_OK;
  IPG_RET(scratch(ctx, (pre + "j").c_str(), pl.npairs + 1, &pl.d_j));
  IPG_RET(scratch(ctx, (pre + "r").c_str(), 3 * pl.npairs + 3, &pl.d_r));
  if (n > 0) {
    if (by_cell && kcap > 0 && (cap > 0 || hmax <= kcap))
      IPG_LAUNCH(ctx, k_pad_compact, nblk(n * kcap, 256), 256, 0, n, kcap, pl.d_off, pad_j, pad_r, pl.d_j, pl.d_r);
    else if (by_cell)
      IPG_LAUNCH(ctx, k_pair_walk_cells<1>, nblk(cl.ncells << split, WALKC_WARPS), WALKC_WARPS * 32, 0, cl.ncells, split,
                 rel_ok, t, cl.d_grid, cl.d_conf, cl.d_cell_start, cl.d_cell_atoms, cl.d_spos, cl.d_srel, nullptr, pl.d_off,
                 pl.d_j, pl.d_r, 0, nullptr);
    else
      IPG_LAUNCH(ctx, k_pair_walk<true>, nblk(32 * n, wt), wt, 0, n, t, cl.d_grid, cl.d_conf, cl.d_cell_start,
                 cl.d_cell_atoms, cl.d_spos, nullptr, pl.d_off, pl.d_j, pl.d_r);
    if (sorted) IPG_LAUNCH(ctx, k_pair_sort, nblk(n, 128), 128, 0, n, pl.d_off, pl.d_j, pl.d_r);
  }
  if (want_transpose) {
    // needed only by the force gather: for one configuration it overlaps the first SNAP
    // kernels on the side stream (+0.6% at 54,000 atoms); for a batch the overlap measured
    // 2.6% slower (512 configurations), so batches build it in order
    const bool side = cl.nconf == 1;
    if (side) IPG_RET(ipg_side_begin(ctx));
    const int st = build_transpose(ctx, pre, n, pl);
    if (side) IPG_RET(ipg_side_end(ctx));
    IPG_RET(st);
  }
  return IPG_OK;
}

int ipg_max_disp2(ipg_ctx* ctx, const CellList& cl, const double* d_pos, const double* d_ref,
                  const int32_t* d_species, const int32_t* d_ref_species, double* out) {
  *out = 0.0;
  if (cl.n == 0) return IPG_OK;
  unsigned long long* d_m;
  IPG_RET(scratch(ctx, "skin_maxdisp", 1, &d_m));
  CUDA_RET(ctx, cudaMemsetAsync(d_m, 0, sizeof(unsigned long long), ctx->stream));
  const int64_t grid = std::min<int64_t>(nblk(cl.n, 256), 4 * ctx->num_sms);
  IPG_LAUNCH(ctx, k_max_disp2, (unsigned)grid, 256, 0, cl.n, cl.d_grid, cl.d_conf, d_pos, d_ref, d_species,
             d_ref_species, d_m);
  unsigned long long h = 0;
  CUDA_RET(ctx, cudaMemcpyAsync(&h, d_m, sizeof(h), cudaMemcpyDeviceToHost, ctx->stream));
  CUDA_RET(ctx, cudaStreamSynchronize(ctx->stream));
  memcpy(out, &h, sizeof(double));
  return IPG_OK;
}

int ipg_filter_pairs(ipg_ctx* ctx, const char* prefix, const CellList& cl, const PairList& cached,
                     const double* d_pos, const int32_t* d_species, int nsp, const double* h_cut, int mode,
                     PairList& pl) {
  IPG_RET(ipg_side_join(ctx));
  std::string pre(prefix);
  PairTest t;
  memset(&t, 0, sizeof(t));
  t.mode = IPG_NLIST_FULL;
  t.literal = (mode & IPG_NLIST_LITERAL_SQRT) ? 1 : 0;
  t.nsp = nsp;
  double cutmax2 = 0.0;
  for (int q = 0; q < nsp * nsp; q++) {
    t.cutsq[q] = h_cut[q];
    cutmax2 = std::max(cutmax2, h_cut[q]);
  }
  const double cutmax = std::sqrt(cutmax2);
  t.rcut = t.literal ? std::sqrt(cutmax) : cutmax;
  t.rcut2_lo = t.rcut * t.rcut * (1.0 - 1e-12);
  t.rcut2_hi = t.rcut * t.rcut * (1.0 + 1e-12);
  const int64_t n = cl.n;
  pl.n = n;
  IPG_RET(scratch(ctx, (pre + "off").c_str(), 2 * n + 1, &pl.d_off));
  pl.d_one = pl.d_off + n + 1;
  CUDA_RET(ctx, cudaMemsetAsync(pl.d_off, 0, sizeof(int64_t) * (2 * n + 1), ctx->stream));
  if (n > 0)
    IPG_LAUNCH(ctx, k_filter_walk<false>, nblk(32 * n, 128), 128, 0, n, t, cl.d_grid, cl.d_conf, cached.d_off,
               cached.d_j, d_pos, d_species, nsp, pl.d_off, nullptr, nullptr, nullptr, ctx->d_status);
  IPG_RET(ipg_scan_i64(ctx, pl.d_off, pl.d_off, n + 1));
  pl.d_np = pl.d_off + n;
  CUDA_RET(ctx, cudaMemcpyAsync(&pl.npairs, pl.d_off + n, sizeof(int64_t), cudaMemcpyDeviceToHost, ctx->stream));
  CUDA_RET(ctx, cudaStreamSynchronize(ctx->stream));
  IPG_RET(scratch(ctx, (pre + "j").c_str(), pl.npairs + 1, &pl.d_j));
  IPG_RET(scratch(ctx, (pre + "r").c_str(), 3 * pl.npairs + 3, &pl.d_r));
  if (n > 0)
    IPG_LAUNCH(ctx, k_filter_walk<true>, nblk(32 * n, 128), 128, 0, n, t, cl.d_grid, cl.d_conf, cached.d_off,
               cached.d_j, d_pos, d_species, nsp, nullptr, pl.d_off, pl.d_j, pl.d_r, ctx->d_status);
  const bool side = cl.nconf == 1;  // as in ipg_build_pairs
  if (side) IPG_RET(ipg_side_begin(ctx));
  const int st = build_transpose(ctx, pre, n, pl);
  if (side) IPG_RET(ipg_side_end(ctx));
  IPG_RET(st);
  return IPG_OK;
}

// ---------------------------------------------------------------------------------
struct ipg_nlist {
  int64_t n = 0, npairs = 0;
  std::vector<int64_t> off;
  std::vector<int32_t> j;
  std::vector<double> r;
};

namespace {

// Validates and uploads the inputs and builds the pair list (or only counts it).
int neighbor_pairs(ipg_ctx* ctx, int64_t n, const double* pos, const double L[3], const int32_t* species,
                   int32_t nspecies, const double* cut, int32_t mode, bool count_only, PairList& pl) {
  if (!ctx || n < 0 || (n > 0 && !pos) || !L || !cut) return IPG_ERR_ARG;
  if (n >= INT32_MAX) return ipg_fail(ctx, IPG_ERR_ARG, "n too large");
  int base = mode & 0xff;
  if (base != IPG_NLIST_HALF && base != IPG_NLIST_FULL) return ipg_fail(ctx, IPG_ERR_ARG, "bad mode");
  if (base == IPG_NLIST_FULL && !species) return ipg_fail(ctx, IPG_ERR_ARG, "full list needs species");
  CUDA_RET(ctx, cudaSetDevice(ctx->device));
  if (!host_all_finite(pos, 3 * n)) return ipg_fail(ctx, IPG_ERR_NONFINITE, "non-finite position");
  if (species && !host_species_ok(species, n, std::max(1, (int)nspecies)))
    return ipg_fail(ctx, IPG_ERR_SPECIES, "species id out of range");
  double *d_pos;
  int32_t* d_sp = nullptr;
  IPG_RET(scratch(ctx, "nl_in_pos", 3 * (size_t)n + 3, &d_pos));
  if (n) CUDA_RET(ctx, cudaMemcpyAsync(d_pos, pos, sizeof(double) * 3 * n, cudaMemcpyHostToDevice, ctx->stream));
  if (species) {
    IPG_RET(scratch(ctx, "nl_in_sp", (size_t)n + 1, &d_sp));
    if (n) CUDA_RET(ctx, cudaMemcpyAsync(d_sp, species, sizeof(int32_t) * n, cudaMemcpyHostToDevice, ctx->stream));
  }
  IPG_RET(ipg_status_reset(ctx));
  int64_t aoff[2] = {0, n};
  double radius;
  if (base == IPG_NLIST_HALF) {
    radius = cut[0];
  } else {
    double m = 0.0;
    for (int q = 0; q < nspecies * nspecies; q++) m = std::max(m, cut[q]);
    radius = std::sqrt(m);
    if (mode & IPG_NLIST_LITERAL_SQRT) radius = std::sqrt(radius);
  }
  if (!(radius >= 0.0)) return ipg_fail(ctx, IPG_ERR_ARG, "cutoff must be >= 0");
  CellList cl;
  IPG_RET(ipg_build_cells(ctx, "nl_", n, d_pos, d_sp, std::max(1, (int)nspecies), 1, aoff, L, radius, cl));
  IPG_RET(ipg_build_pairs(ctx, "nl_", cl, d_sp, std::max(1, (int)nspecies), cut, mode, false, pl, true, 0, 4,
                          count_only));
  return ipg_status_check(ctx, count_only ? "ipg_neighbor_count" : "ipg_neighbor_build");
}

}  // namespace

extern "C" {

int ipg_neighbor_count(ipg_ctx* ctx, int64_t n, const double* pos, const double L[3], const int32_t* species,
                       int32_t nspecies, const double* cut, int32_t mode, int64_t* npairs) {
  if (!npairs) return IPG_ERR_ARG;
  PairList pl;
  IPG_RET(neighbor_pairs(ctx, n, pos, L, species, nspecies, cut, mode, true, pl));
  *npairs = pl.npairs;
  return IPG_OK;
}

int ipg_neighbor_build(ipg_ctx* ctx, int64_t n, const double* pos, const double L[3], const int32_t* species,
                       int32_t nspecies, const double* cut, int32_t mode, ipg_nlist** out) {
  if (!out) return IPG_ERR_ARG;
  PairList pl;
  IPG_RET(neighbor_pairs(ctx, n, pos, L, species, nspecies, cut, mode, false, pl));
  ipg_nlist* nl = new ipg_nlist();
  nl->n = n;
  nl->npairs = pl.npairs;
  nl->off.resize(n + 1);
  nl->j.resize(pl.npairs);
  nl->r.resize(3 * pl.npairs);
  CUDA_RET(ctx, cudaMemcpyAsync(nl->off.data(), pl.d_off, sizeof(int64_t) * (n + 1), cudaMemcpyDeviceToHost,
                                ctx->stream));
  if (pl.npairs) {
    CUDA_RET(ctx, cudaMemcpyAsync(nl->j.data(), pl.d_j, sizeof(int32_t) * pl.npairs, cudaMemcpyDeviceToHost,
                                  ctx->stream));
    CUDA_RET(ctx, cudaMemcpyAsync(nl->r.data(), pl.d_r, sizeof(double) * 3 * pl.npairs, cudaMemcpyDeviceToHost,
                                  ctx->stream));
  }
  int st = ipg_sync(ctx);
  if (st) {
    delete nl;
    return st;
  }
  *out = nl;
  return IPG_OK;
}

int ipg_nlist_size(const ipg_nlist* nl, int64_t* npairs) {
  if (!nl || !npairs) return IPG_ERR_ARG;
  *npairs = nl->npairs;
  return IPG_OK;
}

int ipg_nlist_export(const ipg_nlist* nl, int64_t* offsets, int32_t* j, double* r) {
  if (!nl) return IPG_ERR_ARG;
  if (offsets) memcpy(offsets, nl->off.data(), sizeof(int64_t) * (nl->n + 1));
  if (j && nl->npairs) memcpy(j, nl->j.data(), sizeof(int32_t) * nl->npairs);
  if (r && nl->npairs) memcpy(r, nl->r.data(), sizeof(double) * 3 * nl->npairs);
  return IPG_OK;
}

int ipg_nlist_free(ipg_nlist* nl) {
  if (!nl) return IPG_ERR_ARG;
  delete nl;
  return IPG_OK;
}

}  // extern "C"
