// ipg_snap_y.cu — the Clebsch–Gordan contraction of the SNAP path (twojmax <= YR_MAX_J): Y, Z or
// both from the Utot of 32 atoms per block, one atom per lane (compute_zi of compute_z.jl:5-61,
// compute_yi of compute_yi.jl:86-118); also the tangent of Y along a tangent of Utot.
//
//   Z(j1, j2, j; mb, ma) = sum over mb1 of cg(mb1, mb2) sum over ma1 of cg(ma1, ma2)
//                          U(j1, mb1, ma1) U(j2, mb2, ma2),
//   Y(j; mb, ma) = sum over the triples (j1, j2, j) of coef Z.
//
// In the physical (doubled) indices k = -(2 mb - j) and c = 2 ma - j the sums run over
// m1 + m2 = -k and a1 + a2 = c, whatever j: one product U(j1, mb1, ma1) U(j2, mb2, ma2) feeds
// every level j of the triple at once.  So a warp owns an item (k, YT adjacent columns c), keeps
// the entries of all its levels in registers, and walks the (j1, j2) pairs; per row pair
// (mb1, mb2) it steps through ma1 with a window of YT elements of the second row, one new
// element of each row per step.  A step costs 4 YT FP64 instructions for the products and
// 2 YT per level for their sums; one entry (j, mb, ma) at a time, every use of a product
// formed it anew (6 instructions per use), and every use took its own loads.
//
// The weights cg(mb1, mb2) cg(ma1, ma2) of a step are constants of the basis in exactly the
// order in which the item reads them, so they stream: records of several row pairs, copied two
// records ahead into a ring of each warp's shared memory (cp.async).
// Mirrored rows (beyond the half plane, U(j, mb, ma) = (-1)^(ma+mb) conj(U(j, j-mb, j-ma)))
// are walked backwards, the conjugate taken by an integer flip of the sign bit and the signs kept
// in the weights, so that one step loop per number of levels serves them all: the code of a
// variant per mirror case and four steps at a time no longer fitted the instruction cache (the
// warps of a block run different items) and took 2.5 ms where this takes 1.36 ms; four columns
// per item, half the warps, 3.9 ms.
//
// Bound: issue slots (57% of the active cycles, the FP64 pipe 42%, shared-memory wavefronts 58% of
// their peak; Y at 16,000 atoms) and the latency of shared-memory loads at 16 warps per SM.  Against
// the kernel that formed one row of entries at a time, twojmax 8: Y 1.73 -> 1.36 ms at 54,000 atoms;
// Y 0.60 -> 0.47 ms, Y and Z 0.69 -> 0.58 ms at 16,000.
#include <algorithm>

#include "ipg_snap.cuh"

namespace {

constexpr int YK_WARPS = 8;
// What the two factors of a product are: PL_ONE: both from one Utot.  PL_TWO: the first from one, the second from
// another (the element pairs of chem_flag).  PL_TANGENT: the tangent of PL_ONE's product along Udot,
// U Udot + Udot U (the position pullback).
constexpr int PL_ONE = 0, PL_TWO = 1, PL_TANGENT = 2;
// The tangent as two evaluations, [Y(U + s Udot) - Y(U - s Udot)] / (2s), took 2 x 467 us and 67 us to form
// the two arguments and the difference (16,000 atoms, twojmax 8); in one pass a step forms twice the
// products but sums them into the levels once: 661 us (pullback 3,065 -> 2,720 us a call).  Two planes
// of shared memory leave one block an SM, hence more warps: 16, 12, 10: 2,722, 2,738, 2,785 us a call.
constexpr int YT_WARPS = 16;
constexpr int yk_warps(int pl) { return pl == PL_TANGENT ? YT_WARPS : YK_WARPS; }
constexpr int YK_SLOTS = 3;  // ring: the record in use and two in flight

// Shared memory, in bytes: coefficients of every triple and species | zero guard | half plane of
// the 32 atoms, [u_half][32] double2 | zero guard | energies [items][32] | record rings.
// Window elements before the first or after the last column of a row meet weights of exactly
// zero, so they only have to be finite: neighbors in the half plane (the same atom's), or guard.
// With two sets of Utot (row 1 from one, row 2 from the other) a second half plane and guard follow.
struct YkSmem {
  int coef, guard, u, energy, ring, sets;
  __host__ __device__ int planes() const { return guard + sets * (u + guard); }
  __host__ __device__ int total() const { return coef + planes() + energy + ring; }
};
__host__ __device__ inline YkSmem yk_smem(int nsp, int ntrip, int uh, int nitems, int pl) {
  YkSmem m;
  m.sets = pl != PL_ONE ? 2 : 1;
  m.coef = (8 * nsp * ntrip + 15) & ~15;
  m.guard = YGUARD * YS_ATOMS * 16;
  m.u = uh * YS_ATOMS * 16;
  m.energy = pl == PL_TANGENT ? 0 : nitems * YS_ATOMS * 8;
  m.ring = yk_warps(pl) * YK_SLOTS * YREC * 16;
  return m;
}

__device__ __forceinline__ void cp16(double2* dst, const double2* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src));
}
// Shared-memory loads at 32-bit addresses (immediate offsets, no address arithmetic per load).
template <int OFF>
__device__ __forceinline__ double2 lds2(unsigned addr) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2 + %3];" : "=d"(v.x), "=d"(v.y) : "r"(addr), "n"(OFF));
  return v;
}
constexpr int YE = YS_ATOMS * 16;  // bytes from one half-plane element to the next

__device__ __forceinline__ double2 conj_if(double2 v, unsigned sign) {  // sign: 0, or 0x80000000 for conj(v)
  return make_double2(v.x, __hiloint2double(__double2hiint(v.y) ^ (int)sign, __double2loint(v.y)));
}

// One step: the products of a with the window (w0 the new element, w1 the one before) into the N
// levels, the weights at byte offset WO of wt.  TAN: the tangent of the products, at, v0 and v1 the
// tangents of a, w0 and w1.
template <int N, int WO, bool TAN>
__device__ __forceinline__ void yk_step(const double2 a, const double2 w0, const double2 w1, const double2 at,
                                        const double2 v0, const double2 v1, unsigned wt, double2 (&Z)[YNJ][YT]) {
  static_assert(YT == 2 && YE == 512, "a step holds a window of two elements");
  double px0, py0, px1, py1;
  if (TAN) {
    px0 = fma(at.x, w0.x, fma(-at.y, w0.y, fma(a.x, v0.x, -(a.y * v0.y))));
    py0 = fma(at.x, w0.y, fma(at.y, w0.x, fma(a.x, v0.y, a.y * v0.x)));
    px1 = fma(at.x, w1.x, fma(-at.y, w1.y, fma(a.x, v1.x, -(a.y * v1.y))));
    py1 = fma(at.x, w1.y, fma(at.y, w1.x, fma(a.x, v1.y, a.y * v1.x)));
  } else {
    px0 = fma(a.x, w0.x, -(a.y * w0.y)), py0 = fma(a.x, w0.y, a.y * w0.x);
    px1 = fma(a.x, w1.x, -(a.y * w1.y)), py1 = fma(a.x, w1.y, a.y * w1.x);
  }
  double2 c[N];
#define YK_C(Q) \
  if constexpr (Q < N) c[Q] = lds2<WO + 16 * (Q)>(wt);
  YK_C(0) YK_C(1) YK_C(2) YK_C(3) YK_C(4)
#undef YK_C
#pragma unroll
  for (int q = 0; q < N; q++) {
    Z[q][0].x = fma(c[q].x, px0, Z[q][0].x);
    Z[q][0].y = fma(c[q].x, py0, Z[q][0].y);
    Z[q][1].x = fma(c[q].y, px1, Z[q][1].x);
    Z[q][1].y = fma(c[q].y, py1, Z[q][1].y);
  }
}

// The n steps of one row pair, two at a time (the window moves by renaming).  p1, p2: addresses
// of the rows' first elements, d1, d2 the way to the next ones; m1, m2: the conjugates of a
// mirrored row (its signs are in the weights); wt: address of the weights; tan: from an element of
// U to that of Udot (TAN).
template <int N, bool TAN>
__device__ __forceinline__ void yk_pair(unsigned p1, unsigned p2, int d1, int d2, unsigned m1, unsigned m2,
                                        unsigned wt, int n, unsigned tan, double2 (&Z)[YNJ][YT]) {
  constexpr int DW = N * YT * 8;
  const double2 none = make_double2(0.0, 0.0);
  double2 w1 = conj_if(lds2<0>(p2 - d2), m2), v1 = TAN ? conj_if(lds2<0>(p2 - d2 + tan), m2) : none;
#pragma unroll 1
  for (; n >= 2; n -= 2) {
    const double2 a = conj_if(lds2<0>(p1), m1), w0 = conj_if(lds2<0>(p2), m2);
    const double2 at = TAN ? conj_if(lds2<0>(p1 + tan), m1) : none, v0 = TAN ? conj_if(lds2<0>(p2 + tan), m2) : none;
    p1 += d1;
    p2 += d2;
    const double2 b = conj_if(lds2<0>(p1), m1), bt = TAN ? conj_if(lds2<0>(p1 + tan), m1) : none;
    yk_step<N, 0, TAN>(a, w0, w1, at, v0, v1, wt, Z);
    w1 = conj_if(lds2<0>(p2), m2);
    if (TAN) v1 = conj_if(lds2<0>(p2 + tan), m2);
    p1 += d1;
    p2 += d2;
    yk_step<N, DW, TAN>(b, w1, w0, bt, v1, v0, wt, Z);
    wt += 2 * DW;
  }
  if (n)
    yk_step<N, 0, TAN>(conj_if(lds2<0>(p1), m1), conj_if(lds2<0>(p2), m2), w1,
                       TAN ? conj_if(lds2<0>(p1 + tan), m1) : none, TAN ? conj_if(lds2<0>(p2 + tan), m2) : none, v1, wt,
                       Z);
}

// One record: its m row pairs (from pi on), n steps each, into Z[0 .. N-1] (the N levels of the
// (j1, j2) pair that the item holds).
template <int N, int PL>
__device__ __forceinline__ void yk_record(const YkTab& T, unsigned us, unsigned us2, int pi, int m, int n, bool first,
                                          unsigned wt, unsigned tan,
                                          double2 (&Z)[YNJ][YT]) {
  if (first) {
#pragma unroll
    for (int q = 0; q < N; q++)
#pragma unroll
      for (int t = 0; t < YT; t++) Z[q][t] = make_double2(0.0, 0.0);
  }
  const int wn = n * (N * YT * 8);
#pragma unroll 1
  for (int q = 0; q < m; q++) {
    const int2 x = T.pair[pi + q];
    int d1 = YE - ((x.x & 1) << 10), d2 = ((x.y & 1) << 10) - YE;
    unsigned m1 = (unsigned)x.x << 31, m2 = (unsigned)x.y << 31;
    // kept in registers: the compiler would form them again in every step
    asm volatile("" : "+r"(d1), "+r"(d2), "+r"(m1), "+r"(m2));
    yk_pair<N, PL == PL_TANGENT>(us + (unsigned)(x.x & ~1), us2 + (unsigned)(x.y & ~1), d1, d2, m1, m2, wt, n, tan,
                                 Z);
    wt += wn;
  }
}

// Y of levels LO .. LO + N - 1 of the item += coef Z.
template <int N, int LO>
__device__ __forceinline__ void yk_add(const double* __restrict__ coef, const double2 (&Z)[YNJ][YT],
                                       double2 (&Y)[YNJ][YT]) {
#pragma unroll
  for (int q = 0; q < N; q++) {
    if (LO + q >= YNJ) break;
    const double c = coef[q];
#pragma unroll
    for (int t = 0; t < YT; t++) {
      Y[LO + q][t].x = fma(c, Z[q][t].x, Y[LO + q][t].x);
      Y[LO + q][t].y = fma(c, Z[q][t].y, Y[LO + q][t].y);
    }
  }
}

// The last record of a (j1, j2) pair: its Z goes out and into Y.
template <int YM, int N>
__device__ __forceinline__ void yk_finish(const SnapDev& S, const YkItem& it, int lo, int trip,
                                          const double* __restrict__ coef, int64_t n, int64_t atom, bool valid,
                                          const double2 (&Z)[YNJ][YT], double2 (&Y)[YNJ][YT],
                                          double2* __restrict__ zout) {
  if (YM != YM_Y) {
#pragma unroll
    for (int q = 0; q < N; q++) {
      const int j = it.jmin + 2 * (lo + q), z0 = S.ytrip_jjz[trip + q] + ((j - it.k) >> 1) * (j + 1);
#pragma unroll
      for (int t = 0; t < YT; t++) {
        const int c = it.c0 + 2 * t;
        if (valid && t < it.nt && c <= j && c >= -j) zout[(size_t)(z0 + ((j + c) >> 1)) * n + atom] = Z[q][t];
      }
    }
  }
  if (YM != YM_Z) {
    switch (lo) {
      case 0:
        yk_add<N, 0>(coef + trip, Z, Y);
        break;
      case 1:
        yk_add<N, 1>(coef + trip, Z, Y);
        break;
      case 2:
        yk_add<N, 2>(coef + trip, Z, Y);
        break;
      case 3:
        yk_add<N, 3>(coef + trip, Z, Y);
        break;
      default:
        yk_add<N, 4>(coef + trip, Z, Y);
        break;
    }
  }
}

// YM: YM_Y writes the weighted Y' (yout [u_half][n]) and E_i; YM_Z writes Z (zout [idxz_max][n]);
// YM_YZ both.  gridDim.y > 1 splits the items of a tile over that many blocks, each taking items
// blockIdx.y, blockIdx.y + gridDim.y, ...; the items' energies then go to eitem [items][n] and
// k_snap_yenergy adds them.  An item's result does not depend on the warp that computes it, and
// energies are summed in item order, so neither split nor scheduling changes any bit.
// PL_TWO (Z only): row 2 from a second Utot, for blockIdx.z = p ne + q that of element q against
// element p's (ustride apart; zstride between the pairs' Z).  PL_TANGENT (YM_Y, no energy): utot20 is V
// [u_half][n] of k_snap_vlie, up to the middle element of a level; Udot = -V.
template <int YM, int PL>
__global__ void __launch_bounds__(yk_warps(PL) * 32, PL == PL_TANGENT ? 1 : 2) k_snap_ystream(const __grid_constant__ SnapDev S,
                                                          const __grid_constant__ YkTab T, int64_t n,
                                                          const int32_t* __restrict__ species,
                                                          const double2* __restrict__ utot0,
                                                          const double2* __restrict__ utot20,
                                                          double2* __restrict__ yout, double* __restrict__ Ei,
                                                          double2* __restrict__ zout0, double* __restrict__ eitem,
                                                          int ne, int64_t ustride, int64_t zstride) {
  constexpr bool TWO = PL == PL_TWO;
  constexpr int YK_T = yk_warps(PL) * 32;
  extern __shared__ __align__(16) unsigned char ysh[];
  __shared__ int next_item;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int UH = S.u_half, NI = T.nitem;
  const YkSmem M = yk_smem(S.nsp, S.n_ytrip, UH, NI, PL);
  double* coefs = reinterpret_cast<double*>(ysh);  // [nsp][n_ytrip]
  double2* guard0 = reinterpret_cast<double2*>(ysh + M.coef);
  double2* us = reinterpret_cast<double2*>(ysh + M.coef + M.guard);
  double2* guard1 = reinterpret_cast<double2*>(ysh + M.coef + M.guard + M.u);
  double2* us2 = PL != PL_ONE ? guard1 + YGUARD * YS_ATOMS : us;
  double* erow = reinterpret_cast<double*>(ysh + M.coef + M.planes());
  double2* ring = reinterpret_cast<double2*>(ysh + M.coef + M.planes() + M.energy) + warp * YK_SLOTS * YREC;
  if (YM != YM_Z)
    for (int q = threadIdx.x; q < S.nsp * S.n_ytrip; q += YK_T) {
      const int sp = q / S.n_ytrip, t = q - sp * S.n_ytrip;
      coefs[q] = S.ycoef[(size_t)sp * S.idxz_max + S.ytrip_jjz[t]];
    }
  for (int q = threadIdx.x; q < YGUARD * YS_ATOMS; q += YK_T) {
    guard0[q] = guard1[q] = make_double2(0.0, 0.0);
    if (PL != PL_ONE) us2[UH * YS_ATOMS + q] = make_double2(0.0, 0.0);
  }
  const double2* __restrict__ utot = TWO ? utot0 + (blockIdx.z / ne) * ustride : utot0;
  const double2* __restrict__ utot2 = TWO ? utot20 + (blockIdx.z % ne) * ustride : utot0;
  double2* __restrict__ zout = TWO ? zout0 + blockIdx.z * zstride : zout0;
  const bool split = gridDim.y > 1;
  for (int64_t a0 = (int64_t)blockIdx.x * YS_ATOMS; a0 < n; a0 += (int64_t)gridDim.x * YS_ATOMS) {
    const int na_blk = (int)((n - a0) < YS_ATOMS ? (n - a0) : YS_ATOMS);
    for (int idx = threadIdx.x; idx < UH * YS_ATOMS; idx += YK_T) {
      const int q = idx / YS_ATOMS, l = idx - q * YS_ATOMS;
      const size_t at = (size_t)(a0 + l) * S.idxu_max + S.u_of_h[q];
      us[idx] = l < na_blk ? utot[at] : make_double2(0.0, 0.0);
      if (TWO) us2[idx] = l < na_blk ? utot2[at] : make_double2(0.0, 0.0);
      if (PL == PL_TANGENT) {
        const int hi = S.h_info[q], m = hi & 0xff, j = (hi >> 8) & 0xff;
        const bool mir = !(hi >> 16);  // beyond the middle: (-1)^(ma+mb) conj of the row's mirror element, mb = j / 2
        double2 v = l < na_blk ? utot20[(size_t)(mir ? q - 2 * m + j : q) * n + a0 + l] : make_double2(0.0, 0.0);
        const bool odd = (m + j / 2) & 1;
        us2[idx] = make_double2(mir && odd ? v.x : -v.x, mir && !odd ? v.y : -v.y);
      }
    }
    if (threadIdx.x == 0) next_item = blockIdx.y;
    __syncthreads();
    const int64_t atom = a0 + lane;
    const bool valid = lane < na_blk;
    int si = valid && YM != YM_Z ? species[atom] : 0;
    si = si < 0 ? 0 : (si >= S.nsp ? S.nsp - 1 : si);
    const double* coef = coefs + si * S.n_ytrip;
    const double2* usl = us + lane;
    const unsigned usa = (unsigned)__cvta_generic_to_shared(usl), ringa = (unsigned)__cvta_generic_to_shared(ring);
    const unsigned tan = (unsigned)((us2 - us) * sizeof(double2));
    const unsigned usb = TWO ? (unsigned)__cvta_generic_to_shared(us2 + lane) : usa;
    // items are handed out longest first to whichever warp is free
    for (;;) {
      int r = 0;
      if (lane == 0) r = atomicAdd(&next_item, (int)gridDim.y);
      r = (int)__reduce_max_sync(0xffffffffu, (unsigned)r);  // a uniform register: so are all indices below
      if (r >= NI) break;
      const YkItem& it = T.item[r];
      const double2* src = S.ykstream + it.unit;
      int ri = it.rec, pi = it.pair;
      const int rend = ri + it.nrec;
      __syncwarp();
#pragma unroll
      for (int q = 0; q < 2; q++) {
        const int size = (T.rec[ri + q] >> YF_SIZE) & 0xff;
        if (lane < size) cp16(ring + q * YREC + lane, src + lane);
        if (lane + 32 < size) cp16(ring + q * YREC + lane + 32, src + lane + 32);
        asm volatile("cp.async.commit_group;");
        src += size;
      }
      double2 Z[YNJ][YT], Y[YNJ][YT];
#pragma unroll
      for (int q = 0; q < YNJ; q++)
#pragma unroll
        for (int t = 0; t < YT; t++) Z[q][t] = Y[q][t] = make_double2(0.0, 0.0);
      int slot = 0;
      for (; ri < rend; ri++) {
        __syncwarp();  // every lane is done with the slot that the copy overwrites
        {
          double2* dst = ring + (slot == 0 ? 2 : slot - 1) * YREC;
          const int size = (T.rec[ri + 2] >> YF_SIZE) & 0xff;
          if (lane < size) cp16(dst + lane, src + lane);
          if (lane + 32 < size) cp16(dst + lane + 32, src + lane + 32);
          asm volatile("cp.async.commit_group;");
          src += size;
        }
        asm volatile("cp.async.wait_group 2;" ::: "memory");
        __syncwarp();
        const uint32_t f = T.rec[ri];
        const int m = f & 15, n_steps = (f >> YF_STEPS) & 15, lo = (f >> YF_LO) & 7, trip = f >> YF_TRIP;
        const unsigned wt = ringa + slot * (YREC * 16);
        const bool first = (f & YF_FIRST) != 0, last = (f & YF_LAST) != 0;
        slot = slot == 2 ? 0 : slot + 1;
#define YK_CASE(N)                                                                             \
  case N:                                                                                      \
    yk_record<N, PL>(T, usa, usb, pi, m, n_steps, first, wt, tan, Z);                          \
    if (last) yk_finish<YM, N>(S, it, lo, trip, coef, n, atom, valid, Z, Y, zout);             \
    break;
        switch ((f >> YF_N) & 7) {
          YK_CASE(1)
          YK_CASE(2)
          YK_CASE(3)
          YK_CASE(4)
          YK_CASE(5)
          default:
            break;
        }
#undef YK_CASE
        pi += m;
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      if (YM != YM_Z) {
        double e = 0.0;
#pragma unroll
        for (int q = 0; q < YNJ; q++) {
          const int j = it.jmin + 2 * q;
          if (j > S.J) break;
#pragma unroll
          for (int t = 0; t < YT; t++) {
            const int c = it.c0 + 2 * t;
            if (t >= it.nt || c > j || c < -j) continue;
            const int h = S.half_block[j] + ((j - it.k) >> 1) * (j + 1) + ((j + c) >> 1);
            const double w = it.k == 0 && c == 0 ? 0.5 : 1.0;  // the centre of an even level
            const double2 y = make_double2(w * Y[q][t].x, w * Y[q][t].y);
            if (valid) yout[(size_t)h * n + atom] = y;
            if (PL == PL_TANGENT) continue;
            const double2 u = usl[h * YS_ATOMS];
            e += u.x * y.x + u.y * y.y;
          }
        }
        if (PL == PL_TANGENT) continue;
        if (!split)
          erow[r * YS_ATOMS + lane] = e;
        else if (valid)
          eitem[(size_t)r * n + atom] = e;
      }
    }
    __syncthreads();
    if (YM != YM_Z && PL != PL_TANGENT && !split && warp == 0 && valid) {
      double t = 0.0;
      for (int r = 0; r < NI; r++) t += erow[r * YS_ATOMS + lane];
      Ei[atom] = (2.0 / 3.0) * t + S.ebias[si];
    }
    __syncthreads();
  }
}

// E_i of a split launch: the items' energies in item order.
__global__ void k_snap_yenergy(const __grid_constant__ SnapDev S, int nitem, int64_t n, const int32_t* __restrict__ species,
                               const double* __restrict__ eitem, double* __restrict__ Ei) {
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double t = 0.0;
#pragma unroll 32
  for (int r = 0; r < nitem; r++) t += eitem[(size_t)r * n + i];
  int si = species[i];
  si = si < 0 ? 0 : (si >= S.nsp ? S.nsp - 1 : si);
  Ei[i] = (2.0 / 3.0) * t + S.ebias[si];
}

template <int YM, int PL = PL_ONE>
int launch_ystream_m(ipg_ctx* ctx, const SnapDev& dev, const YkTab& tab, const char* tname, int64_t n,
                     const int32_t* species, const double2* utot, double2* yout, double* Ei, double2* zout,
                     const double2* utot2 = nullptr, int ne = 1, int64_t ustride = 0, int64_t zstride = 0) {
  constexpr int warps = yk_warps(PL), YK_T = warps * 32;
  const auto kernel = k_snap_ystream<YM, PL>;
  const int smem = yk_smem(dev.nsp, dev.n_ytrip, dev.u_half, tab.nitem, PL).total();
  IPG_RET(ipg_smem_limit(ctx, kernel, smem));
  int per_sm = 1;
  CUDA_RET(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, YK_T, smem));
  const int64_t resident = (int64_t)ctx->num_sms * std::max(1, per_sm);
  const int64_t tiles = (n + YS_ATOMS - 1) / YS_ATOMS, pairs = PL == PL_TWO ? (int64_t)ne * ne : 1;
  // Fewer tiles than resident blocks: the items of a tile go to several blocks, at most one
  // block per YK_WARPS items (249 atoms, twojmax 8: 167 us with one block per tile, 74 us split).
  // The tiles of a last, partly filled wave stay whole: split so that the wave ends earlier they
  // took longer (each block stages its tile's Utot again): 3,160 against 3,060 us a pullback of 16,000
  // atoms, 2,544 against 2,520 at 54,000.
  const int64_t most = (tab.nitem + warps - 1) / warps;
  const int64_t nsplit = std::max<int64_t>(1, std::min(most, resident / std::max<int64_t>(1, tiles * pairs)));
  const dim3 grid((unsigned)std::min(tiles, resident), (unsigned)nsplit, (unsigned)pairs);
  double* eitem = nullptr;
  if (YM != YM_Z && PL != PL_TANGENT && nsplit > 1) IPG_RET(scratch(ctx, "snap_yitem", (size_t)tab.nitem * n, &eitem));
  IPG_TIMED_LAUNCH(ctx, tname, kernel, grid, YK_T, smem, dev, tab, n, species, utot, utot2, yout, Ei, zout, eitem, ne,
                   ustride, zstride);
  if (eitem) IPG_LAUNCH(ctx, k_snap_yenergy, (unsigned)((n + 127) / 128), 128, 0, dev, tab.nitem, n, species, eitem, Ei);
  return IPG_OK;
}

}  // namespace

int launch_ystream(ipg_ctx* ctx, const SnapDev& dev, const YkTab& tab, int ym, const char* tname, int64_t n,
                   const int32_t* species, const double2* utot, double2* yout, double* Ei, double2* zout) {
  if (n <= 0) return IPG_OK;
  if (ym == YM_Z) return launch_ystream_m<YM_Z>(ctx, dev, tab, tname, n, species, utot, yout, Ei, zout);
  if (ym == YM_YZ) return launch_ystream_m<YM_YZ>(ctx, dev, tab, tname, n, species, utot, yout, Ei, zout);
  return launch_ystream_m<YM_Y>(ctx, dev, tab, tname, n, species, utot, yout, Ei, zout);
}

int launch_zpairs(ipg_ctx* ctx, const SnapDev& dev, const YkTab& tab, int64_t n, const int32_t* species, int ne,
                  const double2* utot, int64_t ustride, double2* zout, int64_t zstride) {
  if (n <= 0) return IPG_OK;
  constexpr const char* tname = "snap_zrows";
  // Few tiles: every pair in one launch, (p, p) from two copies of the same plane (1,999 atoms, two
  // elements, twojmax 6: 488 -> 392 us a call).  Otherwise one plane for (p, p), which leaves room for more blocks.
  if (ne > 1 && (n + YS_ATOMS - 1) / YS_ATOMS <= ctx->num_sms)
    return launch_ystream_m<YM_Z, PL_TWO>(ctx, dev, tab, tname, n, species, utot, nullptr, nullptr, zout, utot, ne, ustride,
                                        zstride);
  for (int p = 0; p < ne; p++)
    for (int q = 0; q < ne; q++) {
      const double2 *u = utot + p * ustride, *u2 = utot + q * ustride;
      double2* z = zout + (p * ne + q) * zstride;
      IPG_RET(p == q ? (launch_ystream_m<YM_Z>(ctx, dev, tab, tname, n, species, u, nullptr, nullptr, z))
                     : (launch_ystream_m<YM_Z, PL_TWO>(ctx, dev, tab, tname, n, species, u, nullptr, nullptr, z, u2)));
    }
  return IPG_OK;
}

int launch_ytangent(ipg_ctx* ctx, const SnapDev& dev, const YkTab& tab, int64_t n, const int32_t* species,
                    const double2* utot, const double2* V, double2* ydot) {
  if (n <= 0) return IPG_OK;
  return launch_ystream_m<YM_Y, PL_TANGENT>(ctx, dev, tab, "snap_hvp_y", n, species, utot, ydot, nullptr, nullptr, V);
}
