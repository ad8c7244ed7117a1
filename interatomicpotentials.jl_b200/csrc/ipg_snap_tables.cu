// ipg_snap_tables.cu — host construction of the SNAP index and Clebsch–Gordan tables.
//
// The tables are those of initialize_prebuilt_arrays
// (src/BasisSystems/SNAP/types/prebuilt_arrays.jl:48-321): the same enumeration order of
// (j1 >= j2, j = |j1-j2|..min(J, j1+j2) step 2) blocks, the same CG coefficients (factorial
// sums, :250-312) and sqrt(p/q) roots (:314-321), because the descriptors are defined by
// that ordering.  Derived tables (half-plane offsets, the Y gather list, the dB term list)
// are new and serve the CUDA kernels.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "ipg_snap.cuh"

namespace {

// Factorials, up to the largest of delta_cg, as long double (64-bit mantissa): exact wherever the
// reference's Int64 products are exact (twojmax <= 8), and free of Int64 overflow beyond that.
struct Factorials {
  long double f[3 * SNAP_MAX_J / 2 + 2];
  Factorials() {
    f[0] = f[1] = 1.0L;
    for (int k = 2; k < 3 * SNAP_MAX_J / 2 + 2; k++) f[k] = f[k - 1] * k;
  }
  long double operator()(int n) const { return f[n]; }
};

// prebuilt_arrays.jl:250-257
double delta_cg(const Factorials& fact, int j1, int j2, int j) {
  long double den = fact((j1 + j2 + j) / 2 + 1);
  long double num = fact((j1 + j2 - j) / 2) * fact((j1 - j2 + j) / 2) * fact((-j1 + j2 + j) / 2);
  return std::sqrt((double)num / (double)den);
}

}  // namespace

int snap_build_tables(const ipg_snap_params& p, SnapHost& h) {
  const int J = p.twojmax;
  if (J < 0 || J > SNAP_MAX_J) return IPG_ERR_ARG;
  const int jd = J + 1;
  h.J = J;
  auto blk = [jd](int a, int b, int c) { return (a * jd + b) * jd + c; };
  h.idxcg_block.assign(jd * jd * jd, -1);
  h.idxz_block.assign(jd * jd * jd, -1);
  h.idxb_block.assign(jd * jd * jd, -1);
  h.idxu_block.assign(jd, 0);
  h.half_block.assign(jd + 1, 0);

  int cnt = 0;
  for (int j1 = 0; j1 <= J; j1++)
    for (int j2 = 0; j2 <= j1; j2++)
      for (int j = j1 - j2; j <= std::min(J, j1 + j2); j += 2) {
        h.idxcg_block[blk(j1, j2, j)] = cnt;
        cnt += (j1 + 1) * (j2 + 1);
      }
  h.idxcg_max = cnt;

  cnt = 0;
  for (int j = 0; j <= J; j++) {
    h.idxu_block[j] = cnt;
    cnt += (j + 1) * (j + 1);
  }
  h.idxu_max = cnt;

  // half plane: rows mb = 0..j/2 of every level
  cnt = 0;
  h.ext_max = 1;
  for (int j = 0; j <= J; j++) {
    h.half_block[j] = cnt;
    cnt += (j / 2 + 1) * (j + 1);
    h.ext_max = std::max(h.ext_max, ((j + 1) / 2 + 1) * (j + 1));
  }
  h.half_block[jd] = cnt;
  h.u_half = cnt;
  h.h_info.clear();
  h.h_sgen.clear();
  for (int j = 0; j <= J; j++)
    for (int mb = 0; 2 * mb <= j; mb++)
      for (int m = 0; m <= j; m++) {
        const int last = (2 * mb == j) ? mb : j;  // the middle row of an even level is weighted up to mb
        h.h_info.push_back(m | (j << 8) | ((m <= last ? 1 : 0) << 16));
        h.h_sgen.push_back(m < j ? std::sqrt((double)((m + 1) * (j - m))) : 0.0);
        h.h_sgen.push_back(m >= 1 ? std::sqrt((double)(m * (j - m + 1))) : 0.0);
      }

  h.idxb.clear();
  for (int j1 = 0; j1 <= J; j1++)
    for (int j2 = 0; j2 <= j1; j2++)
      for (int j = j1 - j2; j <= std::min(J, j1 + j2); j += 2)
        if (j >= j1) {
          h.idxb_block[blk(j1, j2, j)] = (int)h.idxb.size() / 3;
          h.idxb.push_back(j1);
          h.idxb.push_back(j2);
          h.idxb.push_back(j);
        }
  h.idxb_max = (int)h.idxb.size() / 3;

  h.idxz.clear();
  h.zjju_half.clear();
  for (int j1 = 0; j1 <= J; j1++)
    for (int j2 = 0; j2 <= j1; j2++)
      for (int j = j1 - j2; j <= std::min(J, j1 + j2); j += 2) {
        h.idxz_block[blk(j1, j2, j)] = (int)h.idxz.size();
        for (int mb = 0; 2 * mb <= j; mb++)
          for (int ma = 0; ma <= j; ma++) {
            int ma1min = std::max(0, (2 * ma - j - j2 + j1) / 2);
            int ma2max = (2 * ma - j - (2 * ma1min - j1) + j2) / 2;
            int na = std::min(j1, (2 * ma - j + j2 + j1) / 2) - ma1min + 1;
            int mb1min = std::max(0, (2 * mb - j - j2 + j1) / 2);
            int mb2max = (2 * mb - j - (2 * mb1min - j1) + j2) / 2;
            int nb = std::min(j1, (2 * mb - j + j2 + j1) / 2) - mb1min + 1;
            ZDev z;
            z.j1 = (int8_t)j1;
            z.j2 = (int8_t)j2;
            z.j = (int8_t)j;
            z.na = (int8_t)na;
            z.nb = (int8_t)nb;
            z.pad0 = z.pad1 = z.pad2 = 0;
            z.ma1min = (int8_t)ma1min;
            z.ma2max = (int8_t)ma2max;
            z.mb1min = (int8_t)mb1min;
            z.mb2max = (int8_t)mb2max;
            z.u1base = h.idxu_block[j1] + (j1 + 1) * mb1min + ma1min;
            z.u2base = h.idxu_block[j2] + (j2 + 1) * mb2max + ma2max;
            z.icga0 = ma1min * (j2 + 1) + ma2max;
            z.icgb0 = mb1min * (j2 + 1) + mb2max;
            z.cgoff = h.idxcg_block[blk(j1, j2, j)];
            h.idxz.push_back(z);
            h.zjju_half.push_back(h.half_block[j] + (j + 1) * mb + ma);
          }
      }
  h.idxz_max = (int)h.idxz.size();

  h.rootpq.assign((J + 2) * (J + 2), 0.0);
  for (int a = 1; a <= J; a++)
    for (int b = 1; b <= J; b++) h.rootpq[a * (J + 2) + b] = std::sqrt((double)a / (double)b);

  h.cglist.assign(h.idxcg_max, 0.0);
  const Factorials fact;
  int idx = 0;
  for (int j1 = 0; j1 <= J; j1++)
    for (int j2 = 0; j2 <= j1; j2++)
      for (int j = j1 - j2; j <= std::min(J, j1 + j2); j += 2) {
        const double delta = delta_cg(fact, j1, j2, j);
        for (int m1 = 0; m1 <= j1; m1++) {
          int aa2 = 2 * m1 - j1;
          for (int m2 = 0; m2 <= j2; m2++, idx++) {
            int bb2 = 2 * m2 - j2;
            int m = (aa2 + bb2 + j) / 2;
            if (m < 0 || m > j) continue;
            double sum = 0.0;
            int zmin = std::max(0, std::max(-(j - j2 + aa2) / 2, -(j - j1 - bb2) / 2));
            int zmax = std::min((j1 + j2 - j) / 2, std::min((j1 - aa2) / 2, (j2 + bb2) / 2));
            for (int z = zmin; z <= zmax; z++) {
              long double den = fact(z) * fact((j1 + j2 - j) / 2 - z) * fact((j1 - aa2) / 2 - z) * fact((j2 + bb2) / 2 - z) *
                            fact((j - j2 + aa2) / 2 + z) * fact((j - j1 - bb2) / 2 + z);
              sum += ((z % 2 == 0) ? 1.0 : -1.0) / (double)den;
            }
            int cc2 = 2 * m - j;
            long double sf = fact((j1 + aa2) / 2) * fact((j1 - aa2) / 2) * fact((j2 + bb2) / 2) * fact((j2 - bb2) / 2) *
                         fact((j + cc2) / 2) * fact((j - cc2) / 2) * (long double)(j + 1);
            h.cglist[idx] = sum * delta * std::sqrt((double)sf);
          }
        }
      }

  // bzero (prebuilt_arrays.jl:52-63); wself = 1
  h.bzero.assign(jd, 0.0);
  if (p.bzero_flag)
    for (int j = 0; j <= J; j++) h.bzero[j] = p.bnorm_flag ? 1.0 : (double)(j + 1);

  // dB terms (compute_b.jl:207-400): Z(j1,j2,j) on level j, (j+1)/(j1+1) Z(j,j2,j1) on
  // level j1, (j+1)/(j2+1) Z(j,j1,j2) on level j2 (factors dropped when bnorm_flag).
  h.db.resize(h.idxb_max);
  for (int b = 0; b < h.idxb_max; b++) {
    int j1 = h.idxb[3 * b], j2 = h.idxb[3 * b + 1], j = h.idxb[3 * b + 2];
    DBDev& d = h.db[b];
    d.l[0] = j;
    d.z0[0] = h.idxz_block[blk(j1, j2, j)];
    d.fac[0] = 1.0;
    d.l[1] = j1;
    d.z0[1] = h.idxz_block[blk(j, j2, j1)];
    d.fac[1] = p.bnorm_flag ? 1.0 : (j + 1) / (j1 + 1.0);
    d.l[2] = j2;
    d.z0[2] = h.idxz_block[blk(j, j1, j2)];
    d.fac[2] = p.bnorm_flag ? 1.0 : (j + 1) / (j2 + 1.0);
  }

  // Y = d(beta . B)/dU (design of compute_yi.jl:86-118): each Z entry (J1,J2,J,ma,mb)
  // feeds Y(J,ma,mb) with weight beta[jjb] times multiplicity and (J1+1)/(J+1).
  h.y_jjb.assign(h.idxz_max, 0);
  h.y_mult.assign(h.idxz_max, 0.0);
  for (int z = 0; z < h.idxz_max; z++) {
    int j1 = h.idxz[z].j1, j2 = h.idxz[z].j2, j = h.idxz[z].j;
    int jjb;
    double mult;
    if (j >= j1) {
      jjb = h.idxb_block[blk(j1, j2, j)];
      mult = (j1 == j) ? ((j2 == j) ? 3.0 : 2.0) : 1.0;
    } else if (j >= j2) {
      jjb = h.idxb_block[blk(j, j2, j1)];
      mult = (j2 == j) ? 2.0 : 1.0;
    } else {
      jjb = h.idxb_block[blk(j2, j, j1)];
      mult = 1.0;
    }
    if (!p.bnorm_flag && j1 > j) mult *= (j1 + 1) / (j + 1.0);
    h.y_jjb[z] = jjb;
    h.y_mult[z] = mult;
  }
  h.zfac.assign(h.idxz_max, 0.0);
  for (int j1 = 0; j1 <= J; j1++)
    for (int j2 = 0; j2 <= j1; j2++)
      for (int j = j1 - j2; j <= std::min(J, j1 + j2); j += 2)
        for (int mb = 0; 2 * mb <= j; mb++)
          for (int ma = 0; ma <= j; ma++) {
            const int z = h.idxz_block[blk(j1, j2, j)] + mb * (j + 1) + ma;
            h.zfac[z] = (2 * mb == j && ma == mb ? 1.0 : 2.0) * h.y_mult[z];
          }
  h.y_off.assign(h.u_half + 1, 0);
  for (int z = 0; z < h.idxz_max; z++) h.y_off[h.zjju_half[z] + 1]++;
  for (int q = 0; q < h.u_half; q++) h.y_off[q + 1] += h.y_off[q];
  // Z entries in order of their loop shape, so that the threads of a warp that take
  // consecutive entries run identical (nb, na) trip counts
  {  // counted into the places of each (nb, na), both at most J + 1
    std::vector<int> place((jd + 1) * (jd + 1) + 1, 0);
    auto shape = [&](int z) { return h.idxz[z].nb * (jd + 1) + h.idxz[z].na; };
    for (int z = 0; z < h.idxz_max; z++) place[shape(z) + 1]++;
    for (size_t q = 1; q < place.size(); q++) place[q] += place[q - 1];
    h.zperm.resize(h.idxz_max);
    for (int z = 0; z < h.idxz_max; z++) h.zperm[place[shape(z)]++] = z;
  }
  // Y schedule: every half-plane entry with nonzero weight goes to one of YS_WARPS warps,
  // longest first to the least loaded warp (cost = inner terms of its Z entries)
  {
    h.u_of_h.assign(h.u_half, 0);
    std::vector<std::pair<double, int>> cost;  // (cost, h)
    std::vector<double> wgt(h.u_half, 0.0);
    std::vector<double> hc(h.u_half, 0.0);
    for (int z = 0; z < h.idxz_max; z++) hc[h.zjju_half[z]] += h.idxz[z].nb * (2.0 + h.idxz[z].na) + 2.0;
    for (int j = 0; j <= J; j++)
      for (int mb = 0; 2 * mb <= j; mb++)
        for (int ma = 0; ma <= j; ma++) {
          const int hh = h.half_block[j] + mb * (j + 1) + ma;
          h.u_of_h[hh] = h.idxu_block[j] + mb * (j + 1) + ma;
          wgt[hh] = (2 * mb < j) ? 1.0 : (ma < mb ? 1.0 : (ma == mb ? 0.5 : 0.0));
          if (wgt[hh] != 0.0) cost.push_back({hc[hh], hh});
        }
    std::stable_sort(cost.begin(), cost.end(), [](const std::pair<double, int>& a, const std::pair<double, int>& b) {
      return a.first > b.first;
    });
    std::vector<std::vector<int>> bins(YS_WARPS);
    std::vector<double> load(YS_WARPS, 0.0);
    for (auto& c : cost) {
      int w = (int)(std::min_element(load.begin(), load.end()) - load.begin());
      bins[w].push_back(c.second);
      load[w] += c.first;
    }
    h.ysched_off.assign(YS_WARPS + 1, 0);
    h.ysched_h.clear();
    h.ysched_w.clear();
    for (int w = 0; w < YS_WARPS; w++) {
      std::sort(bins[w].begin(), bins[w].end());
      for (int hh : bins[w]) {
        h.ysched_h.push_back(hh);
        h.ysched_w.push_back(wgt[hh]);
      }
      h.ysched_off[w + 1] = (int)h.ysched_h.size();
    }
  }
  h.y_jjz.assign(h.idxz_max, 0);
  std::vector<int32_t> fill(h.y_off.begin(), h.y_off.end() - 1);
  for (int z = 0; z < h.idxz_max; z++) h.y_jjz[fill[h.zjju_half[z]]++] = z;

  // Streamed Y / Z contraction (layout: ipg_snap.cuh).  Items (k, YT adjacent columns c) in the
  // doubled indices k = -(2 mb - j) >= 0, c = 2 ma - j; the centre row k = 0 needs c <= 0 only.
  memset(&h.yktab, 0, sizeof(h.yktab));
  h.ykstream.clear();
  h.ytrip_jjz.clear();
  h.ytrip_b.clear();
  h.ytrip_fac.clear();
  h.ylev.clear();
  if (J <= YR_MAX_J) {
    std::vector<int32_t> trip_of(jd * jd * jd, -1);
    for (int j1 = 0; j1 <= J; j1++)
      for (int j2 = 0; j2 <= j1; j2++)
        for (int j = j1 - j2; j <= std::min(J, j1 + j2); j += 2) {  // the levels of a pair are adjacent
          trip_of[blk(j1, j2, j)] = (int32_t)h.ytrip_jjz.size();
          h.ytrip_jjz.push_back(h.idxz_block[blk(j1, j2, j)]);
        }
    // the component of each triple and the terms of its derivative (compute_b.jl:104-400) that read it
    h.ytrip_b.assign(h.ytrip_jjz.size(), 0);
    h.ytrip_fac.assign(h.ytrip_jjz.size(), 0.0);
    std::vector<int32_t> trip_at(h.idxz_max, -1);  // by first Z entry
    for (size_t q = 0; q < h.ytrip_jjz.size(); q++) trip_at[h.ytrip_jjz[q]] = (int32_t)q;
    for (int b = 0; b < h.idxb_max; b++)
      for (int t = 0; t < 3; t++) {
        const int q = trip_at[h.db[b].z0[t]];
        h.ytrip_b[q] = b | (((h.ytrip_b[q] >> 16) | (1 << t)) << 16);
        h.ytrip_fac[q] = h.db[b].fac[t];
      }
    h.ylev.assign(J + 2, 0);
    for (int j = 0; j <= J; j++) {
      for (int j1 = 0; j1 <= J; j1++)
        for (int j2 = 0; j2 <= j1; j2++)
          if (j >= j1 - j2 && j <= std::min(J, j1 + j2) && !((j1 + j2 + j) & 1))
            h.ylev.push_back(trip_of[blk(j1, j2, j)]);
      h.ylev[j + 1] = (int32_t)h.ylev.size() - (J + 2);
    }
    struct YkRows {
      int8_t j1, j2, mb1, mb2, lo1, hi1, jlo, N, E, mir;  // mir: the row beyond the half plane (0, 1, 2)
    };
    struct Item {
      YkItem it;
      std::vector<uint32_t> recs;
      std::vector<int2> pairs;
      std::vector<YkRows> rows;  // of every row pair, for its weights
      size_t units = 0;
      double cost = 0.0;
    };
    std::vector<Item> items;
    items.reserve(YK_ITEMS);
    for (int k = 0; k <= J; k++) {
      const int cmax = k == 0 ? 0 : J - ((J - k) & 1);
      for (int c0 = -(J - ((J - k) & 1)); c0 <= cmax; c0 += 2 * YT) {
        items.emplace_back();
        Item& I = items.back();
        memset(&I.it, 0, sizeof(I.it));
        I.recs.reserve(64);
        I.pairs.reserve(128);
        I.rows.reserve(128);
        int nt = 0, jmin = J + 1;
        for (int t = 0; t < YT && c0 + 2 * t <= cmax; t++) {
          nt++;
          jmin = std::min(jmin, std::max(k, std::abs(c0 + 2 * t)));
        }
        I.it.k = (int16_t)k;
        I.it.c0 = (int16_t)c0;
        I.it.nt = (int16_t)nt;
        I.it.jmin = (int16_t)jmin;
        for (int j1 = 0; j1 <= J; j1++)
          for (int j2 = 0; j2 <= j1; j2++) {
            const int jlo = std::max(jmin, j1 - j2), jhi = std::min(J, j1 + j2);
            if (((j1 + j2 - k) & 1) || jlo > jhi) continue;
            const int N = (jhi - jlo) / 2 + 1;
            const int E = (c0 + j1 + j2) / 2;  // ma1 + ma2 of column t is E + t
            const int lo1 = std::max(0, E - j2), hi1 = std::min(j1, E + nt - 1);
            if (lo1 > hi1) continue;
            const size_t first = I.recs.size();
            for (int mb1 = 0; mb1 <= j1; mb1++) {
              const int mb2 = (j1 + j2 - k) / 2 - mb1;
              if (mb2 < 0 || mb2 > j2) continue;
              const bool mir1 = 2 * mb1 > j1, mir2 = 2 * mb2 > j2;  // at most one of them: k >= 0
              const int e1 = h.half_block[j1] + (mir1 ? (j1 - mb1) * (j1 + 1) + j1 - lo1 : mb1 * (j1 + 1) + lo1);
              const int ma2 = E - lo1;  // column t = 0 of the first step
              const int e2 = h.half_block[j2] + (mir2 ? (j2 - mb2) * (j2 + 1) + j2 - ma2 : mb2 * (j2 + 1) + ma2);
              const int steps = hi1 - lo1 + 1, units = steps * N * YT / 2;
              if (I.recs.size() == first || (int)((I.recs.back() >> YF_SIZE) & 0xff) + units > YREC)
                I.recs.push_back((uint32_t)steps << YF_STEPS | (uint32_t)N << YF_N | (uint32_t)((jlo - jmin) / 2) << YF_LO |
                                 (uint32_t)trip_of[blk(j1, j2, jlo)] << YF_TRIP);
              I.recs.back() += 1u | (uint32_t)units << YF_SIZE;
              I.pairs.push_back(make_int2(e1 * YS_ATOMS * 16 | (int)mir1, e2 * YS_ATOMS * 16 | (int)mir2));
              I.rows.push_back({(int8_t)j1, (int8_t)j2, (int8_t)mb1, (int8_t)mb2, (int8_t)lo1, (int8_t)hi1, (int8_t)jlo,
                                (int8_t)N, (int8_t)E, (int8_t)(mir1 ? 1 : (mir2 ? 2 : 0))});
              I.units += units;
              I.cost += steps * YT * (4.0 + 2.0 * N) + 20.0;
            }
            if (I.recs.size() > first) {
              I.recs[first] |= YF_FIRST;
              I.recs.back() |= YF_LAST;
            }
          }
      }
    }
    std::stable_sort(items.begin(), items.end(), [](const Item& a, const Item& b) { return a.cost > b.cost; });
    YkTab& T = h.yktab;
    int nrec = 0, npair = 0;
    size_t nu = 2 * YREC;  // the walk copies up to two records past an item
    for (const Item& I : items) nu += I.units;
    h.ykstream.assign(2 * nu, 0.0);
    double* out = h.ykstream.data();
    if (items.size() > (size_t)YK_ITEMS) return IPG_ERR_UNSUPPORTED;  // sized for YR_MAX_J
    for (Item& I : items) {
      if (nrec + I.recs.size() > (size_t)YK_RECS || npair + I.pairs.size() > (size_t)YK_PAIRS)
        return IPG_ERR_UNSUPPORTED;
      I.it.unit = (int32_t)((out - h.ykstream.data()) / 2);
      I.it.rec = (int16_t)nrec;
      I.it.nrec = (int16_t)I.recs.size();
      I.it.pair = (int16_t)npair;
      for (uint32_t r : I.recs) T.rec[nrec++] = r;
      for (const int2& q : I.pairs) T.pair[npair++] = q;
      T.item[T.nitem++] = I.it;
      for (const YkRows& R : I.rows) {  // its weights, [step][level][YT]
        const double* cgj[YNJ];
        double cb[YNJ];
        for (int q = 0; q < R.N; q++) {
          const int j = R.jlo + 2 * q;
          cgj[q] = h.cglist.data() + h.idxcg_block[blk(R.j1, R.j2, j)];
          cb[q] = cgj[q][R.mb1 * (R.j2 + 1) + R.mb2] * (p.bnorm_flag ? 1.0 / (j + 1) : 1.0);
        }
        for (int ma1 = R.lo1; ma1 <= R.hi1; ma1++, out += R.N * YT)  // zero where an index is out of range
          for (int t = 0; t < I.it.nt; t++) {
            const int m2 = R.E + t - ma1, c = std::abs(I.it.c0 + 2 * t);
            if (m2 < 0 || m2 > R.j2) continue;
            const int sg = R.mir == 1 ? ma1 + R.mb1 : (R.mir == 2 ? m2 + R.mb2 : 0);  // sign of the mirrored element
            for (int q = c > R.jlo ? (c - R.jlo) / 2 : 0; q < R.N; q++)
              out[q * YT + t] = ((sg & 1) ? -cb[q] : cb[q]) * cgj[q][ma1 * (R.j2 + 1) + m2];
          }
      }
    }
  }
  return IPG_OK;
}
