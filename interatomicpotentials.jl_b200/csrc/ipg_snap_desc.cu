// ipg_snap_desc.cu — per-atom force descriptors, virial descriptors and fitting rows from the
// dB/dr of every pair (compute_all_descriptors, snap.jl:226-306; the row layout of
// LAMMPS_SNAP/bispectrum.jl:279-387).
#include <algorithm>

#include "ipg_snap.cuh"

namespace {

constexpr int DG_T = 192;     // threads over the columns (component, direction)
constexpr int DG_PAIRS = 64;  // pairs staged at a time
constexpr int DG_V = 7;       // partial sums per (species, component): W (6) and B

// Sum of dbl over the pairs that end at an atom, have no reverse and an owner of species s (out of line: the
// gather's registers).
__device__ __noinline__ double one_sided_db(int64_t one, const int64_t* __restrict__ rev,
                                            const int64_t* __restrict__ off, int64_t n,
                                            const int32_t* __restrict__ species, int nsp, int s,
                                            const double* __restrict__ dbl, int C) {
  double sum = 0.0;
  for_one_sided(one, rev, [&](int64_t q) {
    int64_t lo = 0, hi = n - 1;  // the owner: the last atom whose pairs start at or before q
    while (lo < hi) {
      const int64_t mid = (lo + hi + 1) / 2;
      if (off[mid] <= q) lo = mid;
      else hi = mid - 1;
    }
    int so = species[lo];
    so = so < 0 ? 0 : (so >= nsp ? nsp - 1 : so);
    if (so == s) sum += dbl[(size_t)q * C];
  });
  return sum;
}

// One block takes one of nchunk chunks of atoms, each of one configuration, and DG_T columns t = 3 b + c
// of dB/dr, dbl [pair][K][3] (chunk + nchunk x tile of columns in blockIdx.x: neither has a limit of its own):
//   dB_k[block s][b][c] = sum over k's pairs, s_k = s, of dbl_p - sum over their reverses and the pairs
//     that end at k without one (k_rev_pair), s_owner = s, of dbl_q (snap.jl:289-290), if dB is wanted;
//   W of the chunk: dB_i/dr_ij (x) (x_i - x_j), absolute positions (snap.jl:292-306), and the sums
//     of B, both per species, into part [chunk][nsp][K][7] (dbl null: the sums of B alone).
// Bound by the reads of dbl: each pair's K x 3 numbers twice (once for its owner, once for its
// neighbor), in rows of 3 K consecutive doubles; W rides on the owner's read.  An atom's pairs are
// staged in shared memory, so the column threads read nothing else.  8,192 atoms, twojmax 8, two
// species: 155 us (plus 26 us of k_desc_reduce) for what a kernel per output did in 570 us; 48
// configurations of at most 250 atoms, twojmax 6: 108 (plus 5) against 2,096 us, nearly all of it
// in a kernel that walked each configuration serially.
template <int NSP>
__global__ void __launch_bounds__(DG_T) k_desc_gather(const int64_t* __restrict__ chunks, int nchunk, int K, int nsp,
                                                      const int64_t* __restrict__ off,
                                                      const int32_t* __restrict__ nbr,
                                                      const int64_t* __restrict__ rev,
                                                      const int64_t* __restrict__ one, int64_t n,
                                                      const int32_t* __restrict__ species,
                                                      const double* __restrict__ pos, const double* __restrict__ dbl,
                                                      const double* __restrict__ B, double* __restrict__ dB, int rows,
                                                      double* __restrict__ part, int want_w) {
  __shared__ double sd[DG_PAIRS][3];
  __shared__ int64_t sp[DG_PAIRS];
  __shared__ int ss[DG_PAIRS];
  const int chunk = blockIdx.x % nchunk;
  const int64_t a0 = chunks[2 * chunk], a1 = chunks[2 * chunk + 1];
  const int col = blockIdx.x / nchunk * DG_T + threadIdx.x, C = 3 * K;
  const bool act = col < C;
  const int b = col / 3, c = col - 3 * b;
  double w[NSP][4];  // per species: the three virial sums of this direction, and B (c = 0)
#pragma unroll
  for (int s = 0; s < NSP; s++) w[s][0] = w[s][1] = w[s][2] = w[s][3] = 0.0;
  for (int64_t i = a0; i < a1; i++) {
    int si = species[i];
    si = si < 0 ? 0 : (si >= nsp ? nsp - 1 : si);
    double acc[NSP];
#pragma unroll
    for (int s = 0; s < NSP; s++) acc[s] = 0.0;
    const double bi = B && act && c == 0 ? B[(size_t)i * K + b] : 0.0;
    const int64_t first = dB ? one[i] : 0;
    double own = 0.0, w0 = 0.0, w1 = 0.0, w2 = 0.0;
    for (int64_t p0 = off[i], p1 = dbl ? off[i + 1] : p0; p0 < p1; p0 += DG_PAIRS) {
      const int m = (int)(p1 - p0 < DG_PAIRS ? p1 - p0 : DG_PAIRS);
      if (want_w) {
        __syncthreads();
        for (int q = threadIdx.x; q < 3 * m; q += DG_T) {
          const int t = q / 3, a = q - 3 * t;
          sd[t][a] = pos[3 * i + a] - pos[3 * (int64_t)nbr[p0 + t] + a];
        }
        __syncthreads();
      }
      if (act) {
        const double* d = dbl + (size_t)p0 * C + col;
        if (want_w) {
#pragma unroll 8
          for (int t = 0; t < m; t++) {
            const double v = d[(size_t)t * C];
            own += v;
            w0 += v * sd[t][c];
            w1 += v * sd[t][2];
            w2 += v * sd[t][1];
          }
        } else {
#pragma unroll 8
          for (int t = 0; t < m; t++) own += d[(size_t)t * C];
        }
      }
    }
#pragma unroll
    for (int s = 0; s < NSP; s++)
      if (s == si) {
        acc[s] = own;
        w[s][0] += w0;
        w[s][1] += w1;
        w[s][2] += w2;
        w[s][3] += bi;
      }
    if (!dB) continue;
    for (int64_t q0 = off[i], q1 = off[i + 1]; q0 < q1; q0 += DG_PAIRS) {
      const int m = (int)(q1 - q0 < DG_PAIRS ? q1 - q0 : DG_PAIRS);
      __syncthreads();
      for (int t = threadIdx.x; t < m; t += DG_T) {
        const int so = species[nbr[q0 + t]];  // the reverse pair's owner
        sp[t] = rev[q0 + t];
        ss[t] = so < 0 ? 0 : (so >= nsp ? nsp - 1 : so);
      }
      __syncthreads();
      if (act) {
#pragma unroll 8
        for (int t = 0; t < m; t++) {
          const double v = sp[t] >= 0 ? dbl[(size_t)sp[t] * C + col] : 0.0;
#pragma unroll
          for (int s = 0; s < NSP; s++) acc[s] -= NSP == 1 || ss[t] == s ? v : 0.0;
        }
      }
    }
    if (first && act) {  // rare
#pragma unroll
      for (int s = 0; s < NSP; s++) acc[s] -= one_sided_db(first, rev, off, n, species, nsp, s, dbl + col, C);
    }
    if (act) {
#pragma unroll
      for (int s = 0; s < NSP; s++)
        if (s < nsp) {
          if (rows)  // [3 n][K nsp]: row 3 i + c
            dB[((size_t)i * 3 + c) * K * nsp + (size_t)s * K + b] = acc[s];
          else  // [n][K nsp][3]
            dB[(size_t)i * C * nsp + (size_t)s * C + col] = acc[s];
        }
    }
  }
  if (!part || !act) return;
  // direction c holds W(c, x_c), W(c, z), W(c, y) of [xx, yy, zz, yz, xz, xy]: xx xz xy | yy yz | zz
#pragma unroll
  for (int s = 0; s < NSP; s++) {
    if (s >= nsp) break;
    double* o = part + (((size_t)chunk * nsp + s) * K + b) * DG_V;
    o[c] = w[s][0];
    if (c == 0) {
      o[4] = w[s][1];
      o[5] = w[s][2];
      o[6] = w[s][3];
    } else if (c == 1) {
      o[3] = w[s][1];
    }
  }
}

// Sums of a configuration's chunks in a fixed order: eight rows of chunks, then the rows (one block a
// configuration and 32 columns, configurations first).
//   Wd [K nsp][6] (one configuration), Aw [nconf][6][K nsp], Ae [nconf][K nsp]; any may be null.
__global__ void __launch_bounds__(256) k_desc_reduce(const int64_t* __restrict__ conf_chunk, int nconf, int KN,
                                                     const double* __restrict__ part, double* __restrict__ Wd,
                                                     double* __restrict__ Aw, double* __restrict__ Ae) {
  __shared__ double sm[8][32];
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5, conf = blockIdx.x % nconf;
  const int t = blockIdx.x / nconf * 32 + x, width = KN * DG_V;
  double v = 0.0;
  if (t < width) {
#pragma unroll 4
    for (int64_t q = conf_chunk[conf] - conf_chunk[0] + y; q < conf_chunk[conf + 1] - conf_chunk[0]; q += 8)
      v += part[(size_t)q * width + t];
  }
  sm[y][x] = v;
  __syncthreads();
  if (y || t >= width) return;
  for (int r = 1; r < 8; r++) v += sm[r][x];
  const int col = t / DG_V, k = t - col * DG_V;
  if (k < 6) {
    if (Wd) Wd[(size_t)col * 6 + k] = v;
    if (Aw) Aw[((size_t)conf * 6 + k) * KN + col] = v;
  } else if (Ae) {
    Ae[(size_t)conf * KN + col] = v;
  }
}

template <int NSP>
int launch_gather(ipg_ctx* ctx, int nchunk, const int64_t* chunks, int64_t n, int K, int nsp, const PairList& pl,
                  const int32_t* species, const double* pos, const double* dbl, const double* B,
                  double* dB, bool rows, double* part, bool want_w) {
  const int ytiles = (3 * K + DG_T - 1) / DG_T;
  IPG_LAUNCH(ctx, k_desc_gather<NSP>, (unsigned)nchunk * ytiles, DG_T, 0, chunks, nchunk, K, nsp, pl.d_off, pl.d_j,
             pl.d_rev, pl.d_one, n, species, pos, dbl, B, dB, rows ? 1 : 0, part, want_w ? 1 : 0);
  return IPG_OK;
}

}  // namespace

int launch_descriptors(ipg_ctx* ctx, int K, int nsp, int nconf, const int64_t* h_off, const PairList& pl,
                       const int32_t* species, const double* pos, const double* dbl,
                       const double* B, double* dB, bool rows, double* Wd, double* Aw, double* Ae) {
  const int64_t n = h_off[nconf];
  const bool sums = Wd || Aw || Ae;
  if (n <= 0 || (!dB && !sums)) return IPG_OK;
  const int ytiles = (3 * K + DG_T - 1) / DG_T, KN = K * nsp;
  // Atoms per chunk: about eight blocks per SM.  The chunks' sums take at most 128 MB (or one
  // configuration's, if that is more: a configuration is at least one chunk), so configurations whose
  // chunks would take more follow in another pair of launches.
  const int64_t width = (int64_t)KN * DG_V, room = std::max<int64_t>(1, (int64_t(16) << 20) / width);
  const int64_t most = std::max<int64_t>(1, std::min<int64_t>((int64_t)ctx->num_sms * 8 / ytiles, room));
  const int64_t per = std::max<int64_t>(1, (n + most - 1) / most);
  std::vector<int64_t> tab;
  std::vector<int64_t> cc(nconf + 1, 0);
  for (int c = 0; c < nconf; c++) {
    for (int64_t a = h_off[c]; a < h_off[c + 1]; a += per) {
      tab.push_back(a);
      tab.push_back(std::min(h_off[c + 1], a + per));
    }
    cc[c + 1] = (int64_t)tab.size() / 2;
  }
  int64_t* hb = host_scratch<int64_t>(ctx, "desc_chunks_h", tab.size() + cc.size());
  memcpy(hb, tab.data(), sizeof(int64_t) * tab.size());
  memcpy(hb + tab.size(), cc.data(), sizeof(int64_t) * cc.size());
  int64_t* d_tab;
  IPG_RET(scratch(ctx, "desc_chunks", tab.size() + cc.size(), &d_tab));
  CUDA_RET(ctx, cudaMemcpyAsync(d_tab, hb, sizeof(int64_t) * (tab.size() + cc.size()), cudaMemcpyHostToDevice,
                                ctx->stream));
  std::vector<int> group = {0};  // first configurations of the launches
  int64_t largest = 0;           // chunks of a group
  for (int c = 0; c < nconf; c++) {
    if (c > group.back() && (cc[c + 1] - cc[group.back()] > room || c - group.back() >= room)) group.push_back(c);
    largest = std::max(largest, cc[c + 1] - cc[group.back()]);
  }
  group.push_back(nconf);
  double* part = nullptr;
  if (sums) IPG_RET(scratch(ctx, "desc_part", (size_t)largest * width, &part));
  const double* Bs = Ae ? B : nullptr;
  const bool want_w = Wd || Aw;
  for (size_t q = 0; q + 1 < group.size(); q++) {
    const int c0 = group[q], nc = group[q + 1] - c0;
    const int nchunk = (int)(cc[group[q + 1]] - cc[c0]);
    const int64_t* chunks = d_tab + 2 * cc[c0];
    const auto gather = nsp == 1 ? launch_gather<1> : nsp == 2 ? launch_gather<2>
                                  : nsp <= 4 ? launch_gather<4> : launch_gather<8>;
    if (nchunk)
      IPG_RET(gather(ctx, nchunk, chunks, n, K, nsp, pl, species, pos, dbl, Bs, dB, rows, part, want_w));
    if (sums)
      IPG_LAUNCH(ctx, k_desc_reduce, (unsigned)nc * (unsigned)((width + 31) / 32), 256, 0, d_tab + tab.size() + c0, nc,
                 KN, part, Wd, Aw ? Aw + (size_t)c0 * 6 * KN : nullptr, Ae ? Ae + (size_t)c0 * KN : nullptr);
  }
  return IPG_OK;
}
