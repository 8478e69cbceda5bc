// pairs.cu -- scores of an explicit pair list (nwg_score_pairs).
//
// pair_wave_kernel<R, P>: one warp per job, a job being P pairs in the halves
// of every register (P = 2, int16x2 lanes: the pairs that provably stay inside
// 16 bits) or one pair on int32 lanes (P = 1).  The warp is a wavefront: lane k
// owns rows [kR, kR + R) of a band of 32R rows, one column behind lane k - 1,
// in the register layout that carries T = H - go (layout 3 of wave_impl.cuh:
// three DPX operations and two adds per word).  Unlike the all-pairs form, no
// two pairs share a Y, so there is no profile to share: each warp builds its
// own, one byte per (letter, row), with its scores made non-negative by a bias
// so that one byte permute yields the word of both pairs.
// Bound by integer issue (about 3.9 instructions a cell with the shuffles and
// loads of a step spread over R = 8 rows).  R = 8 needs 12 KB of profile per
// warp, which leaves 18 warps per SM; R = 4 is for pairs whose Y fits one band
// of 128 rows.  20,000 pairs of about 245 residues, the whole call on a GB300:
// 13.8 ms with one pair per thread and the (H, F) row in global memory (157
// CTAs, one 4-byte-gather chain per cell), 0.99 ms here.
#include <algorithm>
#include <vector>

#include "nwg_ctx.h"
#include "profile8.cuh"
#include "wave_impl.cuh"

namespace nwg {
namespace {

using wave::clamp_code;
using wave::Lanes;
using wave::pick;

constexpr int kPWarps = 2;   // warps per CTA

struct PairWaveArgs {
  const int8_t* codes;
  const int64_t* start;
  const int32_t* len;
  const int32_t* pi;
  const int32_t* pj;
  const int32_t* order;     // the bucket's pairs, P consecutive ones per job
  int32_t* out;
  uint32_t* scratch;        // per warp: 2 buffers x 2 words x scratch_cols (pairs of more than one band)
  unsigned* counter;        // next job
  int npairs;
  int scratch_cols;
  int go, ge;
  int bias;                 // P = 2: added to every score so that it lies in 0 .. 127
  const int8_t* sub;
};

template <int R, int P>
__global__ void __launch_bounds__(32 * kPWarps) pair_wave_kernel(const PairWaveArgs a) {
  using L = Lanes<P>;
  static_assert(R == 4 || R == 8, "rows per lane");
  constexpr int BAND = 32 * R;
  constexpr int PW = kLetters * BAND / 4;                       // profile words of one pair
  __shared__ __align__(16) int8_t s_sub[kLetters * kLetters];
  __shared__ __align__(16) uint32_t s_prof[kPWarps][P][PW];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int e = threadIdx.x; e < kLetters * kLetters; e += blockDim.x)
    s_sub[e] = (int8_t)(a.sub[e] + (P == 2 ? a.bias : 0));
  __syncthreads();
  const uint32_t NGE = L::packed(-a.ge);
  const uint32_t NGO = L::arith(-a.go, -a.go);
  const uint32_t NGEA = L::arith(-a.ge, -a.ge);
  const uint32_t SENT = L::splat(kShortMin + a.ge);
  const int corr = a.go - (P == 2 ? a.bias : 0);                // T + biased score + corr = H + score
  const uint32_t CORR = L::arith(corr, corr);
  const uint32_t zero = P == 2 ? 0x01010101u * (uint32_t)a.bias : 0u;
  uint32_t* scratch = a.scratch + (size_t)(blockIdx.x * kPWarps + warp) * 4 * a.scratch_cols;
  const int njobs = (a.npairs + P - 1) / P;
  for (;;) {
    unsigned job = 0;
    if (lane == 0) job = atomicAdd(a.counter, 1u);
    job = __shfl_sync(0xffffffffu, job, 0);
    if (job >= (unsigned)njobs) break;
    const int8_t* X[P];
    const int8_t* Y[P];
    int Lx[P], Ly[P], id[P];
    int cols = 0, rows = 0, Lmin = 0x7fffffff;
#pragma unroll
    for (int k = 0; k < P; ++k) {
      const int s = (int)job * P + k;
      id[k] = a.order[s < a.npairs ? s : s - 1];               // the odd one out runs in both halves
      const int ix = a.pi[id[k]], iy = a.pj[id[k]];
      X[k] = a.codes + a.start[ix];
      Y[k] = a.codes + a.start[iy];
      Lx[k] = a.len[ix];
      Ly[k] = a.len[iy];
      cols = max(cols, Lx[k]);
      rows = max(rows, Ly[k]);
      Lmin = min(Lmin, Lx[k]);
    }
    const int nb = (rows + BAND - 1) / BAND;
    for (int b = 0; b < nb; ++b) {
      __syncwarp();
#pragma unroll
      for (int k = 0; k < P; ++k)
        build_profile<R>(s_prof[warp][k], s_sub, Y[k], b * BAND + lane * R, Ly[k], zero, lane);
      __syncwarp();
      uint32_t T[R], E[R];
      const int rowbase = b * BAND + lane * R;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        T[r] = L::splat(-a.ge * (rowbase + r + 1) - a.go);       // H[row][-1] - go
        E[r] = SENT;
      }
      // the column after which this lane holds a pair's score in row rr[k], or -1
      int endc[P], rr[P];
#pragma unroll
      for (int k = 0; k < P; ++k) {
        const int r = Ly[k] - 1 - rowbase;
        const bool own = r >= 0 && r < R;
        endc[k] = own ? Lx[k] - 1 : -1;
        rr[k] = r;
      }
      uint32_t hprev = L::splat(-a.ge * rowbase - a.go);
      uint32_t tbot = 0, fbot = 0;
      uint32_t hb = L::splat(-a.ge - a.go);                     // T[-1][c] of lane 0's column (band 0)
      const uint32_t* rd = scratch + ((b + 1) & 1) * 2 * a.scratch_cols;
      uint32_t* wr = scratch + (b & 1) * 2 * a.scratch_cols;
      const bool last_band = b + 1 >= nb;
      int xnext[P];
      uint2 bnext = make_uint2(0u, 0u);
#pragma unroll
      for (int k = 0; k < P; ++k) xnext[k] = lane == 0 ? (int)X[k][0] : 0;
      if (b > 0 && lane == 0) bnext = *reinterpret_cast<const uint2*>(rd);
      auto step = [&](int t, auto ramp, auto tail) {
        const int c = t - lane;
        uint32_t hin = __shfl_up_sync(0xffffffffu, tbot, 1);
        uint32_t f = __shfl_up_sync(0xffffffffu, fbot, 1);
        int xl[P];
#pragma unroll
        for (int k = 0; k < P; ++k) {
          xl[k] = xnext[k];
          if (!decltype(ramp)::value || c + 1 >= 0) xnext[k] = X[k][min(c + 1, Lx[k] - 1)];
        }
        if (lane == 0) {
          hin = b == 0 ? hb : bnext.x;
          f = b == 0 ? SENT : bnext.y;
          if (b > 0 && c + 1 < cols) bnext = *reinterpret_cast<const uint2*>(rd + 2 * (c + 1));
        }
        hb = L::add(hb, NGEA);
        if (!decltype(ramp)::value || c >= 0) {
          uint32_t w[P][R / 4];
#pragma unroll
          for (int k = 0; k < P; ++k) {
            const uint32_t* p = s_prof[warp][k] + (clamp_code(xl[k]) * 32 + lane) * (R / 4);
            if constexpr (R == 8) {
              const uint2 v = *reinterpret_cast<const uint2*>(p);
              w[k][0] = v.x;
              w[k][R / 4 - 1] = v.y;
            } else {
              w[k][0] = *p;
            }
          }
          auto score = [&](int r) -> uint32_t {   // the word of row r: byte r of each pair, sign-extended
            const uint32_t i = r & 3;
            if constexpr (P == 2)
              return perm(w[0][r >> 2], w[P - 1][r >> 2], i | (i | 8) << 4 | (i + 4) << 8 | (i + 4 | 8) << 12);
            else
              return perm(w[0][r >> 2], 0u, i | (i | 8) << 4 | (i | 8) << 8 | (i | 8) << 12);
          };
          uint32_t tup = hin;
          uint32_t hd = hprev + score(0) + CORR;                 // H of the row above at c - 1, plus the score
          hprev = hin;
#pragma unroll
          for (int r = 0; r < R; ++r) {
            f = L::addmax(f, NGE, tup);                          // F[r][c]
            const uint32_t e = L::addmax(E[r], NGE, T[r]);       // E[r][c]
            const uint32_t hn = r + 1 < R ? T[r] + score(r + 1 < R ? r + 1 : 0) + CORR : 0u;
            const uint32_t h = L::max3(e, f, hd);                // H[r][c]
            T[r] = L::add(h, NGO);
            E[r] = e;
            tup = T[r];
            hd = hn;
          }
          tbot = T[R - 1];
          fbot = f;
          if (lane == 31 && !last_band && c < cols) *reinterpret_cast<uint2*>(wr + 2 * c) = make_uint2(tbot, fbot);
          if (decltype(tail)::value) {
#pragma unroll
            for (int k = 0; k < P; ++k)
              if (c == endc[k]) {
                const uint32_t v = pick<R>(T, rr[k]);
                a.out[id[k]] = (k == 0 ? L::lo(v) : L::hi(v)) + a.go;
              }
          }
        }
      };
      // ramp: lanes before column 0; tail: a pair's last column may be reached
      int t = 0;
      const int ramp = min(31, cols + 31);
      for (; t < ramp; ++t) step(t, std::true_type{}, std::true_type{});
#pragma unroll 2
      for (; t < Lmin - 1; ++t) step(t, std::false_type{}, std::false_type{});
      for (; t < cols + 31; ++t) step(t, std::false_type{}, std::true_type{});
    }
  }
}

template <int R, int P>
int pair_ctas_per_sm() {
  static const int n = [] {
    int k = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, pair_wave_kernel<R, P>, 32 * kPWarps, 0) != cudaSuccess) {
      cudaGetLastError();
      return 4;
    }
    return k > 0 ? k : 1;
  }();
  return n;
}

}  // namespace

// One kind of job: rows per lane, pairs per word, its pairs in the order array.
struct PairBucket {
  int R, P, first, count, maxrows, maxcols;
};

int Ctx::score_pairs(const int8_t* codes, const int64_t* offsets, int n, const int32_t* pi, const int32_t* pj,
                     int64_t npairs, int32_t* out, int64_t* pairs16) {
  if (npairs > (int64_t)1 << 30) {   // the kernels index a list with 32 bits
    for (int64_t k = 0; k < npairs; k += (int64_t)1 << 30) {
      const int rc = score_pairs(codes, offsets, n, pi + k, pj + k, std::min(npairs - k, (int64_t)1 << 30), out + k, pairs16);
      if (rc) return rc;
    }
    return NWG_OK;
  }
  const int64_t total = offsets[n];
  std::vector<int32_t> len(n);
  for (int s = 0; s < n; ++s) len[s] = (int32_t)(offsets[s + 1] - offsets[s]);
  // Sixteen bits hold a pair when both lengths are within the context's limit
  // and the most its rows can score is too (the columns may run past its own
  // X, to the other pair's of the word); and the scores must fit seven bits.
  int smin = sub[0], smax = sub[0];
  for (int k = 0; k < kLetters * kLetters; ++k) {
    smin = std::min<int>(smin, sub[k]);
    smax = std::max<int>(smax, sub[k]);
  }
  const bool bytes7 = smax - std::min(smin, 0) <= 127 && smin >= -127;
  const int bias = -std::min(smin, 0);
  auto kind = [&](int64_t k) {   // bucket: (P, R)
    const int Lx = len[pi[k]], Ly = len[pj[k]];
    const bool p2 = bytes7 && std::max(Lx, Ly) <= i16.max_len &&
                    (smax <= 0 || (int64_t)Ly * smax <= i16.max_h);
    return (p2 ? 0 : 2) + (Ly > 128 ? 0 : 1);
  };
  // Order of the list: by bucket, then bands, then X length, longest first
  // (counting sort on X length, then a stable one on the other two), so that
  // the pairs of a word are alike and the long jobs start first.
  int maxlen = 1;
  for (int64_t k = 0; k < npairs; ++k) maxlen = std::max(maxlen, std::max(len[pi[k]], len[pj[k]]));
  const int maxb = (maxlen + 255) / 256;
  const int m = (int)npairs;
  std::vector<int32_t> by_x(m), order(m), slot;
  slot.assign((size_t)maxlen + 2, 0);
  for (int k = 0; k < m; ++k) ++slot[(size_t)(maxlen - len[pi[k]]) + 1];
  for (size_t k = 1; k < slot.size(); ++k) slot[k] += slot[k - 1];
  for (int k = 0; k < m; ++k) by_x[(size_t)slot[(size_t)(maxlen - len[pi[k]])]++] = k;
  auto key = [&](int k) {
    const int b = kind(k);
    return (size_t)b * (maxb + 1) + (size_t)(maxb - (len[pj[k]] + 255) / 256);
  };
  slot.assign((size_t)4 * (maxb + 1) + 1, 0);
  PairBucket bucket[4] = {{8, 2, 0, 0, 1, 1}, {4, 2, 0, 0, 1, 1}, {8, 1, 0, 0, 1, 1}, {4, 1, 0, 0, 1, 1}};
  for (int k = 0; k < m; ++k) {
    ++slot[key(k) + 1];
    PairBucket& b = bucket[kind(k)];
    ++b.count;
    b.maxrows = std::max(b.maxrows, len[pj[k]]);
    b.maxcols = std::max(b.maxcols, len[pi[k]]);
  }
  for (size_t k = 1; k < slot.size(); ++k) slot[k] += slot[k - 1];
  *pairs16 += bucket[0].count + bucket[1].count;
  for (int k = 1; k < 4; ++k) bucket[k].first = bucket[k - 1].first + bucket[k - 1].count;
  for (int k = 0; k < m; ++k) order[(size_t)slot[key(by_x[k])]++] = by_x[k];
  // grids and band-boundary scratch
  int grid[4] = {};
  size_t scratch_words = 1;
  for (int q = 0; q < 4; ++q) {
    const PairBucket& b = bucket[q];
    if (!b.count) continue;
    const int occ = b.P == 2 ? (b.R == 8 ? pair_ctas_per_sm<8, 2>() : pair_ctas_per_sm<4, 2>())
                             : (b.R == 8 ? pair_ctas_per_sm<8, 1>() : pair_ctas_per_sm<4, 1>());
    const int jobs = (b.count + b.P - 1) / b.P;
    grid[q] = std::min((jobs + kPWarps - 1) / kPWarps, sms * occ);
    if (b.maxrows > 32 * b.R)
      scratch_words = std::max(scratch_words, (size_t)grid[q] * kPWarps * 4 * (size_t)b.maxcols);
  }
  int rc;
  if ((rc = b_codes.ensure((size_t)total)) || (rc = b_start.ensure(sizeof(int64_t) * n)) ||
      (rc = b_len.ensure(sizeof(int32_t) * n)) || (rc = b_pi.ensure(sizeof(int32_t) * npairs)) ||
      (rc = b_pj.ensure(sizeof(int32_t) * npairs)) || (rc = b_out.ensure(sizeof(int32_t) * npairs)) ||
      (rc = b_orig.ensure(sizeof(int32_t) * npairs)) || (rc = b_counter.ensure(sizeof(unsigned) * 4)) ||
      (rc = b_pscratch.ensure(sizeof(uint32_t) * scratch_words)))
    return fail(rc, "pair-list allocation");
  cudaStream_t s = stream;
  if ((rc = cuda(cudaMemcpyAsync(b_codes.p, codes, (size_t)total, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemcpyAsync(b_start.p, offsets, sizeof(int64_t) * n, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemcpyAsync(b_len.p, len.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemcpyAsync(b_pi.p, pi, sizeof(int32_t) * npairs, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemcpyAsync(b_pj.p, pj, sizeof(int32_t) * npairs, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemcpyAsync(b_orig.p, order.data(), sizeof(int32_t) * npairs, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemsetAsync(b_counter.p, 0, sizeof(unsigned) * 4, s), "pair-list counters")))
    return rc;
  PairWaveArgs a{};
  a.codes = (const int8_t*)b_codes.p;
  a.start = (const int64_t*)b_start.p;
  a.len = (const int32_t*)b_len.p;
  a.pi = (const int32_t*)b_pi.p;
  a.pj = (const int32_t*)b_pj.p;
  a.out = (int32_t*)b_out.p;
  a.scratch = (uint32_t*)b_pscratch.p;
  a.go = go;
  a.ge = ge;
  a.bias = bias;
  a.sub = (const int8_t*)b_sub.p;
  for (int q = 0; q < 4; ++q) {
    const PairBucket& b = bucket[q];
    if (!b.count) continue;
    a.order = (const int32_t*)b_orig.p + b.first;
    a.npairs = b.count;
    a.scratch_cols = b.maxrows > 32 * b.R ? b.maxcols : 0;
    a.counter = (unsigned*)b_counter.p + q;
    if (b.P == 2 && b.R == 8) pair_wave_kernel<8, 2><<<grid[q], 32 * kPWarps, 0, s>>>(a);
    else if (b.P == 2) pair_wave_kernel<4, 2><<<grid[q], 32 * kPWarps, 0, s>>>(a);
    else if (b.R == 8) pair_wave_kernel<8, 1><<<grid[q], 32 * kPWarps, 0, s>>>(a);
    else pair_wave_kernel<4, 1><<<grid[q], 32 * kPWarps, 0, s>>>(a);
    if ((rc = cuda(cudaGetLastError(), "pair-list launch"))) return rc;
    ++launches;
  }
  if ((rc = cuda(cudaMemcpyAsync(out, b_out.p, sizeof(int32_t) * npairs, cudaMemcpyDeviceToHost, s), "download")) ||
      (rc = cuda(cudaStreamSynchronize(s), "pair-list sync")))
    return rc;
  return NWG_OK;
}

}  // namespace nwg
