// pairs.cu -- scores of an explicit pair list (nwg_score_pairs).
//
// One warp per job, a job being P pairs in the halves of every register (P = 2,
// int16x2 lanes: the pairs that provably stay inside 16 bits) or one pair on
// int32 lanes (P = 1).  The warp is a wavefront: lane k owns rows [kR, kR + R) of
// a band of 32R rows, one column behind lane k - 1.  Unlike the all-pairs form,
// no two pairs share a Y, so there is no profile to share: each warp builds its
// own, one byte per (letter, row), with its scores made non-negative by a bias
// so that one byte permute yields the word of both pairs.  pair7_kernel runs the
// recurrence with the extension cost taken out (layout 7 of wave_impl.cuh);
// pair_wave_kernel, on layout 3 (T = H - go, one add more per word), serves the
// gap models and matrices that layout 7 does not hold.
// Bound by integer issue and the latency of a step (two shuffles, the profile's
// loads, two dependent maxima per row) at 10 to 16 warps per SM, which the
// profiles' shared memory allows.  20,000 pairs of about 245 residues, the whole
// call on a GB300: 13.8 ms with one pair per thread and the (H, F) row in global
// memory (157 CTAs, one 4-byte-gather chain per cell), 0.75 ms on layout 3 (its
// kernels 0.68), 0.64 ms on layout 7 (0.47).
#include <algorithm>
#include <climits>
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

// The same jobs on layout 7 of wave_impl.cuh (the extension cost taken out: three
// DPX operations and one add per word, two dependent ones per row, constant
// borders), where go >= ge, the scores fit the profile's bytes and the borders stay
// above the reference's sentinel.  The codes of the next 32 columns are staged as
// offsets into the profile, as in wave_band7, and R = 12 serves pairs of up to 384
// rows in one band: of 20,000 pairs of 245 residues a quarter have more than 256
// rows, which two bands of 256 computed as 512.  A profile byte is S + 2 ge +
// lift, lift making the least of them 0; rows past a Y and columns past an X have
// the byte `lift`, which adds nothing.
template <int R, int P>
__global__ void __launch_bounds__(32 * kPWarps) pair7_kernel(const PairWaveArgs a) {
  using L = Lanes<P>;
  constexpr int BAND = 32 * R, Q = R / 4;
  constexpr int PW = (kLetters + 1) * BAND / 4;                 // profile words of one pair, a row of `lift` last
  constexpr int SC = 32;                                        // staged columns
  __shared__ __align__(16) int8_t s_sub[kLetters * kLetters];
  __shared__ __align__(16) uint32_t s_prof[kPWarps][P][PW];
  __shared__ __align__(16) int2 s_border[kPWarps][SC];
  __shared__ uint32_t s_codes[kPWarps][P][2 * SC];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int e = threadIdx.x; e < kLetters * kLetters; e += blockDim.x) s_sub[e] = (int8_t)(a.sub[e] + 2 * a.ge + a.bias);
  const uint32_t lifts = 0x01010101u * (uint32_t)a.bias;
#pragma unroll
  for (int k = 0; k < P; ++k)
    for (int e = lane; e < BAND / 4; e += 32) s_prof[warp][k][kLetters * BAND / 4 + e] = lifts;
  __syncthreads();
  const uint32_t NG = L::packed(a.ge - a.go);
  const int zero = P == 2 ? layout7_zero(a.go, a.ge) - 32768 : 0;
  const uint32_t ZERO = L::splat(zero), GAP = L::splat(zero + a.ge - a.go);
  const uint32_t CORR = L::arith(-a.bias, -a.bias);
  int2* scratch = reinterpret_cast<int2*>(a.scratch) + (size_t)(blockIdx.x * kPWarps + warp) * 2 * a.scratch_cols;
  int2* border = s_border[warp];
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
        build_profile<R>(s_prof[warp][k], s_sub, Y[k], b * BAND + lane * R, Ly[k], lifts, lane);
      uint32_t H[R], E[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        H[r] = ZERO;
        E[r] = GAP;
      }
      // the column after which this lane holds a pair's score in row rr[k], or none
      int endc[P], rr[P];
#pragma unroll
      for (int k = 0; k < P; ++k) {
        const int r = Ly[k] - 1 - (b * BAND + lane * R);
        endc[k] = r >= 0 && r < R ? Lx[k] - 1 : INT_MIN;
        rr[k] = r;
      }
      uint32_t hprev = ZERO, hbot = ZERO, fbot = GAP;
      const int2* rd = scratch + (size_t)((b + 1) & 1) * a.scratch_cols;
      int2* wr = scratch + (size_t)(b & 1) * a.scratch_cols - lane;
      const bool store = lane == 31 && b + 1 < nb;
      int nx[P];
      int2 nbd;
      uint32_t last[P];
      auto fetch = [&](int t0) {
        const int c = t0 + lane;
#pragma unroll
        for (int k = 0; k < P; ++k) nx[k] = c < Lx[k] ? (int)clamp_code(X[k][c]) : kLetters;
        nbd = b > 0 && c < cols ? rd[c] : make_int2((int)ZERO, (int)GAP);
      };
#pragma unroll
      for (int k = 0; k < P; ++k) last[k] = kLetters * BAND;     // columns before the first
      fetch(0);
      auto step = [&](int t0, int i, auto tail) {
        constexpr bool kTail = decltype(tail)::value;
        const int c = t0 + i - lane;
        uint32_t hin = __shfl_up_sync(0xffffffffu, hbot, 1);
        uint32_t f = __shfl_up_sync(0xffffffffu, fbot, 1);
        uint32_t w[P][Q];
#pragma unroll
        for (int k = 0; k < P; ++k) {
          const uint32_t* p = s_prof[warp][k] + (s_codes[warp][k][SC - lane + i] >> 2) + lane * Q;
          if constexpr (R == 8) {
            const uint2 v = *reinterpret_cast<const uint2*>(p);
            w[k][0] = v.x;
            w[k][Q - 1] = v.y;
          } else {
#pragma unroll
            for (int q = 0; q < Q; ++q) w[k][q] = p[q];
          }
        }
        if (lane == 0) {
          const int2 bd = border[i];
          hin = (uint32_t)bd.x;
          f = (uint32_t)bd.y;
        }
        if (kTail && c >= cols) return;
        auto score = [&](int r) -> uint32_t {   // the word of row r: byte r of each pair
          const uint32_t i4 = r & 3;
          if constexpr (P == 2)
            return perm(w[0][r >> 2], w[P - 1][r >> 2], i4 | (i4 | 8) << 4 | (i4 + 4) << 8 | (i4 + 4 | 8) << 12);
          else
            return perm(w[0][r >> 2], 0u, i4 | (i4 | 8) << 4 | (i4 | 8) << 8 | (i4 | 8) << 12);
        };
#pragma unroll
        for (int r = R - 1; r >= 0; --r) H[r] = (r > 0 ? H[r > 0 ? r - 1 : 0] : hprev) + score(r) + CORR;
        hprev = hin;
#pragma unroll
        for (int r = 0; r < R; ++r) {
          H[r] = L::max3(E[r], f, H[r]);
          f = L::addmax(H[r], NG, f);
          E[r] = L::addmax(H[r], NG, E[r]);
        }
        hbot = H[R - 1];
        fbot = f;
        if (store && (!kTail || c >= 0)) wr[t0 + i] = make_int2((int)hbot, (int)fbot);
        if (kTail) {
#pragma unroll
          for (int k = 0; k < P; ++k)
            if (c == endc[k]) {
              const uint32_t v = pick<R>(H, rr[k]);
              a.out[id[k]] = (k == 0 ? L::lo(v) : L::hi(v)) - zero - a.ge * (Lx[k] + Ly[k]);
            }
        }
      };
      const int nt = cols + 31;
      for (int t0 = 0; t0 < nt; t0 += SC) {
        __syncwarp();
#pragma unroll
        for (int k = 0; k < P; ++k) {
          s_codes[warp][k][lane] = last[k];
          last[k] = (uint32_t)nx[k] * BAND;
          s_codes[warp][k][SC + lane] = last[k];
        }
        border[lane] = nbd;
        __syncwarp();
        fetch(t0 + SC);
        const int ne = min(nt - t0, SC), ns = min(Lmin - 1 - t0, SC);   // below ns no pair's last column
        for (int i = 0; i < ne;) {
          if (t0 + i >= 31 && i < ns) {
#pragma unroll 4
            for (; i < ns; ++i) step(t0, i, std::false_type{});
          } else {
            step(t0, i, std::true_type{});
            ++i;
          }
        }
      }
    }
  }
}

template <int R, int P, bool Seven>
int pair_ctas_per_sm() {
  static const int n = [] {
    int k = 0;
    const void* fn = nullptr;
    if constexpr (Seven) fn = (const void*)pair7_kernel<R, P>;
    else fn = (const void*)pair_wave_kernel<R, P>;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&k, fn, 32 * kPWarps, 0) != cudaSuccess) {
      cudaGetLastError();
      return 4;
    }
    return k > 0 ? k : 1;
  }();
  return n;
}

// fn(rows per lane, pairs per word, layout 7) as constants.
template <class Fn>
void pair_dispatch(int R, int P, bool seven, Fn&& fn) {
  using std::integral_constant;
  auto with_p = [&](auto p) {
    using B7 = integral_constant<bool, true>;
    using B3 = integral_constant<bool, false>;
    if (seven && R == 12) fn(integral_constant<int, 12>{}, p, B7{});
    else if (seven && R == 8) fn(integral_constant<int, 8>{}, p, B7{});
    else if (seven) fn(integral_constant<int, 4>{}, p, B7{});
    else if (R == 8) fn(integral_constant<int, 8>{}, p, B3{});
    else fn(integral_constant<int, 4>{}, p, B3{});
  };
  if (P == 2) with_p(integral_constant<int, 2>{});
  else with_p(integral_constant<int, 1>{});
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
  int maxlen = 1;
  for (int64_t k = 0; k < npairs; ++k) maxlen = std::max(maxlen, std::max(len[pi[k]], len[pj[k]]));
  // layout 7: its bytes are S + 2 ge, lifted to 0 where the least is below
  const int lift = std::max(0, -(smin + 2 * ge));
  const bool seven = plain7(maxlen) && std::max(smax, 0) + 2 * ge + lift <= 127;
  const bool bytes7 = smax - std::min(smin, 0) <= 127 && smin >= -127;
  const int bias = seven ? lift : -std::min(smin, 0);
  // Bucket of a pair: lanes (int16x2 or int32) and rows per lane, with the fewest
  // rows computed; at equal rows the wider lanes (fewer bands).  12 rows exist on
  // layout 7.
  struct Kind { int R, P; };
  const Kind kinds[6] = {{12, 2}, {8, 2}, {4, 2}, {12, 1}, {8, 1}, {4, 1}};
  auto kind = [&](int64_t k) {
    const int Lx = len[pi[k]], Ly = len[pj[k]];
    const bool p2 = bytes7 && std::max(Lx, Ly) <= i16.max_len && (!seven || Ly <= i16.max_len7) &&
                    (smax <= 0 || (int64_t)Ly * smax <= i16.max_h);
    const int padded12 = (Ly + 383) / 384 * 384, padded8 = (Ly + 255) / 256 * 256;
    return (p2 ? 0 : 3) + (Ly <= 128 ? 2 : seven && padded12 <= padded8 ? 0 : 1);
  };
  // Order of the list: by bucket, then bands, then X length, longest first
  // (counting sort on X length, then a stable one on the other two), so that
  // the pairs of a word are alike and the long jobs start first.
  const int maxb = (maxlen + 255) / 256;
  const int m = (int)npairs;
  std::vector<int32_t> by_x(m), order(m), slot;
  slot.assign((size_t)maxlen + 2, 0);
  for (int k = 0; k < m; ++k) ++slot[(size_t)(maxlen - len[pi[k]]) + 1];
  for (size_t k = 1; k < slot.size(); ++k) slot[k] += slot[k - 1];
  for (int k = 0; k < m; ++k) by_x[(size_t)slot[(size_t)(maxlen - len[pi[k]])]++] = k;
  std::vector<int32_t> key(m);
  slot.assign((size_t)6 * (maxb + 1) + 1, 0);
  PairBucket bucket[6];
  for (int q = 0; q < 6; ++q) bucket[q] = {kinds[q].R, kinds[q].P, 0, 0, 1, 1};
  for (int k = 0; k < m; ++k) {
    const int q = kind(k);
    PairBucket& b = bucket[q];
    key[(size_t)k] = q * (maxb + 1) + (maxb - (len[pj[k]] + 32 * b.R - 1) / (32 * b.R));
    ++slot[(size_t)key[(size_t)k] + 1];
    ++b.count;
    b.maxrows = std::max(b.maxrows, len[pj[k]]);
    b.maxcols = std::max(b.maxcols, len[pi[k]]);
  }
  for (size_t k = 1; k < slot.size(); ++k) slot[k] += slot[k - 1];
  *pairs16 += bucket[0].count + bucket[1].count + bucket[2].count;
  for (int k = 1; k < 6; ++k) bucket[k].first = bucket[k - 1].first + bucket[k - 1].count;
  for (int k = 0; k < m; ++k) order[(size_t)slot[(size_t)key[(size_t)by_x[k]]]++] = by_x[k];
  // grids and band-boundary scratch
  int grid[6] = {}, kinds_used = 0;
  size_t scratch_words = 2, scratch_at[6] = {};   // regions of their own: the buckets run side by side
  for (int q = 0; q < 6; ++q) {
    const PairBucket& b = bucket[q];
    if (!b.count) continue;
    ++kinds_used;
    int occ = 1;
    pair_dispatch(b.R, b.P, seven, [&](auto r, auto p, auto s7) {
      occ = pair_ctas_per_sm<decltype(r)::value, decltype(p)::value, decltype(s7)::value>();
    });
    const int jobs = (b.count + b.P - 1) / b.P;
    grid[q] = std::min((jobs + kPWarps - 1) / kPWarps, sms * occ);
    scratch_at[q] = scratch_words;
    if (b.maxrows > 32 * b.R) scratch_words += (size_t)grid[q] * kPWarps * 4 * (size_t)b.maxcols;
  }
  int rc;
  if ((rc = b_codes.ensure((size_t)total)) || (rc = b_start.ensure(sizeof(int64_t) * n)) ||
      (rc = b_len.ensure(sizeof(int32_t) * n)) || (rc = b_pi.ensure(sizeof(int32_t) * npairs)) ||
      (rc = b_pj.ensure(sizeof(int32_t) * npairs)) || (rc = b_out.ensure(sizeof(int32_t) * npairs)) ||
      (rc = b_orig.ensure(sizeof(int32_t) * npairs)) || (rc = b_counter.ensure(sizeof(unsigned) * 6)) ||
      (rc = b_pscratch.ensure(sizeof(uint32_t) * scratch_words)))
    return fail(rc, "pair-list allocation");
  cudaStream_t s = stream;
  if ((rc = cuda(cudaMemcpyAsync(b_codes.p, codes, (size_t)total, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemcpyAsync(b_start.p, offsets, sizeof(int64_t) * n, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemcpyAsync(b_len.p, len.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemcpyAsync(b_pi.p, pi, sizeof(int32_t) * npairs, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemcpyAsync(b_pj.p, pj, sizeof(int32_t) * npairs, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemcpyAsync(b_orig.p, order.data(), sizeof(int32_t) * npairs, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemsetAsync(b_counter.p, 0, sizeof(unsigned) * 6, s), "pair-list counters")))
    return rc;
  PairWaveArgs a{};
  a.codes = (const int8_t*)b_codes.p;
  a.start = (const int64_t*)b_start.p;
  a.len = (const int32_t*)b_len.p;
  a.pi = (const int32_t*)b_pi.p;
  a.pj = (const int32_t*)b_pj.p;
  a.out = (int32_t*)b_out.p;
  a.go = go;
  a.ge = ge;
  a.bias = bias;
  a.sub = (const int8_t*)b_sub.p;
  // one launch's last jobs beside the next one's first
  const int sides = std::max(0, std::min(kinds_used - 1, (int)branch.size()));
  Fork fork{*this, sides == 0};
  if (sides > 0 && (rc = cuda(cudaEventRecord(fork_ev, s), "pair-list streams"))) return rc;
  for (int k = 0; k < sides; ++k)
    if ((rc = cuda(cudaStreamWaitEvent(branch[k], fork_ev, 0), "pair-list streams"))) return rc;
  int at = 0;
  for (int q = 0; q < 6; ++q) {
    const PairBucket& b = bucket[q];
    if (!b.count) continue;
    const int on = at++ % (sides + 1);
    cudaStream_t bs = on ? branch[on - 1] : s;
    a.scratch = (uint32_t*)b_pscratch.p + scratch_at[q];
    a.order = (const int32_t*)b_orig.p + b.first;
    a.npairs = b.count;
    a.scratch_cols = b.maxrows > 32 * b.R ? b.maxcols : 0;
    a.counter = (unsigned*)b_counter.p + q;
    pair_dispatch(b.R, b.P, seven, [&](auto r, auto p, auto s7) {
      if constexpr (decltype(s7)::value) pair7_kernel<decltype(r)::value, decltype(p)::value><<<grid[q], 32 * kPWarps, 0, bs>>>(a);
      else pair_wave_kernel<decltype(r)::value, decltype(p)::value><<<grid[q], 32 * kPWarps, 0, bs>>>(a);
    });
    if ((rc = cuda(cudaGetLastError(), "pair-list launch"))) return rc;
    ++launches;
  }
  if (sides > 0 && (rc = injected_fork_error())) return rc;
  for (int k = 0; k < sides; ++k)
    if ((rc = cuda(cudaEventRecord(join_ev[k], branch[k]), "pair-list streams")) ||
        (rc = cuda(cudaStreamWaitEvent(s, join_ev[k], 0), "pair-list streams")))
      return rc;
  fork.joined = true;
  if ((rc = cuda(cudaMemcpyAsync(out, b_out.p, sizeof(int32_t) * npairs, cudaMemcpyDeviceToHost, s), "download")) ||
      (rc = cuda(cudaStreamSynchronize(s), "pair-list sync")))
    return rc;
  return NWG_OK;
}

}  // namespace nwg
