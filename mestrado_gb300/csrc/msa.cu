// msa.cu -- progressive alignment along the guide tree.
//
// The reference's AlignmentMatch::computeMSA (AlignmentMatch.cu:320-434) is
// an empty loop, so this is the build's own definition (parity unpinned; the
// oracle's nwo_msa is the same algorithm on the CPU): internal node n+k joins
// left[k] (X, columns) and right[k] (Y, rows).  A profile is its columns'
// letter counts (int16 x 24 per column), in reversed column order like the
// codes.  A merge aligns two profiles with the pairwise recurrence and flags
// of the cherry traceback (NeedlemanWunsch.cu:184-365 and :393-494),
// generalised: cell score sum_x sum_y cX[x] cY[y] S[x][y], gap penalties
// go*kX*kY and ge*kX*kY (k = sequences of a profile), 64-bit integers.  Two
// single sequences therefore align exactly as nwg_align_pairs aligns them.
//
// Device work per tree level (every merge whose children are done):
//  1. msa_score_kernel: every cell's score, over the whole GPU;
//  2. msa_wave_kernel, one CTA per merge: the recurrence as a wavefront of
//     warps, then the walk over its flags;
//  3. msa_build_kernel: the merged profile and, for both children, the map of
//     their columns to the new ones.
// Merges whose differences between neighbouring cells could leave 32 bits, and
// gap models with open < extension, take msa_dp_kernel (64-bit cells) in
// place of 1 and 2.
// At the end the final position of every column is resolved parents first
// (msa_pos_kernel) and every leaf's residues are scattered into its row.
#include <algorithm>
#include <cstring>
#include <numeric>
#include <vector>

#include "nwg_ctx.h"
#include "walk.cuh"

namespace nwg {
namespace {

constexpr int kMR = 256;   // rows per strip = threads per CTA of the 64-bit form

struct MergeDesc {
  int64_t xoff, yoff, ooff;   // first column of X, Y and the new profile in the count pool
  int64_t xmap, ymap;         // X's and Y's column maps (written here)
  int64_t nib;                // first flag byte
  int64_t src;                // first entry of the alignment's columns (capacity lx + ly)
  int64_t scratch;            // 64-bit form: first (H, F) pair of the strip-boundary scratch (lx entries)
  int64_t score;              // wave form: first int4 of the cell scores
  int64_t bnd;                // wave form: first entry of the band-boundary row (lx entries)
  int32_t lx, ly, kx, ky;
  int32_t nsup;               // wave form: supersteps of a band
  int32_t tile0;              // wave form: first CTA of the score kernel
  int32_t mac32;              // kx * ky * max|S| < 2^31: a cell's score sum fits int32
  int32_t pad;
};

__device__ __forceinline__ int64_t mx64(int64_t a, int64_t b) { return a > b ? a : b; }

__device__ __forceinline__ unsigned msa_nib(const uint8_t* nib, int lx, int x, int y) {
  if (y < 0) return x < 0 ? 0u : 9u;     // row -1: left + continue-left; corner: stop
  if (x < 0) return 6u;                  // column -1: up + continue-up
  const int s = y / kMR, yl = y - s * kMR;
  return nib[(size_t)s * (size_t)(lx + kMR - 1) * kMR + (size_t)(x + yl) * kMR + yl];
}

// The traceback rules of the cherry alignment over the merge's flags (one
// thread): the alignment's columns in forward order as (X column, Y column),
// -1 for a gap; returns their number.
__device__ int msa_walk(const MergeDesc& m, const uint8_t* nib, int2* src) {
  const int lx = m.lx, ly = m.ly;
  const uint8_t* nb = nib + m.nib;
  int2* op = src + m.src;
  int x = lx - 1, y = ly - 1, k = 0;
  unsigned prev = 12u;
  unsigned cell = msa_nib(nb, lx, x, y);
  while ((cell & 12u) && k < lx + ly) {
    unsigned todo;
    if (((prev & 12u) == 4u) && (prev & 2u)) todo = 4u;
    else if (((prev & 12u) == 8u) && (prev & 1u)) todo = 8u;
    else if ((cell & 12u) == 4u) todo = 4u;
    else if ((cell & 12u) == 8u) todo = 8u;
    else todo = 12u;
    if ((todo != 4u && x < 0) || (todo != 8u && y < 0)) break;
    bool stop = false;
    op[k++] = make_int2((todo & 8u) ? x : -1, (todo & 4u) ? y : -1);
    if (todo == 8u) {
      --x;
    } else if (todo == 4u) {
      --y;
      stop = y < 0;
    } else {
      --x;
      --y;
    }
    prev = todo | (cell & 3u);
    cell = stop ? 0u : msa_nib(nb, lx, x, y);
  }
  for (; x >= 0 && k < lx + ly; --x) op[k++] = make_int2(x, -1);   // columns the walk left, opposite gaps
  for (; y >= 0 && k < lx + ly; --y) op[k++] = make_int2(-1, y);
  return k;
}

// The 64-bit form: 256 rows per strip, one thread per row, an anti-diagonal
// step per __syncthreads; thread r keeps W[x] = sum_y cY[r][y] S[x][y] in
// registers, with the next column's counts loaded a step ahead; (H, F) of the
// row above comes through shared memory, the bottom row of a strip through
// global scratch; the 4 flag bits of every cell are stored one byte per cell,
// anti-diagonal major; then thread 0 walks them.  About 0.4 us a step: it
// remains for the merges that the wave form's 32-bit differences cannot hold.
__global__ void __launch_bounds__(kMR) msa_dp_kernel(const MergeDesc* md, const int16_t* __restrict__ cnt, uint8_t* nib,
                                                     longlong2* __restrict__ scratch, const int8_t* __restrict__ sub,
                                                     int go, int ge, int2* __restrict__ src,
                                                     int32_t* __restrict__ nops) {
  __shared__ int8_t s_sub[kLetters * kLetters];
  __shared__ int64_t sh_h[2][kMR], sh_f[2][kMR];
  const MergeDesc m = md[blockIdx.x];
  for (int e = threadIdx.x; e < kLetters * kLetters; e += blockDim.x) s_sub[e] = sub[e];
  __syncthreads();
  const int lx = m.lx, ly = m.ly;
  const int64_t kk = (int64_t)m.kx * m.ky;
  const int64_t GO = (int64_t)go * kk, GE = (int64_t)ge * kk;
  const int64_t kSent = -(((int64_t)1) << 60);
  const int16_t* X = cnt + m.xoff * kLetters;
  const int16_t* Y = cnt + m.yoff * kLetters;
  longlong2* bnd = scratch + m.scratch;
  const int tid = threadIdx.x;
  const int nstrips = (ly + kMR - 1) / kMR;
  for (int sidx = 0; sidx < nstrips; ++sidx) {
    const int r = sidx * kMR + tid;       // this thread's row
    const bool live = r < ly;
    int32_t W[kLetters];
#pragma unroll
    for (int x = 0; x < kLetters; ++x) W[x] = 0;
    if (live) {
      const int16_t* cy = Y + (size_t)r * kLetters;
      for (int b = 0; b < kLetters; ++b) {
        const int c = cy[b];
        if (c == 0) continue;
#pragma unroll
        for (int x = 0; x < kLetters; ++x) W[x] += c * (int)s_sub[b * kLetters + x];
      }
    }
    int64_t hleft = -GE * (r + 1), eleft = kSent;
    int64_t diag = -GE * r;               // H[r-1][-1] (0 for row 0)
    uint8_t* nb = nib + m.nib + (size_t)sidx * (size_t)(lx + kMR - 1) * kMR;
    const int steps = lx + kMR - 1;
    // the counts of this thread's column, loaded one step ahead
    auto load_col = [&](int c, uint4 (&v)[3]) {
      if (c >= 0 && c < lx) {
        const uint4* p = reinterpret_cast<const uint4*>(X + (size_t)c * kLetters);
        v[0] = p[0];
        v[1] = p[1];
        v[2] = p[2];
      }
    };
    uint4 cur[3] = {}, nxt[3] = {};
    load_col(-tid, cur);
    for (int t = 0; t < steps; ++t) {
      const int c = t - tid;
      const int par = t & 1;
      load_col(c + 1, nxt);
      if (live && c >= 0 && c < lx) {
        int64_t hup, fup;
        if (tid == 0) {
          if (sidx == 0) {
            hup = -GE * (c + 1);
            fup = kSent;
          } else {
            const longlong2 v = bnd[c];
            hup = v.x;
            fup = v.y;
          }
        } else {
          hup = sh_h[par ^ 1][tid - 1];
          fup = sh_f[par ^ 1][tid - 1];
        }
        int64_t s = 0;
        if (m.mac32) {   // |s| <= kx * ky * max|S| < 2^31
          int32_t s32 = 0;
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const uint32_t w[4] = {cur[q].x, cur[q].y, cur[q].z, cur[q].w};
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              s32 += (int32_t)(int16_t)(w[h] & 0xFFFFu) * W[q * 8 + 2 * h];
              s32 += (int32_t)(int16_t)(w[h] >> 16) * W[q * 8 + 2 * h + 1];
            }
          }
          s = s32;
        } else {
#pragma unroll
          for (int q = 0; q < 3; ++q) {
            const uint32_t w[4] = {cur[q].x, cur[q].y, cur[q].z, cur[q].w};
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              s += (int64_t)(int16_t)(w[h] & 0xFFFFu) * W[q * 8 + 2 * h];
              s += (int64_t)(int16_t)(w[h] >> 16) * W[q * 8 + 2 * h + 1];
            }
          }
        }
        const int64_t f = mx64(fup - GE, hup - GO);
        const uint32_t cu = f == fup - GE;
        const int64_t e = mx64(eleft - GE, hleft - GO);
        const uint32_t cl = e == eleft - GE;
        const int64_t sim = diag + s;
        const int64_t h = mx64(mx64(e, f), sim);
        const uint32_t L = ((h == e) && (h != f)) || (h == sim);
        const uint32_t U = (h == f) || (h == sim);
        nb[(size_t)t * kMR + tid] = (uint8_t)((L << 3) | (U << 2) | (cu << 1) | cl);
        diag = hup;
        hleft = h;
        eleft = e;
        sh_h[par][tid] = h;
        sh_f[par][tid] = f;
        if (tid == kMR - 1 && sidx + 1 < nstrips) bnd[c] = make_longlong2(h, f);
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) cur[q] = nxt[q];
      __syncthreads();
    }
  }
  // the walk, while the merge's flags are still in L2 (the CTA barrier above
  // makes every thread's flags visible to thread 0)
  if (tid == 0) nops[blockIdx.x] = msa_walk(m, nib, src);
}

// ---- the wave form ------------------------------------------------------------
// Every value of the recurrence is held relative to a neighbouring cell, in 32
// bits: with u(r,c) = H(r,c) - H(r-1,c), v(r,c) = H(r,c) - H(r,c-1),
// a = F - H and b = E - H of a cell, and H(r-1,c-1) as the zero,
//   F = v(r-1,c) + max(a(r-1,c) - GE, -GO),   E = u(r,c-1) + max(b(r,c-1) - GE, -GO),
//   H = max(E, F, S),  u = H - v(r-1,c),  v = H - u(r,c-1)
// -- the same comparisons, so the same flags.  With GO >= GE every one of
// these lies within k * (max S + |min S| + 4 go), k = kX * kY: u, v >= -GO from
// H >= F >= Hup - GO (and likewise E); u <= max S + GO, since a diagonal step
// gives u = S - v(r-1,c), an F step u <= 0, and an E step no more than the cell
// where its gap opened; the others follow.  The host takes this form while that
// bound stays below 2^30 (a set of 8,000 sequences under the usual penalties).
//
// A band is 128 rows, four per lane of a warp, lane l a column behind lane
// l - 1; v and a of a lane's bottom row go to the next lane by shuffle, of a
// band's bottom row to the next warp through a ring in shared memory (to the
// first warp, for more bands than warps, through a row in global memory).  The
// CTA's warps work on consecutive bands kLag supersteps of kStep columns
// apart, one CTA barrier per superstep.  A tree's deep levels hold one or two
// merges, so a level costs one merge's chain of steps: 0.21 ms for 560 columns
// x 560 rows of 8,000 sequences (0.43 ms at 339 columns with 64-bit cells, one
// row per thread and a barrier per anti-diagonal).  The whole alignment of
// 8,000 sequences of 100-300 residues: 22.1 to 10.2 ms.
constexpr int kWRows = 4;                  // rows per lane
constexpr int kWBand = 32 * kWRows;        // rows per band
constexpr int kStep = 8;                   // columns per superstep
constexpr int kLag = 5;                    // supersteps between the bands of consecutive warps: the
                                           // last lane is 31 columns behind the first
constexpr int kWMax = 8;                   // warps per CTA, at most
constexpr int kRing = 64;                  // ring columns: the 8 being read to the 8 being written span 40
constexpr int kScoreSteps = 16;            // steps per warp of the score kernel
constexpr int kScoreWarps = 8;
constexpr int kWinSteps = 16;              // supersteps of flags in the walk's window
constexpr int kDiffSent = -(1 << 30);      // a and b of the cells above row 0 and left of column 0

// Scores of the cells of a level's merges in the wave kernel's order: int4
// (g * nsup * 8 + t) * 32 + l of a merge holds rows 128 g + 4 l .. + 3 at
// column t - l (0 outside).  One CTA per 128 rows x 128 steps: the rows' scores
// against each letter, W[x] = sum_y cY[y] S[y][x], go to shared memory once,
// then each warp runs 16 steps with its lanes' 4 x 24 of them in registers:
// 96 multiply-adds for three 16-byte loads of column counts.
__global__ void __launch_bounds__(32 * kScoreWarps) msa_score_kernel(const MergeDesc* __restrict__ md, int nm,
                                                                    const int16_t* __restrict__ cnt,
                                                                    const int8_t* __restrict__ sub,
                                                                    int4* __restrict__ score) {
  __shared__ int8_t s_sub[kLetters * kLetters];
  __shared__ int s_w[kLetters][kWBand];
  int lo = 0, hi = nm - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (md[mid].tile0 <= (int)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  const MergeDesc m = md[lo];
  const int nchunk = (m.nsup * kStep + kScoreSteps * kScoreWarps - 1) / (kScoreSteps * kScoreWarps);
  const int tile = (int)blockIdx.x - m.tile0;
  const int g = tile / nchunk, chunk = tile - g * nchunk;
  for (int e = threadIdx.x; e < kLetters * kLetters; e += blockDim.x) s_sub[e] = sub[e];
  __syncthreads();
  {
    // two threads per row, twelve letters each
    const int row = threadIdx.x % kWBand, x0 = (threadIdx.x / kWBand) * 12;
    int w[12];
#pragma unroll
    for (int x = 0; x < 12; ++x) w[x] = 0;
    const int r = g * kWBand + row;
    if (r < m.ly) {
      const int16_t* cy = cnt + (m.yoff + r) * kLetters;
      for (int b = 0; b < kLetters; ++b) {
        const int c = cy[b];
        if (c == 0) continue;
#pragma unroll
        for (int x = 0; x < 12; ++x) w[x] += c * (int)s_sub[b * kLetters + x0 + x];
      }
    }
#pragma unroll
    for (int x = 0; x < 12; ++x) s_w[x0 + x][row] = w[x];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int t0 = (chunk * kScoreWarps + warp) * kScoreSteps;
  const int t1 = min(t0 + kScoreSteps, m.nsup * kStep);
  if (t0 >= t1) return;
  int4 W[kLetters];
#pragma unroll
  for (int x = 0; x < kLetters; ++x) W[x] = *reinterpret_cast<const int4*>(&s_w[x][kWRows * lane]);
  const uint4* X = reinterpret_cast<const uint4*>(cnt + m.xoff * kLetters);   // 48 bytes a column
  int4* out = score + m.score + ((int64_t)g * m.nsup * kStep + t0) * 32 + lane;
  uint4 nxt[3] = {};
  auto load = [&](int t) {
    const int c = t - lane;
    const bool in = c >= 0 && c < m.lx;
#pragma unroll
    for (int q = 0; q < 3; ++q) nxt[q] = in ? X[(int64_t)c * 3 + q] : make_uint4(0u, 0u, 0u, 0u);
  };
  load(t0);
  for (int t = t0; t < t1; ++t) {
    const uint4 cur[3] = {nxt[0], nxt[1], nxt[2]};
    if (t + 1 < t1) load(t + 1);
    int4 s = make_int4(0, 0, 0, 0);
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const uint32_t w[4] = {cur[q].x, cur[q].y, cur[q].z, cur[q].w};
#pragma unroll
      for (int h = 0; h < 8; ++h) {
        const int n = (h & 1) ? (int)w[h >> 1] >> 16 : (int)(int16_t)(w[h >> 1] & 0xFFFFu);
        const int4 k = W[q * 8 + h];
        s.x += n * k.x;
        s.y += n * k.y;
        s.z += n * k.z;
        s.w += n * k.w;
      }
    }
    *out = s;
    out += 32;
  }
}

// The walk's window over a merge's flags: up to kWinSteps supersteps of one band.
struct MsaWindow {
  const uint4* flags;    // the merge's flags
  uint4* win;            // shared: [kWinSteps][32]
  int nsup;
  int g = -1, j0 = 0;    // band, first superstep held
  static __device__ __forceinline__ int superstep(int x, int y) { return (x + ((y & (kWBand - 1)) >> 2)) >> 3; }
  __device__ __forceinline__ bool covers(int x, int y) const {
    const int j = superstep(x, y) - j0;
    return (y >> 7) == g && j >= 0 && j < kWinSteps;
  }
  __device__ __forceinline__ unsigned cell(int x, int y) const {
    const int l = (y & (kWBand - 1)) >> 2, t = x + l, i = t & 7;
    const uint32_t* w = reinterpret_cast<const uint32_t*>(win + ((t >> 3) - j0) * 32 + l);
    return (w[i >> 1] >> (4 * (7 - ((i & 1) * 4 + (y & 3))))) & 15u;
  }
  __device__ __forceinline__ void load(int x, int y) {
    const int lane = threadIdx.x & 31;
    g = y >> 7;
    j0 = superstep(x, y) - (kWinSteps - 1);
    __syncwarp();
    uint4 v[kWinSteps];
#pragma unroll
    for (int k = 0; k < kWinSteps; ++k)
      if (j0 + k >= 0) v[k] = flags[((int64_t)g * nsup + j0 + k) * 32 + lane];
#pragma unroll
    for (int k = 0; k < kWinSteps; ++k)
      if (j0 + k >= 0) win[k * 32 + lane] = v[k];
    __syncwarp();
  }
};

__global__ void __launch_bounds__(32 * kWMax) msa_wave_kernel(const MergeDesc* __restrict__ md,
                                                             const int4* __restrict__ score, uint4* flags,
                                                             int2* bnd, int2* __restrict__ src,
                                                             int32_t* __restrict__ nops, int go, int ge) {
  __shared__ int2 s_ring[kWMax][kRing];
  __shared__ uint4 s_win[kWinSteps * 32];
  const MergeDesc m = md[blockIdx.x];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const int kk = m.kx * m.ky;
  const int GO = go * kk, GE = ge * kk;
  const int nb = (m.ly + kWBand - 1) / kWBand, nsup = m.nsup;
  // warp w runs bands w, w + nwarp, ..: band p * nwarp + w from superstep p * period + kLag * w on
  const int period = max(nsup, kLag * nwarp);
  const int last = (nb - 1) / nwarp * period + (nb - 1) % nwarp * kLag + nsup;
  uint4* fl = flags + m.nib / 16;
  const int4* sc = score + m.score + lane;
  int2* bd = bnd + m.bnd;
  const int2* in_ring = s_ring[warp == 0 ? nwarp - 1 : warp - 1];
  int uL[kWRows], bL[kWRows];
  int vbot = 0, abot = 0;
  int4 cur[kStep];
  int g = warp, j = -kLag * warp;
  for (int q = 0; q < last; ++q) {
    if (j >= 0 && j < nsup && g < nb) {
      const int4* band = sc + (int64_t)g * nsup * kStep * 32;
      if (j == 0) {
#pragma unroll
        for (int i = 0; i < kStep; ++i) cur[i] = band[i * 32];
#pragma unroll
        for (int r = 0; r < kWRows; ++r) {
          uL[r] = -GE;
          bL[r] = kDiffSent;
        }
      }
      int4 nxt[kStep];
      if (j + 1 < nsup) {
#pragma unroll
        for (int i = 0; i < kStep; ++i) nxt[i] = band[((j + 1) * kStep + i) * 32];
      }
      if (warp == 0 && g > 0) {   // the row above, left in global memory by the last warp
        const int c = j * kStep + lane;
        if (lane < kStep && c < m.lx) s_ring[nwarp - 1][c & (kRing - 1)] = bd[c];
        __syncwarp();
      }
      uint32_t word[kStep / 2] = {};
      auto steps = [&](auto checked) {
#pragma unroll
        for (int i = 0; i < kStep; ++i) {
          const int t = j * kStep + i;
          int vU = __shfl_up_sync(0xffffffffu, vbot, 1);
          int aU = __shfl_up_sync(0xffffffffu, abot, 1);
          if (g == 0) {
            if (lane == 0) {
              vU = -GE;
              aU = kDiffSent;
            }
          } else {
            const int2 in = in_ring[t & (kRing - 1)];
            if (lane == 0) {
              vU = in.x;
              aU = in.y;
            }
          }
          if (decltype(checked)::value && t == lane) {   // the lane's column 0: what came before was no cell
#pragma unroll
            for (int r = 0; r < kWRows; ++r) {
              uL[r] = -GE;
              bL[r] = kDiffSent;
            }
          }
          const int sv[kWRows] = {cur[i].x, cur[i].y, cur[i].z, cur[i].w};
          uint32_t w = word[i >> 1];
#pragma unroll
          for (int r = 0; r < kWRows; ++r) {
            // flags as sign bits, appended by funnel shifts: cU = a(up) - GE >= -GO,
            // cL likewise, F >= E, H == S; then U = ps || pf, L = ps || !pf
            const uint32_t xcu = (uint32_t)(GE - GO - 1 - aU);
            const int F = vU + __viaddmax_s32(aU, -GE, -GO);
            const uint32_t xcl = (uint32_t)(GE - GO - 1 - bL[r]);
            const int E = uL[r] + __viaddmax_s32(bL[r], -GE, -GO);
            const uint32_t xpf = (uint32_t)(E - F - 1);
            const int h = __vimax3_s32(E, F, sv[r]);
            const uint32_t xps = (uint32_t)(h - sv[r] - 1);
            w = __funnelshift_l(xps | ~xpf, w, 1);   // L
            w = __funnelshift_l(xps | xpf, w, 1);    // U
            w = __funnelshift_l(xcu, w, 1);          // cU
            w = __funnelshift_l(xcl, w, 1);          // cL
            const int v = h - uL[r];
            uL[r] = h - vU;
            aU = F - h;
            bL[r] = E - h;
            vU = v;
          }
          word[i >> 1] = w;
          vbot = vU;
          abot = aU;
          const int c = t - 31;
          if (lane == 31 && c >= 0 && c < m.lx) {
            if (warp + 1 < nwarp) s_ring[warp][c & (kRing - 1)] = make_int2(vbot, abot);
            else if (g + 1 < nb) bd[c] = make_int2(vbot, abot);
          }
        }
      };
      if (j < 32 / kStep) steps(std::true_type{});
      else steps(std::false_type{});
      fl[((int64_t)g * nsup + j) * 32 + lane] = make_uint4(word[0], word[1], word[2], word[3]);
#pragma unroll
      for (int i = 0; i < kStep; ++i) cur[i] = nxt[i];
    }
    if (++j == period) {
      j = 0;
      g += nwarp;
    }
    __syncthreads();
  }
  if (warp != 0) return;
  // the walk: the alignment's columns in forward order (X column, Y column; -1 a gap)
  MsaWindow win{fl, s_win, nsup};
  int2* out = src + m.src;
  WalkPos p = run_walk(win, m.lx, m.ly, m.lx + m.ly, [&](int k, int n, int x, int y, int sx, int sy) {
    if (lane < n) out[k + lane] = make_int2(sx ? x - lane : -1, sy ? y - lane : -1);
  });
  // columns the walk left, opposite gaps
  for (int i = lane; i <= p.x; i += 32) out[p.k + i] = make_int2(p.x - i, -1);
  p.k += p.x + 1;
  for (int i = lane; i <= p.y; i += 32) out[p.k + i] = make_int2(-1, p.y - i);
  p.k += p.y + 1;
  if (lane == 0) nops[blockIdx.x] = p.k;
}

// Merged profile and child maps: three threads per column, eight letters each
// (the counts of both children are added as packed 16-bit halves).
constexpr int kBuildCols = 64;
__global__ void __launch_bounds__(3 * kBuildCols) msa_build_kernel(const MergeDesc* __restrict__ md, int16_t* cnt,
                                                                  int32_t* __restrict__ maps,
                                                                  const int2* __restrict__ src,
                                                                  const int32_t* __restrict__ nops) {
  const int k = nops[blockIdx.x];
  const int j = blockIdx.y * kBuildCols + threadIdx.x / 3, part = threadIdx.x % 3;
  if (j >= k) return;
  const MergeDesc& m = md[blockIdx.x];
  const int2 s = src[m.src + j];
  const int col = k - 1 - j;   // reversed storage
  const uint4* pool = reinterpret_cast<const uint4*>(cnt);
  uint4 v = make_uint4(0u, 0u, 0u, 0u);
  if (s.x >= 0) v = pool[(m.xoff + s.x) * 3 + part];
  if (s.y >= 0) {
    const uint4 w = pool[(m.yoff + s.y) * 3 + part];
    v = make_uint4(v.x + w.x, v.y + w.y, v.z + w.z, v.w + w.w);
  }
  reinterpret_cast<uint4*>(cnt)[(m.ooff + col) * 3 + part] = v;
  if (part == 0) {
    if (s.x >= 0) maps[m.xmap + s.x] = col;
    if (s.y >= 0) maps[m.ymap + s.y] = col;
  }
}

// Leaf profiles: one column per residue (reversed codes), count 1.
__global__ void msa_leaf_kernel(const int8_t* __restrict__ codes, int64_t total, int16_t* cnt) {
  const int64_t c = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= total) return;
  int16_t* o = cnt + c * kLetters;
  int x = codes[c];
  if (x < 0 || x >= kLetters) x = kLetters - 1;
#pragma unroll
  for (int k = 0; k < kLetters; ++k) o[k] = (int16_t)(k == x);
}

struct PosJob {
  int64_t parent_pos;   // parent's positions (first column)
  int64_t child_pos;    // child's positions (written)
  int64_t child_map;    // child's column -> parent column
  int32_t len;          // child columns
  int32_t pad;
};

// pos[child][c] = pos[parent][map[c]]; one CTA per (parent, child).
__global__ void msa_pos_kernel(const PosJob* __restrict__ jobs, int32_t* pos, const int32_t* __restrict__ maps) {
  const PosJob j = jobs[blockIdx.x];
  for (int c = threadIdx.x; c < j.len; c += blockDim.x) pos[j.child_pos + c] = pos[j.parent_pos + maps[j.child_map + c]];
}

__global__ void msa_root_kernel(int32_t* pos, int64_t root_pos, int len) {
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c < len) pos[root_pos + c] = len - 1 - c;
}

// Rows: out[v][pos[v][c]] = letter of residue c of leaf v (one CTA per leaf).
__global__ void msa_rows_kernel(const int8_t* __restrict__ codes, const int64_t* __restrict__ off,
                                const int32_t* __restrict__ pos, char* out, int64_t L) {
  const int v = blockIdx.x;
  const int64_t a = off[v], b = off[v + 1];
  const char kDec[kLetters + 1] = "ARNDCQEGHILKMFPSTWYVBZX*";
  for (int64_t c = a + threadIdx.x; c < b; c += blockDim.x) {
    int x = codes[c];
    if (x < 0 || x >= kLetters) x = kLetters - 1;
    out[(int64_t)v * L + pos[c]] = kDec[x];
  }
}

}  // namespace

struct MsaState {
  DevBuf codes, off, cnt, maps, pos, nib, src, scratch, score, bnd, nops, md, pj, out;
  int n = 0;
  int64_t L = 0;
  ~MsaState() {
    for (DevBuf* b : {&codes, &off, &cnt, &maps, &pos, &nib, &src, &scratch, &score, &bnd, &nops, &md, &pj, &out}) b->release();
  }
};

void Ctx::msa_release() {
  delete reinterpret_cast<MsaState*>(msa_state);
  msa_state = nullptr;
}

int Ctx::msa(const int8_t* codes, const int64_t* offsets, int n, const int32_t* left, const int32_t* right,
             int64_t* msa_len, nwg_stats* st) {
  if (!codes || !offsets || n < 1 || (n > 1 && (!left || !right)) || !msa_len) return fail(NWG_ERR_INVALID, "msa arguments");
  const int nn = 2 * n - 1;
  // the tree: children, heights (levels), each node a child at most once
  std::vector<int> height(nn, 0), used(nn, 0), kseq(nn, 1);
  std::vector<int64_t> len(nn, 0);
  for (int v = 0; v < n; ++v) {
    len[v] = offsets[v + 1] - offsets[v];
    if (len[v] <= 0) return fail(NWG_ERR_EMPTY_SEQ, "zero-length sequence");
  }
  int levels = 0;
  for (int k = 0; k < n - 1; ++k) {
    const int a = left[k], b = right[k], v = n + k;
    if (a < 0 || b < 0 || a >= b || b >= v || used[a] || used[b]) return fail(NWG_ERR_INVALID, "malformed guide tree");
    used[a] = used[b] = 1;
    height[v] = 1 + std::max(height[a], height[b]);
    kseq[v] = kseq[a] + kseq[b];
    levels = std::max(levels, height[v]);
  }
  if (!msa_state) msa_state = new MsaState();
  MsaState& M = *reinterpret_cast<MsaState*>(msa_state);
  const int64_t total = offsets[n] - offsets[0];
  std::vector<int64_t> off0(n + 1);
  for (int v = 0; v <= n; ++v) off0[v] = offsets[v] - offsets[0];
  cudaStream_t s = stream;
  int rc;
  // column pool: leaves first (their columns = residues), internal nodes appended per level
  std::vector<int64_t> col(nn, -1);
  for (int v = 0; v < n; ++v) col[v] = off0[v];
  int64_t pool = total;
  if ((rc = M.codes.ensure((size_t)std::max<int64_t>(total, 1))) || (rc = M.off.ensure(sizeof(int64_t) * (n + 1))))
    return fail(rc, "msa allocation");
  if ((rc = cuda(cudaMemcpyAsync(M.codes.p, codes + offsets[0], (size_t)total, cudaMemcpyHostToDevice, s), "msa upload")) ||
      (rc = cuda(cudaMemcpyAsync(M.off.p, off0.data(), sizeof(int64_t) * (n + 1), cudaMemcpyHostToDevice, s),
                 "msa upload")))
    return rc;
  // worst-case pool: every internal node at most the sum of its leaves' lengths
  std::vector<int64_t> leafsum(nn, 0);
  for (int v = 0; v < n; ++v) leafsum[v] = len[v];
  int64_t cap = total;
  for (int k = 0; k < n - 1; ++k) {
    leafsum[n + k] = leafsum[left[k]] + leafsum[right[k]];
    cap += leafsum[n + k];
  }
  if ((rc = M.cnt.ensure(sizeof(int16_t) * kLetters * (size_t)std::max<int64_t>(cap, 1))) ||
      (rc = M.maps.ensure(sizeof(int32_t) * (size_t)std::max<int64_t>(cap, 1))) ||
      (rc = M.pos.ensure(sizeof(int32_t) * (size_t)std::max<int64_t>(cap, 1))))
    return fail(rc, "msa allocation");
  if (st) cudaEventRecord(ev0, s);
  msa_leaf_kernel<<<(unsigned)((total + 255) / 256), 256, 0, s>>>((const int8_t*)M.codes.p, total, (int16_t*)M.cnt.p);
  ++launches;
  std::vector<std::vector<int>> bylevel(levels + 1);
  for (int k = 0; k < n - 1; ++k) bylevel[height[n + k]].push_back(n + k);
  int64_t cells = 0;
  int64_t smax = 1;   // largest |S| of the context's matrix
  for (int k = 0; k < kLetters * kLetters; ++k) smax = std::max<int64_t>(smax, sub[k] < 0 ? -sub[k] : sub[k]);
  const int64_t diff_bound = 2 * smax + 4 * (int64_t)go;   // the wave form's differences, per kX * kY
  constexpr int64_t kScoreBatch = (int64_t)1 << 25;        // int4 scores of one batch of merges (512 MiB)
  constexpr int64_t kScoreMax = (int64_t)1 << 29;          // of one merge (8 GiB; beyond, the 64-bit form)
  std::vector<MergeDesc> md;
  std::vector<int32_t> nops;
  for (int l = 1; l <= levels; ++l) {
    // wave-form merges first, most supersteps first; then the 64-bit ones
    std::vector<int>& nodes = bylevel[l];
    const int nm = (int)nodes.size();
    auto shape = [&](int v, int64_t& bands, int64_t& nsup) {
      bands = (len[right[v - n]] + kWBand - 1) / kWBand;
      nsup = (len[left[v - n]] + 31 + kStep - 1) / kStep;
    };
    auto is_wave = [&](int v) {
      int64_t bands, nsup;
      shape(v, bands, nsup);
      return go >= ge && (int64_t)kseq[left[v - n]] * kseq[right[v - n]] * diff_bound < ((int64_t)1 << 30) &&
             bands * nsup * kStep * 32 <= kScoreMax;
    };
    const int nwave = (int)(std::stable_partition(nodes.begin(), nodes.end(), is_wave) - nodes.begin());
    std::stable_sort(nodes.begin(), nodes.begin() + nwave, [&](int u, int v) {
      int64_t bu, su, bv, sv;
      shape(u, bu, su);
      shape(v, bv, sv);
      return bu != bv ? bu > bv : su > sv;
    });
    md.assign(nm, MergeDesc{});
    int64_t nib_total = 0, src_total = 0, scr_total = 0, score_cap = 0, bnd_total = 0;
    // batches of wave merges that share the score buffer (on one stream, so one after another)
    struct Batch {
      int first, count, tiles, warps;
    };
    std::vector<Batch> batches;
    int64_t score_used = 0;
    int maxcols = 1;
    for (int q = 0; q < nm; ++q) {
      const int v = nodes[q], a = left[v - n], b = right[v - n];
      MergeDesc& d = md[q];
      d.xoff = col[a];
      d.yoff = col[b];
      d.lx = (int)len[a];
      d.ly = (int)len[b];
      d.kx = kseq[a];
      d.ky = kseq[b];
      d.mac32 = (int64_t)d.kx * d.ky * smax < ((int64_t)1 << 31) ? 1 : 0;
      d.xmap = col[a];
      d.ymap = col[b];
      d.ooff = pool;
      col[v] = pool;
      pool += len[a] + len[b];   // capacity; the walk's length is read back below
      d.nib = nib_total;
      d.src = src_total;
      src_total += d.lx + d.ly;
      maxcols = std::max(maxcols, d.lx + d.ly);
      cells += (int64_t)d.lx * d.ly;
      if (q < nwave) {
        int64_t bands, nsup;
        shape(v, bands, nsup);
        d.nsup = (int)nsup;
        const int64_t words = bands * nsup * kStep * 32;
        if (batches.empty() || score_used + words > kScoreBatch) {
          batches.push_back({q, 0, 0, 1});
          score_used = 0;
        }
        Batch& bt = batches.back();
        d.score = score_used;
        score_used += words;
        score_cap = std::max(score_cap, score_used);
        d.tile0 = bt.tiles;
        bt.tiles += (int)(bands * ((nsup * kStep + kScoreSteps * kScoreWarps - 1) / (kScoreSteps * kScoreWarps)));
        bt.count += 1;
        bt.warps = std::max(bt.warps, (int)std::min<int64_t>(bands, kWMax));
        d.bnd = bnd_total;
        if (bands > kWMax) bnd_total += d.lx;
        nib_total += bands * nsup * 512;
      } else {
        const int nstr = (d.ly + kMR - 1) / kMR;
        nib_total += ((int64_t)nstr * (d.lx + kMR - 1) * kMR + 15) / 16 * 16;
        d.scratch = scr_total;
        scr_total += d.lx;
      }
    }
    if ((rc = M.nib.ensure((size_t)std::max<int64_t>(nib_total, 1))) ||
        (rc = M.src.ensure(sizeof(int2) * (size_t)std::max<int64_t>(src_total, 1))) ||
        (rc = M.scratch.ensure(sizeof(longlong2) * (size_t)std::max<int64_t>(scr_total, 1))) ||
        (rc = M.score.ensure(sizeof(int4) * (size_t)std::max<int64_t>(score_cap, 1))) ||
        (rc = M.bnd.ensure(sizeof(int2) * (size_t)std::max<int64_t>(bnd_total, 1))) ||
        (rc = M.nops.ensure(sizeof(int32_t) * nm)) || (rc = M.md.ensure(sizeof(MergeDesc) * nm)))
      return fail(rc, "msa allocation");
    if ((rc = cuda(cudaMemcpyAsync(M.md.p, md.data(), sizeof(MergeDesc) * nm, cudaMemcpyHostToDevice, s), "msa upload")))
      return rc;
    const MergeDesc* dmd = (const MergeDesc*)M.md.p;
    for (const Batch& b : batches) {
      msa_score_kernel<<<b.tiles, 32 * kScoreWarps, 0, s>>>(dmd + b.first, b.count, (const int16_t*)M.cnt.p,
                                                            (const int8_t*)b_sub.p, (int4*)M.score.p);
      msa_wave_kernel<<<b.count, 32 * b.warps, 0, s>>>(dmd + b.first, (const int4*)M.score.p, (uint4*)M.nib.p,
                                                       (int2*)M.bnd.p, (int2*)M.src.p, (int32_t*)M.nops.p + b.first,
                                                       go, ge);
      launches += 2;
    }
    if (nwave < nm) {
      msa_dp_kernel<<<nm - nwave, kMR, 0, s>>>(dmd + nwave, (const int16_t*)M.cnt.p, (uint8_t*)M.nib.p,
                                               (longlong2*)M.scratch.p, (const int8_t*)b_sub.p, go, ge,
                                               (int2*)M.src.p, (int32_t*)M.nops.p + nwave);
      ++launches;
    }
    msa_build_kernel<<<dim3((unsigned)nm, (unsigned)((maxcols + kBuildCols - 1) / kBuildCols)), 3 * kBuildCols, 0, s>>>(
        dmd, (int16_t*)M.cnt.p, (int32_t*)M.maps.p, (const int2*)M.src.p, (const int32_t*)M.nops.p);
    ++launches;
    if ((rc = cuda(cudaGetLastError(), "msa launch"))) return rc;
    // the new profiles' lengths (the next level sizes its work with them)
    nops.resize(nm);
    if ((rc = cuda(cudaMemcpyAsync(nops.data(), M.nops.p, sizeof(int32_t) * nm, cudaMemcpyDeviceToHost, s), "msa")) ||
        (rc = cuda(cudaStreamSynchronize(s), "msa sync")))
      return rc;
    for (int q = 0; q < nm; ++q) len[nodes[q]] = nops[q];
  }
  // final positions, parents first, then the rows
  const int root = nn - 1;
  const int64_t L = len[root];
  std::vector<PosJob> pj;
  if ((rc = cuda(cudaMemsetAsync(M.pos.p, 0, sizeof(int32_t) * (size_t)std::max<int64_t>(pool, 1), s), "msa"))) return rc;
  msa_root_kernel<<<(unsigned)((L + 255) / 256), 256, 0, s>>>((int32_t*)M.pos.p, col[root], (int)L);
  ++launches;
  if ((rc = M.pj.ensure(sizeof(PosJob) * (size_t)std::max(2 * n, 2)))) return fail(rc, "msa allocation");
  for (int l = levels; l >= 1; --l) {
    pj.clear();
    for (int v : bylevel[l]) {
      const int a = left[v - n], b = right[v - n];
      pj.push_back(PosJob{col[v], col[a], col[a], (int32_t)len[a], 0});
      pj.push_back(PosJob{col[v], col[b], col[b], (int32_t)len[b], 0});
    }
    if ((rc = cuda(cudaMemcpyAsync(M.pj.p, pj.data(), sizeof(PosJob) * pj.size(), cudaMemcpyHostToDevice, s), "msa")))
      return rc;
    msa_pos_kernel<<<(unsigned)pj.size(), 256, 0, s>>>((const PosJob*)M.pj.p, (int32_t*)M.pos.p,
                                                      (const int32_t*)M.maps.p);
    ++launches;
    // the job list is reused by the next level: wait for this launch
    if ((rc = cuda(cudaStreamSynchronize(s), "msa sync"))) return rc;
  }
  if ((rc = M.out.ensure((size_t)std::max<int64_t>((int64_t)n * L, 1)))) return fail(rc, "msa allocation");
  if ((rc = cuda(cudaMemsetAsync(M.out.p, '-', (size_t)n * L, s), "msa"))) return rc;
  msa_rows_kernel<<<n, 256, 0, s>>>((const int8_t*)M.codes.p, (const int64_t*)M.off.p, (const int32_t*)M.pos.p,
                                    (char*)M.out.p, L);
  ++launches;
  if (st) cudaEventRecord(ev1, s);
  if ((rc = cuda(cudaStreamSynchronize(s), "msa sync"))) return rc;
  M.n = n;
  M.L = L;
  *msa_len = L;
  if (st) {
    float ms = 0;
    cudaEventElapsedTime(&ms, ev0, ev1);
    st->kernel_ms = ms;
    st->cells = cells;
    st->pairs = n - 1;
  }
  return NWG_OK;
}

int Ctx::msa_rows(char* out, int64_t stride) {
  MsaState* M = reinterpret_cast<MsaState*>(msa_state);
  if (!M || !M->n || !out || stride < M->L) return fail(NWG_ERR_INVALID, "msa rows");
  int rc;
  if ((rc = cuda(cudaMemcpy2DAsync(out, (size_t)stride, M->out.p, (size_t)M->L, (size_t)M->L, (size_t)M->n,
                                   cudaMemcpyDeviceToHost, stream),
                 "msa download")) ||
      (rc = cuda(cudaStreamSynchronize(stream), "msa sync")))
    return rc;
  return NWG_OK;
}

}  // namespace nwg

using nwg::Ctx;

extern "C" {

int nwg_msa(nwg_ctx* ctx, const int8_t* codes, const int64_t* offsets, int n, const int32_t* left,
            const int32_t* right, int64_t* msa_len, nwg_stats* stats) {
  if (!ctx) return NWG_ERR_INVALID;
  Ctx* c = reinterpret_cast<Ctx*>(ctx);
  if (stats) std::memset(stats, 0, sizeof(*stats));
  c->launches = 0;
  const int rc = c->msa(codes, offsets, n, left, right, msa_len, stats);
  if (stats) stats->launches = c->launches;
  return rc;
}

int nwg_msa_rows(nwg_ctx* ctx, char* out, int64_t row_stride) {
  if (!ctx) return NWG_ERR_INVALID;
  return reinterpret_cast<Ctx*>(ctx)->msa_rows(out, row_stride);
}

}  // extern "C"
