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
//  2. msa_wave_kernel, one cluster per merge: the recurrence as a wavefront of
//     warps, then the walk over its flags;
//  3. msa_build_kernel: the merged profile and, for both children, the map of
//     their columns to the new ones.
// Merges whose differences between neighbouring cells could leave 32 bits or
// whose scores find no memory, and gap models with open < extension, take
// msa_dp_kernel (64-bit cells) in place of 1 and 2.
// At the end the final position of every column is resolved parents first
// (msa_pos_kernel) and every leaf's residues are scattered into its row.
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <numeric>
#include <vector>

#include "nwg_ctx.h"
#include "pipe.cuh"
#include "profile8.cuh"

namespace nwg {
namespace {

constexpr int kMR = 256;   // rows per strip = threads per CTA of the 64-bit form

struct MergeDesc {
  int64_t xoff, yoff, ooff;   // first column of X, Y and the new profile in the count pool
  int64_t xmap, ymap;         // X's and Y's column maps (written here)
  int64_t nib;                // first flag byte
  int64_t src;                // first entry of the alignment's columns (capacity lx + ly)
  int64_t scratch;            // 64-bit form: first (H, F) pair of the strip-boundary scratch (lx entries)
  int64_t score;              // wave form: first int of the cell scores
  int64_t bnd;                // wave form: first entry of the band-boundary row (lx entries)
  int32_t lx, ly, kx, ky;
  int32_t tile0;              // wave form: first CTA of the score kernel
  int32_t mac32;              // kx * ky * max|S| < 2^31: a cell's score sum fits int32
  int32_t bytes;              // wave form: X's counts fit a byte and Y's row scores this many (0: they don't)
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
// The pipeline of pipe.cuh in 32 bits: its values lie within
// kX kY (2 max|S| + 4 go), and the host takes this form while that stays
// below 2^31 (a set of 8,000 sequences under the usual penalties).  A tree's
// deep levels hold one or two merges, so such a level costs one merge's chain
// of steps.  Four rows per lane: two give a shorter step but more hops between
// bands and more instructions a cell, and measured the same on a deep level.
// A level of one merge of 560 columns x 560 rows takes 82 us, of which the walk
// 10 (207 us with one CTA barrier per eight steps on a single SM and the scores
// in registers; 0.43 ms at 339 columns with 64-bit cells, one row per thread
// and a barrier per anti-diagonal).
constexpr int kScoreSteps = 32;            // steps per warp of the score kernel
constexpr int kScoreWarps = 4;
constexpr int kMsaWindow = 8192;           // bytes of flags in the walk's window

constexpr int kRows = 4;                   // rows per lane of the pipeline

// Sum of four products of unsigned bytes of a with signed (unsigned) bytes of b.
__device__ __forceinline__ int dot4_us(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}
__device__ __forceinline__ int dot4_uu(uint32_t a, uint32_t b, int c) {
  int d;
  asm("dp4a.u32.u32 %0, %1, %2, %3;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
  return d;
}

// The steps [t0, t1) of one warp of the score kernel.  Bytes: 0 for any counts
// and row scores (24 multiply-adds a cell); 1 when X's counts fit a byte and
// the row scores a signed one (6 four-byte dot products); 2 when the row scores
// need two (6 with the high bytes, 6 with the low).
template <int Bytes>
__device__ __forceinline__ void score_steps(const MergeDesc& m, const int (*s_w)[32 * kRows],
                                            const int16_t* __restrict__ cnt, int4* __restrict__ out, int base, int t0,
                                            int t1) {
  constexpr int R = kRows;
  const int lane = threadIdx.x & 31;
  constexpr int kW = Bytes == 0 ? kLetters : kLetters / 4;
  int W[kW][R], V[Bytes == 2 ? kW : 1][R];   // row scores (their high and low bytes)
#pragma unroll
  for (int q = 0; q < kLetters / 4; ++q) {
    int w[4][R];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
      const int4 v = *reinterpret_cast<const int4*>(&s_w[4 * q + x][R * lane]);
      w[x][0] = v.x, w[x][1] = v.y, w[x][2] = v.z, w[x][3] = v.w;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if constexpr (Bytes == 0) {
#pragma unroll
        for (int x = 0; x < 4; ++x) W[4 * q + x][r] = w[x][r];
      } else {
        const uint32_t lo = perm(perm(w[0][r], w[1][r], 0x0040), perm(w[2][r], w[3][r], 0x0040), 0x5410);
        if constexpr (Bytes == 2) {
          W[q][r] = (int)perm(perm(w[0][r], w[1][r], 0x0051), perm(w[2][r], w[3][r], 0x0051), 0x5410);
          V[q][r] = (int)lo;
        } else {
          W[q][r] = (int)lo;
        }
      }
    }
  }
  const uint4* X = reinterpret_cast<const uint4*>(cnt + m.xoff * kLetters);   // 48 bytes a column
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
    int s[R];
#pragma unroll
    for (int r = 0; r < R; ++r) s[r] = Bytes == 2 ? 0 : base;
    if constexpr (Bytes == 0) {
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const uint32_t w[4] = {cur[q].x, cur[q].y, cur[q].z, cur[q].w};
#pragma unroll
        for (int h = 0; h < 8; ++h) {
          const int n = (h & 1) ? (int)w[h >> 1] >> 16 : (int)(int16_t)(w[h >> 1] & 0xFFFFu);
#pragma unroll
          for (int r = 0; r < R; ++r) s[r] += n * W[q * 8 + h][r];
        }
      }
    } else {
      uint32_t n[kW];   // the column's counts, a byte each
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        n[2 * q] = perm(cur[q].x, cur[q].y, 0x6420);
        n[2 * q + 1] = perm(cur[q].z, cur[q].w, 0x6420);
      }
#pragma unroll
      for (int q = 0; q < kW; ++q)
#pragma unroll
        for (int r = 0; r < R; ++r) s[r] = dot4_us(n[q], (uint32_t)W[q][r], s[r]);
      if constexpr (Bytes == 2) {
#pragma unroll
        for (int r = 0; r < R; ++r) s[r] = s[r] * 256 + base;
#pragma unroll
        for (int q = 0; q < kW; ++q)
#pragma unroll
          for (int r = 0; r < R; ++r) s[r] = dot4_uu(n[q], (uint32_t)V[q][r], s[r]);
      }
    }
    out[(int64_t)t * 32] = make_int4(s[0], s[1], s[2], s[3]);
  }
}

// Scores of the cells of a level's merges in the wave kernel's order: entry
// (g * nsup * 8 + t) * 32 + l of a merge holds rows 128 g + 4 l .. + 3 at column
// t - l (2 GE outside).  One CTA per 128 rows x 128 steps: the rows' scores
// against each letter, W[x] = sum_y cY[y] S[y][x], go to shared memory once,
// then each warp runs 32 steps with its lanes' in registers, for three 16-byte
// loads of column counts a step.  Where counts and row scores fit bytes (a
// tree's lower levels, most of the cells) four products are one instruction.
// The lowest level of 8,000 sequences (2.7e8 padded cells, 1.1 GB of scores):
// 0.64 to 0.35 ms, 3.1 TB/s of stores; the whole tree 2.3 to 1.4 ms.
__global__ void __launch_bounds__(32 * kScoreWarps) msa_score_kernel(const MergeDesc* __restrict__ md, int nm,
                                                                    const int16_t* __restrict__ cnt,
                                                                    const int8_t* __restrict__ sub, int ge,
                                                                    int* __restrict__ score) {
  constexpr int kBand = 32 * kRows;
  static_assert(kBand == 32 * kScoreWarps, "one thread per row");
  __shared__ __align__(16) int8_t s_sub[kLetters * kLetters];
  __shared__ __align__(16) int s_w[kLetters][kBand];
  int lo = 0, hi = nm - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (md[mid].tile0 <= (int)blockIdx.x) lo = mid;
    else hi = mid - 1;
  }
  const MergeDesc m = md[lo];
  const int steps = pipe::supersteps_of(m.lx) * pipe::kStep;
  const int nchunk = (steps + kScoreSteps * kScoreWarps - 1) / (kScoreSteps * kScoreWarps);
  const int tile = (int)blockIdx.x - m.tile0;
  const int g = tile / nchunk, chunk = tile - g * nchunk;
  for (int e = threadIdx.x; e < kLetters * kLetters / 4; e += blockDim.x)
    reinterpret_cast<int*>(s_sub)[e] = reinterpret_cast<const int*>(sub)[e];
  __syncthreads();
  {
    int w[kLetters];
#pragma unroll
    for (int x = 0; x < kLetters; ++x) w[x] = 0;
    const int r = g * kBand + threadIdx.x;
    if (r < m.ly) {
      const uint4* cy = reinterpret_cast<const uint4*>(cnt + (m.yoff + r) * kLetters);
      const uint4 v[3] = {cy[0], cy[1], cy[2]};
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        const uint32_t h[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
        for (int b = 0; b < 8; ++b) {
          const int c = (b & 1) ? (int)h[b >> 1] >> 16 : (int)(int16_t)(h[b >> 1] & 0xFFFFu);
          if (c == 0) continue;
          const int* row = reinterpret_cast<const int*>(s_sub + (q * 8 + b) * kLetters);
#pragma unroll
          for (int x4 = 0; x4 < kLetters / 4; ++x4) {
            const int p = row[x4];
#pragma unroll
            for (int x = 0; x < 4; ++x) w[4 * x4 + x] += c * (int)(int8_t)(p >> (8 * x));
          }
        }
      }
    }
#pragma unroll
    for (int x = 0; x < kLetters; ++x) s_w[x][threadIdx.x] = w[x];
  }
  __syncthreads();
  const int t0 = (chunk * kScoreWarps + (int)(threadIdx.x >> 5)) * kScoreSteps;
  const int t1 = min(t0 + kScoreSteps, steps);
  if (t0 >= t1) return;
  int4* out = reinterpret_cast<int4*>(score + m.score) + (int64_t)g * steps * 32 + (threadIdx.x & 31);
  const int base = 2 * ge * m.kx * m.ky;   // the pipeline's S' = S + 2 GE
  if (m.bytes == 1) score_steps<1>(m, s_w, cnt, out, base, t0, t1);
  else if (m.bytes == 2) score_steps<2>(m, s_w, cnt, out, base, t0, t1);
  else score_steps<0>(m, s_w, cnt, out, base, t0, t1);
}

// The pipeline's scores: a superstep's are one block of 4 KB, copied to shared
// memory kSlots supersteps ahead by one bulk copy (a superstep takes about as
// long as a read from the far L2, so registers loaded one ahead left the warp
// waiting, and two ahead cost 64 of them).
struct MsaScore {
  static constexpr int kSlots = 3;
  static constexpr int kBytes = pipe::kStep * 32 * (int)sizeof(int4);
  struct Ring {
    int4 v[kSlots][pipe::kStep * 32];
    unsigned long long bar[kSlots];
  };
  Ring* ring;           // this warp's, in shared memory
  const int4* base;     // the merge's scores
  int nsup;
  const int4* band = nullptr;
  const int4* cur = nullptr;
  unsigned used = 0;    // supersteps begun
  __device__ __forceinline__ void ask(int j, unsigned use) {
    pipe::bar_expect(&ring->bar[use % kSlots], kBytes);
    pipe::copy_bulk(ring->v[use % kSlots], band + (int64_t)j * pipe::kStep * 32, kBytes, &ring->bar[use % kSlots]);
  }
  __device__ __forceinline__ void load(int g) {
    band = base + (int64_t)g * nsup * pipe::kStep * 32;
    if ((threadIdx.x & 31) == 0)
      for (int j = 0; j < kSlots && j < nsup; ++j) ask(j, used + j);
  }
  __device__ __forceinline__ void begin(int, pipe::Link& ln) {
    ln.wait(&ring->bar[used % kSlots], (used / kSlots) & 1);
    cur = ring->v[used % kSlots] + (threadIdx.x & 31);
  }
  __device__ __forceinline__ void get(int i, int, int (&s)[kRows]) const {
    const int4 v = cur[i * 32];
    s[0] = v.x, s[1] = v.y, s[2] = v.z, s[3] = v.w;
  }
  __device__ __forceinline__ void end(int j) {
    __syncwarp();
    if ((threadIdx.x & 31) == 0 && j + kSlots < nsup) ask(j + kSlots, used + kSlots);
    ++used;
  }
  __device__ __forceinline__ void column_done(int, const int (&)[kRows]) const {}
  __device__ __forceinline__ void band_done() const {}
};

// C CTAs (one cluster) per merge; dynamic shared memory: a score ring per warp,
// then the walk's window in its place.
__global__ void __launch_bounds__(32 * pipe::kWarps, 4) msa_wave_kernel(const MergeDesc* __restrict__ md, int C,
                                                                       const int* __restrict__ score,
                                                                       uint32_t* flags, int2* bnd, unsigned* done,
                                                                       int2* __restrict__ src,
                                                                       int32_t* __restrict__ nops, int* err, int go,
                                                                       int ge) {
  using Ring = MsaScore::Ring;
  static_assert(sizeof(Ring) >= kMsaWindow, "the window takes a ring's place");
  __shared__ pipe::Inbox s_box[pipe::kWarps];
  extern __shared__ __align__(128) unsigned char s_dyn[];
  Ring* s_ring = reinterpret_cast<Ring*>(s_dyn);
  const int q = blockIdx.x / C, rank = blockIdx.x - q * C;
  const MergeDesc m = md[q];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpc = blockDim.x >> 5;
  const int gw = rank * wpc + warp, nwarp = C * wpc;
  if (threadIdx.x == 0)
    for (int w = 0; w < wpc; ++w)
      for (int k = 0; k < MsaScore::kSlots; ++k) pipe::bar_init(&s_ring[w].bar[k]);
  pipe::init_inboxes(s_box, wpc);
  pipe::Link ln;
  ln.in = &s_box[warp];
  ln.out = pipe::cluster_addr(pipe::smem_addr(&s_box[(gw + 1) % wpc]), (gw + 1) % nwarp / wpc);
  ln.back = pipe::cluster_addr(pipe::smem_addr(&s_box[(gw + nwarp - 1) % wpc]), (gw + nwarp - 1) % nwarp / wpc);
  ln.err = err;
  const int nsup = pipe::supersteps_of(m.lx);
  uint32_t* fl = flags + m.nib / 4;
  MsaScore sc;
  sc.ring = s_ring + warp;
  sc.base = reinterpret_cast<const int4*>(score + m.score);
  sc.nsup = nsup;
  pipe::run_bands<kRows>(ln, pipe::Wrap{bnd + m.bnd, done + q}, sc, fl, m.lx, m.ly, (go - ge) * m.kx * m.ky, gw, nwarp);
  pipe::cluster_barrier();   // every band's flags are written, every copy has arrived
  if (rank != 0 || warp != 0) return;
  // the walk: the alignment's columns in forward order (X column, Y column; -1 a gap)
  pipe::Window<kRows, kMsaWindow> win{fl, reinterpret_cast<uint32_t*>(s_dyn), nsup};
  int2* out = src + m.src;
  WalkPos p = run_walk(win, m.lx, m.ly, m.lx + m.ly, [&](int k, int n, int x, int y, int sx, int sy) {
    if (lane < n) out[k + lane] = make_int2(sx ? x - lane : -1, sy ? y - lane : -1);
  });
  // columns the walk left, opposite gaps
  for (int i = lane; i <= p.x; i += 32) out[p.k + i] = make_int2(p.x - i, -1);
  p.k += p.x + 1;
  for (int i = lane; i <= p.y; i += 32) out[p.k + i] = make_int2(-1, p.y - i);
  p.k += p.y + 1;
  if (lane == 0) nops[q] = p.k;
}

cudaError_t launch_msa_wave(const MergeDesc* md, int count, int warps, const int* score, uint32_t* flags, int2* bnd,
                            unsigned* done, int2* src, int32_t* nops, int* err, int go, int ge, cudaStream_t s) {
  const int C = (warps + pipe::kWarps - 1) / pipe::kWarps;
  const int wpc = (warps + C - 1) / C;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(count * C));
  cfg.blockDim = dim3((unsigned)(32 * wpc));
  cfg.dynamicSmemBytes = sizeof(MsaScore::Ring) * wpc;
  cfg.stream = s;
  const cudaError_t e = allow_smem((const void*)msa_wave_kernel);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)C;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, msa_wave_kernel, md, C, score, flags, bnd, done, src, nops, err, go, ge);
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

// Leaf profiles: one column per residue (reversed codes), count 1; three
// threads per column, so a warp's stores are whole lines (1.6 million residues:
// 210 to 18 us).
__global__ void msa_leaf_kernel(const int8_t* __restrict__ codes, int64_t total, uint4* __restrict__ cnt) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= 3 * total) return;
  const int64_t c = e / 3;
  int x = codes[c];
  if (x < 0 || x >= kLetters) x = kLetters - 1;
  x -= 8 * (int)(e - 3 * c);   // the letter's place among this thread's eight
  const uint32_t one = (x & 1) ? 0x10000u : 1u;
  cnt[e] = make_uint4(x >> 1 == 0 ? one : 0u, x >> 1 == 1 ? one : 0u, x >> 1 == 2 ? one : 0u, x >> 1 == 3 ? one : 0u);
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
  msa_leaf_kernel<<<(unsigned)((3 * total + 255) / 256), 256, 0, s>>>((const int8_t*)M.codes.p, total,
                                                                     (uint4*)M.cnt.p);
  ++launches;
  std::vector<std::vector<int>> bylevel(levels + 1);
  for (int k = 0; k < n - 1; ++k) bylevel[height[n + k]].push_back(n + k);
  int64_t cells = 0;
  int64_t smax = 1;   // largest |S| of the context's matrix
  for (int k = 0; k < kLetters * kLetters; ++k) smax = std::max<int64_t>(smax, sub[k] < 0 ? -sub[k] : sub[k]);
  const int64_t diff_bound = 2 * smax + 4 * (int64_t)go;   // the wave form's values, per kX * kY
  constexpr int64_t kScoreBatch = (int64_t)1 << 27;        // cell scores of one batch of merges (512 MiB)
  constexpr int64_t kScoreMax = (int64_t)1 << 31;          // of one merge (8 GiB; beyond, the 64-bit form)
  std::vector<MergeDesc> md;
  std::vector<int32_t> nops;
  // Cell scores that one merge may take.  Where there is no memory for a level's,
  // its merges beyond a batch, then all, take the 64-bit form, which needs none.
  int64_t score_max = kScoreMax;
  // failure injection for the tests: more scores than this do not fit
  const char* inject = std::getenv("NWG_MSA_INJECT_SCORE_OOM");
  const int64_t score_room = inject ? std::atoll(inject) : INT64_MAX;
  // batches of wave merges that share the score buffer (on one stream, so one after another)
  struct Batch {
    int first, count, tiles, warps;
  };
  std::vector<Batch> batches;
  for (int l = 1; l <= levels; ++l) {
    // wave-form merges first, most supersteps first; then the 64-bit ones
    std::vector<int>& nodes = bylevel[l];
    const int nm = (int)nodes.size();
    constexpr int kBand = 32 * kRows;
    auto padded = [&](int v) {   // cell scores of a merge
      return (int64_t)((len[right[v - n]] + kBand - 1) / kBand) * kBand * pipe::supersteps_of((int)len[left[v - n]]) *
             pipe::kStep;
    };
    auto is_wave = [&](int v) {
      return go >= ge && (int64_t)kseq[left[v - n]] * kseq[right[v - n]] * diff_bound < ((int64_t)1 << 31) &&
             padded(v) <= score_max;
    };
    int nwave = 0, maxcols = 1;
    const int64_t pool0 = pool, cells0 = cells;
    for (;;) {
      nwave = (int)(std::stable_partition(nodes.begin(), nodes.end(), is_wave) - nodes.begin());
      std::stable_sort(nodes.begin(), nodes.begin() + nwave, [&](int u, int v) {
        const int64_t bu = (len[right[u - n]] + kBand - 1) / kBand, bv = (len[right[v - n]] + kBand - 1) / kBand;
        return bu != bv ? bu > bv : len[left[u - n]] > len[left[v - n]];
      });
      md.assign(nm, MergeDesc{});
      batches.clear();
      pool = pool0;
      cells = cells0;
      int64_t nib_total = 0, src_total = 0, scr_total = 0, score_cap = 0, score_used = 0, bnd_total = 0;
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
        d.bytes = d.kx > 255 ? 0 : d.ky * smax <= 127 ? 1 : d.ky * smax <= 32767 ? 2 : 0;
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
          const int64_t bands = (d.ly + kBand - 1) / kBand, nsup = pipe::supersteps_of(d.lx);
          const int64_t words = padded(v);
          if (batches.empty() || score_used + words > kScoreBatch) {
            batches.push_back({q, 0, 0, 1});
            score_used = 0;
          }
          Batch& bt = batches.back();
          d.score = score_used;
          score_used += words;
          score_cap = std::max(score_cap, score_used);
          d.tile0 = bt.tiles;
          bt.tiles += (int)(bands * ((nsup * pipe::kStep + kScoreSteps * kScoreWarps - 1) / (kScoreSteps * kScoreWarps)));
          bt.count += 1;
          bt.warps = std::max(bt.warps, (int)std::min<int64_t>(bands, pipe::kWarps * pipe::kCluster));
          d.bnd = bnd_total;
          if (bands > pipe::kWarps * pipe::kCluster) bnd_total += d.lx;
          nib_total += bands * nsup * 128 * kRows;
        } else {
          const int nstr = (d.ly + kMR - 1) / kMR;
          nib_total += ((int64_t)nstr * (d.lx + kMR - 1) * kMR + 15) / 16 * 16;
          d.scratch = scr_total;
          scr_total += d.lx;
        }
      }
      rc = score_cap > score_room ? NWG_ERR_OOM : NWG_OK;
      if (rc || (rc = M.nib.ensure((size_t)std::max<int64_t>(nib_total, 1))) ||
          (rc = M.src.ensure(sizeof(int2) * (size_t)std::max<int64_t>(src_total, 1))) ||
          (rc = M.scratch.ensure(sizeof(longlong2) * (size_t)std::max<int64_t>(scr_total, 1))) ||
          (rc = M.bnd.ensure(sizeof(int2) * (size_t)std::max<int64_t>(bnd_total, 1))) ||
          (rc = M.nops.ensure(sizeof(int32_t) * (2 * (size_t)nm + 1))) || (rc = M.md.ensure(sizeof(MergeDesc) * nm)) ||
          (rc = M.score.ensure(sizeof(int) * (size_t)std::max<int64_t>(score_cap, 1)))) {
        if (rc != NWG_ERR_OOM || score_max == 0) return fail(rc, "msa allocation");
        M.score.release();
        score_max = score_cap > kScoreBatch ? kScoreBatch : 0;
        continue;
      }
      break;
    }
    if ((rc = cuda(cudaMemcpyAsync(M.md.p, md.data(), sizeof(MergeDesc) * nm, cudaMemcpyHostToDevice, s), "msa upload")))
      return rc;
    const MergeDesc* dmd = (const MergeDesc*)M.md.p;
    // nops: the merges' lengths, an error flag, the wave form's wrap counters
    int32_t* dnops = (int32_t*)M.nops.p;
    int* derr = (int*)dnops + nm;
    unsigned* ddone = (unsigned*)dnops + nm + 1;
    if ((rc = cuda(cudaMemsetAsync(derr, 0, sizeof(int) * ((size_t)nm + 1), s), "msa"))) return rc;
    for (const Batch& b : batches) {
      const MergeDesc* bmd = dmd + b.first;
      msa_score_kernel<<<b.tiles, 32 * kScoreWarps, 0, s>>>(bmd, b.count, (const int16_t*)M.cnt.p,
                                                            (const int8_t*)b_sub.p, ge, (int*)M.score.p);
      if ((rc = cuda(launch_msa_wave(bmd, b.count, b.warps, (const int*)M.score.p, (uint32_t*)M.nib.p, (int2*)M.bnd.p,
                                     ddone + b.first, (int2*)M.src.p, dnops + b.first, derr, go, ge, s),
                     "msa launch")))
        return rc;
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
    nops.resize((size_t)nm + 1);
    if ((rc = cuda(cudaMemcpyAsync(nops.data(), M.nops.p, sizeof(int32_t) * ((size_t)nm + 1), cudaMemcpyDeviceToHost, s),
                   "msa")) ||
        (rc = cuda(cudaStreamSynchronize(s), "msa sync")))
      return rc;
    if (nops[nm]) return fail(NWG_ERR_TIMEOUT, "progressive alignment: a bounded device wait ran out");
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
  // scores beyond a batch's (one large merge) are not kept for the next call
  if (M.score.cap > sizeof(int) * (size_t)kScoreBatch) M.score.release();
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
