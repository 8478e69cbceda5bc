// trace.cu -- pairwise alignment with traceback for guide-tree cherries.
//
// Replaces AlignmentMatch::computePairwise (AlignmentMatch.cu:140-317) with
// its three kernels: NeedlemanWunschGlobalMatchKernel (NeedlemanWunsch.cu:
// 184-365), NeedlemanWunschGlobalBackKernel (:393-494) and
// reorderMatchesMemory (:496-563).
//
// match_kernel<W>: a wavefront of W lanes per pair (W = 32, 16 or 8: 32/W
//   pairs per warp), int32 lanes; lane k of a front owns 8 rows of a band of
//   8W rows, one column behind lane k-1, bottom (H, F) passed by
//   __shfl_up_sync within the front.  Narrow fronts cut the rows computed
//   past the end of Y (the last band) and the ramp of W-1 columns per band.
//   Every cell yields the reference's 4-bit flags
//     bit3 L  = (H==E && H!=F) || H==diag        (:330)
//     bit2 U  = H==F || H==diag                  (:332)
//     bit1 cU = F == F_up - ge                   (:315-316, :334)
//     bit0 cL = E == E_left - ge                 (:336)
//   from the sign bits of four differences, appended by funnel shifts.
//   A lane's 8 rows of one column make one 32-bit word; the W lanes of a
//   front store W consecutive words per step: word (b*(Lx+W-1) + t)*W + k
//   holds rows b*8W + 8k .. +7 at column t-k, a byte per flag (L highest),
//   row r in bit 7-r.
// trace_pipe_kernel: one pair as a pipeline of warps over a cluster (pipe.cuh),
//   four rows per lane, for launches whose pairs do not fill the chip.
// The walk runs in the warp right after the pair's last band, while its flags
//   are still in L2, from (Lx-1, Ly-1), in runs (walk.cuh), over a window of
//   4 or 8 KB of flags staged in shared memory.  The moves go through a small
//   queue in shared memory, so that the residues' loads and the characters'
//   stores are 128 at a time.  Characters come out in forward order, so the
//   reorder/byte-swap pass is not needed.
#include <algorithm>
#include <cstring>
#include <vector>

#include "nwg_ctx.h"
#include "pipe.cuh"
#include "profile8.cuh"

namespace nwg {

namespace {

constexpr int kTR = 8;                               // rows per lane
constexpr int kTWarps = 4;                           // warps per CTA
constexpr int kTProfBytes = kLetters * 32 * kTR;     // profile bytes per warp (6 KB, every W)

struct TraceArgs {
  const int8_t* codes;
  const int64_t* start;
  const int32_t* len;
  const int32_t* px;
  const int32_t* py;
  const int32_t* order;     // slot -> pair: pairs of similar lengths share a warp
  const int64_t* nib_off;   // per pair: first word of its nibble array
  uint32_t* nib;
  int32_t* scratch;         // per pair slot: 2 buffers x 2 ints x maxlen
  int32_t* score;
  char* outx;
  char* outy;
  int32_t* outlen;
  int64_t stride;
  int npairs;
  int scratch_cols;
  int go, ge;
  const int8_t* sub;
  // pipeline form
  unsigned* done;           // per pair: columns handed on through the scratch row
  int* err;                 // set when a wait runs out
};

__device__ __forceinline__ unsigned tclamp(int c) {
  const unsigned u = (unsigned)c;
  return u < (unsigned)kLetters ? u : (unsigned)(kLetters - 1);
}

static_assert(kTR == 8, "a lane's scores of one column are one 8-byte load");

// The gapped strings of one walk: its moves queue in shared memory and leave
// 128 at a time (a load and a store per move on the walk itself would make
// every run wait for memory).
constexpr int kQueue = 256;
__device__ const char d_dec[kLetters + 1] = "ARNDCQEGHILKMFPSTWYVBZX*";   // code -> letter
struct TextOut {
  const int8_t* X;
  const int8_t* Y;
  char* ox;
  char* oy;
  int2* queue;      // shared, kQueue entries: the move's column and row, -1 for a gap
  int done = 0;     // moves written out
  static __device__ __forceinline__ char letter(int c) { return d_dec[tclamp(c)]; }
  __device__ __forceinline__ void flush(int count) {
    const int lane = threadIdx.x & 31;
    __syncwarp();
    int cx[4], cy[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = q * 32 + lane;
      cx[q] = cy[q] = -1;
      if (e < count) {
        const int2 p = queue[(done + e) % kQueue];
        if (p.x >= 0) cx[q] = tclamp(X[p.x]);
        if (p.y >= 0) cy[q] = tclamp(Y[p.y]);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = q * 32 + lane;
      if (e < count) {
        ox[done + e] = cx[q] >= 0 ? letter(cx[q]) : '-';
        oy[done + e] = cy[q] >= 0 ? letter(cy[q]) : '-';
      }
    }
    done += count;
    __syncwarp();
  }
  __device__ __forceinline__ void operator()(int k, int m, int x, int y, int sx, int sy) {
    const int lane = threadIdx.x & 31;
    if (lane < m) queue[(k + lane) % kQueue] = make_int2(sx ? x - lane : -1, sy ? y - lane : -1);
    if (k + m - done >= 128) flush(128);
  }
  // the last moves, the terminators
  __device__ __forceinline__ void finish(int k) {
    flush(k - done);
    if ((threadIdx.x & 31) == 0) ox[k] = oy[k] = 0;
  }
};

// Window over a pair's flags in the match kernel's layout: 1,024 words, the
// steps of one band that end at the walk's cell.
template <int W>
struct MatchWindow {
  static constexpr int kSteps = 1024 / W;
  const uint32_t* nib;
  uint32_t* win;           // shared, 1,024 words
  int Lx;
  int b = -1, t0 = 0;      // band, first step held
  __device__ __forceinline__ bool covers(int x, int y) const {
    const int t = x + y % (8 * W) / 8 - t0;
    return y / (8 * W) == b && t >= 0 && t < kSteps;
  }
  __device__ __forceinline__ unsigned cell(int x, int y) const {
    const int k = y % (8 * W) / 8;
    const uint32_t w = win[(x + k - t0) * W + k] >> (7 - (y & 7));
    return (w >> 24 & 1u) << 3 | (w >> 16 & 1u) << 2 | (w >> 8 & 1u) << 1 | (w & 1u);
  }
  __device__ __forceinline__ void load(int x, int y) {
    const int lane = threadIdx.x & 31;
    b = y / (8 * W);
    t0 = x + y % (8 * W) / 8 - (kSteps - 1);
    __syncwarp();
    const uint32_t* src = nib + ((int64_t)b * (Lx + W - 1) + t0) * W;
    uint4 v[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = (q * 32 + lane) * 4;
      if (t0 + e / W >= 0) v[q] = *reinterpret_cast<const uint4*>(src + e);
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int e = (q * 32 + lane) * 4;
      if (t0 + e / W >= 0) *reinterpret_cast<uint4*>(win + e) = v[q];
    }
    __syncwarp();
  }
};

// One pair's walk by one warp.
template <class Window>
__device__ void walk_pair(const TraceArgs& a, int p, Window& win, int2* queue) {
  const int ix = a.px[p], iy = a.py[p];
  TextOut out{a.codes + a.start[ix], a.codes + a.start[iy], a.outx + (size_t)p * a.stride,
              a.outy + (size_t)p * a.stride, queue};
  const int Lx = a.len[ix], Ly = a.len[iy];
  const WalkPos w = run_walk(win, Lx, Ly, Lx + Ly, out);
  out.finish(w.k);
  if ((threadIdx.x & 31) == 0) a.outlen[p] = w.k;
}

template <int W>
__global__ void __launch_bounds__(32 * kTWarps) match_kernel(const TraceArgs a) {
  constexpr int S = 32 / W;         // fronts (pairs) per warp
  constexpr int BAND = W * kTR;     // rows per band
  __shared__ int8_t s_sub[kLetters * kLetters];
  __shared__ __align__(16) int8_t s_prof[kTWarps][kTProfBytes];   // per front [letter][band row]
  for (int e = threadIdx.x; e < kLetters * kLetters; e += blockDim.x) s_sub[e] = a.sub[e];
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int front = lane / W, sl = lane % W;
  const int wslot = (blockIdx.x * kTWarps + warp) * S;
  if (wslot >= a.npairs) return;    // the whole warp is idle
  const int slot = wslot + front;
  const int p = slot < a.npairs ? a.order[slot] : -1;
  const int8_t* X = nullptr;
  const int8_t* Y = nullptr;
  int Lx = 0, Ly = 0;
  if (p >= 0) {
    const int ix = a.px[p], iy = a.py[p];
    X = a.codes + a.start[ix];
    Y = a.codes + a.start[iy];
    Lx = a.len[ix];
    Ly = a.len[iy];
  }
  const int go = a.go, ge = a.ge;
  const int nb = (Ly + BAND - 1) / BAND;
  const int nb_max = __reduce_max_sync(0xffffffffu, (unsigned)nb);
  const int lx_max = __reduce_max_sync(0xffffffffu, (unsigned)Lx);
  int8_t* prof = s_prof[warp] + front * (kLetters * BAND);
  int32_t* scr = p >= 0 ? a.scratch + (size_t)p * 4 * a.scratch_cols : nullptr;
  uint32_t* nib = p >= 0 ? a.nib + a.nib_off[p] : nullptr;
  const int kSent = kShortMin + ge;
  int H[kTR], E[kTR];
  for (int b = 0; b < nb_max; ++b) {
    const bool band_on = b < nb;
    __syncwarp();
    if (band_on)
      for (int e = sl; e < kLetters * BAND; e += W) {
        const int x = e / BAND, row = e - x * BAND, grow = b * BAND + row;
        prof[e] = grow < Ly ? s_sub[tclamp(Y[grow]) * kLetters + x] : (int8_t)0;
      }
    __syncwarp();
    const int rowbase = b * BAND + sl * kTR;
#pragma unroll
    for (int r = 0; r < kTR; ++r) {
      H[r] = -ge * (rowbase + r + 1);
      E[r] = kSent;
    }
    int hprev = -ge * rowbase;
    int hbot = 0, fbot = 0;
    const int32_t* rd = scr + ((b + 1) & 1) * 2 * a.scratch_cols;
    int32_t* wr = scr + (b & 1) * 2 * a.scratch_cols;
    uint32_t* nb_base = nib + (size_t)b * (Lx + W - 1) * W;
    for (int t = 0; t < lx_max + W - 1; ++t) {
      const int c = t - sl;
      int hin = __shfl_up_sync(0xffffffffu, hbot, 1, W);
      int fin = __shfl_up_sync(0xffffffffu, fbot, 1, W);
      if (band_on && c >= 0 && c < Lx) {
        if (sl == 0) {
          if (b == 0) {
            hin = -ge * (c + 1);
            fin = kSent;
          } else {
            hin = rd[2 * c];
            fin = rd[2 * c + 1];
          }
        }
        // the lane's 8 scores of column c: one 8-byte load
        const uint2 pw = *reinterpret_cast<const uint2*>(prof + tclamp(X[c]) * BAND + sl * kTR);
        int diag = hprev;
        hprev = hin;
        int f = fin, hup = hin;
        uint32_t aL = 0, aU = 0, aCu = 0, aCl = 0;
#pragma unroll
        for (int r = 0; r < kTR; ++r) {
          // Each flag is the sign bit of one difference (a - b - 1 < 0 <=> a <= b):
          // cu = (F_up - ge >= H_up - go), cl = (E_left - ge >= H_left - go),
          // pf = (F >= E), ps = (diag + S >= max(F, E)), i.e. H == diag + S;
          // then U = ps || pf and L = ps || !pf, since otherwise H = max(F, E)
          // and H == F <=> pf, (H == E && H != F) <=> !pf.  The bits are
          // appended by funnel shifts to a word per flag (one word for all
          // would chain 32 shifts a step), the words' low bytes then joined:
          // L, U, cU, cL of row r land in bits 31-r, 23-r, 15-r and 7-r.
          const int fo = f - ge, hgo = hup - go;
          const uint32_t xcu = (uint32_t)(hgo - fo - 1);
          f = max(fo, hgo);
          const int eo = E[r] - ge, ego = H[r] - go;
          const uint32_t xcl = (uint32_t)(ego - eo - 1);
          const int e = max(eo, ego);
          const int sv = (int)(int8_t)((r < 4 ? pw.x : pw.y) >> (8 * (r & 3)));
          const int sim = diag + sv;
          const uint32_t xpf = (uint32_t)(e - f - 1);
          const int t2 = max(f, e);
          const uint32_t xps = (uint32_t)(t2 - sim - 1);
          const int h = max(sim, t2);
          aL = __funnelshift_l(xps | ~xpf, aL, 1);
          aU = __funnelshift_l(xps | xpf, aU, 1);
          aCu = __funnelshift_l(xcu, aCu, 1);
          aCl = __funnelshift_l(xcl, aCl, 1);
          diag = H[r];
          H[r] = h;
          E[r] = e;
          hup = h;
        }
        nb_base[(size_t)t * W + sl] = perm(perm(aCl, aCu, 0x0040), perm(aU, aL, 0x0040), 0x5410);
        hbot = H[kTR - 1];
        fbot = f;
        if (sl == W - 1 && b + 1 < nb) {
          wr[2 * c] = hbot;
          wr[2 * c + 1] = fbot;
        }
      }
    }
    if (band_on) {
      const int rr = (Ly - 1) - b * BAND;
      if (rr >= 0 && rr < BAND && sl == rr / kTR) {
        int v = 0;
#pragma unroll
        for (int r = 0; r < kTR; ++r)
          if (r == rr % kTR) v = H[r];
        a.score[p] = v;
      }
    }
  }
  // the walks, one after another, while the pairs' flags are still in L2 (the
  // warp's stores are visible to the warp after the warp barrier); window and
  // queue take the place of the fronts' profiles
  __syncwarp();
  static_assert(4096 + kQueue * sizeof(int2) <= kTProfBytes, "window and queue fit the profile's space");
  for (int f = 0; f < S; ++f) {
    const int q = __shfl_sync(0xffffffffu, p, f * W);
    if (q < 0) break;   // pairs fill the fronts from the first on
    MatchWindow<W> win{a.nib + a.nib_off[q], reinterpret_cast<uint32_t*>(s_prof[warp]), a.len[a.px[q]]};
    walk_pair(a, q, win, reinterpret_cast<int2*>(s_prof[warp] + 4096));
  }
}

// ---- the pipeline form ------------------------------------------------------------

// The pipeline's scores: a byte profile of the warp's band (S' = S + 2 ge, as a
// signed byte) and the CTA's copy of X's codes, both in shared memory.
struct TraceScore {
  uint32_t* prof;        // this warp's, [letter][lane] words of four rows
  const int8_t* xs;      // X's codes from column -32 on
  const int8_t* s_sub;   // the matrix plus 2 ge
  const int8_t* Y;
  int lx, ly;
  uint32_t zero;         // 2 ge in every byte: rows past Y
  int row0 = 0, sum = 0; // first row of the lane; sum of u(r, lx - 1) over its rows
  __device__ __forceinline__ void load(int g) {
    const int lane = threadIdx.x & 31;
    row0 = g * 128 + 4 * lane;
    __syncwarp();
    build_profile<4>(prof, s_sub, Y, row0, ly, zero, lane);
    __syncwarp();
  }
  __device__ __forceinline__ void begin(int, pipe::Link&) const {}
  __device__ __forceinline__ void end(int) const {}
  __device__ __forceinline__ void get(int, int t, int (&s)[4]) const {
    const int lane = threadIdx.x & 31;
    const uint32_t w = prof[(int)xs[32 + t - lane] * 32 + lane];
#pragma unroll
    for (int r = 0; r < 4; ++r) s[r] = (int)perm(w, 0u, r | (r | 8) << 4 | (r | 8) << 8 | (r | 8) << 12);
  }
  __device__ __forceinline__ void column_done(int t, const int (&n)[4]) {
    if (t >= lx - 1 && t - (int)(threadIdx.x & 31) == lx - 1) {
#pragma unroll
      for (int r = 0; r < 4; ++r)
        if (row0 + r < ly) sum -= n[r];
    }
  }
  __device__ __forceinline__ void band_done() const {}
};

constexpr int kTraceWindow = 8192;   // bytes of flags in the walk's window

// Dynamic shared memory of a pipeline CTA: profiles, then X's codes; the walk's
// window and queue take their place.
inline size_t trace_pipe_smem(int wpc, int lx_max) {
  const size_t score = (size_t)wpc * kLetters * 128 + (size_t)(lx_max + 128);
  const size_t walk = kTraceWindow + kQueue * sizeof(int2);
  return (std::max(score, walk) + 127) / 128 * 128;
}

// C CTAs (one cluster) per pair.
__global__ void __launch_bounds__(32 * pipe::kWarps, 4) trace_pipe_kernel(const TraceArgs a, int C) {
  __shared__ pipe::Inbox s_box[pipe::kWarps];
  __shared__ __align__(16) int8_t s_sub[kLetters * kLetters];
  extern __shared__ __align__(128) unsigned char s_dyn[];
  const int p = a.order[blockIdx.x / C], rank = blockIdx.x % C;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, wpc = blockDim.x >> 5;
  const int gw = rank * wpc + warp, nwarp = C * wpc;
  const int ix = a.px[p], iy = a.py[p];
  const int8_t* X = a.codes + a.start[ix];
  const int Lx = a.len[ix], Ly = a.len[iy];
  int8_t* xs = reinterpret_cast<int8_t*>(s_dyn) + wpc * kLetters * 128;
  for (int e = threadIdx.x; e < kLetters * kLetters; e += blockDim.x) s_sub[e] = (int8_t)(a.sub[e] + 2 * a.ge);
  for (int e = threadIdx.x; e < Lx + 80; e += blockDim.x)   // 32 before column 0, past the last superstep
    xs[e] = e >= 32 && e - 32 < Lx ? (int8_t)tclamp(X[e - 32]) : (int8_t)0;
  pipe::init_inboxes(s_box, wpc);
  pipe::Link ln;
  ln.in = &s_box[warp];
  ln.out = pipe::cluster_addr(pipe::smem_addr(&s_box[(gw + 1) % wpc]), (gw + 1) % nwarp / wpc);
  ln.back = pipe::cluster_addr(pipe::smem_addr(&s_box[(gw + nwarp - 1) % wpc]), (gw + nwarp - 1) % nwarp / wpc);
  ln.err = a.err;
  TraceScore sc{reinterpret_cast<uint32_t*>(s_dyn) + warp * kLetters * 32, xs, s_sub, a.codes + a.start[iy], Lx, Ly,
                0x01010101u * (uint32_t)(2 * a.ge & 255)};
  uint32_t* fl = a.nib + a.nib_off[p];
  pipe::run_bands<4>(ln, pipe::Wrap{reinterpret_cast<int2*>(a.scratch + (size_t)p * 4 * a.scratch_cols), a.done + p},
                     sc, fl, Lx, Ly, a.go - a.ge, gw, nwarp);
  // H(Ly-1, Lx-1): the last column's sum of u, less the free extension's ge a cell
  const int sum = __reduce_add_sync(0xffffffffu, sc.sum) - (gw == 0 ? a.ge * (Lx + Ly) : 0);
  if (lane == 0 && sum != 0) atomicAdd(&a.score[p], sum);
  pipe::cluster_barrier();   // every band's flags are written
  if (rank != 0 || warp != 0) return;
  pipe::Window<4, kTraceWindow> win{fl, reinterpret_cast<uint32_t*>(s_dyn), pipe::supersteps_of(Lx)};
  walk_pair(a, p, win, reinterpret_cast<int2*>(s_dyn + kTraceWindow));
}

}  // namespace

struct TraceState {
  DevBuf codes, start, len, px, py, order, off, nib, scratch, score, outx, outy, outlen, done;
  ~TraceState() {
    for (DevBuf* b : {&codes, &start, &len, &px, &py, &order, &off, &nib, &scratch, &score, &outx, &outy, &outlen, &done})
      b->release();
  }
};

namespace {

// Front width of the match kernel: 16 lanes (two pairs a warp, bands of 128
// rows, ramps of 15 columns) for short Y, else 32.  Kernel times on a GB300 at
// W = 32 / 16 / 8, ms: 4,000 pairs of 60 residues 0.143 / 0.092 / 0.151, 1,000
// of 100 0.086 / 0.156 / 0.252, 4,000 of 190 0.44 / 0.66 / 1.25 (a second band
// of a narrow front waits for the first one's row).
constexpr int kShortRows = 80;
int trace_lanes(double mean_rows) { return mean_rows <= kShortRows ? 16 : 32; }

// Whether the pipeline form gives this context's alignments of sequences up to
// maxlen: it needs open >= extension, scores that fit a signed byte with the
// extension folded in, X's codes in shared memory, and lengths at which the
// recurrence's finite sentinel (-32768 + ge before row 0 and column 0) never
// beats a gap opened at the border.
bool pipe_ok(const Ctx& c, int maxlen) {
  int smin = 127, smax = -128;
  for (int k = 0; k < kLetters * kLetters; ++k) {
    smin = std::min<int>(smin, c.sub[k]);
    smax = std::max<int>(smax, c.sub[k]);
  }
  return c.go >= c.ge && smin + 2 * c.ge >= -128 && smax + 2 * c.ge <= 127 && 2 * c.ge <= 127 && maxlen <= 100000 &&
         (int64_t)c.ge * (maxlen + 1) + c.go < 32768;
}

cudaError_t launch_pipe(const TraceArgs& a, int first, int count, int warps, int lx_max, cudaStream_t s) {
  const int C = (warps + pipe::kWarps - 1) / pipe::kWarps;
  const int wpc = (warps + C - 1) / C;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(count * C));
  cfg.blockDim = dim3((unsigned)(32 * wpc));
  cfg.dynamicSmemBytes = trace_pipe_smem(wpc, lx_max);
  cfg.stream = s;
  const cudaError_t e = allow_smem((const void*)trace_pipe_kernel);
  if (e != cudaSuccess) return e;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)C;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  TraceArgs b = a;
  b.order += first;
  return cudaLaunchKernelEx(&cfg, trace_pipe_kernel, b, C);
}

cudaError_t launch_match(int W, const TraceArgs& a, cudaStream_t s) {
  const int per_cta = kTWarps * (32 / W);
  const int grid = (a.npairs + per_cta - 1) / per_cta;
  if (W == 8) match_kernel<8><<<grid, 32 * kTWarps, 0, s>>>(a);
  else if (W == 16) match_kernel<16><<<grid, 32 * kTWarps, 0, s>>>(a);
  else match_kernel<32><<<grid, 32 * kTWarps, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace

// The pipeline launches of one batch (pairs in order: most bands first).  A
// pair takes one warp per band over as many CTAs (of four warps) as that needs,
// at most so many that all pairs' CTAs come to about five an SM; a deeper pair
// runs its bands in passes.  With one CTA a pair, pairs of one or two bands go
// to CTAs of as many warps, in launches of their own side by side (a launch's
// shape is its first pair's).  Kernel times on a GB300 against one warp per
// pair: 4,000 pairs of 210 residues 0.71 to 0.38 ms, 200 of 867 4.0 to 0.40 ms,
// 200 of 2,000 21.1 to 1.6 ms (one CTA each 3.3), 1,500 of 867 4.45 to 1.43 ms
// (two CTAs each 2.0), one of 2,000 5.3 to 0.40 ms.
static int launch_pipes(Ctx* c, const TraceArgs& a, const std::vector<int32_t>& order,
                        const std::vector<int32_t>& len, const int32_t* px, const int32_t* py, cudaStream_t s) {
  const int m = (int)order.size();
  auto bands = [&](int k) { return (len[py[order[(size_t)k]]] + 127) / 128; };
  int lx = 1;
  for (int k = 0; k < m; ++k) lx = std::max(lx, len[px[k]]);
  const int ctas = std::min(std::max((5 * c->sms + m / 2) / m, 1), pipe::kCluster);
  int rc;
  if (ctas > 1) return c->cuda(launch_pipe(a, 0, m, std::min(bands(0), ctas * pipe::kWarps), lx, s), "traceback launch");
  int first[4] = {0, 0, 0, m};   // pairs of three bands or more, of two, of one
  while (first[1] < m && bands(first[1]) > 2) ++first[1];
  first[2] = first[1];
  while (first[2] < m && bands(first[2]) > 1) ++first[2];
  for (int g = 2; g > 0; --g)   // a group that would not fill the SMs joins the wider one
    if (first[g + 1] - first[g] < c->sms) first[g] = first[g + 1];
  // the first non-empty group stays on the stream, the others fork from it
  if ((rc = c->cuda(cudaEventRecord(c->fork_ev, s), "fork"))) return rc;
  Ctx::Fork fork{*c};
  int used = 0, b = -1;
  for (int g = 0; g < 3; ++g) {
    const int count = first[g + 1] - first[g];
    if (count == 0) continue;
    cudaStream_t bs = s;
    if (b >= 0) {
      bs = c->branch[(size_t)b];
      if ((rc = c->cuda(cudaStreamWaitEvent(bs, c->fork_ev, 0), "fork"))) return rc;
    }
    if ((rc = c->cuda(launch_pipe(a, first[g], count, std::min(bands(first[g]), pipe::kWarps), lx, bs),
                      "traceback launch")))
      return rc;
    if (b >= 0 && (rc = c->cuda(cudaEventRecord(c->join_ev[(size_t)b], bs), "join"))) return rc;
    if (used++) ++c->launches;   // the caller counts the first
    ++b;
  }
  if (b > 0 && (rc = c->injected_fork_error())) return rc;
  for (int k = 0; k < b; ++k)
    if ((rc = c->cuda(cudaStreamWaitEvent(s, c->join_ev[(size_t)k], 0), "join"))) return rc;
  fork.joined = true;
  return NWG_OK;
}

void Ctx::extra_release() {
  delete reinterpret_cast<TraceState*>(trace_state);
  trace_state = nullptr;
  nj_release();
  ingest_release();
  msa_release();
}

int Ctx::align_pairs(const int8_t* codes, const int64_t* offsets, int n, const int32_t* px, const int32_t* py,
                     int npairs, char* outx, char* outy, int64_t stride, int32_t* outlen, int32_t* score,
                     nwg_stats* st) {
  if (!codes || !offsets || n < 1 || npairs < 0 || (npairs > 0 && (!px || !py || !outx || !outy || !outlen)))
    return fail(NWG_ERR_INVALID, "align_pairs arguments");
  int maxlen = 0;
  for (int s = 0; s < n; ++s) {
    const int64_t L = offsets[s + 1] - offsets[s];
    if (L <= 0) return fail(NWG_ERR_EMPTY_SEQ, "zero-length sequence");
    maxlen = std::max<int>(maxlen, (int)L);
  }
  for (int k = 0; k < npairs; ++k) {
    if (px[k] < 0 || px[k] >= n || py[k] < 0 || py[k] >= n) return fail(NWG_ERR_INVALID, "pair index");
    if (stride < offsets[px[k] + 1] - offsets[px[k]] + offsets[py[k] + 1] - offsets[py[k]] + 1)
      return fail(NWG_ERR_INVALID, "output stride shorter than Lx + Ly + 1");
  }
  if (npairs == 0) return NWG_OK;
  const int64_t total = offsets[n];
  if (!residues_ok(codes, total)) return fail(NWG_ERR_BAD_RESIDUE, "residue code outside 0..23");
  if (!trace_state) trace_state = new TraceState();
  TraceState& T = *reinterpret_cast<TraceState*>(trace_state);
  std::vector<int32_t> len(n);
  for (int s = 0; s < n; ++s) len[s] = (int32_t)(offsets[s + 1] - offsets[s]);
  int rc;
  if ((rc = T.codes.ensure((size_t)total)) || (rc = T.start.ensure(sizeof(int64_t) * n)) ||
      (rc = T.len.ensure(sizeof(int32_t) * n)))
    return fail(rc, "traceback allocation");
  cudaStream_t s = stream;
  if ((rc = cuda(cudaMemcpyAsync(T.codes.p, codes, (size_t)total, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemcpyAsync(T.start.p, offsets, sizeof(int64_t) * n, cudaMemcpyHostToDevice, s), "upload")) ||
      (rc = cuda(cudaMemcpyAsync(T.len.p, len.data(), sizeof(int32_t) * n, cudaMemcpyHostToDevice, s), "upload")))
    return rc;
  // batches bounded by the nibble memory (~1 GiB of words per batch)
  const int64_t kBudgetWords = (int64_t)1 << 28;
  // statistics: kernel_ms = the match kernels alone, d2h_ms = the downloads
  cudaEvent_t ev_copied = nullptr;
  if (st && (rc = cuda(cudaEventCreate(&ev_copied), "traceback event"))) return rc;
  struct EventGuard {
    cudaEvent_t e;
    ~EventGuard() {
      if (e) cudaEventDestroy(e);
    }
  } guard{ev_copied};
  double mean_rows = 0.0;
  for (int k = 0; k < npairs; ++k) mean_rows += len[py[k]];
  mean_rows /= npairs;
  const int W = trace_lanes_forced ? trace_lanes_forced : trace_lanes(mean_rows);
  // the pipeline form, except for many short pairs (4,000 of 60 residues: 0.111
  // against 0.092 ms with two pairs a warp; 2,000: 0.054 against 0.067)
  const bool piped = !trace_lanes_forced && pipe_ok(*this, maxlen) &&
                     !(mean_rows <= kShortRows && npairs > 4 * pipe::kWarps * sms);
  const int band = piped ? 128 : 8 * W;
  int k0 = 0;
  while (k0 < npairs) {
    std::vector<int64_t> off;
    int64_t words = 0;
    int k1 = k0;
    while (k1 < npairs) {
      const int Lx = len[px[k1]], Ly = len[py[k1]];
      const int64_t w = piped ? (int64_t)((Ly + band - 1) / band) * pipe::supersteps_of(Lx) * 128
                              : (int64_t)((Ly + band - 1) / band) * (Lx + W - 1) * W;
      if (k1 > k0 && words + w > kBudgetWords) break;
      off.push_back(words);
      words += w;
      ++k1;
    }
    const int m = k1 - k0;
    // pairs of similar band counts and X lengths share a warp
    std::vector<int32_t> order((size_t)m);
    for (int k = 0; k < m; ++k) order[(size_t)k] = k;
    std::stable_sort(order.begin(), order.end(), [&](int u, int v) {
      const int bu = (len[py[k0 + u]] + band - 1) / band, bv = (len[py[k0 + v]] + band - 1) / band;
      if (bu != bv) return bu > bv;
      return len[px[k0 + u]] > len[px[k0 + v]];
    });
    if ((rc = T.px.ensure(sizeof(int32_t) * m)) || (rc = T.py.ensure(sizeof(int32_t) * m)) ||
        (rc = T.order.ensure(sizeof(int32_t) * m)) ||
        (rc = T.off.ensure(sizeof(int64_t) * m)) || (rc = T.nib.ensure(sizeof(uint32_t) * (size_t)words)) ||
        (rc = T.scratch.ensure(sizeof(int32_t) * 4 * (size_t)m * maxlen)) ||
        (rc = T.score.ensure(sizeof(int32_t) * m)) || (rc = T.outx.ensure((size_t)m * stride)) ||
        (rc = T.outy.ensure((size_t)m * stride)) || (rc = T.outlen.ensure(sizeof(int32_t) * m)) ||
        (rc = T.done.ensure(sizeof(int32_t) * ((size_t)m + 1))))
      return fail(rc, "traceback allocation");
    if ((rc = cuda(cudaMemcpyAsync(T.px.p, px + k0, sizeof(int32_t) * m, cudaMemcpyHostToDevice, s), "upload")) ||
        (rc = cuda(cudaMemcpyAsync(T.py.p, py + k0, sizeof(int32_t) * m, cudaMemcpyHostToDevice, s), "upload")) ||
        (rc = cuda(cudaMemcpyAsync(T.off.p, off.data(), sizeof(int64_t) * m, cudaMemcpyHostToDevice, s), "upload")) ||
        (rc = cuda(cudaMemcpyAsync(T.order.p, order.data(), sizeof(int32_t) * m, cudaMemcpyHostToDevice, s),
                   "upload")))
      return rc;
    TraceArgs a{};
    a.codes = (const int8_t*)T.codes.p;
    a.start = (const int64_t*)T.start.p;
    a.len = (const int32_t*)T.len.p;
    a.px = (const int32_t*)T.px.p;
    a.py = (const int32_t*)T.py.p;
    a.order = (const int32_t*)T.order.p;
    a.nib_off = (const int64_t*)T.off.p;
    a.nib = (uint32_t*)T.nib.p;
    a.scratch = (int32_t*)T.scratch.p;
    a.score = (int32_t*)T.score.p;
    a.outx = (char*)T.outx.p;
    a.outy = (char*)T.outy.p;
    a.outlen = (int32_t*)T.outlen.p;
    a.stride = stride;
    a.npairs = m;
    a.scratch_cols = maxlen;
    a.go = go;
    a.ge = ge;
    a.sub = (const int8_t*)b_sub.p;
    a.done = (unsigned*)T.done.p;
    a.err = (int*)T.done.p + m;
    if (piped && ((rc = cuda(cudaMemsetAsync(T.done.p, 0, sizeof(int32_t) * ((size_t)m + 1), s), "traceback")) ||
                  (rc = cuda(cudaMemsetAsync(T.score.p, 0, sizeof(int32_t) * m, s), "traceback"))))
      return rc;
    if (st) cudaEventRecord(ev0, s);
    ++launches;
    if (piped) {
      if ((rc = launch_pipes(this, a, order, len, px + k0, py + k0, s))) return rc;
    } else if ((rc = cuda(launch_match(W, a, s), "traceback launch"))) {
      return rc;
    }
    if (st) cudaEventRecord(ev1, s);
    if ((rc = cuda(cudaMemcpyAsync(outx + (size_t)k0 * stride, T.outx.p, (size_t)m * stride, cudaMemcpyDeviceToHost, s),
                   "download")) ||
        (rc = cuda(cudaMemcpyAsync(outy + (size_t)k0 * stride, T.outy.p, (size_t)m * stride, cudaMemcpyDeviceToHost, s),
                   "download")) ||
        (rc = cuda(cudaMemcpyAsync(outlen + k0, T.outlen.p, sizeof(int32_t) * m, cudaMemcpyDeviceToHost, s),
                   "download")))
      return rc;
    if (score &&
        (rc = cuda(cudaMemcpyAsync(score + k0, T.score.p, sizeof(int32_t) * m, cudaMemcpyDeviceToHost, s), "download")))
      return rc;
    int err = 0;
    if (piped && (rc = cuda(cudaMemcpyAsync(&err, a.err, sizeof(err), cudaMemcpyDeviceToHost, s), "download"))) return rc;
    if (st) cudaEventRecord(ev_copied, s);
    if ((rc = cuda(cudaStreamSynchronize(s), "traceback sync"))) return rc;
    if (err) return fail(NWG_ERR_TIMEOUT, "traceback: a bounded device wait ran out");
    if (st) {
      for (int k = k0; k < k1; ++k) st->cells += (int64_t)len[px[k]] * len[py[k]];
      float ms = 0.f, ms2 = 0.f;
      cudaEventElapsedTime(&ms, ev0, ev1);
      cudaEventElapsedTime(&ms2, ev1, ev_copied);
      st->kernel_ms += ms;
      st->d2h_ms += ms2;
    }
    k0 = k1;
  }
  if (st) {
    st->pairs = npairs;
    st->pairs_int32 = npairs;
  }
  return NWG_OK;
}

}  // namespace nwg

namespace {

// Post-order walk of TreeNode::getNodes (TreeNode.cpp:91-117) over the join
// records: left subtree, right subtree, then the node; a node whose two
// children are leaves is a cherry (AlignmentMatch.cu:167-186, vecSize == 2).
int cherries(const int32_t* left, const int32_t* right, int nleaves, int32_t* node, int32_t* l, int32_t* r) {
  if (nleaves < 2) return 0;
  const int nn = 2 * nleaves - 1;
  std::vector<int> stack;
  std::vector<char> expanded((size_t)nn, 0);
  stack.push_back(nn - 1);
  int cnt = 0;
  while (!stack.empty()) {
    const int v = stack.back();
    if (v < nleaves) {
      stack.pop_back();
      continue;
    }
    const int k = v - nleaves;
    if (!expanded[(size_t)v]) {
      expanded[(size_t)v] = 1;
      stack.push_back(right[k]);
      stack.push_back(left[k]);
      continue;
    }
    stack.pop_back();
    if (left[k] < nleaves && right[k] < nleaves) {
      if (node) {
        node[cnt] = v;
        l[cnt] = left[k];
        r[cnt] = right[k];
      }
      ++cnt;
    }
  }
  return cnt;
}

}  // namespace

extern "C" int nwg_cherries(const int32_t* left, const int32_t* right, int nleaves, int32_t* node, int32_t* l,
                            int32_t* r) {
  if (!left || !right || nleaves < 0) return -NWG_ERR_INVALID;
  for (int k = 0; k + 1 < nleaves; ++k) {
    if (left[k] < 0 || right[k] < 0 || left[k] >= nleaves + k || right[k] >= nleaves + k) return -NWG_ERR_INVALID;
  }
  return cherries(left, right, nleaves, node, l, r);
}

extern "C" int nwg_set_trace_lanes(nwg_ctx* ctx, int lanes) {
  if (!ctx || !(lanes == 0 || lanes == 8 || lanes == 16 || lanes == 32)) return NWG_ERR_INVALID;
  reinterpret_cast<nwg::Ctx*>(ctx)->trace_lanes_forced = lanes;
  return NWG_OK;
}

extern "C" int nwg_align_pairs(nwg_ctx* ctx, const int8_t* codes, const int64_t* offsets, int n, const int32_t* px,
                               const int32_t* py, int npairs, char* outx, char* outy, int64_t stride, int32_t* len,
                               int32_t* score, nwg_stats* stats) {
  if (!ctx) return NWG_ERR_INVALID;
  nwg::Ctx* c = reinterpret_cast<nwg::Ctx*>(ctx);
  if (stats) std::memset(stats, 0, sizeof(*stats));
  c->launches = 0;
  const int rc = c->align_pairs(codes, offsets, n, px, py, npairs, outx, outy, stride, len, score, stats);
  if (stats) stats->launches = c->launches;
  return rc;
}
