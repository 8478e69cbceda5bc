// pipe.cuh -- one alignment with flags as a pipeline of warps over the SMs of
// a thread-block cluster.
//
// Two changes of variables.  H'(r,c) = H(r,c) + GE (r + c + 2) makes extension
// free: with S' = S + 2 GE and GD = GO - GE, F' = max(F'up, H'up - GD), E'
// likewise, and both boundaries are 0.  And every value is held relative to a
// neighbouring cell: with u(r,c) = H'(r,c) - H'(r-1,c), v(r,c) = H'(r,c) -
// H'(r,c-1), and F, E, H of a cell counted from H'(r-1,c-1),
//   m = max(E, S'),  H = max(F, m),  u = H - v(r-1,c),  v = H - u(r,c-1),
//   F(r+1,c) = max(F, m - GD) - u(r,c-1),   E(r,c+1) = max(E, H - GD) - v(r-1,c)
// -- the same comparisons as on the values themselves, so the same flags: 17
// integer operations a cell, two of them on the way from a row's F to the next
// row's (the F line uses GD >= 0: F - GD never beats F).  Difference recurrences
// for affine gaps are published (Suzuki and Kasahara, BMC Bioinformatics 19:45,
// 2018).  With GO >= GE, u and v lie in [-GD, max S' + GD] (H >= F >= Hup - GD; a
// diagonal step gives u = S' - v(r-1,c), an F step u <= 0, an E step no more than
// the cell where its gap opened), and everything else within 2 max|S| + 4 GO.
//
// A band is 32 R rows, R per lane of a warp, lane l one column behind lane
// l - 1.  Consecutive bands run on consecutive warps, four to a CTA (one per
// scheduler: the step is bound by the integer pipe of its scheduler) and up to
// eight CTAs to a cluster.  A band's bottom row goes to the next warp, eight
// columns at a time, by asynchronous stores that count bytes on a barrier in
// the receiving CTA's shared memory (a ring of eight stages, each given back by
// a remote arrive), so no barrier couples the warps.  Past 32
// bands the first warp takes the next one; its row above is in global memory.
//
// Flags: four raw bits a cell, sign bits of differences appended by funnel
// shifts to a word per kind, so that the shifts of a row do not wait for one
// another: H != S, F < E, no continue up, no continue left.  Eight columns of a
// lane's R rows make R words (bit (kind * 8 + step) * R + row, from the top),
// band-major, superstep (eight steps) by superstep.
//
// The step is bound by its instructions at one warp per scheduler (185 cycles
// for four rows, 2 cycles an instruction), not by memory.  Measured on the way,
// cycles a step: a release arrive per stage 440, flags in one word 310, values
// with GE in every difference 250, scores loaded one superstep ahead 193.
#pragma once

#include <cstddef>
#include <type_traits>

#include "nwg_internal.h"
#include "walk.cuh"

namespace nwg {
namespace pipe {

constexpr int kStep = 8;          // columns per superstep and per ring stage
constexpr int kStages = 8;        // ring stages per warp
constexpr int kWarps = 4;         // warps per CTA, at most
constexpr int kCluster = 8;       // CTAs per cluster, at most
constexpr long long kWaitCycles = 4000000000ll;   // about two seconds: no wait takes a millisecond

// Supersteps of a band over lx columns: the last lane is 31 columns behind.
__host__ __device__ __forceinline__ int stages_of(int lx) { return (lx + kStep - 1) / kStep; }
__host__ __device__ __forceinline__ int supersteps_of(int lx) { return stages_of(lx) + 32 / kStep; }

// Shared memory of one warp as a receiver of the row above its band.
struct alignas(16) Inbox {
  int2 ring[kStages * kStep];
  unsigned long long full[kStages];    // bytes of the stage have arrived
  unsigned long long empty[kStages];   // this warp's receiver has read the stage it sent
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned cluster_addr(unsigned a, int rank) {
  unsigned r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}

__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

__device__ __forceinline__ void bar_init(unsigned long long* b) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(b)) : "memory");
}

__device__ __forceinline__ void bar_expect(unsigned long long* b, int bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void bar_arrive_remote(unsigned addr) {
  asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}

__device__ __forceinline__ bool bar_try(unsigned long long* b, int parity) {
  unsigned ok;
  asm volatile(
      "{\n.reg .pred p;\n"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      "selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_addr(b)), "r"(parity)
      : "memory");
  return ok != 0;
}

__device__ __forceinline__ void store_async(unsigned addr, int x, int y, int z, int w, unsigned bar) {
  asm volatile(
      "st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(addr),
      "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar)
      : "memory");
}

// Copy of a contiguous block to this CTA's shared memory, counted on a barrier.
__device__ __forceinline__ void copy_bulk(void* dst, const void* src, int bytes, unsigned long long* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(bar))
               : "memory");
}

// The warp's place in the pipeline and its ends.
struct Link {
  Inbox* in;              // this warp's
  unsigned out;           // the next warp's inbox (cluster address)
  unsigned back;          // the previous warp's inbox (cluster address)
  int* err;               // set when a wait runs out
  unsigned sent = 0;      // stages sent / received so far
  unsigned taken = 0;
  bool dead = false;      // a wait ran out: no more waits, no more sends

  __device__ __forceinline__ void wait(unsigned long long* b, int parity) {
    if (dead || bar_try(b, parity)) return;
    const long long t0 = clock64();
    while (!bar_try(b, parity))
      if (clock64() - t0 > kWaitCycles) {
        dead = true;
        atomicExch(err, 1);
        return;
      }
  }
};

// Barriers of the CTA's inboxes; every thread of the cluster calls it.
__device__ __forceinline__ void init_inboxes(Inbox* box, int nwarp) {
  if (threadIdx.x == 0) {
    for (int w = 0; w < nwarp; ++w)
      for (int s = 0; s < kStages; ++s) {
        bar_init(&box[w].full[s]);
        bar_init(&box[w].empty[s]);
      }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int w = 0; w < nwarp; ++w)
      for (int s = 0; s < kStages; ++s) bar_expect(&box[w].full[s], kStep * (int)sizeof(int2));
  }
  cluster_barrier();
}

// The row that the last warp leaves in global memory for the first one.
struct Wrap {
  int2* row;              // lx entries
  unsigned* done;         // columns written so far, over all passes (starts at 0)
};

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// One lane's rows.
template <int R>
struct Rows {
  int n[R];             // -u(r, c-1)
  int e[R];             // E(r, c)
  int cl[R];            // negative: no continue-left flag at (r, c)
};

// All bands of one warp.  Score: load(g) before a band; begin(j, ln) and end(j)
// around a superstep; get(i, t, s) the R scores at its step i, the warp's step
// t; column_done(t, n) after a step.
// flags: the alignment's flag words; GD: open - extension; gw of nwarp: this warp.
template <int R, class Score>
__device__ void run_bands(Link& ln, const Wrap& wrap, Score& score, uint32_t* __restrict__ flags, int lx, int ly,
                          int GD, int gw, int nwarp) {
  static_assert(R == 4, "a superstep's bits of one kind are one word");
  const int lane = threadIdx.x & 31;
  const int nb = (ly + 32 * R - 1) / (32 * R);
  const int nst = stages_of(lx), nsup = supersteps_of(lx);
  for (int g = gw, pass = 0; g < nb; g += nwarp, ++pass) {
    const bool from_wrap = gw == 0 && g > 0;
    const bool from_prev = gw > 0;
    const bool to_next = gw + 1 < nwarp && g + 1 < nb;
    const bool to_wrap = gw + 1 == nwarp && g + 1 < nb;
    Rows<R> st;
    int pk = 0, fb = 0;        // the bottom row's 2 v + (no continue-up flag below), F of the row below
    auto reset = [&]() {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        st.n[r] = 0;
        st.e[r] = -GD;           // E(r, 0): a gap opened at column -1
        st.cl[r] = -1;
      }
    };
    reset();
    score.load(g);
    // a stage holds the columns of one superstep of the warp above, from its
    // fourth on: 8 q - 7 .. 8 q, so a superstep here takes the last entry of
    // one stage and the first seven of the next
    int2 carry = make_int2(1, -GD);   // row -1: v = 0, no continue flag, a gap opened there
    auto receive = [&](int2 (&in)[kStep]) {
      const unsigned s = ln.taken % kStages;
      ln.wait(&ln.in->full[s], (ln.taken / kStages) & 1);
      in[0] = carry;
#pragma unroll
      for (int i = 0; i + 1 < kStep; ++i) in[i + 1] = ln.in->ring[s * kStep + i];
      carry = ln.in->ring[s * kStep + kStep - 1];
    };
    auto give_back = [&]() {   // every lane has used the stage: arm it again and give it back
      const unsigned s = ln.taken % kStages;
      __syncwarp();
      if (lane == 0) {
        bar_expect(&ln.in->full[s], kStep * (int)sizeof(int2));
        bar_arrive_remote(ln.back + (unsigned)offsetof(Inbox, empty) + 8u * s);
      }
      ++ln.taken;
    };
    if (from_prev) {
      int2 none[kStep];
      receive(none);
      give_back();
    }
    auto superstep = [&](int j, auto ramp) {
      int2 in[kStep];
#pragma unroll
      for (int i = 0; i < kStep; ++i) in[i] = make_int2(1, -GD);
      const bool got = from_prev && j < nst;
      if (got) {
        receive(in);
      } else if (from_wrap && j < nst) {
        const unsigned need = (unsigned)(pass - 1) * (unsigned)(nst * kStep) + (unsigned)((j + 1) * kStep);
        const long long t0 = clock64();
        while (!ln.dead && (int)(ld_acquire(wrap.done) - need) < 0)
          if (clock64() - t0 > kWaitCycles) {
            ln.dead = true;
            atomicExch(ln.err, 1);
          }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < kStep; ++i)
          if (j * kStep + i < lx) in[i] = __ldcg(wrap.row + j * kStep + i);
      }
      score.begin(j, ln);
      uint32_t acc[4] = {};   // a word per kind
      int op[kStep], of[kStep];
#pragma unroll
      for (int i = 0; i < kStep; ++i) {
        const int t = j * kStep + i;
        int p = __shfl_up_sync(0xffffffffu, pk, 1);
        int F = __shfl_up_sync(0xffffffffu, fb, 1);
        p = lane == 0 ? in[i].x : p;
        F = lane == 0 ? in[i].y : F;
        if (decltype(ramp)::value && t == lane) reset();   // the lane's column 0: what came before was no cell
        int vU = p >> 1;
        int ncu = p << 31;
        int s[R];
        score.get(i, t, s);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int E = st.e[r], n = st.n[r];
          const int m = max(E, s[r]);
          const int h = max(F, m);
          const int hg = h - GD;
          // sign bits: H != S', F < E, no continue up, no continue left
          acc[0] = __funnelshift_l((uint32_t)(s[r] - h), acc[0], 1);
          acc[1] = __funnelshift_l((uint32_t)(F - E), acc[1], 1);
          acc[2] = __funnelshift_l((uint32_t)ncu, acc[2], 1);
          acc[3] = __funnelshift_l((uint32_t)st.cl[r], acc[3], 1);
          ncu = F - hg;                                     // the row below
          st.cl[r] = E - hg;                                // the next column
          st.e[r] = max(E, hg) - vU;
          st.n[r] = vU - h;
          F = __viaddmax_s32(m, -GD, F) + n;
          vU = h + n;
        }
        op[i] = pk = (int)__funnelshift_l((uint32_t)ncu, (uint32_t)vU, 1);
        of[i] = fb = F;
        score.column_done(t, st.n);
      }
      uint32_t* fw = flags + (((int64_t)g * nsup + j) * 32 + lane) * R;
      *reinterpret_cast<uint4*>(fw) = make_uint4(acc[0], acc[1], acc[2], acc[3]);
      score.end(j);
      if (got) give_back();
      if (to_next && j >= 3) {
        const unsigned k = ln.sent + (unsigned)(j - 3), q = k % kStages;
        // room for this stage and the next three (stages are given back in order)
        if (k % 4 == 0 && k + 3 >= kStages) ln.wait(&ln.in->empty[(k + 3) % kStages], ((k + 3) / kStages - 1) & 1);
        if (lane == 31 && !ln.dead) {
#pragma unroll
          for (int i = 0; i < kStep; i += 2)
            store_async(ln.out + 8u * (q * kStep + i), op[i], of[i], op[i + 1], of[i + 1],
                        ln.out + (unsigned)offsetof(Inbox, full) + 8u * q);
        }
      } else if (to_wrap) {
        const int c0 = j * kStep - 31;
        if (lane == 31) {
#pragma unroll
          for (int i = 0; i < kStep; ++i)
            if (c0 + i >= 0 && c0 + i < lx) wrap.row[c0 + i] = make_int2(op[i], of[i]);
          // tell the first warp, every 32 columns
          if (j % 4 == 3 || j + 1 == nsup)
            st_release(wrap.done, (unsigned)pass * (unsigned)(nst * kStep) + (unsigned)min(max(c0 + kStep, 0), nst * kStep));
        }
      }
    };
    for (int j = 0; j < 32 / kStep; ++j) superstep(j, std::true_type{});
    for (int j = 32 / kStep; j < nsup; ++j) superstep(j, std::false_type{});
    if (to_next) ln.sent += (unsigned)nst + 1;
    score.band_done();
  }
}

// The walk's window over an alignment's flags: kBytes of supersteps of one band.
template <int R, int kBytes>
struct Window {
  static constexpr int kSup = kBytes / (128 * R);   // supersteps held
  static_assert(kSup >= 4, "window");
  const uint32_t* flags;
  uint32_t* win;          // shared, kBytes
  int nsup;
  int g = -1, j0 = 0;     // band, first superstep held
  static __device__ __forceinline__ int superstep(int x, int y) { return (x + (y % (32 * R)) / R) / kStep; }
  __device__ __forceinline__ bool covers(int x, int y) const {
    const int j = superstep(x, y) - j0;
    return y / (32 * R) == g && j >= 0 && j < kSup;
  }
  __device__ __forceinline__ unsigned cell(int x, int y) const {
    const int l = (y % (32 * R)) / R, t = x + l;
    const uint32_t* w = win + ((t / kStep - j0) * 32 + l) * R;
    auto bit = [&](int kind) {
      const int k = (kind * kStep + t % kStep) * R + y % R;
      return (w[k >> 5] >> (31 - (k & 31))) & 1u;
    };
    // U: H == F or H == S; L: H == S or else H == E
    const unsigned ns = bit(0), nf = bit(1);
    return ((ns ^ 1u) | nf) << 3 | ((ns & nf) ^ 1u) << 2 | (bit(2) ^ 1u) << 1 | (bit(3) ^ 1u);
  }
  __device__ __forceinline__ void load(int x, int y) {
    const int lane = threadIdx.x & 31;
    g = y / (32 * R);
    j0 = superstep(x, y) - (kSup - 1);
    __syncwarp();
    const uint4* src = reinterpret_cast<const uint4*>(flags + ((int64_t)g * nsup + j0) * 32 * R);
    uint4* dst = reinterpret_cast<uint4*>(win);
    constexpr int kPer = 8 * R;             // 16-byte units per superstep
#pragma unroll
    for (int k = 0; k < kSup * kPer / 32; k += 8) {
      uint4 v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int e = (k + q) * 32 + lane;
        if (k + q < kSup * kPer / 32 && j0 + e / kPer >= 0) v[q] = __ldcg(src + e);
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int e = (k + q) * 32 + lane;
        if (k + q < kSup * kPer / 32 && j0 + e / kPer >= 0) dst[e] = v[q];
      }
    }
    __syncwarp();
  }
};

}  // namespace pipe
}  // namespace nwg
