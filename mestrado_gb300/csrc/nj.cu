// nj.cu -- neighbor joining on the device: the join loop of
// SpeciesBlock::buildTree (SpeciesBlock.cpp:845-1343) with modifyMatrix
// (:710-842), buildGblRowSums (:426-453) and TreeNode::join (TreeNode.cpp:
// 31-58), for one process and one GPU.
//
// Semantics kept from the reference:
//  * D is float, row/column slots; the new node takes the slot of the smaller
//    id and keeps its stale diagonal (:787-841, :952, :1186);
//  * T is double: T[k] += (float)(tmp - (Dik + Djk)) with tmp the float
//    ((Dik + Djk) - d) / 2 (:793-801); the new node's T is the sequential
//    double sum of its tmp values in ascending id order (:799, :818); rebuilds
//    recompute every T as a sequential double sum of its row over active
//    nodes in ascending id order, diagonal included (:432-452);
//  * rebuilds after max(n0*0.5, 200) joins, then every n*0.5, never below
//    200 active nodes (:864, :1226-1247);
//  * the pair chosen is the minimum of q = ((double)d*(n-2) - T[a]) - T[b]
//    with (a, b) the order of the reference's Dij record (node-id order for
//    records made by buildBins, :549-558; row-slot order for records made when
//    a node is inserted, :1280-1292), ties to the larger max(i,j) then the
//    larger min(i,j) (:1165-1179).
// The reference reaches that minimum through bins and heaps (:456-674,
// :1019-1144), which only prune -- except that a pair popped from a heap is
// valued as d*(n-2) - (T[a] + T[b]) (:1119-1121) and more than QDA=8 equal
// values are cut by nth_element (:1148).  Each step therefore also checks
// whether any other pair comes within the two roundings of the winner, or
// more than four pairs tie exactly; such a step is counted as ambiguous (its
// pick is still the exact-argmin one).  The heap-size rebuild trigger
// (:1206-1223) cannot fire while the heaps hold at most the entries pushed
// since the last build; that bound is tracked and any check it cannot exclude
// is counted.
//
// Search per join: q in float, fl(fl(fl(d*(n-2)) - Tf_r) - Tf_c) with Tf the
// float copy of T, is within E = 8 * 2^-24 * M of the exact q, M the largest
// |d|(n-2) + |T_r| + |T_c|.  The candidates are the pairs whose float q is at most
// the smallest + 3E; each gets its exact double q in both roundings.  One CTA
// looks at every pair for every join; a team of CTAs keeps a lower bound per row
// and looks only at the rows whose bound reaches the best known pair (the section
// on the lazy search).
// The winner follows the tie-break; the ambiguity check runs over the
// candidates: any pair left out has q > winner + E, beyond reach of either
// rounding.  All floating-point operations use the _rn intrinsics in the
// reference's evaluation order (no contraction).
//
// Three launch forms run a job's whole join loop (several jobs per launch in
// the serving loop):
//  * one CTA with the job in its shared memory (up to 136 taxa);
//  * one thread-block cluster, the matrix in L2 (up to 600 taxa, and every larger
//    job of the serving loop);
//  * the whole GPU, one cooperative launch per segment between compactions (to
//    the live slots, in slot order), above that.
#include <algorithm>
#include <cfloat>
#include <climits>
#include <cstdlib>
#include <cstring>
#include <vector>

#include <cooperative_groups.h>
#include <math_constants.h>

#include "nwg_ctx.h"

namespace nwg {

namespace {

constexpr int kNJMaxN = 8192;
constexpr float kFloatTop = 1.329228e36f;   // 2^120: the float search holds q and T up to here
constexpr int kNoPair = 0x7F7FFFFF;    // ford(FLT_MAX): a row without a pair
constexpr int kCandCap = 2048;         // candidate list capacity per join (longer lists are not read)

struct NJDev {
  float* D;            // n0 x ld, slots
  double* T;           // per slot
  float* Tf;           // per slot, (float)T; NaN at dead and padding slots (ld entries)
  int* slot;           // per node id (2n0-1), -1 dead
  int* node;           // per slot: node id, -1 dead
  int* act;            // active node ids ascending [n0 + 1]
  int* na;             // active count
  int* g32;            // [2][4]: ties, ambiguous pairs and candidates of the fallback scan
  unsigned long long* stats;  // [0] ambiguous steps, [1] tie steps, [2] internal errors,
                              // [3] open heap-size checks, [4] rebuilds (cluster form)
  nwg_join* joins;
  int* prow;           // slot -> its row's place in D (n0: xrow); [n0] the free place
  float* xrow;         // one more row (ld floats)
  double* tx;          // [2 * n0]: every slot's T for the exchanges of even and of odd number
  int n0;              // slots
  int ld;              // row stride of D (floats), a multiple of 4
  int cand_cap;        // candidate list capacity
  int pad;
};

// Row at place q of the matrix.
__device__ __forceinline__ float* row_at(const NJDev& s, int q) {
  return q < s.n0 ? s.D + (size_t)q * s.ld : s.xrow;
}

__device__ __forceinline__ int ford(float f) {
  // order-preserving map float -> int (for atomicMin / atomicMax)
  const int b = __float_as_int(f);
  return b >= 0 ? b : b ^ 0x7FFFFFFF;
}


// Exponent of the lowest set bit of a nonzero float (INT_MAX for zero).
__device__ __forceinline__ int low_bit_exp(float f) {
  const unsigned b = __float_as_uint(f) & 0x7FFFFFFFu;
  if (b == 0) return INT_MAX;
  const unsigned e = b >> 23, m = b & 0x7FFFFFu;
  if (e == 0) return -149 + __ffs(m) - 1;
  return (int)e - 150 + __ffs(m | 0x800000u) - 1;
}

// Exponent of the highest set bit of |f| (f = m * 2^(e) with m in [1, 2)),
// INT_MIN for 0.
__device__ __forceinline__ int top_bit_exp(float f) {
  const unsigned b = __float_as_uint(f) & 0x7FFFFFFFu;
  if (b == 0) return INT_MIN;
  const unsigned e = b >> 23, m = b & 0x7FFFFFu;
  if (e == 0) return -149 + (31 - __clz(m));
  return (int)e - 127;
}

// f as a signed integer count of 2^lowexp (exact: lowexp is at most the
// lowest set bit of f, and |f| < 2^(lowexp + 49) is checked by the caller).
__device__ __forceinline__ long long float_units(float f, int lowexp) {
  const unsigned b = __float_as_uint(f);
  const unsigned e = (b >> 23) & 0xFFu, m = b & 0x7FFFFFu;
  if (e == 0 && m == 0) return 0;
  const long long mant = e == 0 ? (long long)m : (long long)(m | 0x800000u);
  const int sh = (e == 0 ? -149 : (int)e - 150) - lowexp;   // value = mant * 2^(sh + lowexp)
  // a right shift drops only zero bits: lowexp <= the lowest set bit of f
  const long long v = sh >= 0 ? mant << sh : mant >> (-sh);
  return (b >> 31) ? -v : v;
}

// A sequential double sum of floats equals any-order sum when every partial
// sum is exact: all terms are multiples of 2^lowexp and sum|x| < 2^(53+lowexp)
// (a multiple of 2^lowexp below that magnitude has at most 53 significant
// bits).  absum is itself a rounded sum, hence the 1e-12 slack.
__device__ __forceinline__ bool sum_is_exact(double absum, int lowexp) {
  if (lowexp == INT_MAX) return true;   // every term is zero
  return absum * (1.0 + 1e-12) < ldexp(1.0, 53 + lowexp);
}

// Sequential row sums (buildGblRowSums): one warp per active row; the lanes'
// any-order sum is used when it is provably exact, else lane 0 sums in order.
__global__ void rowsum_kernel(NJDev s, const int* abort) {
  if (*(volatile const int*)abort) return;   // a segment gave up: the lists were never written
  const int na = *s.na;
  const int lane = threadIdx.x & 31;
  const int k = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
  if (k >= na) return;
  const int sk = s.slot[s.act[k]];
  const float* row = row_at(s, s.prow[sk]);
  double part = 0.0, ab = 0.0;
  int lowexp = INT_MAX;
  for (int j = lane; j < na; j += 32) {
    const float x = row[s.slot[s.act[j]]];
    part = __dadd_rn(part, (double)x);
    ab = __dadd_rn(ab, (double)fabsf(x));
    lowexp = min(lowexp, low_bit_exp(x));
  }
  for (int o = 16; o > 0; o >>= 1) {
    part = __dadd_rn(part, __shfl_down_sync(0xffffffffu, part, o));
    ab = __dadd_rn(ab, __shfl_down_sync(0xffffffffu, ab, o));
    lowexp = min(lowexp, __shfl_down_sync(0xffffffffu, lowexp, o));
  }
  if (lane == 0) {
    double sum = part;
    if (!sum_is_exact(ab, lowexp)) {
      sum = 0.0;
      for (int j = 0; j < na; ++j) sum = __dadd_rn(sum, (double)row[s.slot[s.act[j]]]);
    }
    s.T[sk] = sum;
    s.Tf[sk] = (float)sum;
  }
}

// The pick's outcome: the winner's position among the candidates, the
// candidates within rounding of it (itself included) as ties or as pairs the
// reference's heap rounding could have preferred, and a failed pick.
struct PickOut {
  int idx;
  unsigned ties, amb;
  bool error;       // no candidate, or the list overflowed
};

// The pick's statistics: ambiguous step, tie step or internal error.
__device__ __forceinline__ void record_pick(const NJDev& s, const PickOut& r) {
  if (r.error) atomicAdd(&s.stats[2], 1ull);
  else if (r.amb > 0 || r.ties > 4) atomicAdd(&s.stats[0], 1ull);
  else if (r.ties > 1) atomicAdd(&s.stats[1], 1ull);
}

// ---- candidates, the grid barrier ------------------------------------------

struct GCand {
  long long k1, k2;   // order-preserving integer keys of q1 and q2
  double q1;          // record-order rounding of q (SpeciesBlock.cpp:1051)
  double ta, tb;      // T of the slots of a and b
  int a, b;           // node ids, a < b
  int sa, sb;         // their slots
  float d;
  int pad;
};

// An entry of the fallback scan's list: the keys and the nodes, each as its id
// above its slot (in the order of the ids; the winner's d and row sums are read
// again after the pick).
struct KCand {
  long long k1, k2;
  int a, b;
};
constexpr int kSlotBits = 13;
static_assert(kNJMaxN <= 1 << kSlotBits, "slots");
__device__ __forceinline__ int slot_of(int packed) { return packed & ((1 << kSlotBits) - 1); }
__device__ __forceinline__ KCand kc_of(const GCand& c) {
  return KCand{c.k1, c.k2, c.a << kSlotBits | c.sa, c.b << kSlotBits | c.sb};
}

struct GridNJ {
  unsigned* bar;        // [0] barrier arrivals, [1] publications (both count up from 0 per launch)
  int* abort;           // set when a wait gave up or a pick failed; every CTA and queued kernel then leaves
  float4* gather;       // [2 * CTAs]: the grid's exchanges
  KCand* cand;          // the candidate list of the fallback scan
  KCand* cbest;         // [CTAs]: per CTA its first candidate of the fallback scan
  int stall;            // failure injection: the first CTA never publishes
  int pad;
};

constexpr int kAbortWait = 1, kAbortPick = 2;
constexpr long long kBarrierSpinCycles = 4000000000ll;   // about two seconds: no phase takes a millisecond
constexpr int kFastRows = 32;                             // candidate rows the direct pick evaluates

__device__ __forceinline__ unsigned ld_acquire_u32(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void red_release_add(unsigned* p, unsigned v) {
  asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// Grid barrier of a cooperative launch (all CTAs resident): arrivals count up,
// the k-th barrier waits for k * gridDim.x arrivals.  A wait that exceeds the
// spin limit, or sees another CTA's abort, sets the abort flag and returns
// false; the caller then leaves the kernel.
__device__ bool grid_barrier(const GridNJ& g, unsigned& target) {
  __shared__ int s_ok;
  __syncthreads();
  target += gridDim.x;
  if (threadIdx.x == 0) {
    // release: this CTA's writes (ordered before by the CTA barrier) are
    // visible to every CTA that acquires the count
    red_release_add(&g.bar[0], 1u);
    int ok = 1;
    const long long t0 = clock64();
    while ((int)(ld_acquire_u32(&g.bar[0]) - target) < 0) {
      if (*(volatile int*)g.abort) {
        ok = 0;
        break;
      }
      if (clock64() - t0 > kBarrierSpinCycles) {
        atomicExch(g.abort, kAbortWait);
        ok = 0;
        break;
      }
    }
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// The CTAs that run one job's join loop: the whole cooperative grid (large n)
// or one thread-block cluster (a job per cluster).
struct Team {
  int rank, size;
};

template <bool CL>
__device__ __forceinline__ bool team_sync(const GridNJ& g, unsigned& target) {
  if constexpr (CL) {
    cooperative_groups::this_cluster().sync();
    return true;
  } else {
    return grid_barrier(g, target);
  }
}

// Order-preserving map double -> int64 (finite values; -0 and +0 map alike).
__device__ __forceinline__ long long dkey(double q) {
  long long b = __double_as_longlong(q);
  if ((b & 0x7FFFFFFFFFFFFFFFll) == 0) b = 0;
  return b >= 0 ? b : b ^ 0x7FFFFFFFFFFFFFFFll;
}

// Exact double of u * 2^e (|u| < 2^53, the result a normal double).
__device__ __forceinline__ double units_to_double(long long u, int e) {
  if (u == 0) return 0.0;
  const unsigned long long m = (unsigned long long)(u < 0 ? -u : u);
  const int msb = 63 - __clzll((long long)m);
  const unsigned long long bits = ((unsigned long long)(msb + e + 1023) << 52) |
                                  ((m << (52 - msb)) & 0xFFFFFFFFFFFFFull) | (u < 0 ? (1ull << 63) : 0ull);
  return __longlong_as_double(bits);
}

// One element of P: q, the row's two smallest (with the column of the
// smallest) and the magnitude |x| + |tc| (the row's |tr| is added per row).
// At a dead or padding slot tc is NaN: q and the magnitude are NaN and drop
// out (comparisons with NaN are false; fmaxf ignores NaN).
__device__ __forceinline__ void pass_elem(float d, float tc, int c, float tr, float nm2f, float& m1, float& m2,
                                          int& c1, float& mag) {
  const float x = __fmul_rn(d, nm2f);
  const float q = __fsub_rn(__fsub_rn(x, tr), tc);
  const bool lt = q < m1;
  m2 = lt ? m1 : fminf(m2, q);
  c1 = lt ? c : c1;
  m1 = lt ? q : m1;
  mag = fmaxf(mag, __fadd_rn(fabsf(x), fabsf(tc)));
}

// A candidate from its pair: slots r, c with their node ids, T and d.
__device__ __forceinline__ GCand make_cand(int r, int c, int ur, int uc, double Tr, double Tc, float d, double nm2,
                                           int watermark) {
  GCand cd;
  const bool rfirst = ur < uc;
  cd.a = rfirst ? ur : uc;
  cd.b = rfirst ? uc : ur;
  cd.sa = rfirst ? r : c;
  cd.sb = rfirst ? c : r;
  cd.ta = rfirst ? Tr : Tc;
  cd.tb = rfirst ? Tc : Tr;
  cd.d = d;
  cd.pad = 0;
  // record order (SpeciesBlock.cpp:1051): node-id order, except for a record
  // made when the newer node was inserted (row-slot order)
  const bool swap = cd.b >= watermark && cd.sb < cd.sa;
  const double nmd = __dmul_rn((double)d, nm2);
  cd.q1 = swap ? __dsub_rn(__dsub_rn(nmd, cd.tb), cd.ta) : __dsub_rn(__dsub_rn(nmd, cd.ta), cd.tb);
  cd.k1 = dkey(cd.q1);
  cd.k2 = dkey(__dsub_rn(nmd, __dadd_rn(cd.ta, cd.tb)));   // heap rounding (:1119-1121)
  return cd;
}

// Winner (smallest q1, then larger b, then larger a) and the ambiguity / tie
// counts over nc candidates, by one warp; load(k) gives candidate k.
template <class Load>
__device__ PickOut pick_keys(int nc, Load&& load) {   // load(k) has k1, k2, a, b
  const int l = threadIdx.x & 31;
  long long bk = LLONG_MAX, bk2 = LLONG_MAX;
  int ba = INT_MAX, bb = -1, bi = -1;
  for (int k = l; k < nc; k += 32) {
    const auto c = load(k);
    if (c.k1 < bk || (c.k1 == bk && (c.b > bb || (c.b == bb && c.a > ba)))) {
      bk = c.k1;
      bk2 = c.k2;
      ba = c.a;
      bb = c.b;
      bi = k;
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    const long long q = __shfl_xor_sync(0xffffffffu, bk, o);
    const long long q2 = __shfl_xor_sync(0xffffffffu, bk2, o);
    const int a2 = __shfl_xor_sync(0xffffffffu, ba, o);
    const int b2 = __shfl_xor_sync(0xffffffffu, bb, o);
    const int i2 = __shfl_xor_sync(0xffffffffu, bi, o);
    if (q < bk || (q == bk && (b2 > bb || (b2 == bb && a2 > ba)))) {
      bk = q;
      bk2 = q2;
      ba = a2;
      bb = b2;
      bi = i2;
    }
  }
  // every lane holds the winner; any other candidate whose smaller rounding
  // reaches the winner's larger one could have been picked by the reference
  const long long hiw = max(bk, bk2);
  const bool robust_w = bk == bk2;
  unsigned ties = 0, amb = 0;
  for (int k = l; k < nc; k += 32) {
    const auto c = load(k);
    if (min(c.k1, c.k2) > hiw) continue;
    if (c.a == ba && c.b == bb) ++ties;
    else if (robust_w && c.k1 == c.k2 && c.k1 == bk) ++ties;
    else ++amb;
  }
  for (int o = 16; o > 0; o >>= 1) {
    ties += __shfl_xor_sync(0xffffffffu, ties, o);
    amb += __shfl_xor_sync(0xffffffffu, amb, o);
  }
  PickOut r;
  r.idx = bi;
  r.ties = ties;
  r.amb = amb;
  r.error = bb < 0;
  return r;
}

// Long candidate lists (wide exact ties, e.g. hundreds of identical
// sequences, whose pairs all tie): above kListPickMax candidates one warp's
// pick over the list would be slow, and the list does not hold them.  Instead
// every CTA reduces its threads' first candidates in the pick's order, the
// winner is the first of those, and a second scan counts the ties and
// ambiguous pairs against it with pick_keys' rule.  (The one-CTA form always
// picks this way, without the list.)
constexpr int kListPickMax = kCandCap;

__device__ __forceinline__ KCand kc_none() { return KCand{LLONG_MAX, LLONG_MAX, INT_MAX, -1}; }

// x before y in the pick's order: smaller q1 key, then larger b, then larger a.
__device__ __forceinline__ bool kc_first(const KCand& x, const KCand& y) {
  return x.k1 < y.k1 || (x.k1 == y.k1 && (x.b > y.b || (x.b == y.b && x.a > y.a)));
}

__device__ __forceinline__ KCand ld_kcand(const KCand* p) {   // written by other CTAs: from L2
  return KCand{__ldcg(&p->k1), __ldcg(&p->k2), __ldcg(&p->a), __ldcg(&p->b)};
}

__device__ __forceinline__ KCand warp_first(KCand x) {
  for (int o = 16; o > 0; o >>= 1) {
    KCand y;
    y.k1 = __shfl_xor_sync(0xffffffffu, x.k1, o);
    y.k2 = __shfl_xor_sync(0xffffffffu, x.k2, o);
    y.a = __shfl_xor_sync(0xffffffffu, x.a, o);
    y.b = __shfl_xor_sync(0xffffffffu, x.b, o);
    if (kc_first(y, x)) x = y;
  }
  return x;
}

// The CTA's first candidate, valid in warp 0 (sw: 32 entries of shared memory,
// not reused before the next CTA barrier).
__device__ KCand cta_first(KCand x, KCand* sw) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = ((int)blockDim.x + 31) >> 5;
  x = warp_first(x);
  if (lane == 0) sw[warp] = x;
  __syncthreads();
  if (warp == 0) x = warp_first(lane < nw ? sw[lane] : kc_none());
  return x;
}

// pick_keys' tie and ambiguity rule for candidate c against the winner w.
__device__ __forceinline__ void count_vs(const KCand& c, const KCand& w, unsigned& ties, unsigned& amb) {
  if (min(c.k1, c.k2) > max(w.k1, w.k2)) return;
  if (c.a == w.a && c.b == w.b) ++ties;
  else if (w.k1 == w.k2 && c.k1 == c.k2 && c.k1 == w.k1) ++ties;
  else ++amb;
}

// A warp's candidates of one scan step into the list, one atomic per warp.
// *count ends at the number of candidates when that is at most
// kListPickMax, else above kListPickMax: a warp that saw the count pass it
// stops counting (full, the same in the warp).
__device__ __forceinline__ void list_push(const NJDev& s, const GridNJ& g, int* count, bool pred, const KCand& c, bool& full) {
  const unsigned bal = __ballot_sync(0xffffffffu, pred);
  if (bal == 0 || full) return;
  const int lane = threadIdx.x & 31;
  int base = 0;
  if (lane == 0) base = atomicAdd(count, __popc(bal));
  base = __shfl_sync(0xffffffffu, base, 0);
  const int idx = base + __popc(bal & ((1u << lane) - 1u));
  if (pred && idx < s.cand_cap) g.cand[idx] = c;
  full = base + __popc(bal) > kListPickMax;
}

// An exact sum of floats as u * 2^e (|u| < 2^62), with a = sum of |values| in
// the same units and t the highest exponent; e = INT_MAX for no values.  A
// sum whose values span 48 bits or more is not kept (the row's range then
// rules out the integer sum anyway; e and t stay exact).
struct USum {
  long long u, a;
  int e, t;
};

__device__ __forceinline__ void usum_add(USum& x, const USum& y) {
  if (y.e == INT_MAX) return;
  if (x.e == INT_MAX) {
    x = y;
    return;
  }
  const int e = min(x.e, y.e), t = max(x.t, y.t);
  if (t - e >= 48) {
    x.u = x.a = 0;
  } else {
    const long long mx = 1ll << (x.e - e), my = 1ll << (y.e - e);
    x.u = x.u * mx + y.u * my;
    x.a = x.a * mx + y.a * my;
  }
  x.e = e;
  x.t = t;
}

__device__ __forceinline__ void usum_warp(USum& x) {
  for (int o = 16; o > 0; o >>= 1) {
    USum y;
    y.u = __shfl_xor_sync(0xffffffffu, x.u, o);
    y.a = __shfl_xor_sync(0xffffffffu, x.a, o);
    y.e = __shfl_xor_sync(0xffffffffu, x.e, o);
    y.t = __shfl_xor_sync(0xffffffffu, x.t, o);
    usum_add(x, y);
  }
}

// ---- lazy search: one job per team of CTAs, one exchange per join --------------
// The team is the whole cooperative grid or one thread-block cluster.  Two
// things keep a join short.
//
// Replicated state.  Every CTA holds the slot -> node map and T of the whole job
// in its shared memory, T as the sum of two floats, and applies every join to
// its own copy: it reads the two joined rows, updates every T, and forms the new
// node's row sum itself (in integers).  The copies are the same in every CTA, so
// a join needs no exchange but the search's: one all-gather of each CTA's best
// pair.  The exact double T of row r is kept by the row's owner (CTA r modulo the
// team's size) and read from global memory where a pick needs it; only the owner
// writes row r of the matrix.  A new node's row goes to a free place (the one
// that the last join's row left), since the other CTAs may still be reading the
// joined rows.  (With the double T in every copy a join of 8,000 taxa spent 8 us
// in the FP64 pipe.)
//
// Lower bounds.  A join changes q(r,c) = d (n-2) - T_r - T_c by
// -(d(r,c) + dT_r + dT_c), so a lower bound L_r of row r's smallest q moves by
// at most dmax_r + dT_r + max dT (dmax_r: the row's largest d), rounded down.
// The pair of r and the new node is looked at itself.  A row is scanned again
// only when L_r reaches the best pair known: the smallest current q among the
// CTA's own rows' last best pairs and the pairs that the CTAs published for the
// last join.  8,000 sequences scan 1.2 % of the live rows a join, 1,000 about a
// tenth.
//
// What bounds it: a chain of a few dependent steps per join (pick, the two rows
// through L2, the update and its reduction, the scan, the exchange), each a CTA
// barrier or an L2 round trip; 5-9 us.  Against one streaming pass over the
// whole live triangle per join with three to four barriers, which it replaced
// (bounded by L2 and HBM bandwidth at 8,000 taxa, by its barriers below 2,000),
// whole job, matrix on the device: 15.3 -> 7.7 ms at 1,200 taxa, 130 -> 70.5 ms at
// 8,000.  Where many pairs tie, exactly or within rounding, the candidate scan
// decides: 16-byte loads, several in flight, few rows split over the warps, and a
// count that stops at five ties (400 taxa in copies 8.1 -> 5.5 ms, the full pass
// 6.2; 8,000 taxa that tie within rounding 1,030 -> 367, the full pass 730).
//
// The pick is exact as with a full pass: every float q is within E of the exact
// q; every pair whose float q is at most the smallest + 3E lies in a row whose
// bound reaches the best known pair + 5E, so it was scanned for this join.  A CTA
// publishes its smallest q and its second smallest (of the same row or another
// row); when no second is within the threshold, the published pairs within it
// are all the candidates.  Otherwise the CTAs scan their rows within the
// threshold into the candidate list.
// Threads per CTA, at most.  A thread per own row, so 512 do for 16 CTAs or more
// and for 8 up to 4,096 taxa, with 128 registers: one CTA of 512 threads an SM, two
// of 256.  Bounded at 1,024 the kernels have 64 registers and spill in the candidate
// scan (400 taxa: 2.5 instead of 2.2 ms), but four CTAs of 256 threads fit an SM:
// for launches of more clusters than that (100 jobs of 140 to 300 taxa: 14.8 instead
// of 24.7 ms).
constexpr int kLazyThreads = 512, kLazyThreadsMax = 1024;
constexpr int kLazyMaxCtas = 160;         // team size, at most
// From kCompactN slots on, the matrix is also compacted whenever one in
// kCompactPart of them is dead: every CTA reads and updates all slots for every
// join, and a new segment costs one scan of all rows.  8,000 taxa: 78.1 ms at
// rebuilds only, 73.5 / 72.9 / 74.0 / 75.2 with a part of 4 / 8 / 16 / 24; 2,100:
// 14.57 / 14.28 / 14.30 / 14.42 / 14.65.
constexpr int kCompactN = 2048, kCompactPart = 8;

struct LazyLayout {
  size_t tf, tl, tv, node, prow, ord, made, row, town, parts, bytes;
  int rows;                                // own rows per CTA
};

__host__ __device__ inline LazyLayout lazy_layout(int n0, int ld, int size) {
  auto al = [](size_t x) { return (x + 15) / 16 * 16; };
  LazyLayout L;
  L.rows = (n0 + size - 1) / size;
  size_t o = 0;
  L.tf = o; o += al(sizeof(float) * ld);
  L.tl = o; o += al(sizeof(float) * ld);
  L.tv = o; o += al(sizeof(float) * ld);
  L.node = o; o += al(sizeof(int16_t) * ld);
  L.prow = o; o += al(sizeof(int16_t) * n0);
  L.ord = o; o += al(sizeof(int16_t) * n0);
  L.made = o; o += al(sizeof(int16_t) * n0);
  L.row = o; o += al((sizeof(float) * 5 + sizeof(int)) * L.rows);
  L.town = o; o += al(sizeof(double) * L.rows);
  L.parts = o; o += al(sizeof(float4) * 2 * size);
  L.bytes = o;
  return L;
}

// Threads per CTA, between 256 and 512 (more make every CTA barrier dearer than
// their loads in flight save), at least one per own row and per CTA of the team, a
// multiple of 32: one per four slots over the whole GPU, one per slot in a
// cluster with the GPU to itself, whose CTAs have more rows to scan (500 taxa that tie within rounding:
// 4.7 ms instead of 5.0, with distances of 1 to 999 2.73 instead of 2.82).  The
// serving loop's batches share the GPU: 16 jobs of up to 512 taxa 12.2 ms, 12.8 with
// the wide form where a batch is small.
inline int lazy_threads(int ld, int rows, int size, bool alone) {
  const int want = size <= 16 && alone ? ld : ld / 4;
  const int t = std::max(std::max(std::min(std::max(want, 256), 512), rows), size);
  return (t + 31) / 32 * 32;
}

// The job's state in the CTA's shared memory.
struct LazyMem {
  float* Tf;        // T = Tf + Tl; NaN at dead and padding slots
  float* Tl;
  float* tv;        // the join's new values
  int16_t* node;    // slot -> node id, -1 dead or padding
  int16_t* prow;    // slot -> its row's place
  int16_t* ord;     // slots by ascending node id at the segment's start
  int16_t* made;    // slots of the nodes made since, in order
  // own rows (row l * size + rank)
  double* To;       // exact T
  float* L;         // lower bound of the row's smallest exact q
  float* U;         // float q of its last best pair (FLT_MAX: none)
  float* d1;        // that pair's d and column
  int* c1;
  float* dmax;      // the row's largest d
  float* m2;        // its second smallest q if scanned for this join, else FLT_MAX
  float4* parts;    // [2][size]: per CTA smallest q, second, pair (r | c << 16), d
};

// What every CTA knows alike.
struct LazyRep {
  float dabs;       // largest |d| of any pair so far
  float tabs;       // largest |T| of a live slot
  int elow;         // every d is a multiple of 2^elow (INT_MAX: all zero)
};

__device__ __forceinline__ float lazy_err(const LazyRep& k, float nm2f) {   // E for this join's float q
  const float m = __fadd_ru(__fmul_ru(k.dabs, fabsf(nm2f)), __fmul_ru(2.f, k.tabs));
  return __fadd_ru(__fmul_ru(8.f * 5.9604645e-8f, m), 1e-30f);
}

// Whether floats do not hold this join's q and T (undefined or infinite values
// among them, or too near the overflow for one more join's growth): the search
// is then exact, over every pair.
__device__ __forceinline__ bool lazy_wide(const LazyRep& k, float nm2f) {
  return !(__fadd_ru(__fmul_ru(k.dabs, fmaxf(nm2f, 1.f)), __fmul_ru(2.f, k.tabs)) <= kFloatTop);
}

__device__ __forceinline__ float lazy_q(float d, float tr, float tc, float nm2f) {
  return __fsub_rn(__fsub_rn(__fmul_rn(d, nm2f), tr), tc);
}

__device__ __forceinline__ float unford(int i) { return __int_as_float(i >= 0 ? i : i ^ 0x7FFFFFFF); }

// One row's two smallest q and largest d (and, at a segment's start, largest
// |d| and lowest exponent).
struct RowScan {
  float m1, m2, d1, mx, ma;   // d1: d of the smallest (in column c1)
  int c1, el;
};

__device__ __forceinline__ RowScan scan_none() { return RowScan{FLT_MAX, FLT_MAX, 0.f, -FLT_MAX, 0.f, -1, INT_MAX}; }

template <bool First>
__device__ __forceinline__ void scan_elem(RowScan& x, float d, float tc, int c, float tr, float nm2f) {
  const float q = lazy_q(d, tr, tc, nm2f);   // NaN at dead and padding slots: drops out below
  const bool lt = q < x.m1;
  x.m2 = lt ? x.m1 : fminf(x.m2, q);
  x.c1 = lt ? c : x.c1;
  x.d1 = lt ? d : x.d1;
  x.m1 = lt ? q : x.m1;
  if (tc == tc) {
    x.mx = fmaxf(x.mx, d);
    if (First) {
      x.ma = fmaxf(x.ma, fabsf(d));
      x.el = min(x.el, low_bit_exp(d));
    }
  }
}

// Warp `sub` of the `wpr` that scan row r.
template <bool First>
__device__ RowScan scan_row_part(const NJDev& s, const LazyMem& m, int r, int sub, int wpr, float nm2f) {
  const int lane = threadIdx.x & 31;
  RowScan x = scan_none();
  const float tr = m.Tf[r];
  if (tr != tr) return x;   // dead
  const float* row = row_at(s, m.prow[r]);
  const int c0 = r + 1, v0 = (c0 + 3) >> 2, nv = s.ld >> 2;
  if (sub == 0 && lane < 4 * v0 - c0 && c0 + lane < s.n0)
    scan_elem<First>(x, __ldcg(row + c0 + lane), m.Tf[c0 + lane], c0 + lane, tr, nm2f);
  const float4* row4 = reinterpret_cast<const float4*>(row);
  const float4* Tf4 = reinterpret_cast<const float4*>(m.Tf);
#pragma unroll 4
  for (int v = v0 + sub * 32 + lane; v < nv; v += 32 * wpr) {
    const float4 d = __ldcg(row4 + v);
    const float4 tc = Tf4[v];
    scan_elem<First>(x, d.x, tc.x, 4 * v, tr, nm2f);
    scan_elem<First>(x, d.y, tc.y, 4 * v + 1, tr, nm2f);
    scan_elem<First>(x, d.z, tc.z, 4 * v + 2, tr, nm2f);
    scan_elem<First>(x, d.w, tc.w, 4 * v + 3, tr, nm2f);
  }
  return x;
}

// Two smallest (an equal pair makes m2 = m1; of equal ones the lowest lane's
// first), the largest and the lowest over the lanes.
template <bool First>
__device__ __forceinline__ void scan_warp(RowScan& x) {
  const int lane = threadIdx.x & 31;
  const int key = ford(x.m1);
  const int k1 = __reduce_min_sync(0xffffffffu, key);
  const int first = __ffs(__ballot_sync(0xffffffffu, key == k1)) - 1;
  // the second: the first lane's own second, or another lane's smallest
  const int k2 = __reduce_min_sync(0xffffffffu, lane == first ? ford(x.m2) : key);
  x.m1 = unford(k1);
  x.m2 = unford(k2);
  x.c1 = __shfl_sync(0xffffffffu, x.c1, first);
  x.d1 = __shfl_sync(0xffffffffu, x.d1, first);
  x.mx = unford(__reduce_max_sync(0xffffffffu, ford(x.mx)));
  if (First) {
    x.ma = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(x.ma)));
    x.el = __reduce_min_sync(0xffffffffu, x.el);
  }
}

// Scans the own rows row_of(0) .. row_of(cnt - 1) (the same in every warp): U,
// d1, c1, dmax, m2, and L = m1 - E.  Few rows are split over the CTA's warps (a
// power of two per row).  First: the largest |d| and lowest exponent go to ma /
// el.  Every thread calls it; the results are visible after the caller's next
// CTA barrier.
template <bool First, class Rows>
__device__ void scan_rows(const NJDev& s, const LazyMem& m, Team tm, Rows&& row_of, int cnt, float nm2f, float E,
                          int* ma, int* el) {
  __shared__ RowScan part[32];
  const int lane = threadIdx.x & 31, warp = (int)threadIdx.x >> 5, nw = (int)blockDim.x >> 5;
  if (cnt == 0) return;   // the same in the CTA
  int wpr = 1;
  while (2 * wpr * cnt <= nw) wpr *= 2;
  const int per = nw / wpr;   // rows at a time
  for (int k0 = 0; k0 < cnt; k0 += per) {
    const int k = k0 + warp / wpr, sub = warp % wpr;
    const bool mine = k < cnt && warp / wpr < per;
    const int l = mine ? row_of(k) : 0;
    RowScan x = scan_none();
    if (mine) {
      x = scan_row_part<First>(s, m, l * tm.size + tm.rank, sub, wpr, nm2f);
      scan_warp<First>(x);
    }
    if (wpr > 1) {
      if (lane == 0) part[warp] = x;
      __syncthreads();
      if (mine && sub == 0) {
        x = lane < wpr ? part[warp + lane] : scan_none();
        scan_warp<First>(x);
      }
    }
    if (mine && sub == 0 && lane == 0) {
      m.U[l] = x.m1;
      m.m2[l] = x.m2;
      m.c1[l] = x.c1;
      m.d1[l] = x.d1;
      m.dmax[l] = x.c1 >= 0 ? x.mx : 0.f;
      m.L[l] = x.c1 >= 0 ? __fsub_rd(x.m1, E) : FLT_MAX;
      if (First) {
        atomicMax(ma, __float_as_int(x.ma));
        atomicMin(el, x.el);
      }
    }
    if (wpr > 1 && k0 + per < cnt) __syncthreads();   // part is free again
  }
}

// Exchange of the CTAs' published float4 through global memory (the grid): the
// value, then an arrival count that one thread of each CTA polls, then all the
// values at once.  (Polling the values themselves, 152 readers of 152 lines,
// kept the L2 slices that hold them busy: 12,000 cycles an exchange.)
// Publishing: one thread, after a CTA barrier that follows the CTA's writes to
// global memory.
__device__ __forceinline__ void grid_publish(const GridNJ& g, Team tm, unsigned seq, float4 v) {
  g.gather[(size_t)(seq & 1) * tm.size + tm.rank] = v;
  red_release_add(&g.bar[1], 1u);
}

// Every CTA's published value into parts' half seq & 1; every thread calls it.
// False when a wait ran out or another CTA gave up.
__device__ bool grid_gather(const GridNJ& g, Team tm, unsigned seq, float4* parts) {
  int bad = 0;
  if (threadIdx.x == 0) {
    const unsigned target = seq * (unsigned)tm.size;
    const long long t0 = clock64();
    while ((int)(ld_acquire_u32(&g.bar[1]) - target) < 0) {
      if (*(volatile int*)g.abort) bad = 1;
      else if (clock64() - t0 > kBarrierSpinCycles) {
        atomicExch(g.abort, kAbortWait);
        bad = 1;
      }
      if (bad) break;
    }
  }
  if (__syncthreads_or(bad)) return false;
  const size_t at = (size_t)(seq & 1) * tm.size + threadIdx.x;
  if ((int)threadIdx.x < tm.size) parts[at] = __ldcg(g.gather + at);
  __syncthreads();
  return true;
}

// Publishes this CTA's value (v, in warp 0's lanes) and gathers every CTA's into
// m.parts' half seq & 1; every thread calls it, after a CTA barrier that follows
// the CTA's writes to global memory.
template <bool CL>
__device__ bool team_exchange(const GridNJ& g, const LazyMem& m, Team tm, unsigned seq, float4 v) {
  if constexpr (CL) {
    if ((int)threadIdx.x < tm.size)
      cooperative_groups::this_cluster().map_shared_rank(m.parts, threadIdx.x)[(seq & 1) * tm.size + tm.rank] = v;
    cooperative_groups::this_cluster().sync();
    return true;
  } else {
    if (threadIdx.x == 0 && !(g.stall && tm.rank == 0)) grid_publish(g, tm, seq, v);
    return grid_gather(g, tm, seq, m.parts);
  }
}

// The CTA's smallest and second smallest q over its own rows, by one warp (the
// result in every lane).
__device__ __forceinline__ float4 cta_best(const LazyMem& m, Team tm, int rows) {
  const int lane = threadIdx.x & 31;
  float b1 = FLT_MAX, b2 = FLT_MAX;
  int bl = 0;
  for (int l = lane; l < rows; l += 32) {
    const float u = m.U[l], v = m.m2[l];
    const bool lt = u < b1;
    b2 = lt ? fminf(b1, v) : fminf(b2, u);
    bl = lt ? l : bl;
    b1 = lt ? u : b1;
  }
  const int key = ford(b1);
  const int k1 = __reduce_min_sync(0xffffffffu, key);
  const int first = __ffs(__ballot_sync(0xffffffffu, key == k1)) - 1;
  const int k2 = __reduce_min_sync(0xffffffffu, lane == first ? ford(b2) : key);
  bl = __shfl_sync(0xffffffffu, bl, first);
  return make_float4(unford(k1), unford(k2), __uint_as_float((unsigned)(bl * tm.size + tm.rank) | (unsigned)m.c1[bl] << 16),
                     m.d1[bl]);
}

// Candidate scan of the fallback: this CTA's own rows within the threshold,
// visit(pred, candidate) by whole warps.  tx: every slot's exact T.  wide: every
// live row's pairs, without a look at the floats; a pair whose q is undefined or
// +infinity is none, as in the reference's comparisons.  A warp stops when visit
// returns false (the same in the warp).  Every thread calls it.
template <class Visit>
__device__ void lazy_cand_scan(const NJDev& s, const LazyMem& m, Team tm, int rows, const double* tx, float nm2f,
                               double nm2, int watermark, float thr, bool wide, Visit&& visit) {
  __shared__ int16_t s_rows[1024];
  const int lane = threadIdx.x & 31, warp = (int)threadIdx.x >> 5, nw = (int)blockDim.x >> 5;
  int cnt = 0;   // the rows, counted by every warp for itself
  for (int l0 = 0; l0 < rows; l0 += 32) {
    const int l = l0 + lane, r = l * tm.size + tm.rank;
    const bool in = l < rows && (wide ? r < s.n0 && m.node[r] >= 0 : m.U[l] <= thr);
    const unsigned bal = __ballot_sync(0xffffffffu, in);
    if (warp == 0 && in) s_rows[cnt + __popc(bal & ((1u << lane) - 1u))] = (int16_t)l;
    cnt += __popc(bal);
  }
  __syncthreads();
  if (cnt == 0) return;
  int wpr = 1;   // few rows are split over the warps
  while (2 * wpr * cnt <= nw) wpr *= 2;
  const int per = nw / wpr, sub = warp % wpr, nv = s.ld >> 2;
  if (warp / wpr >= per) return;
  constexpr int kAhead = 2;   // 16-byte loads of a lane in flight
  const float4* Tf4 = reinterpret_cast<const float4*>(m.Tf);
  for (int k = warp / wpr; k < cnt; k += per) {
    const int l = s_rows[k], r = l * tm.size + tm.rank, ur = m.node[r];
    const float tr = m.Tf[r];
    const double Tr = m.To[l];
    const float4* row4 = reinterpret_cast<const float4*>(row_at(s, m.prow[r]));
    for (int v0 = ((r + 1) >> 2) + 32 * sub; v0 < nv; v0 += 32 * wpr * kAhead) {
      float4 d4[kAhead];
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int v = v0 + 32 * wpr * u + lane;
        d4[u] = v < nv ? __ldcg(row4 + v) : make_float4(0.f, 0.f, 0.f, 0.f);
      }
#pragma unroll
      for (int u = 0; u < kAhead; ++u) {
        const int v = v0 + 32 * wpr * u + lane;
        const float4 t4 = Tf4[min(v, nv - 1)];
        const float d[4] = {d4[u].x, d4[u].y, d4[u].z, d4[u].w}, tc[4] = {t4.x, t4.y, t4.z, t4.w};
        unsigned in = 0;   // the candidates among the four columns
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int c = 4 * v + e;   // q is NaN at dead and padding slots
          const bool is = wide ? c < s.n0 && m.node[c] >= 0 : lazy_q(d[e], tr, tc[e], nm2f) <= thr;
          if (v < nv && c > r && is) in |= 1u << e;
        }
        if (!__any_sync(0xffffffffu, in)) continue;
        double Tc[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) Tc[e] = in >> e & 1 ? __ldcg(tx + 4 * v + e) : 0.0;
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          bool pred = in >> e & 1;
          KCand kc = kc_none();
          if (pred) {
            const GCand cd = make_cand(r, 4 * v + e, ur, m.node[4 * v + e], Tr, Tc[e], d[e], nm2, watermark);
            kc = kc_of(cd);
            pred = !wide || cd.q1 < DBL_MAX;
          }
          if (!visit(pred, kc)) return;
        }
      }
    }
  }
}

// The pick when the published pairs do not decide it alone (several within the
// threshold, or a CTA's second): the winner in *win and *pk, the same in every
// CTA.  False when a wait ran out.
template <bool CL>
__device__ bool lazy_pick_slow(const NJDev& s, const GridNJ& g, const LazyMem& m, Team tm, int rows,
                               const float4* parts, const double* tx, float thr, bool listed, bool wide, float nm2f,
                               double nm2, int watermark, GCand* win, PickOut* pk, unsigned& picks, unsigned& target) {
  __shared__ GCand fc[32];
  const int lane = threadIdx.x & 31;
  if (listed) {   // at most 32 published pairs are all the candidates
    if (threadIdx.x < 32) {
      int base = 0;
      for (int b0 = 0; b0 < tm.size; b0 += 32) {
        const float4 v = b0 + lane < tm.size ? parts[b0 + lane] : make_float4(FLT_MAX, FLT_MAX, 0.f, 0.f);
        const bool in = b0 + lane < tm.size && v.x <= thr;
        const unsigned bal = __ballot_sync(0xffffffffu, in);
        if (in) {
          const unsigned rc = __float_as_uint(v.z);
          const int r = rc & 0xFFFFu, c = rc >> 16;
          fc[base + __popc(bal & ((1u << lane) - 1u))] =
              make_cand(r, c, m.node[r], m.node[c], __ldcg(tx + r), __ldcg(tx + c), v.w, nm2, watermark);
        }
        base += __popc(bal);
      }
      __syncwarp();
      const PickOut r = pick_keys(base, [&](int k) { return fc[k]; });
      if (lane == 0) {
        *pk = r;
        *win = fc[r.idx];
      }
    }
    __syncthreads();
    return true;
  }
  // the counts alternate between two sets: this pick's are zero, the last one's
  // are read by nobody any more once every CTA is here
  int* const cnt = s.g32 + 4 * (picks & 1);
  int* const old = s.g32 + 4 * (picks + 1 & 1);
  ++picks;
  KCand first = kc_none();
  bool full = false;
  lazy_cand_scan(s, m, tm, rows, tx, nm2f, nm2, watermark, thr, wide, [&](bool pred, const KCand& c) {
    list_push(s, g, &cnt[2], pred, c, full);
    if (pred && kc_first(c, first)) first = c;
    return true;
  });
  if (!team_sync<CL>(g, target)) return false;
  if (tm.rank == 0 && threadIdx.x == 0) old[0] = old[1] = old[2] = 0;
  // the winner's pair again, as the scan read it (row = the smaller slot)
  auto rederive = [&](const KCand& w) {
    const int sa = slot_of(w.a), sb = slot_of(w.b);
    const int r0 = min(sa, sb), c0 = max(sa, sb);
    *win = make_cand(r0, c0, m.node[r0], m.node[c0], __ldcg(tx + r0), __ldcg(tx + c0),
                     __ldcg(row_at(s, m.prow[r0]) + c0), nm2, watermark);
  };
  const int ncount = __ldcg(&cnt[2]);   // the same in every CTA
  if (ncount <= min(s.cand_cap, kListPickMax)) {
    if (threadIdx.x < 32) {
      const PickOut r = pick_keys(ncount, [&](int k) { return ld_kcand(&g.cand[k]); });
      if (lane == 0) {
        *pk = r;
        if (!r.error) rederive(ld_kcand(&g.cand[r.idx]));
      }
    }
  } else {
    __shared__ KCand sw[32];
    __shared__ KCand sfirst;
    const KCand cf = cta_first(first, sw);
    if (threadIdx.x == 0) g.cbest[tm.rank] = cf;
    if (!team_sync<CL>(g, target)) return false;
    if (threadIdx.x < 32) {
      const PickOut r = pick_keys(tm.size, [&](int k) { return ld_kcand(&g.cbest[k]); });
      if (lane == 0) sfirst = r.error ? kc_none() : ld_kcand(&g.cbest[r.idx]);
    }
    __syncthreads();
    const KCand w = sfirst;
    unsigned ties = 0, amb = 0;
    lazy_cand_scan(s, m, tm, rows, tx, nm2f, nm2, watermark, thr, wide, [&](bool pred, const KCand& c) {
      // one ambiguous pair, or five ties, decide the step's statistics
      unsigned t = 0, a = 0;
      if (pred) count_vs(c, w, t, a);
      ties += __popc(__ballot_sync(0xffffffffu, t));
      amb |= __any_sync(0xffffffffu, a);
      return ties <= 4 && !amb;
    });
    if (lane == 0 && (ties | amb)) {   // the warp's
      atomicAdd(&cnt[0], (int)ties);
      atomicAdd(&cnt[1], (int)amb);
    }
    if (!team_sync<CL>(g, target)) return false;
    if (threadIdx.x == 0) {
      pk->idx = 0;
      pk->ties = (unsigned)__ldcg(&cnt[0]);
      pk->amb = (unsigned)__ldcg(&cnt[1]);
      pk->error = w.b < 0;
      if (!pk->error) rederive(w);
    }
  }
  return true;
}

// The sequential double sum of the join's values over the active nodes in
// ascending id order (SpeciesBlock.cpp:799, :818), by one thread.
__device__ double lazy_seq_sum(const LazyMem& m, int n_ord, int id0, int n_made, int si, int sj) {
  double sum = 0.0;
  for (int k = 0; k < n_ord; ++k) {
    const int p = m.ord[k], v = m.node[p];
    if (v >= 0 && v < id0 && p != si && p != sj) sum = __dadd_rn(sum, (double)m.tv[p]);
  }
  for (int k = 0; k < n_made; ++k) {
    const int p = m.made[k];
    if (m.node[p] == id0 + k && p != si && p != sj) sum = __dadd_rn(sum, (double)m.tv[p]);
  }
  return sum;
}

// Joins step0 .. step1 - 1 of an n-taxon job by one team (the active count
// before join t is n - t); T, Tf, node, prow, slot and the active list come from
// and go back to global memory.  seq: exchanges so far.  False when the team
// stops (a wait ran out, the pick failed) -- the same in every CTA.
template <bool CL>
__device__ bool lazy_segment(const NJDev& s, const GridNJ& g, Team tm, unsigned char* smem, int step0, int step1, int n,
                             int watermark, unsigned& seq, unsigned& target) {
  const int tid = (int)threadIdx.x, nth = (int)blockDim.x, lane = tid & 31, warp = tid >> 5, nw = nth >> 5;
  const int n0 = s.n0, ld = s.ld, nv = ld >> 2;
  LazyMem m;
  int rows;
  {
    const LazyLayout Y = lazy_layout(n0, ld, tm.size);
    rows = Y.rows;
    m.Tf = reinterpret_cast<float*>(smem + Y.tf);
    m.Tl = reinterpret_cast<float*>(smem + Y.tl);
    m.tv = reinterpret_cast<float*>(smem + Y.tv);
    m.node = reinterpret_cast<int16_t*>(smem + Y.node);
    m.prow = reinterpret_cast<int16_t*>(smem + Y.prow);
    m.ord = reinterpret_cast<int16_t*>(smem + Y.ord);
    m.made = reinterpret_cast<int16_t*>(smem + Y.made);
    m.To = reinterpret_cast<double*>(smem + Y.town);
    m.L = reinterpret_cast<float*>(smem + Y.row);
    m.U = m.L + rows;
    m.d1 = m.U + rows;
    m.dmax = m.d1 + rows;
    m.m2 = m.dmax + rows;
    m.c1 = reinterpret_cast<int*>(m.m2 + rows);
    m.parts = reinterpret_cast<float4*>(smem + Y.parts);
  }
  __shared__ int s_ma, s_el, s_hint;
  __shared__ int16_t s_list[1024];         // own rows to scan
  __shared__ GCand swin;
  __shared__ PickOut spick;
  __shared__ double s_seq;
  __shared__ float s_thr;
  __shared__ int s_cands;
  __shared__ float4 s_pair;
  __shared__ LazyRep s_rep;
  __shared__ long long w_u[32];            // per warp: the join's integer sum,
  __shared__ long long w_u2[32], w_a2[32]; // the second sum and its values' magnitudes
  __shared__ int4 w_x[32];                 // largest dT (ordered), |T|, |tmp|, lowest exponent
  unsigned picks = 0;                      // slow picks over the candidate scan so far
  if (tm.rank == 0 && tid < 8) s.g32[tid] = 0;   // before the first exchange
  const int id0 = n + step0;               // ids from here on are made in this segment
  const int n_ord = __ldcg(s.na);
  int spare = __ldcg(s.prow + n0);         // the free place
  float ta = 0.f;
  for (int p = tid; p < ld; p += nth) {
    const int v = p < n0 ? __ldcg(s.node + p) : -1;
    m.node[p] = (int16_t)v;
    if (p < n0) m.prow[p] = (int16_t)__ldcg(s.prow + p);
    const double t = v >= 0 ? __ldcg(s.T + p) : 0.0;
    const float hi = __double2float_rn(t);
    ta = fmaxf(ta, fabsf(hi) <= FLT_MAX ? fabsf(hi) : CUDART_INF_F);
    m.Tf[p] = v >= 0 ? hi : __int_as_float(0x7FC00000);
    m.Tl[p] = __double2float_rn(__dsub_rn(t, (double)hi));
    m.tv[p] = 0.f;
  }
  for (int k = tid; k < n_ord; k += nth) m.ord[k] = (int16_t)__ldcg(s.slot + __ldcg(s.act + k));
  for (int l = tid; l < rows; l += nth) {
    m.L[l] = m.U[l] = m.m2[l] = FLT_MAX;
    m.d1[l] = m.dmax[l] = 0.f;
    m.c1[l] = 0;
    const int r = l * tm.size + tm.rank;
    const bool live = r < n0 && __ldcg(s.node + r) >= 0;
    m.To[l] = live ? __ldcg(s.T + r) : 0.0;
    // the exact T that go with the first exchange of pairs (seq + 2)
    if (live) s.tx[(size_t)(seq & 1) * n0 + r] = m.To[l];
  }
  if (tid == 0) {
    s_ma = 0;
    s_el = INT_MAX;
  }
  ta = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(ta)));
  if (lane == 0) w_x[warp].x = __float_as_int(ta);
  __syncthreads();
  // ---- every own row once: best pairs, bounds; the largest |d|, |T| and the
  // lowest exponent of the whole job
  LazyRep rep{0.f, 0.f, INT_MAX};
  float nm2f = (float)(n - step0 - 2);
  {
    const int own = n0 > tm.rank ? (n0 - tm.rank + tm.size - 1) / tm.size : 0;   // dead rows scan to nothing
    scan_rows<true>(s, m, tm, [](int k) { return k; }, own, nm2f, 0.f, &s_ma, &s_el);
    __syncthreads();
    for (int w = 0; w < nw; ++w) rep.tabs = fmaxf(rep.tabs, __int_as_float(w_x[w].x));
    rep.tabs = __fmul_ru(rep.tabs, 1.000001f);
    if (!team_exchange<CL>(g, m, tm, ++seq, make_float4(__int_as_float(s_ma), 0.f, __int_as_float(s_el), 0.f)))
      return false;
    const float4* pp = m.parts + (seq & 1) * tm.size;
    for (int b = 0; b < tm.size; ++b) {
      rep.dabs = fmaxf(rep.dabs, pp[b].x);
      rep.elow = min(rep.elow, __float_as_int(pp[b].z));
    }
    const float E = lazy_err(rep, nm2f);
    for (int l = tid; l < rows; l += nth)
      if (m.U[l] < FLT_MAX) m.L[l] = __fsub_rd(m.U[l], E);
    __syncthreads();
  }
  float4 pub = make_float4(FLT_MAX, FLT_MAX, 0.f, 0.f);
  if (warp == 0) pub = cta_best(m, tm, rows);
  if (!team_exchange<CL>(g, m, tm, ++seq, pub)) return false;
  for (int step = step0; step < step1; ++step) {
    const int m_n = n - step, next = n + step;
    const double nm2 = (double)(m_n - 2);
    const float4* const parts = m.parts + (seq & 1) * tm.size;
    const double* const tx = s.tx + (size_t)(seq & 1) * n0;
    // ---- pick: the published pairs within the threshold
    const bool wide = lazy_wide(rep, nm2f);   // the same in every thread of the team
    if (warp == 0) {
      const float E = lazy_err(rep, nm2f);
      constexpr int kPer = kLazyMaxCtas / 32;
      float x[kPer], own = FLT_MAX;
      int at = 0, cands = 0;
#pragma unroll
      for (int t = 0; t < kPer; ++t) {
        const int b = lane + 32 * t;
        x[t] = b < tm.size ? parts[b].x : FLT_MAX;
        if (x[t] < own) {
          own = x[t];
          at = b;
        }
      }
      const float q = unford(__reduce_min_sync(0xffffffffu, ford(own)));
      const float thr = q < FLT_MAX ? __fadd_ru(q, __fmul_ru(3.f, E)) : -FLT_MAX;
      bool second = false;
#pragma unroll
      for (int t = 0; t < kPer; ++t) {
        const bool in = lane + 32 * t < tm.size && x[t] <= thr;
        if (in) second |= parts[lane + 32 * t].y <= thr;
        cands += __popc(__ballot_sync(0xffffffffu, in));
      }
      if (__any_sync(0xffffffffu, second)) cands = -1;
      const unsigned has = __ballot_sync(0xffffffffu, own <= thr);
      if (lane == (has ? __ffs(has) - 1 : 0)) {
        s_thr = thr;
        s_cands = cands;
        s_pair = parts[at];
      }
    }
    __syncthreads();
    const float thr = s_thr;
    const int cands = s_cands;
    const unsigned rc = __float_as_uint(s_pair.z);
    float dmin = s_pair.w;
    int i, j, si, sj;
    const bool fast = cands == 1 && !wide;
    if (fast) {
      const int r = rc & 0xFFFFu, c = rc >> 16;
      const int ur = m.node[r], uc = m.node[c];
      i = min(ur, uc);
      j = max(ur, uc);
      si = ur < uc ? r : c;
      sj = ur < uc ? c : r;
    } else {
      if (!lazy_pick_slow<CL>(s, g, m, tm, rows, parts, tx, thr, cands >= 1 && cands <= 32 && !wide, wide, nm2f, nm2,
                              watermark, &swin, &spick, picks, target))
        return false;
      __syncthreads();
      if (spick.error) {   // the same in every CTA
        if (tm.rank == 0 && tid == 0) {
          record_pick(s, spick);
          // nothing goes back to global memory: what is queued behind this
          // segment must not read the lists, it leaves as after a wait that ran out
          if constexpr (!CL) atomicExch(g.abort, kAbortPick);
        }
        return false;
      }
      i = swin.a;
      j = swin.b;
      si = swin.sa;
      sj = swin.sb;
      dmin = swin.d;
    }
    // ---- the join, in every CTA: modifyMatrix (SpeciesBlock.cpp:787-841) on its
    // copy of T; the owners write the new row and their rows' new column
    const bool own_si = si % tm.size == tm.rank;
    const int place = m.prow[si];
    const float* const rowi = row_at(s, place);
    float* const newrow = row_at(s, spare);
    // every new value is a multiple of 2^eu, and at most 1.5 dabs (rounding aside)
    const int eu = rep.elow == INT_MAX ? 0 : rep.elow - 1;
    const int span_max = rep.dabs > 0.f ? top_bit_exp(rep.dabs) + 3 - eu : 0;
    const bool u32 = !wide && span_max <= 30 && eu >= -100 && eu <= 100;
    const bool u64 = !wide && span_max < 47;
    const float scale = u32 ? __int_as_float((127 - eu) << 23) : 0.f;
    long long u = 0;
    int x_el = INT_MAX, x_or = 0;
    float x_t = 0.f, x_d = 0.f, x_dt = -FLT_MAX;
    const float* const rowj = row_at(s, m.prow[sj]);
    // this thread's own row: the new column's value and the change of T
    const int r_own = tid * tm.size + tm.rank;
    const bool has_own = tid < rows && r_own < n0;
    const float a_own = has_own ? __ldcg(rowi + r_own) : 0.f, b_own = has_own ? __ldcg(rowj + r_own) : 0.f;
    for (int v = tid; v < nv; v += nth) {
      const float4 a4 = __ldcg(reinterpret_cast<const float4*>(rowi) + v);
      const float4 b4 = __ldcg(reinterpret_cast<const float4*>(rowj) + v);
      const float4 h4 = reinterpret_cast<const float4*>(m.Tf)[v], l4 = reinterpret_cast<const float4*>(m.Tl)[v];
      const float a[4] = {a4.x, a4.y, a4.z, a4.w}, b[4] = {b4.x, b4.y, b4.z, b4.w};
      const float hi[4] = {h4.x, h4.y, h4.z, h4.w}, lo[4] = {l4.x, l4.y, l4.z, l4.w};
      float nh[4], nl[4], nt[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float sumf = __fadd_rn(a[k], b[k]);
        const float tmp = __fmul_rn(__fsub_rn(sumf, dmin), 0.5f);
        const float dt = __fsub_rn(tmp, sumf);
        // T as two floats: two-sum, then the carry (NaN stays NaN at dead
        // slots; si's and sj's are set below)
        const float sm = __fadd_rn(hi[k], dt), bb = __fsub_rn(sm, hi[k]);
        const float c = __fadd_rn(lo[k], __fadd_rn(__fsub_rn(hi[k], __fsub_rn(sm, bb)), __fsub_rn(dt, bb)));
        nh[k] = __fadd_rn(sm, c);
        nl[k] = __fsub_rn(c, __fsub_rn(nh[k], sm));
        nt[k] = tmp;
        const int p = 4 * v + k;
        if (hi[k] == hi[k] && p != si && p != sj) {
          x_dt = fmaxf(x_dt, dt);
          x_t = fmaxf(x_t, fabsf(nh[k]));
          x_d = fmaxf(x_d, fabsf(tmp));
          if (u32) {
            const int y = __float2int_rn(__fmul_rn(tmp, scale));   // exact
            u += y;
            x_or |= y;
          } else {
            x_el = min(x_el, low_bit_exp(tmp));
            if (u64) u += float_units(tmp, eu);
          }
        }
      }
      reinterpret_cast<float4*>(m.Tf)[v] = make_float4(nh[0], nh[1], nh[2], nh[3]);
      reinterpret_cast<float4*>(m.Tl)[v] = make_float4(nl[0], nl[1], nl[2], nl[3]);
      reinterpret_cast<float4*>(m.tv)[v] = make_float4(nt[0], nt[1], nt[2], nt[3]);
      if (own_si) reinterpret_cast<float4*>(newrow)[v] = make_float4(nt[0], nt[1], nt[2], nt[3]);
    }
    const float sum_own = __fadd_rn(a_own, b_own);
    const float nd = __fmul_rn(__fsub_rn(sum_own, dmin), 0.5f), dt = __fsub_rn(nd, sum_own);
    const bool upd = has_own && m.node[r_own] >= 0 && r_own != si && r_own != sj;
    if (upd) row_at(s, m.prow[r_own])[si] = nd;
    for (int o = 16; o > 0; o >>= 1) u += __shfl_xor_sync(0xffffffffu, u, o);
    if (x_or) x_el = eu + __ffs(x_or) - 1;
    x_el = __reduce_min_sync(0xffffffffu, x_el);
    int k_dt = __reduce_max_sync(0xffffffffu, ford(x_dt));
    x_t = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(x_t)));
    x_d = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(x_d)));
    if (lane == 0) {
      w_u[warp] = u;
      w_x[warp] = make_int4(k_dt, __float_as_int(x_t), __float_as_int(x_d), x_el);
    }
    if (tid == 0) s_hint = 0x7F7FFFFF;
    __syncthreads();
    // the whole CTA's, in the warps that go on with it
    const bool lead = warp * 32 < max(rows, tm.size) || warp == nw - 1;
    double tsum = 0.0;
    float tsf = 0.f, drift = 0.f;
    if (lead) {
      const int4 y = lane < nw ? w_x[lane] : make_int4(ford(-FLT_MAX), 0, 0, INT_MAX);
      u = lane < nw ? w_u[lane] : 0;
      for (int o = 16; o > 0; o >>= 1) u += __shfl_xor_sync(0xffffffffu, u, o);
      k_dt = __reduce_max_sync(0xffffffffu, y.x);
      x_t = __uint_as_float(__reduce_max_sync(0xffffffffu, (unsigned)y.y));
      x_d = __uint_as_float(__reduce_max_sync(0xffffffffu, (unsigned)y.z));
      x_el = __reduce_min_sync(0xffffffffu, y.w);
    } else {
      // whether the sequential sum is needed is the same in every warp
      const int4 y = lane < nw ? w_x[lane] : make_int4(0, 0, 0, INT_MAX);
      x_d = __uint_as_float(__reduce_max_sync(0xffffffffu, (unsigned)y.z));
      x_el = __reduce_min_sync(0xffffffffu, y.w);
    }
    // the new node's row sum: the integer sum when every partial sum of the
    // sequential double sum is exact (all terms multiples of 2^eu, together
    // below 2^53 of them), else a sum in finer units or the sequential sum itself
    const int span = x_el == INT_MAX ? 0 : top_bit_exp(x_d) + 1 - eu;
    if (!wide && x_el == INT_MAX) {
      // every value is zero
    } else if (u64 && x_el >= eu && span <= span_max && span + 32 - __clz(m_n) <= 53) {
      tsum = units_to_double(u, eu);
    } else {
      // Real-valued distances: halving every join takes elow below what the job's
      // largest value leaves room for, but the values of one join span less.  A
      // second sum in units of their own lowest bit, exact under the same rule:
      // 16 ms instead of 75 (a sequential sum per join) for 1,200 taxa.
      bool exact = false;
      if (!wide && top_bit_exp(x_d) - x_el < 48) {   // |value| < 2^49 units, 8,192 of them
        long long u2 = 0, a2 = 0;
        for (int v = tid; v < nv; v += nth) {   // the slots that this thread has just updated
          const float4 h4 = reinterpret_cast<const float4*>(m.Tf)[v], t4 = reinterpret_cast<const float4*>(m.tv)[v];
          const float hi[4] = {h4.x, h4.y, h4.z, h4.w}, val[4] = {t4.x, t4.y, t4.z, t4.w};
#pragma unroll
          for (int k = 0; k < 4; ++k)
            if (hi[k] == hi[k] && 4 * v + k != si && 4 * v + k != sj) {
              const long long y = float_units(val[k], x_el);
              u2 += y;
              a2 += y < 0 ? -y : y;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
          u2 += __shfl_xor_sync(0xffffffffu, u2, o);
          a2 += __shfl_xor_sync(0xffffffffu, a2, o);
        }
        if (lane == 0) {
          w_u2[warp] = u2;
          w_a2[warp] = a2;
        }
        __syncthreads();
        u2 = lane < nw ? w_u2[lane] : 0;
        a2 = lane < nw ? w_a2[lane] : 0;
        for (int o = 16; o > 0; o >>= 1) {
          u2 += __shfl_xor_sync(0xffffffffu, u2, o);
          a2 += __shfl_xor_sync(0xffffffffu, a2, o);
        }
        exact = a2 < (1ll << 53);
        if (exact) tsum = units_to_double(u2, x_el);
      }
      if (!exact) {   // the same in the CTA
        if (tid == 0) s_seq = lazy_seq_sum(m, n_ord, id0, step - step0, si, sj);
        __syncthreads();
        tsum = s_seq;
      }
    }
    if (lead) {
      rep.dabs = wide ? CUDART_INF_F : fmaxf(rep.dabs, x_d);   // wide up to the segment's end: Tf no longer says who lives
      rep.elow = min(rep.elow, x_el);
      tsf = __double2float_rn(tsum);
      rep.tabs = __fmul_ru(fmaxf(x_t, fabsf(tsf)), 1.000001f);
      drift = k_dt == ford(-FLT_MAX) ? 0.f : unford(k_dt);
    }
    if (warp == nw - 1 && lane == 0 && tm.rank == 0) {   // the join record
      nwg_join& J = s.joins[step];
      J.i = i;
      J.j = j;
      J.node = next;
      J.n = m_n;
      J.d = dmin;
      J.pad = 0.f;
      if (fast) {
        const int r = min(si, sj), c = max(si, sj);
        const GCand cd = make_cand(r, c, r == si ? i : j, r == si ? j : i, __ldcg(tx + r), __ldcg(tx + c), dmin, nm2,
                                   watermark);
        J.q = cd.q1;
        J.ti = cd.ta;
        J.tj = cd.tb;
      } else {
        J.q = swin.q1;
        J.ti = swin.ta;
        J.tj = swin.tb;
        record_pick(s, spick);
      }
      s.slot[j] = -1;
      s.slot[i] = -1;
      s.slot[next] = si;
    }
    if (tid == 0) {   // read again only after the next barrier
      s_rep = rep;
      if (own_si) newrow[si] = __ldcg(rowi + si);   // the diagonal keeps i's value
      m.Tf[si] = tsf;
      m.Tl[si] = __double2float_rn(__dsub_rn(tsum, (double)tsf));
      m.Tf[sj] = __int_as_float(0x7FC00000);   // dead: NaN
      m.node[si] = (int16_t)next;
      m.node[sj] = -1;
      m.prow[si] = (int16_t)spare;
      m.made[step - step0] = (int16_t)si;
    }
    spare = place;
    nm2f = (float)(m_n - 3);
    // ---- the rows' bounds and best pairs under the new T; the best pair known
    int hint = 0x7F7FFFFF;
    if (tid < rows) {
      const int l = tid;
      m.m2[l] = FLT_MAX;
      float L = FLT_MAX, U = FLT_MAX;
      if (r_own == si) {
        L = -FLT_MAX;   // the new row: scanned below
        m.To[l] = tsum;
        s.tx[(size_t)((seq + 1) & 1) * n0 + r_own] = tsum;
      } else if (upd) {
        const float tr = m.Tf[r_own];
        const double t = __dadd_rn(m.To[l], (double)dt);
        m.To[l] = t;
        s.tx[(size_t)((seq + 1) & 1) * n0 + r_own] = t;
        const int c1 = m.c1[l];
        L = m.L[l];
        if (L < FLT_MAX) L = __fsub_rd(L, __fadd_ru(m.dmax[l], __fadd_ru(dt, drift)));
        if (m.U[l] < FLT_MAX && c1 != si && c1 != sj) U = lazy_q(m.d1[l], tr, m.Tf[c1], nm2f);
        if (r_own < si) {
          const float q = lazy_q(nd, tr, tsf, nm2f);
          L = fminf(L, __fsub_rd(q, lazy_err(rep, nm2f)));
          m.dmax[l] = fmaxf(m.dmax[l], nd);
          if (q < U) {
            U = q;
            m.c1[l] = si;
            m.d1[l] = nd;
          }
        }
        hint = ford(U);
      }
      m.L[l] = L;
      m.U[l] = U;
    }
    if (tid < tm.size) {   // the pairs published for this join that still stand
      const float4 v = parts[tid];
      const unsigned e = __float_as_uint(v.z);
      const int r = e & 0xFFFFu, c = e >> 16;
      if (v.x < FLT_MAX && r != si && r != sj && c != si && c != sj)
        hint = min(hint, ford(lazy_q(v.w, m.Tf[r], m.Tf[c], nm2f)));
    }
    if (warp * 32 < max(rows, tm.size)) {
      hint = __reduce_min_sync(0xffffffffu, hint);
      if (lane == 0) atomicMin(&s_hint, hint);
    }
    __syncthreads();
    if (step + 1 == step1) break;
    // ---- the rows whose bound reaches it, counted by every warp for itself
    rep = s_rep;
    const bool search = !lazy_wide(rep, nm2f);
    const float E = lazy_err(rep, nm2f);
    const float best = unford(s_hint);
    const float reach = best < FLT_MAX ? __fadd_ru(best, __fmul_ru(5.f, E)) : FLT_MAX;
    int cnt = 0;
    for (int l0 = 0; search && l0 < rows; l0 += 32) {
      const float L = l0 + lane < rows ? m.L[l0 + lane] : FLT_MAX;
      cnt += __popc(__ballot_sync(0xffffffffu, L <= reach && L < FLT_MAX));
    }
    if (cnt) {   // the same in every warp
      if (warp == 0) {
        int base = 0;
        for (int l0 = 0; l0 < rows; l0 += 32) {
          const float L = l0 + lane < rows ? m.L[l0 + lane] : FLT_MAX;
          const bool in = L <= reach && L < FLT_MAX;
          const unsigned bal = __ballot_sync(0xffffffffu, in);
          if (in) s_list[base + __popc(bal & ((1u << lane) - 1u))] = (int16_t)(l0 + lane);
          base += __popc(bal);
        }
      }
      __syncthreads();   // also: the bounds are read before the scan changes them
      scan_rows<false>(s, m, tm, [&](int k) { return (int)s_list[k]; }, cnt, nm2f, E, nullptr, nullptr);
      __syncthreads();
    }
    if (warp == 0) pub = cta_best(m, tm, rows);
    if (!team_exchange<CL>(g, m, tm, ++seq, pub)) return false;
  }
  // ---- back to global memory: T, maps and the active list (ascending ids)
  for (int l = tid; l < rows; l += nth) {
    const int r = l * tm.size + tm.rank;
    if (r < n0 && m.node[r] >= 0) s.T[r] = m.To[l];
  }
  if (tm.rank == 0) {
    for (int p = tid; p < n0; p += nth) {
      s.Tf[p] = m.Tf[p];
      s.node[p] = m.node[p];
      s.prow[p] = m.prow[p];
    }
    if (tid == 0) s.prow[n0] = spare;
    __shared__ int w_cnt[33];
    const int ids = n + step1, per = (ids + nth - 1) / nth;
    const int a0 = min(tid * per, ids), a1 = min(a0 + per, ids);
    int keep = 0;
    for (int v = a0; v < a1; ++v) keep += __ldcg(s.slot + v) >= 0;
    int incl = keep;
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) w_cnt[warp] = incl;
    __syncthreads();
    int off = incl - keep;
    for (int w = 0; w < warp; ++w) off += w_cnt[w];
    for (int v = a0; v < a1; ++v)
      if (__ldcg(s.slot + v) >= 0) s.act[off++] = v;
    if (tid == 0) *s.na = n - step1;
  }
  return true;
}

// Joins step0 .. step1-1 of an n-taxon job over the whole GPU (one cooperative
// launch between two rebuilds).
__global__ void __launch_bounds__(kLazyThreads, 1) nj_lazy_grid_kernel(NJDev s, GridNJ g, int step0, int step1, int n,
                                                                       int watermark) {
  extern __shared__ __align__(16) unsigned char smem[];
  if (*(volatile int*)g.abort) return;   // an earlier segment gave up: every CTA leaves
  const Team tm{(int)blockIdx.x, (int)gridDim.x};
  unsigned seq = 0, target = 0;
  lazy_segment<false>(s, g, tm, smem, step0, step1, n, watermark, seq, target);
}

// TreeNode::join (TreeNode.cpp:31-58) for a recorded join: L_i = (d + (T_i -
// T_j)/(n-2)) / 2, L_j likewise, n = 2 gives d/2 each, a negative side is
// clamped to 0 and moved to the other.
__device__ void join_lengths(nwg_join& J) {
  const double half = 0.5;
  double li, lj;
  if (J.n == 2) {
    li = lj = __dmul_rn((double)J.d, half);
  } else {
    const double nm2 = (double)(J.n - 2);
    li = __dmul_rn(half, __dadd_rn((double)J.d, __ddiv_rn(__dsub_rn(J.ti, J.tj), nm2)));
    lj = __dmul_rn(half, __dadd_rn((double)J.d, __ddiv_rn(__dsub_rn(J.tj, J.ti), nm2)));
  }
  if (li < 0.0) {
    lj = __dsub_rn(lj, li);
    li = 0.0;
  } else if (lj < 0.0) {
    li = __dsub_rn(li, lj);
    lj = 0.0;
  }
  J.len_i = li;
  J.len_j = lj;
}

__global__ void nj_lengths_kernel(nwg_join* joins, int count) {
  const int k = blockIdx.x * blockDim.x + threadIdx.x;
  if (k < count) join_lengths(joins[k]);
}

// Compaction, part 1 (one CTA): map[p] = new slot of live slot p (ascending),
// T / Tf / node into the new slots, slot[v] of every live node remapped.
__global__ void __launch_bounds__(1024) compact_map_kernel(NJDev s, int* map, double* T2, float* Tf2, int* node2,
                                                           int nslots, const int* abort) {
  if (*(volatile const int*)abort) return;
  __shared__ int wsum[33];
  const int n0 = s.n0;
  const int chunk = (n0 + blockDim.x - 1) / blockDim.x;
  const int p0 = threadIdx.x * chunk;
  int keep = 0;
  for (int p = p0; p < p0 + chunk && p < n0; ++p) keep += s.node[p] >= 0;
  int incl = keep;
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if ((threadIdx.x & 31) >= o) incl += y;
  }
  if ((threadIdx.x & 31) == 31) wsum[threadIdx.x >> 5] = incl;
  __syncthreads();
  if (threadIdx.x == 0) {
    int acc = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
      const int t = wsum[w];
      wsum[w] = acc;
      acc += t;
    }
    wsum[32] = acc;
  }
  __syncthreads();
  int q = wsum[threadIdx.x >> 5] + incl - keep;
  for (int p = p0; p < p0 + chunk && p < n0; ++p) {
    const int v = s.node[p];
    if (v >= 0) {
      map[p] = q;
      T2[q] = s.T[p];
      Tf2[q] = s.Tf[p];
      node2[q] = v;
      ++q;
    } else {
      map[p] = -1;
    }
  }
  __syncthreads();
  for (int v = threadIdx.x; v < nslots; v += blockDim.x) {
    const int p = s.slot[v];
    if (p >= 0) s.slot[v] = map[p];
  }
}

// Compaction, part 2: D2[map[p]][map[c]] = D[p][c] for live p, c (one block per old row).
__global__ void __launch_bounds__(256) compact_copy_kernel(NJDev s, const int* map, float* D2, int ld2,
                                                           const int* abort) {
  if (*(volatile const int*)abort) return;
  const int p = blockIdx.x;
  const int np = map[p];
  if (np < 0) return;
  const float* row = row_at(s, s.prow[p]);
  float* out = D2 + (size_t)np * ld2;
  for (int c = threadIdx.x; c < s.n0; c += blockDim.x) {
    const int nc = map[c];
    if (nc >= 0) out[nc] = row[c];
  }
}

// Every row of the compacted matrix at its slot's place.
__global__ void compact_rows_kernel(int* prow, int n0, const int* abort) {
  if (*(volatile const int*)abort) return;
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p <= n0) prow[p] = p;
}

// ---- one job per thread-block cluster ------------------------------------------
// The lazy search with the C CTAs of a cluster as the team; the exchange goes
// through distributed shared memory, and the reference's rebuild schedule runs
// inside the kernel (row sums over the cluster, no compaction: the matrix stays
// in L2).  Against holding the matrix in the cluster's shared memory and passing
// over all of it for every join (the form this replaced, up to 768 taxa): 2.31 ms
// instead of 2.81 for 400 taxa, 3.70 / 4.72 for 600; against a full pass over L2
// for every join, see the thresholds at cluster_nj_max_n.

struct NJJob {
  NJDev s;
  GridNJ g;
  int n;
  int pad;
};

// Sequential row sums (buildGblRowSums, SpeciesBlock.cpp:426-453) over the
// active list, one warp per row, warps w0, w0 + wstride, ...; the lanes'
// any-order sum is used when it is provably exact, else lane 0 sums in order.
__device__ void team_rowsums(const NJDev& s, const int* act, int w0, int wstride) {
  const int na = *s.na;
  const int lane = threadIdx.x & 31;
  for (int k = w0; k < na; k += wstride) {
    const int sk = s.slot[act[k]];
    const float* row = row_at(s, s.prow[sk]);
    double part = 0.0, ab = 0.0;
    int lowexp = INT_MAX;
    for (int j = lane; j < na; j += 32) {
      const float x = row[s.slot[act[j]]];
      part = __dadd_rn(part, (double)x);
      ab = __dadd_rn(ab, (double)fabsf(x));
      lowexp = min(lowexp, low_bit_exp(x));
    }
    for (int o = 16; o > 0; o >>= 1) {
      part = __dadd_rn(part, __shfl_down_sync(0xffffffffu, part, o));
      ab = __dadd_rn(ab, __shfl_down_sync(0xffffffffu, ab, o));
      lowexp = min(lowexp, __shfl_down_sync(0xffffffffu, lowexp, o));
    }
    if (lane == 0) {
      double sum = part;
      if (!sum_is_exact(ab, lowexp)) {
        sum = 0.0;
        for (int j = 0; j < na; ++j) sum = __dadd_rn(sum, (double)row[s.slot[act[j]]]);
      }
      s.T[sk] = sum;
      s.Tf[sk] = __double2float_rn(sum);
    }
  }
}

template <int C, int Threads>
__global__ void __cluster_dims__(C, 1, 1) __launch_bounds__(Threads, 1) nj_cluster_kernel(const NJJob* jobs,
                                                                                              int njobs) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ NJJob sjob;   // the job's descriptor (shared memory keeps registers free)
  const int job = (int)blockIdx.x / C;   // the same for every CTA of the cluster
  if (job >= njobs) return;
  if (threadIdx.x == 0) sjob = jobs[job];
  __syncthreads();
  const NJDev& s = sjob.s;
  const GridNJ& g = sjob.g;
  const int n = sjob.n;
  const Team tm{(int)cooperative_groups::this_cluster().block_rank(), C};
  const int w0 = tm.rank * (int)(blockDim.x >> 5) + (int)(threadIdx.x >> 5);
  const int wstride = C * (int)(blockDim.x >> 5);
  const int t0 = tm.rank * (int)blockDim.x + (int)threadIdx.x, tstride = C * (int)blockDim.x;
  unsigned seq = 0, target = 0;
  for (int k = t0; k < 2 * n - 1; k += tstride) s.slot[k] = k < n ? k : -1;
  for (int k = t0; k < n; k += tstride) {
    s.node[k] = k;
    s.act[k] = k;
  }
  for (int k = t0; k <= n; k += tstride) s.prow[k] = k;
  if (tm.rank == 0 && threadIdx.x == 0) {
    *s.na = n;
    s.stats[0] = s.stats[1] = s.stats[2] = s.stats[3] = s.stats[4] = 0;
  }
  cooperative_groups::this_cluster().sync();
  if (n < 2) return;
  team_rowsums(s, s.act, w0, wstride);
  cooperative_groups::this_cluster().sync();
  // the reference's schedule (SpeciesBlock.cpp:864, :1206-1247)
  const int kBinT = 30 * 31 / 2;
  int steps = max((int)((float)n * 0.5f), 200);
  int pq_ck = 500;
  long long ave0 = (((long long)(n - 1) * n) / 2) / kBinT;
  long long ub = ((long long)n * (n - 1)) / 2;
  int watermark = n;
  for (int step = 0; step < n - 1;) {
    const int seg_end = steps == INT_MAX ? n - 1 : min(n - 1, step + steps + 1);
    const bool ok = lazy_segment<true>(s, g, tm, smem, step, seg_end, n, watermark, seq, target);
    cooperative_groups::this_cluster().sync();   // the state is back in global memory; no CTA writes another's memory
    if (!ok) return;
    bool rebuild = false;
    for (; step < seg_end; ++step) {
      if (--pq_ck == 0) {
        pq_ck = 500;
        if (steps > 0 && (double)(ub / kBinT) / (double)ave0 > 2.0 && tm.rank == 0 && threadIdx.x == 0) s.stats[3] += 1;
      }
      const int m_after = n - step - 1;
      if (steps == 0) {
        rebuild = true;
      } else {
        if (steps != INT_MAX) --steps;
        ub += m_after - 1;
      }
    }
    if (rebuild) {
      const int m_after = n - step;
      team_rowsums(s, s.act, w0, wstride);
      if (tm.rank == 0 && threadIdx.x == 0) s.stats[4] += 1;
      watermark = n + step;
      steps = (m_after < 200) ? INT_MAX : (int)((float)m_after * 0.5f);
      ave0 = (((long long)(m_after - 1) * m_after) / 2) / kBinT;
      ub = ((long long)m_after * (m_after - 1)) / 2;
      cooperative_groups::this_cluster().sync();
    }
  }
  for (int k = t0; k < n - 1; k += tstride) join_lengths(s.joins[k]);
}

// ---- small jobs: the whole join loop in one CTA ----------------------------
// Up to kCtaNJMax taxa one CTA holds the job in its shared memory: the rows,
// T, the float row sums, the maps and the active lists.  A thread scans its
// own folded row pair sequentially (no per-row warp reduction), and every
// phase boundary is a CTA barrier; the new node's row sum is complete when the
// join share's block reduction is.  The arithmetic is that of the other forms.

constexpr int kCtaNJMax = 160;       // at most: shared memory
// Up to here the CTA is faster than a cluster, whose join costs nearly the same at
// any small size.  Whole-number distances, ms (CTA / cluster): 0.79 / 0.71 at 137
// taxa, 0.88 / 0.77 at 150, 1.03 / 0.82 at 160; points on a line 0.72 / 0.74, 0.79 /
// 0.80, 0.98 / 0.85.
constexpr int kCtaNJDefault = 136;
constexpr int kCtaThreads = 256;

struct CtaLayout {
  int ldl;
  size_t rows, tf, t, node, slot, act_a, act_b, grm, grc, tv, bytes;
};

__host__ __device__ inline CtaLayout cta_layout(int n) {
  auto al = [](size_t x) { return (x + 15) / 16 * 16; };
  CtaLayout L;
  L.ldl = (n + 3) & ~3;
  size_t o = 0;
  L.rows = o; o += al(sizeof(float) * (size_t)n * L.ldl);
  L.tf = o; o += al(sizeof(float) * L.ldl);
  L.t = o; o += al(sizeof(double) * n);
  L.node = o; o += al(sizeof(int) * n);
  L.slot = o; o += al(sizeof(int) * 2 * n);
  L.act_a = o; o += al(sizeof(int) * (n + 1));
  L.act_b = o; o += al(sizeof(int) * (n + 1));
  L.grm = o; o += al(sizeof(int) * n);
  L.grc = o; o += al(sizeof(int4) * n);
  L.tv = o; o += al(sizeof(float) * n);
  L.bytes = o;
  return L;
}

// Block-wide reduction of a USum over kCtaThreads threads (result in thread 0).
__device__ __forceinline__ USum cta_usum(USum x, USum* swarp) {
  usum_warp(x);
  if ((threadIdx.x & 31) == 0) swarp[threadIdx.x >> 5] = x;
  __syncthreads();
  if (threadIdx.x == 0)
    for (int w = 1; w < kCtaThreads / 32; ++w) usum_add(x, swarp[w]);
  return x;
}

__global__ void __launch_bounds__(kCtaThreads, 1) nj_cta_kernel(const NJJob* jobs, int njobs) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ NJJob sjob;
  __shared__ float wq[kCtaThreads / 32], wm[kCtaThreads / 32];
  __shared__ USum swarp[kCtaThreads / 32];
  __shared__ int rows_sel[kFastRows];
  __shared__ GCand fc[kFastRows];
  __shared__ int nsel, s_ok;
  __shared__ PickOut spick;
  __shared__ GCand swin;
  __shared__ float sthr;
  __shared__ bool s_wide;   // floats do not hold this join's q: every live pair is looked at, exactly
  if ((int)blockIdx.x >= njobs) return;
  if (threadIdx.x == 0) sjob = jobs[blockIdx.x];
  __syncthreads();
  const NJDev& s = sjob.s;
  const int n = sjob.n;
  const CtaLayout L = cta_layout(n);
  const int ldl = L.ldl;
  float* rows = reinterpret_cast<float*>(smem + L.rows);
  float* Tf = reinterpret_cast<float*>(smem + L.tf);
  double* T = reinterpret_cast<double*>(smem + L.t);
  int* node = reinterpret_cast<int*>(smem + L.node);
  int* slot = reinterpret_cast<int*>(smem + L.slot);
  int* act = reinterpret_cast<int*>(smem + L.act_a);
  int* act2 = reinterpret_cast<int*>(smem + L.act_b);
  int* grm = reinterpret_cast<int*>(smem + L.grm);
  int4* grc = reinterpret_cast<int4*>(smem + L.grc);
  float* tv = reinterpret_cast<float*>(smem + L.tv);
  const int tid = (int)threadIdx.x, nth = kCtaThreads;
  const int lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < n * ldl; e += nth) {
    const int r = e / ldl, c = e - r * ldl;
    rows[e] = c < n ? s.D[(size_t)r * s.ld + c] : 0.f;
  }
  for (int k = tid; k < ldl; k += nth) Tf[k] = __int_as_float(0x7FC00000);
  for (int k = tid; k < 2 * n; k += nth) slot[k] = k < n ? k : -1;
  for (int k = tid; k < n; k += nth) {
    node[k] = k;
    act[k] = k;
  }
  if (tid == 0) {
    s.stats[0] = s.stats[1] = s.stats[2] = s.stats[3] = s.stats[4] = 0;
  }
  __syncthreads();
  // row sums (buildGblRowSums): a thread per row, the reference's sequential
  // double sum over the active list in ascending id order
  auto rowsums = [&](int na) {
    for (int k = tid; k < na; k += nth) {
      const int r = slot[act[k]];
      const float* row = rows + (size_t)r * ldl;
      double sum = 0.0;
      for (int j = 0; j < na; ++j) sum = __dadd_rn(sum, (double)row[slot[act[j]]]);
      T[r] = sum;
      Tf[r] = __double2float_rn(sum);
    }
    __syncthreads();
  };
  if (n >= 2) rowsums(n);
  const int kBinT = 30 * 31 / 2;
  int steps = max((int)((float)n * 0.5f), 200);
  int pq_ck = 500;
  long long ave0 = (((long long)(n - 1) * n) / 2) / kBinT;
  long long ub = ((long long)n * (n - 1)) / 2;
  int watermark = n;
  const int npairs = (n + 1) / 2;
  for (int step = 0; step < n - 1; ++step) {
    const int m_n = n - step, next = n + step;
    const float nm2f = (float)(m_n - 2);
    const double nm2 = (double)(m_n - 2);
    // ---- pass: a thread per folded row pair, its rows scanned sequentially
    float qmin = FLT_MAX, mmax = 0.f;
    if (tid < npairs) {
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        const int r = h ? n - 1 - tid : tid;
        if (h && r == tid) break;
        const float tr = Tf[r];
        if (tr != tr) {   // dead
          grm[r] = kNoPair;
          continue;
        }
        const float* row = rows + (size_t)r * ldl;
        float m1 = FLT_MAX, m2 = FLT_MAX, mag = 0.f;
        int c1 = -1;
        // columns r+1 .. up to the next multiple of 4 one by one, then 16-byte
        // vectors (rows padded to ldl floats, the padding's row sums NaN)
        const int v0 = (r + 4) >> 2;
        for (int c = r + 1; c < 4 * v0 && c < n; ++c) pass_elem(row[c], Tf[c], c, tr, nm2f, m1, m2, c1, mag);
        const float4* row4 = reinterpret_cast<const float4*>(row);
        const float4* Tf4 = reinterpret_cast<const float4*>(Tf);
#pragma unroll 2
        for (int v = v0; v < (ldl >> 2); ++v) {
          const float4 d = row4[v];
          const float4 tc = Tf4[v];
          pass_elem(d.x, tc.x, 4 * v, tr, nm2f, m1, m2, c1, mag);
          pass_elem(d.y, tc.y, 4 * v + 1, tr, nm2f, m1, m2, c1, mag);
          pass_elem(d.z, tc.z, 4 * v + 2, tr, nm2f, m1, m2, c1, mag);
          pass_elem(d.w, tc.w, 4 * v + 3, tr, nm2f, m1, m2, c1, mag);
        }
        grm[r] = ford(m1);
        grc[r] = make_int4(ford(m2), c1, __float_as_int(c1 >= 0 ? row[c1] : 0.f), 0);
        qmin = fminf(qmin, m1);
        mmax = fmaxf(mmax, __fadd_rn(mag, fabsf(tr)));
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      qmin = fminf(qmin, __shfl_xor_sync(0xffffffffu, qmin, o));
      mmax = fmaxf(mmax, __shfl_xor_sync(0xffffffffu, mmax, o));
    }
    if (lane == 0) {
      wq[warp] = qmin;
      wm[warp] = mmax;
    }
    __syncthreads();
    if (tid == 0) {
      float q = FLT_MAX, mm = 0.f;
      for (int w = 0; w < nth / 32; ++w) {
        q = fminf(q, wq[w]);
        mm = fmaxf(mm, wm[w]);
      }
      sthr = q + 3.f * (8.f * 5.9604645e-8f * mm) + 1e-30f;
      s_wide = !(mm <= kFloatTop);
      nsel = 0;
    }
    __syncthreads();
    // ---- pick
    const float thr = sthr;
    const bool wide = s_wide;
    const int othr = ford(thr);
    for (int r = tid; r < n; r += nth) {
      if (grm[r] <= othr && grm[r] != kNoPair) {
        const int k = atomicAdd(&nsel, 1);
        if (k < kFastRows) rows_sel[k] = r;
      }
    }
    __syncthreads();
    const int nr = nsel;
    if (warp == 0) {
      int ok = nr >= 1 && nr <= kFastRows && !wide;
      if (ok && lane < nr) {
        const int r = rows_sel[lane];
        const int4 rec = grc[r];
        const int c = rec.y;
        if (rec.x <= othr || c < 0) {
          ok = 0;   // a second pair of the row within the threshold
        } else {
          fc[lane] = make_cand(r, c, node[r], node[c], T[r], T[c], __int_as_float(rec.z), nm2, watermark);
        }
      }
      ok = __all_sync(0xffffffffu, ok);
      PickOut pr{};
      if (ok && nr == 1) {
        pr.idx = 0;
        pr.ties = 1;
        pr.amb = 0;
        pr.error = false;
      } else if (ok) {
        pr = pick_keys(nr, [&](int k) { return fc[k]; });
      }
      if (lane == 0) {
        s_ok = ok;
        if (ok) {
          spick = pr;
          swin = fc[pr.idx];
        }
      }
    }
    __syncthreads();
    if (!s_ok) {
      // fallback: the selected rows' pairs within the threshold, scanned
      // twice: the first candidate in the pick's order (block reduction),
      // then the ties and ambiguous pairs against it (pick_keys' rule)
      auto scan = [&](auto&& visit, auto&& go_on) {
        for (int r = 0; r < n; ++r) {
          if (!(wide || grm[r] <= othr) || node[r] < 0) continue;
          if (!go_on()) break;
          const int ur = node[r];
          const float tr = Tf[r];
          const float* row = rows + (size_t)r * ldl;
          for (int c = r + 1 + tid; c < n; c += nth) {
            const int uc = node[c];
            if (uc < 0) continue;
            const float d = row[c];
            const float q = __fsub_rn(__fsub_rn(__fmul_rn(d, nm2f), tr), Tf[c]);
            if (!wide && !(q <= thr)) continue;
            const GCand cd = make_cand(r, c, ur, uc, T[r], T[c], d, nm2, watermark);
            if (wide && !(cd.q1 < DBL_MAX)) continue;
            visit(kc_of(cd));
          }
        }
      };
      __shared__ KCand skw[32];
      __shared__ KCand sfirst;
      __shared__ unsigned scnt[2];
      KCand first = kc_none();
      scan([&](const KCand& c) {
        if (kc_first(c, first)) first = c;
      }, [] { return true; });
      first = cta_first(first, skw);
      if (tid == 0) {
        sfirst = first;
        scnt[0] = scnt[1] = 0;
      }
      __syncthreads();
      const KCand wk = sfirst;
      unsigned ties = 0, amb = 0;
      // one ambiguous pair, or five ties, decide the step's statistics
      if (wk.b >= 0)
        scan([&](const KCand& c) { count_vs(c, wk, ties, amb); },
             [&] { return !__any_sync(0xffffffffu, amb) && __popc(__ballot_sync(0xffffffffu, ties)) <= 4; });
      for (int o = 16; o > 0; o >>= 1) {
        ties += __shfl_xor_sync(0xffffffffu, ties, o);
        amb += __shfl_xor_sync(0xffffffffu, amb, o);
      }
      if (lane == 0 && (ties | amb)) {
        atomicAdd(&scnt[0], ties);
        atomicAdd(&scnt[1], amb);
      }
      __syncthreads();
      if (tid == 0) {
        spick.idx = 0;
        spick.ties = scnt[0];
        spick.amb = scnt[1];
        spick.error = wk.b < 0;
        if (!spick.error) {
          // the winner's pair again, as the scan read it (row = the smaller slot)
          const int sa = slot_of(wk.a), sb = slot_of(wk.b);
          const int r0 = min(sa, sb), c0 = max(sa, sb);
          swin = make_cand(r0, c0, node[r0], node[c0], T[r0], T[c0], rows[(size_t)r0 * ldl + c0], nm2, watermark);
        }
      }
      __syncthreads();
      if (spick.error) {
        if (tid == 0) record_pick(s, spick);
        break;
      }
    }
    // ---- join share: a thread per slot
    const GCand w = swin;
    const int i = w.a, j = w.b, si = w.sa, sj = w.sb;
    USum x;
    x.u = x.a = 0;
    x.e = INT_MAX;
    x.t = INT_MIN;
    for (int p = tid; p < n; p += nth) {
      if (node[p] < 0 || p == si || p == sj) continue;
      float* row = rows + (size_t)p * ldl;
      const float sumf = __fadd_rn(row[si], row[sj]);
      const float tmp = __fmul_rn(__fsub_rn(sumf, w.d), 0.5f);
      const double t = __dadd_rn(T[p], (double)__fsub_rn(tmp, sumf));
      T[p] = t;
      Tf[p] = __double2float_rn(t);
      row[si] = tmp;
      rows[(size_t)si * ldl + p] = tmp;
      tv[p] = tmp;
      if (tmp != 0.f) {
        USum y;
        y.e = low_bit_exp(tmp);
        y.t = top_bit_exp(tmp);
        y.u = float_units(tmp, y.e);
        y.a = y.u < 0 ? -y.u : y.u;
        usum_add(x, y);
      }
    }
    for (int k = tid; k < m_n; k += nth) {
      const int v = act[k];
      if (v != i && v != j) act2[k - (v > i) - (v > j)] = v;
    }
    x = cta_usum(x, swarp);   // ends with every thread past the share
    if (tid == 0) {
      double sum;
      if (x.e == INT_MAX) {
        sum = 0.0;
      } else if (x.t - x.e < 48 && x.a < (1ll << 53) && x.t < 128) {   // 128: infinite or undefined
        sum = units_to_double(x.u, x.e);   // exact: the sequential sum's value
      } else {
        sum = 0.0;   // the reference's loop: active ids ascending, i and j skipped
        for (int k = 0; k < m_n; ++k) {
          const int v = act[k];
          if (v != i && v != j) sum = __dadd_rn(sum, (double)tv[slot[v]]);
        }
      }
      T[si] = sum;
      Tf[si] = __double2float_rn(sum);
      Tf[sj] = __int_as_float(0x7FC00000);
      node[sj] = -1;
      node[si] = next;
      slot[j] = -1;
      slot[i] = -1;
      slot[next] = si;
      act2[m_n - 2] = next;
      nwg_join& J = s.joins[step];
      J.i = i;
      J.j = j;
      J.node = next;
      J.n = m_n;
      J.d = w.d;
      J.pad = 0.f;
      J.q = w.q1;
      J.ti = w.ta;
      J.tj = w.tb;
      record_pick(s, spick);
    }
    {
      int* t = act;
      act = act2;
      act2 = t;
    }
    // ---- the reference's rebuild schedule (SpeciesBlock.cpp:864, :1206-1247)
    if (--pq_ck == 0) {
      pq_ck = 500;
      if (steps > 0 && (double)(ub / kBinT) / (double)ave0 > 2.0 && tid == 0) s.stats[3] += 1;
    }
    const int m_after = m_n - 1;
    __syncthreads();
    if (steps == 0) {
      rowsums(m_after);
      if (tid == 0) s.stats[4] += 1;
      watermark = next + 1;
      steps = (m_after < 200) ? INT_MAX : (int)((float)m_after * 0.5f);
      ave0 = (((long long)(m_after - 1) * m_after) / 2) / kBinT;
      ub = ((long long)m_after * (m_after - 1)) / 2;
    } else {
      --steps;
      ub += m_after - 1;
    }
  }
  __syncthreads();
  for (int k = tid; k < n - 1; k += nth) join_lengths(s.joins[k]);
}

}  // namespace

struct NJState {
  DevBuf D, jobws, desc;
  // whole-GPU form: row sums, maps, compaction buffers, candidates, exchanges and barrier words
  DevBuf T, Tf, slot, node, act, na, g32, stats, joins, cand, cbest;
  DevBuf D2, T2, Tf2, node2, map, prow, xrow, tx, gather, gbar;
  ~NJState() {
    for (DevBuf* b : {&D, &jobws, &desc, &T, &Tf, &slot, &node, &act, &na, &g32, &stats, &joins, &cand, &cbest, &D2, &T2,
                      &Tf2, &node2, &map, &prow, &xrow, &tx, &gather, &gbar})
      b->release();
  }
};

// Up to this many taxa one cluster runs the whole join loop; larger matrices
// take the whole GPU.  A cluster's exchange is the cheaper one, the whole GPU
// has fewer rows to rescan per CTA: 5.5 us a join in the cluster at 500 taxa, 5.8 at
// 600, 6.2 on the whole GPU at 650 to 1,000.  The
// environment variable NWG_NJ_CLUSTER_MAX_N overrides the threshold (both forms
// give the same joins; the tests run each form on the same inputs).
int cluster_nj_max_n() {
  static const int v = [] {
    const char* e = std::getenv("NWG_NJ_CLUSTER_MAX_N");
    return e ? std::atoi(e) : 600;
  }();
  return v;
}

void Ctx::nj_release() {
  delete reinterpret_cast<NJState*>(nj_state);
  nj_state = nullptr;
}

int Ctx::nj(const float* D, int64_t ld, int n, bool device_D, nwg_join* joins, nwg_nj_stats* st) {
  if (n < 1 || !D || ld < n || (!joins && n > 1)) return fail(NWG_ERR_INVALID, "nj arguments");
  if (n > kNJMaxN) return fail(NWG_ERR_INVALID, "neighbor joining on the device supports n <= 8192");
  nwg_nj_stats stats;
  std::memset(&stats, 0, sizeof(stats));
  if (n == 1) {
    stats.reference_identical = 1;
    if (st) *st = stats;
    return NWG_OK;
  }
  if (!nj_state) nj_state = new NJState();
  NJState& S = *reinterpret_cast<NJState*>(nj_state);
  const int nn = 2 * n - 1;
  const bool big = n > cluster_nj_max_n();
  const int ldd = nj_row_stride(n);   // rows padded to a multiple of 4 floats (16-byte loads)
  int rc;
  if ((rc = S.D.ensure(sizeof(float) * (size_t)n * ldd))) return fail(rc, "nj allocation");
  cudaStream_t s = stream;
  const cudaMemcpyKind kind = device_D ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
  if ((rc = cuda(cudaMemcpy2DAsync(S.D.p, sizeof(float) * ldd, D, sizeof(float) * ld, sizeof(float) * n, n, kind, s),
                 "nj upload")))
    return rc;
  const void* jsrc;   // join records and statistics on the device
  const void* ssrc;
  if (!big) {
    if ((rc = S.jobws.ensure(nj_job_workspace(n))) || (rc = S.desc.ensure(sizeof(NJJob))))
      return fail(rc, "nj allocation");
    NJJob J{};
    nwg_join* jp;
    unsigned long long* sp;
    nj_job_setup(&J, (float*)S.D.p, n, ldd, (char*)S.jobws.p, &jp, &sp);
    jsrc = jp;
    ssrc = sp;
    // the descriptor travels in the stream (a pageable copy is staged at once)
    if ((rc = cuda(cudaMemcpyAsync(S.desc.p, &J, sizeof(J), cudaMemcpyHostToDevice, s), "nj upload"))) return rc;
    if (st) cudaEventRecord(ev0, s);
    if ((rc = cuda(n <= cta_nj_max_n() ? launch_nj_cta(S.desc.p, 1, n, s)
                                       : launch_nj_cluster(S.desc.p, 1, n, nj_cluster_size(), sms, true, s),
                   "nj launch")))
      return rc;
    ++launches;
  } else {
    // one CTA per SM (cooperative launch)
    const int grid = std::min(sms, kLazyMaxCtas);
    if ((rc = S.T.ensure(sizeof(double) * n)) || (rc = S.Tf.ensure(sizeof(float) * ldd)) ||
        (rc = S.slot.ensure(sizeof(int) * nn)) || (rc = S.node.ensure(sizeof(int) * n)) ||
        (rc = S.act.ensure(sizeof(int) * (n + 1))) || (rc = S.na.ensure(sizeof(int))) ||
        (rc = S.g32.ensure(sizeof(int) * 8)) || (rc = S.stats.ensure(sizeof(unsigned long long) * 5)) ||
        (rc = S.joins.ensure(sizeof(nwg_join) * (n - 1))) || (rc = S.cand.ensure(sizeof(KCand) * kCandCap)) ||
        (rc = S.cbest.ensure(sizeof(KCand) * grid)) || (rc = S.D2.ensure(sizeof(float) * (size_t)n * ldd)) ||
        (rc = S.T2.ensure(sizeof(double) * n)) || (rc = S.Tf2.ensure(sizeof(float) * ldd)) ||
        (rc = S.node2.ensure(sizeof(int) * n)) || (rc = S.map.ensure(sizeof(int) * n)) ||
        (rc = S.prow.ensure(sizeof(int) * (n + 1))) || (rc = S.xrow.ensure(sizeof(float) * ldd)) ||
        (rc = S.tx.ensure(sizeof(double) * 2 * n)) ||
        (rc = S.gather.ensure(sizeof(float4) * 2 * grid)) || (rc = S.gbar.ensure(sizeof(int) * 4)))
      return fail(rc, "nj allocation");
    NJDev d{};
    d.D = (float*)S.D.p;
    d.T = (double*)S.T.p;
    d.Tf = (float*)S.Tf.p;
    d.slot = (int*)S.slot.p;
    d.node = (int*)S.node.p;
    d.act = (int*)S.act.p;
    d.na = (int*)S.na.p;
    d.g32 = (int*)S.g32.p;
    d.stats = (unsigned long long*)S.stats.p;
    d.joins = (nwg_join*)S.joins.p;
    d.prow = (int*)S.prow.p;
    d.xrow = (float*)S.xrow.p;
    d.tx = (double*)S.tx.p;
    d.n0 = n;
    d.ld = ldd;
    d.cand_cap = kCandCap;
    jsrc = S.joins.p;
    ssrc = S.stats.p;
    std::vector<int> slot0(nn, -1), act0(n + 1, n);   // act0: the identity, for the lists and maps
    for (int k = 0; k < n; ++k) slot0[k] = k, act0[k] = k;
    const int na0 = n;
    if ((rc = cuda(cudaMemcpyAsync(S.slot.p, slot0.data(), sizeof(int) * nn, cudaMemcpyHostToDevice, s), "nj upload")) ||
        (rc = cuda(cudaMemcpyAsync(S.node.p, act0.data(), sizeof(int) * n, cudaMemcpyHostToDevice, s), "nj upload")) ||
        (rc = cuda(cudaMemcpyAsync(S.act.p, act0.data(), sizeof(int) * (n + 1), cudaMemcpyHostToDevice, s), "nj upload")) ||
        (rc = cuda(cudaMemcpyAsync(S.prow.p, act0.data(), sizeof(int) * (n + 1), cudaMemcpyHostToDevice, s), "nj upload")) ||
        (rc = cuda(cudaMemcpyAsync(S.na.p, &na0, sizeof(int), cudaMemcpyHostToDevice, s), "nj upload")) ||
        (rc = cuda(cudaMemsetAsync(S.stats.p, 0, sizeof(unsigned long long) * 5, s), "nj upload")) ||
        (rc = cuda(cudaStreamSynchronize(s), "nj upload")))   // the host vectors above are local
      return rc;
    const int smem = (int)lazy_layout(n, ldd, grid).bytes;   // the first segment's: later ones have fewer slots
    int blocks_per_sm = 0;
    if ((rc = cuda(allow_smem((const void*)nj_lazy_grid_kernel), "nj occupancy")) ||
        (rc = cuda(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks_per_sm, nj_lazy_grid_kernel, kLazyThreads, smem),
                   "nj occupancy")))
      return rc;
    if (blocks_per_sm < 1) return fail(NWG_ERR_CUDA, "neighbor-joining grid kernel does not fit");
    float* Dalt = (float*)S.D2.p;
    double* Talt = (double*)S.T2.p;
    float* Tfalt = (float*)S.Tf2.p;
    int* nodealt = (int*)S.node2.p;
    GridNJ g{};
    g.bar = (unsigned*)S.gbar.p;
    g.abort = (int*)S.gbar.p + 2;
    g.gather = (float4*)S.gather.p;
    g.cbest = (KCand*)S.cbest.p;
    g.cand = (KCand*)S.cand.p;
    // NaN (all bits set) float row sums at the padding slots; rowsum_kernel
    // fills the live ones
    if ((rc = cuda(cudaMemsetAsync(S.gbar.p, 0, sizeof(int) * 4, s), "nj upload")) ||
        (rc = cuda(cudaMemsetAsync(S.Tf.p, 0xFF, sizeof(float) * ldd, s), "nj upload")))
      return rc;
    if (st) cudaEventRecord(ev0, s);
    rowsum_kernel<<<(n + 7) / 8, 256, 0, s>>>(d, g.abort);
    ++launches;
    // The reference's schedule (deterministic in n): rebuild after
    // max(n*0.5, 200) joins, then every m*0.5 joins, none below 200 active
    // nodes; the joins between two rebuilds are one cooperative launch.
    const int kBinT = 30 * 31 / 2;
    int steps = std::max((int)((float)n * 0.5f), 200);
    int pq_ck = 500;
    long long ave0 = (((long long)(n - 1) * n) / 2) / kBinT;
    long long ub = ((long long)n * (n - 1)) / 2;
    int watermark = n, m_n = n;
    // compaction to the live slots, in slot order (every slot comparison of
    // the record-order rounding is unchanged, so it may run at any step)
    auto compact = [&](int na) -> int {
      const int ld2 = (na + 3) & ~3;
      int e;
      if ((e = cuda(cudaMemsetAsync(Tfalt, 0xFF, sizeof(float) * ld2, s), "nj launch"))) return e;
      compact_map_kernel<<<1, 1024, 0, s>>>(d, (int*)S.map.p, Talt, Tfalt, nodealt, nn, g.abort);
      compact_copy_kernel<<<d.n0, 256, 0, s>>>(d, (const int*)S.map.p, Dalt, ld2, g.abort);
      compact_rows_kernel<<<(na + 256) / 256, 256, 0, s>>>(d.prow, na, g.abort);
      launches += 3;
      std::swap(d.D, Dalt);
      std::swap(d.T, Talt);
      std::swap(d.Tf, Tfalt);
      std::swap(d.node, nodealt);
      d.n0 = na;
      d.ld = ld2;
      return NWG_OK;
    };
    int step = 0;
    while (step < n - 1) {
      // the segment ends with the join after which the countdown reaches 0
      const int sched_end = steps == INT_MAX ? n - 1 : std::min(n - 1, step + steps + 1);
      const int seg_end = d.n0 >= kCompactN ? std::min(sched_end, step + d.n0 / kCompactPart) : sched_end;
      if ((rc = cuda(cudaMemsetAsync(S.gbar.p, 0, sizeof(unsigned) * 2, s), "nj launch"))) return rc;
      // failure injection for the tests (NWG_NJ_INJECT_BARRIER_STALL=1): in the
      // first segment the first CTA never publishes, so the first exchange never
      // completes and every CTA gives up after the spin limit
      const char* inject = std::getenv("NWG_NJ_INJECT_BARRIER_STALL");
      g.stall = step == 0 && inject && std::atoi(inject) == 1 ? 1 : 0;
      {
        int a0 = step, a1 = seg_end, an = n, aw = watermark;
        const int threads = lazy_threads(d.ld, (d.n0 + grid - 1) / grid, grid, true);
        void* args[] = {&d, &g, &a0, &a1, &an, &aw};
        if ((rc = cuda(cudaLaunchCooperativeKernel((const void*)nj_lazy_grid_kernel, dim3(grid), dim3(threads), args,
                                                   (size_t)smem, s),
                       "nj launch")))
          return rc;
        ++launches;
      }
      bool rebuild = false;
      for (; step < seg_end; ++step) {
        if (--pq_ck == 0) {
          pq_ck = 500;
          if (steps > 0) {
            const double r = (double)(ub / kBinT) / (double)ave0;
            if (r > 2.0) ++stats.pq_trigger_open;
          }
        }
        --m_n;
        if (steps == 0) {
          rebuild = true;
        } else {
          if (steps != INT_MAX) --steps;
          ub += m_n - 1;
        }
      }
      if (rebuild) {
        rowsum_kernel<<<(m_n + 7) / 8, 256, 0, s>>>(d, g.abort);
        ++launches;
        if ((rc = compact(m_n))) return rc;
        ++stats.rebuilds;
        watermark = n + step;
        steps = (m_n < 200) ? INT_MAX : (int)((float)m_n * 0.5f);
        ave0 = (((long long)(m_n - 1) * m_n) / 2) / kBinT;
        ub = ((long long)m_n * (m_n - 1)) / 2;
      } else if (step < n - 1 && (rc = compact(m_n))) {
        return rc;
      }
      if ((rc = cuda(cudaGetLastError(), "nj launch"))) return rc;
    }
    nj_lengths_kernel<<<(n - 1 + 255) / 256, 256, 0, s>>>(d.joins, n - 1);
    ++launches;
    if ((rc = cuda(cudaGetLastError(), "nj launch"))) return rc;
  }
  if (st) cudaEventRecord(ev1, s);
  unsigned long long dst[5] = {0, 0, 0, 0, 0};
  if ((rc = cuda(cudaMemcpyAsync(joins, jsrc, sizeof(nwg_join) * (n - 1), cudaMemcpyDeviceToHost, s), "nj download")) ||
      (rc = cuda(cudaMemcpyAsync(dst, ssrc, sizeof(dst), cudaMemcpyDeviceToHost, s), "nj download")) ||
      (rc = cuda(cudaStreamSynchronize(s), "nj sync")))
    return rc;
  if (dst[2]) return fail(NWG_ERR_CUDA, "neighbor joining candidate list empty or overflowing");
  if (big) {
    int gb[4];
    if ((rc = cuda(cudaMemcpy(gb, S.gbar.p, sizeof(gb), cudaMemcpyDeviceToHost), "nj download"))) return rc;
    if (gb[2] == kAbortWait) return fail(NWG_ERR_CUDA, "neighbor-joining grid barrier timed out");
  }
  stats.ambiguous_steps = (int64_t)dst[0];
  stats.tie_steps = (int64_t)dst[1];
  if (!big) {
    stats.pq_trigger_open = (int64_t)dst[3];
    stats.rebuilds = (int64_t)dst[4];
  }
  stats.reference_identical = stats.ambiguous_steps == 0 && stats.pq_trigger_open == 0;
  if (st) {
    float ms = 0;
    cudaEventElapsedTime(&ms, ev0, ev1);
    stats.device_ms = ms;
    *st = stats;
  }
  return NWG_OK;
}

// Workspace of one job of the cluster forms, laid out from `base` (256-byte
// aligned pieces); fills *J when given.  The job's matrix is separate (n rows
// of ld floats, ld a multiple of 4; the cluster form modifies it in place, the
// one-CTA form only reads it).
static size_t job_layout(int n, int ld, char* base, NJJob* J) {
  auto al = [](size_t x) { return (x + 255) / 256 * 256; };
  const size_t cap = std::min<size_t>(kCandCap, (size_t)n * (n - 1) / 2 + 1);
  constexpr int kC = 16;   // the largest cluster
  size_t off = 0;
  auto take = [&](size_t bytes) {
    char* q = base ? base + off : nullptr;
    off += al(bytes);
    return q;
  };
  char* T = take(sizeof(double) * n);
  char* Tf = take(sizeof(float) * ld);
  char* slot = take(sizeof(int) * (2 * n));
  char* node = take(sizeof(int) * n);
  char* act = take(sizeof(int) * (n + 1));
  char* na = take(sizeof(int) * 4);
  char* g32 = take(sizeof(int) * 8);
  char* stats = take(sizeof(unsigned long long) * 5);
  char* cand = take(sizeof(KCand) * cap);
  char* cbest = take(sizeof(KCand) * kC);
  char* joins = take(sizeof(nwg_join) * (n > 1 ? n - 1 : 1));
  char* prow = take(sizeof(int) * (n + 1));
  char* xrow = take(sizeof(float) * ld);
  char* tx = take(sizeof(double) * 2 * n);
  if (J) {
    J->s.prow = (int*)prow;
    J->s.xrow = (float*)xrow;
    J->s.tx = (double*)tx;
    J->s.T = (double*)T;
    J->s.Tf = (float*)Tf;
    J->s.slot = (int*)slot;
    J->s.node = (int*)node;
    J->s.act = (int*)act;
    J->s.na = (int*)na;
    J->s.g32 = (int*)g32;
    J->s.stats = (unsigned long long*)stats;
    J->s.joins = (nwg_join*)joins;
    J->s.n0 = n;
    J->s.ld = ld;
    J->s.cand_cap = (int)cap;
    J->g.cand = (KCand*)cand;
    J->g.cbest = (KCand*)cbest;
    J->n = n;
  }
  return off;
}

size_t nj_job_workspace(int n) { return job_layout(n, nj_row_stride(n), nullptr, nullptr); }

// Fill the job descriptor for a job of n nodes with matrix D (row stride ld)
// and workspace at base; returns the addresses of its join records and
// statistics.
void nj_job_setup(void* job_out, float* D, int n, int ld, char* base, nwg_join** joins, unsigned long long** stats) {
  NJJob J{};
  job_layout(n, ld, base, &J);
  J.s.D = D;
  *joins = J.s.joins;
  *stats = J.s.stats;
  std::memcpy(job_out, &J, sizeof(J));
}

size_t nj_job_desc_bytes() { return sizeof(NJJob); }

// One job per cluster of C CTAs (C = 8 or 16); nmax: the largest job; alone: no other
// launch shares the SMs.
cudaError_t launch_nj_cluster(const void* d_jobs, int njobs, int nmax, int C, int sms, bool alone, cudaStream_t s) {
  if (njobs <= 0) return cudaSuccess;
  const NJJob* jobs = reinterpret_cast<const NJJob*>(d_jobs);
  const int ld = nj_row_stride(nmax);
  const int bytes = (int)lazy_layout(nmax, ld, C).bytes;
  const int threads = lazy_threads(ld, (nmax + C - 1) / C, C, alone);
  const bool most = (int64_t)njobs * C > 2 * (int64_t)sms || threads > kLazyThreads;
  const auto fn = C == 16 ? (most ? nj_cluster_kernel<16, kLazyThreadsMax> : nj_cluster_kernel<16, kLazyThreads>)
                          : (most ? nj_cluster_kernel<8, kLazyThreadsMax> : nj_cluster_kernel<8, kLazyThreads>);
  cudaError_t e;
  if ((C == 16 && (e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1))) ||
      (e = allow_smem((const void*)fn)))
    return e;
  fn<<<njobs * C, threads, bytes, s>>>(jobs, njobs);
  return cudaGetLastError();
}

// Jobs of at most this many taxa run the join loop in one CTA
// (nj_cta_kernel); NWG_NJ_CTA_MAX_N overrides it (0: never).
int cta_nj_max_n() {
  static const int v = [] {
    const char* e = std::getenv("NWG_NJ_CTA_MAX_N");
    return e ? std::min(std::atoi(e), kCtaNJMax) : kCtaNJDefault;
  }();
  return v;
}

cudaError_t launch_nj_cta(const void* d_jobs, int njobs, int nmax, cudaStream_t s) {
  if (njobs <= 0) return cudaSuccess;
  const int bytes = (int)cta_layout(std::max(nmax, 2)).bytes;
  const cudaError_t e = allow_smem((const void*)nj_cta_kernel);
  if (e != cudaSuccess) return e;
  nj_cta_kernel<<<njobs, kCtaThreads, bytes, s>>>(reinterpret_cast<const NJJob*>(d_jobs), njobs);
  return cudaGetLastError();
}

// The largest cluster (16, else 8) that the device schedules for the join loop.
int nj_cluster_size() {
  static int best = 0;
  if (best) return best;
  best = 8;
  const void* fn = (const void*)nj_cluster_kernel<16, kLazyThreads>;
  if (cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(16);
    cfg.blockDim = dim3(kLazyThreads);
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = 16;
    at.val.clusterDim.y = 1;
    at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int clusters = 0;
    if (cudaOccupancyMaxActiveClusters(&clusters, fn, &cfg) == cudaSuccess && clusters > 0) best = 16;
  }
  cudaGetLastError();
  return best;
}

}  // namespace nwg

extern "C" int nwg_nj(nwg_ctx* ctx, const float* D, int64_t ld, int n, nwg_join* joins, nwg_nj_stats* stats) {
  if (!ctx) return NWG_ERR_INVALID;
  nwg::Ctx* c = reinterpret_cast<nwg::Ctx*>(ctx);
  c->launches = 0;
  const int rc = c->nj(D, ld, n, false, joins, stats);
  if (stats) stats->launches = c->launches;
  return rc;
}

extern "C" int nwg_nj_dev(nwg_ctx* ctx, const float* d_D, int64_t ld, int n, nwg_join* joins, nwg_nj_stats* stats) {
  if (!ctx) return NWG_ERR_INVALID;
  nwg::Ctx* c = reinterpret_cast<nwg::Ctx*>(ctx);
  c->launches = 0;
  const int rc = c->nj(d_D, ld, n, true, joins, stats);
  if (stats) stats->launches = c->launches;
  return rc;
}
