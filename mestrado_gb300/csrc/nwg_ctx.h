// nwg_ctx.h -- the context behind the opaque nwg_ctx handle (not installed).
#pragma once

#include <algorithm>
#include <string>
#include <vector>

#include "nwg_internal.h"

namespace nwg {

// Grow-only device buffer owned by a context.
struct DevBuf {
  void* p = nullptr;
  size_t cap = 0;
  int ensure(size_t bytes);
  void release();
};

// One sequence set as the kernels see it: sorted by length (descending).
struct SetView {
  int n = 0;
  int maxlen = 0;
  std::vector<int32_t> len, orig, bound;
  std::vector<int64_t> start;
  const int8_t* d_codes = nullptr;
  const int64_t* d_start = nullptr;
  const int32_t* d_len = nullptr;
  const int32_t* d_orig = nullptr;
};

const int8_t* builtin_matrix();
const char* letter_order();

struct TuneChoice {
  int R;   // rows per lane (4 to 32, even; not a multiple of 4, or 28: layouts 2 to 4 and 7 on int16x2 lanes only)
  int V;   // register layout (0 to 7)
  int W;   // lanes per wavefront (32, 16, 8): band of W*R rows; 1: one pair per thread, bands of R rows
};
// Rows a Y of `rows` residues occupies under choice t (whole bands).
inline int padded_rows(const TuneChoice& t, int rows) {
  const int band = t.W * t.R;
  return (rows + band - 1) / band * band;
}
// The same band on full-width fronts, for groups that run on int32 lanes
// (the narrow fronts and the rows per lane that are not multiples of 4 exist
// for int16x2 lanes only).
// Layout 7 has no sentinel at the borders, which on int32 lanes the reference's
// -32768 + ge can reach: it needs ge * length + go below it (plain7).
inline TuneChoice int32_choice(TuneChoice t, bool plain7) {
  if (t.V == 6) t.V = 3;   // the split strips exist for int16x2 lanes only
  if (t.V == 3 || t.V == 7) t.V = plain7 ? 7 : 3;
  if (t.W == 32 && t.R % 4 == 0 && t.R != 28) return t;
  const int band = t.W * t.R;
  int R = 32;
  for (int r : {4, 8, 12, 16, 20, 24, 32})
    if (32 * r >= band) { R = r; break; }
  return {R, t.V == 1 ? 0 : t.V, 32};
}
constexpr int kTuneClasses = NWG_TUNE_CLASSES;
// Upper bound of the Y rows of each class; the last class takes every longer Y.
constexpr int kClassRows[kTuneClasses] = {64,  96,  128, 160, 192, 224, 256,  320,
                                          384, 448, 512, 640, 768, 1024, 1536, 1 << 30};
// Defaults before tuning, measured on a GB300.  Where layout 7 is exact (go >=
// ge, see Int16Limits), each class has the candidates that are the fastest for
// some Y of the class, with their rates in GCUPS over band-padded rows: the plan
// takes the one with the least estimated time per Y group, as after tuning.
// Layout 7 is the fastest in every class (at 450 rows 9.1 TCUPS against 7.6 for
// layout 3, at 2,000 10.1 against 8.4); up to 64 rows with one pair per thread.
struct RatedChoice {
  int R, W, gcups;
};
constexpr int kRatedMax = 6;
constexpr RatedChoice kDefaultRated[kTuneClasses][kRatedMax] = {
    {{32, 1, 6324}, {16, 1, 5010}, {24, 1, 6110}},
    {{12, 8, 7298}, {24, 1, 5742}},
    {{16, 8, 8474}},
    {{20, 8, 8907}, {18, 8, 8672}},
    {{24, 8, 8996}, {22, 8, 8823}},
    {{28, 8, 8907}, {26, 8, 9161}},
    {{16, 8, 8898}},
    {{20, 8, 8838}, {18, 16, 8816}},
    {{24, 16, 9266}, {22, 16, 9102}},
    {{28, 16, 9143}, {26, 16, 9148}, {18, 8, 8907}},
    {{16, 32, 8755}, {30, 16, 8620}},
    {{20, 16, 9461}, {18, 16, 9409}},
    {{24, 16, 9875}, {22, 16, 9778}},
    {{32, 32, 9808}, {30, 32, 9791}, {26, 16, 9804}, {18, 16, 9678}, {28, 16, 9787}},
    {{24, 16, 10136}, {22, 16, 10060}, {26, 16, 9923}, {28, 16, 9915}, {20, 32, 9635}, {30, 16, 9669}},
    {{30, 32, 10106}, {26, 32, 10082}, {32, 32, 10066}, {28, 32, 10032}, {22, 32, 9952}, {24, 32, 9909}}};
// The wavefronts for latency-bound callers (the serving loop): one pair per
// thread needs 256 X per CTA and streams a Y in bands, so it wins on throughput
// over many X but lengthens a small job; one band per Y up to 1,024 rows.
constexpr TuneChoice kDefaultTuneWave7[kTuneClasses] = {
    {8, 7, 8},   {12, 7, 8},  {16, 7, 8},  {20, 7, 8},  {24, 7, 8},  {28, 7, 8},  {16, 7, 16}, {20, 7, 16},
    {24, 7, 16}, {28, 7, 16}, {16, 7, 32}, {20, 7, 32}, {24, 7, 32}, {32, 7, 32}, {24, 7, 32}, {32, 7, 32}};
// Without layout 7: one choice per class, mostly the layouts with 1.5 ALU
// operations per cell (3, and 6 where R is a multiple of 8).
constexpr TuneChoice kDefaultTune[kTuneClasses] = {
    {32, 4, 1},  {32, 4, 1},  {16, 5, 8},  {20, 3, 8},  {24, 6, 8},  {28, 3, 8},  {32, 6, 8},  {20, 3, 16},
    {24, 6, 16}, {28, 3, 16}, {32, 6, 16}, {20, 3, 32}, {24, 6, 16}, {32, 3, 32}, {24, 6, 16}, {32, 3, 32}};
constexpr TuneChoice kDefaultTuneWave[kTuneClasses] = {
    {8, 5, 8},   {12, 0, 8},  {16, 5, 8},  {20, 3, 8},  {24, 6, 8},  {28, 3, 8},  {32, 6, 8},  {20, 3, 16},
    {24, 6, 16}, {28, 3, 16}, {32, 6, 16}, {20, 3, 32}, {24, 6, 16}, {32, 3, 32}, {24, 6, 16}, {32, 3, 32}};
int tune_class(int rows);

struct BatchPlan;
struct Ctx;
void destroy_plans(Ctx* c);

struct Ctx {
  int go = 10, ge = 2;
  int8_t sub[kLetters * kLetters];
  Int16Limits i16{kInt16MaxLen, 32756 - 11, 0, 0, false};   // set from (go, ge, sub) at creation
  int device = 0, sms = 1;
  cudaStream_t own_stream = nullptr;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  std::string last_err;
  int launches = 0;
  // Kernel choice per length class of the Y rows (rows <= kClassRows[k]):
  // rows per lane and register layout, set by the autotuner (tune.cu).
  TuneChoice tune[kTuneClasses];
  // The fastest wavefront (W >= 8) per class, for the serving loop, whose
  // small jobs are latency-bound (one pair per thread lengthens them).
  TuneChoice tune_wave[kTuneClasses];
  // Every candidate the autotuner timed per class, with its rate in computed
  // cells per second (band-padded rows x columns / time); before tuning the
  // defaults' rates.  Empty when the table was set by hand (or without layout 7
  // before tuning): tune[] is then used as it is.
  struct Cand {
    TuneChoice t;
    double rate;
  };
  std::vector<Cand> cands[kTuneClasses];
  // The tables before tuning.
  void default_tuning() {
    for (int k = 0; k < kTuneClasses; ++k) {
      const bool seven = i16.max_len7 > 0;
      cands[k].clear();
      tune[k] = seven ? TuneChoice{kDefaultRated[k][0].R, 7, kDefaultRated[k][0].W} : kDefaultTune[k];
      tune_wave[k] = seven ? kDefaultTuneWave7[k] : kDefaultTuneWave[k];
      if (!seven) continue;
      for (const RatedChoice& r : kDefaultRated[k])
        if (r.R > 0) cands[k].push_back({{r.R, 7, r.W}, 1e9 * r.gcups});
    }
  }
  // The choice for a Y group of this many rows: the class's candidate with
  // the least estimated time (its padded rows / its rate), the class's
  // fastest at the class bound unless another is estimated 2 % faster.
  // Layout 4 is exact only when go >= ge and falls back to layout 2; layout 7
  // falls back to layout 3 beyond its range.
  TuneChoice choice(int rows) const {
    const int k = tune_class(rows);
    TuneChoice t = tune[k], fastest = t;
    double pick_est = 0.0, min_est = 0.0;
    for (const Cand& c : cands[k]) {
      const double est = padded_rows(c.t, rows) / c.rate;
      if (c.t.R == t.R && c.t.V == t.V && c.t.W == t.W) pick_est = est;
      if (min_est == 0.0 || est < min_est) {
        min_est = est;
        fastest = c.t;
      }
    }
    if (pick_est > 0.0 && min_est < 0.98 * pick_est) t = fastest;
    return allowed(t, rows);
  }
  // The choice when the whole set is `cells` cells over columns up to `cols`: a
  // small set does not fill the GPU with warps, and what counts is how long one
  // warp takes for its Y, a chain of two maxima per row (10 cycles) and about 90
  // cycles per column.  The wavefronts with few rows per lane are then the
  // faster ones; the estimate is the longer of that chain and the set's time at
  // the candidate's rate, and a quarter of the shorter.  All pairs of 64 x 300
  // residues: 52 us with 12 rows on 32 lanes, 62 with 18 on 16, 86 with two
  // bands of 20 on 8.
  static double chain_s(const TuneChoice& t, int rows, int cols) {   // seconds
    return padded_rows(t, rows) / (t.W * t.R) * (cols + t.W - 1) * (10.0 * t.R + 90.0) / 2.0e9;
  }
  // fitted: the template that is the fastest for each length, else the class's first
  // for all its Y.
  double rate_of(const TuneChoice& t, int rows) const {   // cells/s over padded rows, about
    for (const Cand& c : cands[tune_class(rows)])
      if (c.t.R == t.R && c.t.V == t.V && c.t.W == t.W) return c.rate;
    return small_rate(t.R);
  }
  static double small_rate(int R) {   // the wavefronts of few rows per lane, measured
    constexpr double kSlow[] = {4.2e12, 6.5e12, 7.9e12, 8.4e12};   // at 4, 8, 12, 16 rows
    return R < 20 ? kSlow[R / 4 - 1] : 9.0e12;
  }
  TuneChoice choice_set(int rows, int cols, double cells, bool fitted) const {
    const TuneChoice t = fitted ? choice(rows) : allowed(tune[tune_class(rows)], rows);
    if (t.V != 7 || cands[tune_class(rows)].empty()) return t;
    const auto est = [&](const TuneChoice& c, double rate) {
      const double chain = chain_s(c, rows, cols);
      const double whole = cells * padded_rows(c, rows) / rows / rate;
      return std::max(chain, whole) + 0.25 * std::min(chain, whole);
    };
    const double rate = rate_of(t, rows);
    // a set of many waves of jobs: the shortest chain would not show
    if (cells * padded_rows(t, rows) / rows / rate > 20.0 * chain_s(t, rows, cols)) return t;
    TuneChoice best = t;
    double best_est = 0.95 * est(t, rate);   // not for less than a twentieth
    for (int W : {8, 32})   // few templates: the first use of each in a process loads it (0.5 to 1 ms)
      for (int R : {4, 8, 12, 16, 24, 32}) {
        const TuneChoice c{R, 7, W};
        const double e = est(c, small_rate(R));
        if (e < best_est) {
          best_est = e;
          best = c;
        }
      }
    return best;
  }
  TuneChoice allowed(TuneChoice t, int rows) const {
    if (t.V == 4 && go < ge) t.V = 2;
    if (t.V == 7 && rows > i16.max_len7) t.V = 3;
    return t;
  }
  // Layout 7 on int32 lanes: no border value of sequences up to maxlen falls to
  // the reference's sentinel.
  bool plain7(int maxlen) const { return go >= ge && (int64_t)ge * maxlen + go < 32700; }
  TuneChoice choice_wave(int rows) const {
    return allowed(tune_wave[tune_class(rows)], rows);
  }
  uint64_t tune_version = 0;        // bumped on every change (part of the plan key)
  bool tuned = false;

  DevBuf b_codes, b_start, b_len, b_orig, b_bound, b_bad;
  DevBuf b_start2, b_len2, b_orig2;
  DevBuf b_gy, b_gy2, b_gx, b_jobs, b_counter, b_wscratch, b_pscratch, b_yprefix;
  DevBuf b_D, b_sub, b_rowmax;
  DevBuf b_pi, b_pj, b_out;
  // per-launch event timing (nwg_set_launch_timing)
  bool launch_timing = false;
  std::vector<nwg_launch_rec> recs;
  std::vector<cudaEvent_t> evpool;
  int rec_begin(const nwg_launch_rec& r);   // records the start event; returns record index
  int rec_end(int idx);
  int rec_finalize();
  // batched-form plans (batched.cu): [0] all-pairs triangle, [1] block
  BatchPlan* plans[2] = {nullptr, nullptr};
  bool use_graphs = true;
  std::vector<cudaStream_t> branch;     // parallel branches for bucket launches
  cudaEvent_t fork_ev = nullptr;
  std::vector<cudaEvent_t> join_ev;
  int autotune(bool force, nwg_tune_result* out);
  bool tune_from_cache(nwg_tune_result* res);
  int batched(const int8_t* d_codes, const int64_t* xoff, int nx, const int64_t* yoff, int ny, bool triangle,
              float* d_D, int64_t ld, int64_t col0, int mode, nwg_stats* st);
  // traceback / neighbor joining state (trace.cu, nj.cu)
  void* trace_state = nullptr;
  void* nj_state = nullptr;
  void* ingest_state = nullptr;
  void* msa_state = nullptr;
  void extra_release();
  void nj_release();
  void ingest_release();
  void msa_release();
  int msa(const int8_t* codes, const int64_t* offsets, int n, const int32_t* left, const int32_t* right,
          int64_t* msa_len, nwg_stats* st);
  int msa_rows(char* out, int64_t stride);
  int nj(const float* D, int64_t ld, int n, bool device_D, nwg_join* joins, nwg_nj_stats* st);
  // Work forked from the stream to the branch streams: a call that returns before it
  // has joined them waits for them here, since the next call reuses its buffers.
  struct Fork {
    Ctx& c;
    bool joined = false;
    ~Fork() {
      if (!joined)
        for (cudaStream_t b : c.branch) cudaStreamSynchronize(b);
    }
  };
  // Failure injection for the tests (NWG_INJECT_FORK_ERROR=1): an error between the
  // last launch on a branch stream and the join.
  int injected_fork_error();
  int score_pairs(const int8_t* codes, const int64_t* offsets, int n, const int32_t* pi, const int32_t* pj,
                  int64_t npairs, int32_t* out, int64_t* pairs16);   // pairs.cu
  int trace_lanes_forced = 0;   // front width of the traceback kernel (0: chosen per call)
  int align_pairs(const int8_t* codes, const int64_t* offsets, int n, const int32_t* px, const int32_t* py,
                  int npairs, char* outx, char* outy, int64_t stride, int32_t* outlen, int32_t* score,
                  nwg_stats* st);

  ~Ctx();
  int fail(int status, const char* what, cudaError_t e = cudaSuccess);
  int cuda(cudaError_t e, const char* what);
  int prepare_set(const int8_t* d_codes, const int64_t* offsets, int n, SetView& v, DevBuf& bstart,
                  DevBuf& blen, DevBuf& borig, bool want_bounds);
  int run_plain(const SetView& X, const SetView& Y, bool triangle, float* d_D, int64_t ld,
                int64_t col0, nwg_stats* st);
  int score_all_dev(const int8_t* d_codes, const int64_t* offsets, int n, float* d_D, int64_t ld,
                    int mode, nwg_stats* st);
};

}  // namespace nwg
