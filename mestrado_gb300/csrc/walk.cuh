// walk.cuh -- the backtrace walk over 4-bit cell flags, by one warp, in runs.
//
// The rules are those of NeedlemanWunschGlobalBackKernel (NeedlemanWunsch.cu:
// 393-494): the continue flags of the previous move first, then up, then left,
// else diagonal; row -1 reads as left + continue, column -1 as up + continue;
// an up move out of row 0 ends the walk.  Taken one cell at a time they are a
// chain of dependent reads (about 60 cycles a move from shared memory).  But
// after a diagonal move the next move depends on the next cell alone, and an
// up (left) move goes on while the cells passed carry the continue flag.  So
// the lanes read the next 32 cells along the diagonal, or along the gap, at
// once, and a ballot gives the length of the run: one step of the chain per
// run, not per move.
#pragma once

#include <cstdint>

namespace nwg {

// The walk's place and what it has emitted.
struct WalkPos {
  int x, y;         // next cell, -1 past the first row / column
  int k;            // moves emitted
};

// win.covers(x, y): whether the window holds cell (x, y); win.cell(x, y): its
// flags (L 8, U 4, cU 2, cL 1); win.load(x, y): (whole warp) reload the window
// so that it ends at (x, y).  emit(k, m, x, y, sx, sy): (whole warp) moves k ..
// k + m - 1 start at (x, y) and take sx columns and sy rows each (0 or 1).
// cap: the most moves.  Every lane returns the same state.
template <class Window, class Emit>
__device__ WalkPos run_walk(Window& win, int lx, int ly, int cap, Emit&& emit) {
  const int lane = threadIdx.x & 31;
  int x = lx - 1, y = ly - 1, k = 0;
  bool go_up = false, go_left = false;   // the previous move's continue flags
  while (x >= 0 && y >= 0 && k < cap) {
    if (!win.covers(x, y)) win.load(x, y);
    unsigned first = 12u;
    if (!go_up && !go_left) {
      // the diagonal from (x, y): a run of cells that send the walk diagonally
      const int cx = x - lane, cy = y - lane;
      const bool in = cx >= 0 && cy >= 0 && win.covers(cx, cy);
      const unsigned n = in ? win.cell(cx, cy) : 0u;
      first = __shfl_sync(0xffffffffu, n, 0) & 12u;
      if (first == 12u) {
        const unsigned run = __ballot_sync(0xffffffffu, in && (n & 12u) == 12u && k + lane < cap);
        const int m = run == 0xffffffffu ? 32 : __ffs(~run) - 1;
        emit(k, m, x, y, 1, 1);
        x -= m;
        y -= m;
        k += m;
        continue;
      }
      if (first == 0u) break;   // no direction: never set by a recurrence
    }
    // a gap: the first move is taken, the next ones while the cells passed
    // carry the continue flag
    const bool up = go_up || (!go_left && first == 4u);
    const int cx = up ? x : x - lane, cy = up ? y - lane : y;
    const bool in = cx >= 0 && cy >= 0 && win.covers(cx, cy) && k + lane < cap;
    const unsigned n = in ? win.cell(cx, cy) : 0u;
    const unsigned on = __ballot_sync(0xffffffffu, in && (n & (up ? 2u : 1u)));
    const unsigned have = __ballot_sync(0xffffffffu, in);
    const int last = on == 0xffffffffu ? 31 : __ffs(~on) - 1;   // the cell that ends the run
    const int avail = have == 0xffffffffu ? 32 : __ffs(~have) - 1;
    const int m = last + 1 < avail ? last + 1 : avail;
    const bool cont = (on >> (m - 1)) & 1u;                      // the run goes on past this read
    emit(k, m, x, y, up ? 0 : 1, up ? 1 : 0);
    if (up) y -= m;
    else x -= m;
    k += m;
    go_up = up && cont;
    go_left = !up && cont;
    if (up && y < 0) return {x, y, k};   // an up move out of row 0 ends the walk
  }
  if (y < 0) {
    // row -1: left to the corner (unless a continued up move wanted more rows: ended above)
    while (x >= 0 && k < cap) {
      const int m = min(32, min(x + 1, cap - k));
      emit(k, m, x, y, 1, 0);
      x -= m;
      k += m;
    }
  } else if (x < 0 && !go_left) {
    // column -1: up to the corner; a continued left move has nowhere to go and ends the walk
    while (y >= 0 && k < cap) {
      const int m = min(32, min(y + 1, cap - k));
      emit(k, m, x, y, 0, 1);
      y -= m;
      k += m;
    }
  }
  return {x, y, k};
}

}  // namespace nwg
