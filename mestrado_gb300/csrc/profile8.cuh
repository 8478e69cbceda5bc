// profile8.cuh -- one warp's score profile of a band of 32 R rows, a byte per
// (letter, row), in shared memory.
#pragma once

#include "nwg_internal.h"

namespace nwg {

// Byte permute; a selector nibble with bit 3 set replicates its byte's sign.
__device__ __forceinline__ uint32_t perm(uint32_t a, uint32_t b, uint32_t sel) {
  uint32_t r;
  asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(sel));
  return r;
}

// A bad code reads as the last letter: nothing outside the tables is addressed.
__device__ __forceinline__ unsigned profile_code(int c) {
  const unsigned u = (unsigned)c;
  return u < (unsigned)kLetters ? u : (unsigned)(kLetters - 1);
}

// The lane's R bytes of each letter of one pair's band, into prof[letter][lane][R].
template <int R>
__device__ __forceinline__ void build_profile(uint32_t* prof, const int8_t* s_sub, const int8_t* Y, int row0, int Ly,
                                              uint32_t zero, int lane) {
  uint32_t y[R];
#pragma unroll
  for (int r = 0; r < R; ++r) y[r] = row0 + r < Ly ? profile_code(Y[row0 + r]) * kLetters : 0xFFFFu;
#pragma unroll
  for (int x4 = 0; x4 < kLetters; x4 += 4) {
    uint32_t w[4][R / 4];
#pragma unroll
    for (int q = 0; q < R / 4; ++q) {
      uint32_t v[4];   // four letters of rows 4q .. 4q + 3
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const uint32_t o = y[4 * q + k];
        v[k] = o != 0xFFFFu ? *reinterpret_cast<const uint32_t*>(s_sub + o + x4) : zero;
      }
      const uint32_t t0 = perm(v[0], v[1], 0x5140), t1 = perm(v[2], v[3], 0x5140);
      const uint32_t t2 = perm(v[0], v[1], 0x7362), t3 = perm(v[2], v[3], 0x7362);
      w[0][q] = perm(t0, t1, 0x5410);
      w[1][q] = perm(t0, t1, 0x7632);
      w[2][q] = perm(t2, t3, 0x5410);
      w[3][q] = perm(t2, t3, 0x7632);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      uint32_t* d = prof + ((x4 + k) * 32 + lane) * (R / 4);
      if constexpr (R == 8) {
        *reinterpret_cast<uint2*>(d) = make_uint2(w[k][0], w[k][1]);
      } else {
#pragma unroll
        for (int q = 0; q < R / 4; ++q) d[q] = w[k][q];
      }
    }
  }
}

}  // namespace nwg
