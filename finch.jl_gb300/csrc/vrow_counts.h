// Two counts to a 64-bit word, as the virtual-row schedules scan them.
#pragma once

#include <cstdint>

#ifdef __CUDACC__
#define FGB_HD __host__ __device__ __forceinline__
#else
#define FGB_HD inline
#endif

namespace fgb {

FGB_HD int64_t vr_pack(int64_t lo, int64_t hi) { return (int64_t)((uint64_t)lo | (uint64_t)hi << 32); }
FGB_HD int64_t vr_lo(int64_t w) { return w & 0xffffffffll; }
FGB_HD int64_t vr_hi(int64_t w) { return (int64_t)((uint64_t)w >> 32); }

// Whether the bands' virtual rows, counted apart in 64 bits, are no more than
// a schedule's 32-bit indices reach.  Every other count is smaller, so the
// words' halves have not run over where this holds; the words themselves
// cannot tell (2^32 + 7 rows leave 7 in the low half).
inline bool vrow_fits(const unsigned long long* band_rows, int nbands) {
  unsigned long long all = 0;
  for (int b = 0; b < nbands; ++b) {
    if (band_rows[b] > INT32_MAX) return false;
    all += band_rows[b];
  }
  return all <= INT32_MAX;
}

}  // namespace fgb
