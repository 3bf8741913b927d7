// The fibers of a run of stored entries, for kernels that walk entries and
// need the fiber of each.
#pragma once

#include "fgb_internal.cuh"

namespace fgb {

constexpr int FC_THREADS = 256;
constexpr int FC_ENTRIES = 2048;  // entries per block
constexpr int FC_FEW = 256;       // the same where those blocks would leave SMs idle
constexpr int FC_FIBERS = 2048;   // fiber starts kept in shared memory

// Entries [p0, p0 + n) of a compressed matrix, by a block of FC_THREADS: two
// searches of ptr, 256 probes a round, bound their fibers, whose starts are
// then read once, coalesced; an entry's fiber is found among those (a binary
// search of all of ptr per entry, 20 dependent loads on a million fibers,
// was most of the kernels that did it).
template <class PtrT>
struct FiberChunk {
  const PtrT* ptr;
  int base;
  int64_t p0, f0;
  int count;      // fibers f0 .. f0 + count - 1 hold the entries
  const int* s;   // their starts from p0, where they fit

  // Number of fibers f < nf with ptr[f] - base <= p (block-uniform).
  static __device__ int64_t starts_up_to(const PtrT* ptr, int64_t nf, int base, int64_t p) {
    int64_t lo = 0, hi = nf;
    while (lo < hi) {
      const int64_t step = (hi - lo + FC_THREADS - 1) / FC_THREADS;
      const int64_t q = lo + threadIdx.x * step;
      const int n = __syncthreads_count(q < hi && ld_ptr(ptr, q) - base <= p);
      const int64_t next = lo + n * step;
      if (n == 0) {
        hi = lo;
      } else {
        lo += (n - 1) * step + 1;
        if (next < hi) hi = next;
      }
    }
    return lo;
  }

  // s_starts: FC_FIBERS ints of shared memory.  Ends with a barrier.
  __device__ FiberChunk(const PtrT* ptr_, int64_t nf, int base_, int64_t p0_, int n, int* s_starts)
      : ptr(ptr_), base(base_), p0(p0_) {
    f0 = starts_up_to(ptr, nf, base, p0) - 1;
    const int64_t f1 = starts_up_to(ptr, nf, base, p0 + n - 1);
    count = (int)(f1 - f0);
    s = nullptr;
    if (count <= FC_FIBERS) {
      for (int k = threadIdx.x; k < count; k += FC_THREADS)
        s_starts[k] = k == 0 ? 0 : (int)(ld_ptr(ptr, f0 + k) - base - p0);
      s = s_starts;
    }
    __syncthreads();
  }

  // Fiber of entry p0 + e: the last that starts at or before it.
  __device__ int64_t of(int e) const {
    int lo = 0, hi = count;
    if (s) {
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (s[mid] <= e) lo = mid;
        else hi = mid;
      }
    } else {
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (ld_ptr(ptr, f0 + mid) - base - p0 <= e) lo = mid;
        else hi = mid;
      }
    }
    return f0 + lo;
  }
};

// Whether blocks of FC_ENTRIES are fewer than the SMs (8,000 entries in 4
// blocks: masked scaling 117 us, in 32 of FC_FEW 96).
inline bool fc_few(int64_t nnz, int num_sms) { return nnz < (int64_t)FC_ENTRIES * num_sms; }

inline int64_t fc_blocks(int64_t nnz, int run) { return (nnz + run - 1) / run; }

}  // namespace fgb
