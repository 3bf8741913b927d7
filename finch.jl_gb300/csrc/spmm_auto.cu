// CSR SpMM of aligned operands with no schedule given: whole rows, blocks of
// equal work.
//
// Row r sits at step r + ptr[r] of the walk over rows and stored entries, and
// a block owns the rows that begin in its share of the steps; it searches ptr
// for the first of them.  A group of G lanes (V columns a lane) folds one row
// at a time, one running sum per output, with up to 8 gathers of B in flight;
// the groups of a warp are never made to meet.  A row of more than SA_LONG
// entries is listed, and when the block's other rows are done the whole block
// folds each listed row, an equal part per group, the parts added in a fixed
// order.  No row is split between blocks: no scratch, no second launch, and
// results are the same run to run.
//
// Bound: latency of the B-row gathers (8 a lane in flight, 2 blocks of 126
// registers an SM: 3 or 4 blocks spill and measured 137 and 116 us where 2
// take 102), FP64 also by its pipe.  GB300, per call, against the merge-path
// items it replaces as the default (the warp's sub-groups met at every row
// end, and carries were fixed up afterwards): 150,011 rows, 120,007 columns,
// 12 entries a row, k = 64: F32 Zipf 194 -> 102 us, uniform 152 -> 90; F64
// Zipf 414 -> 295, uniform 406 -> 262.  20,000 Zipf rows 102 -> 31; 100,000
// rows of 20, k = 128, 234 -> 139; 500,000 rows of 8, k = 32, 279 -> 174.
#include <algorithm>

#include "spmm_common.cuh"

namespace fgb {

constexpr int SA_THREADS = 256;
constexpr int SA_LONG = 64;
constexpr int SA_LIST = 64;  // more than a share holds; a full list would cost speed only
// A block's share: an equal one of all steps while that keeps every block in
// the first wave, at most SA_MAX_STEPS (4096: 500,000 rows of 8 189 us).
constexpr int64_t SA_MIN_STEPS = 256, SA_MAX_STEPS = 2048;

template <class T, class VT, class PtrT, int G, int V>
__global__ void __launch_bounds__(SA_THREADS, 2) spmm_csr_auto(
    int64_t nrows, const PtrT* __restrict__ ptr, const int* __restrict__ idx, const VT* __restrict__ val,
    const T* __restrict__ B, int64_t ldb, T* __restrict__ C, int64_t ldc, int64_t c0, int64_t nk, int base,
    int accumulate) {
  constexpr int NG = SA_THREADS / G, WARPS = SA_THREADS / 32;
  __shared__ int64_t s_long[SA_LIST];
  __shared__ int s_n;
  __shared__ VecT<T, V> s_part[2][WARPS][G];
  const int tid = threadIdx.x, lane = tid % G, g = tid / G;
  const unsigned gmask = group_mask<G>();
  const int64_t col = c0 + (int64_t)lane * V;
  const bool active = col < nk;  // V divides nk - c0
  const T* Bc = B + col;
  const uint64_t pol_stream = policy_evict_first();
  const uint64_t pol_keep = policy_evict_last();
  const int64_t f0 = ld_ptr(ptr, 0);
  const int64_t steps = ld_ptr(ptr, nrows) - f0 + nrows;
  const int64_t per = (steps + gridDim.x - 1) / gridDim.x;
  const int64_t first = blockIdx.x * per, end = first + per;
  if (tid == 0) s_n = 0;
  // first row whose step is at least `first` (nrows if none): 256 probes a round
  int64_t lo = 0, hi = nrows;
  while (lo < hi) {  // block-uniform
    const int64_t step = (hi - lo + SA_THREADS - 1) / SA_THREADS;
    const int64_t q = lo + tid * step;
    const int n = __syncthreads_count(q < hi && ld_ptr(ptr, q) - f0 + q < first);
    const int64_t next = lo + n * step;
    if (n == 0) {
      hi = lo;
    } else {
      lo += (n - 1) * step + 1;
      if (next < hi) hi = next;
    }
  }
  __syncthreads();

  // Entries [p, p1) of a row by the group, in storage order.
  auto fold = [&](VecT<T, V>& acc, int64_t p, int64_t p1) {
    for (int64_t pb = p; pb < p1; pb += G) {
      const int64_t pe = pb + lane;
      int my_j = 0;
      T my_a = T(0);
      if (pe < p1) {
        my_j = ld_stream_i32(idx + pe, pol_stream) - base;
        my_a = load_val<T, VT>(val, pe, pol_stream);
      }
      const int cnt = p1 - pb < (int64_t)G ? (int)(p1 - pb) : G;
      int t = 0;
      if constexpr (G >= 8)
        for (; t + 8 <= cnt; t += 8)
          pull_batch<T, G, V, 8, FM_FMA>(acc, t, my_j, my_a, Bc, ldb, active, gmask, pol_keep);
      if (t + 4 <= cnt) {
        pull_batch<T, G, V, 4, FM_FMA>(acc, t, my_j, my_a, Bc, ldb, active, gmask, pol_keep);
        t += 4;
      }
      if (t + 2 <= cnt) {
        pull_batch<T, G, V, 2, FM_FMA>(acc, t, my_j, my_a, Bc, ldb, active, gmask, pol_keep);
        t += 2;
      }
      if (t < cnt) pull_batch<T, G, V, 1, FM_FMA>(acc, t, my_j, my_a, Bc, ldb, active, gmask, pol_keep);
    }
  };
  auto store = [&](int64_t row, VecT<T, V> acc) {
    T* dst = C + row * ldc + col;
    if (accumulate) {
      const VecT<T, V> old = load_out<T, V>(dst);
#pragma unroll
      for (int q = 0; q < V; ++q) acc.v[q] += old.v[q];
    }
    store_out<T, V>(dst, acc, pol_stream);
  };

  for (int64_t row = lo + g; row < nrows; row += NG) {
    const int64_t p0 = ld_ptr(ptr, row), p1 = ld_ptr(ptr, row + 1);
    if (p0 - f0 + row >= end) break;
    if (p1 - p0 > SA_LONG) {
      int kept = 0;
      if (lane == 0) {
        const int at = atomicAdd(&s_n, 1);
        if (at < SA_LIST) s_long[at] = row;
        kept = at < SA_LIST;
      }
      if (__shfl_sync(gmask, kept, 0, G)) continue;
    }
    VecT<T, V> acc;
#pragma unroll
    for (int q = 0; q < V; ++q) acc.v[q] = T(0);
    fold(acc, p0 - base, p1 - base);
    if (active) store(row, acc);
  }
  __syncthreads();
  const int nlong = s_n < SA_LIST ? s_n : SA_LIST;
  for (int l = 0; l < nlong; ++l) {  // block-uniform
    const int64_t row = s_long[l];
    const int64_t p0 = ld_ptr(ptr, row) - base, p1 = ld_ptr(ptr, row + 1) - base;
    const int64_t part = ((p1 - p0 + NG - 1) / NG + 7) / 8 * 8;
    const int64_t q0 = p0 + g * part, q1 = q0 + part < p1 ? q0 + part : p1;
    VecT<T, V> acc;
#pragma unroll
    for (int q = 0; q < V; ++q) acc.v[q] = T(0);
    fold(acc, q0, q1);
    __syncwarp();
#pragma unroll
    for (int m = G; m < 32; m <<= 1)
#pragma unroll
      for (int q = 0; q < V; ++q) acc.v[q] += __shfl_xor_sync(0xffffffffu, acc.v[q], m);
    if ((tid & 31) < G) s_part[l & 1][tid >> 5][lane] = acc;
    __syncthreads();
    if (tid < G && active) {
#pragma unroll
      for (int w = 1; w < WARPS; ++w)
#pragma unroll
        for (int q = 0; q < V; ++q) acc.v[q] += s_part[l & 1][w][lane].v[q];
      store(row, acc);
    }
  }
}

template <class T, class VT, class PtrT, int G>
static int launch_auto(fgb_ctx* ctx, const fgb_sparse* A, const T* B, int64_t ldb, int64_t nk, T* C, int64_t ldc,
                       int accumulate, cudaStream_t s) {
  constexpr int V = sizeof(T) == 4 ? 4 : 2;
  auto kern = spmm_csr_auto<T, VT, PtrT, G, V>;
  static const int occ = [&] {  // once per process (one device model); thread-safe
    int o = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kern, SA_THREADS, 0);
    return o > 0 ? o : 1;
  }();
  const int64_t steps = A->nrows + A->nnz;
  const int64_t share = std::clamp(steps / ((int64_t)occ * ctx->num_sms), SA_MIN_STEPS, SA_MAX_STEPS);
  const int grid = (int)std::min<int64_t>((steps + share - 1) / share, INT32_MAX);
  for (int64_t c0 = 0; c0 < nk; c0 += G * V) {
    kern<<<grid, SA_THREADS, 0, s>>>(A->nrows, (const PtrT*)A->ptr, (const int*)A->idx, (const VT*)A->val, B, ldb, C,
                                     ldc, c0, nk, A->index_base, accumulate);
    const int rc = check_launch("spmm_csr_auto");
    if (rc) return rc;
  }
  return FGB_OK;
}

template <class T, class VT>
static int auto_typed(fgb_ctx* ctx, const fgb_sparse* A, const void* B, int64_t ldb, int64_t nk, void* C, int64_t ldc,
                      int accumulate, cudaStream_t s) {
  constexpr int V = sizeof(T) == 4 ? 4 : 2;
  const int64_t need = (nk + V - 1) / V;  // lanes that cover a row of B, at most a warp
  auto go = [&](auto ptr_t) -> int {
    using P = decltype(ptr_t);
    if (need <= 4) return launch_auto<T, VT, P, 4>(ctx, A, (const T*)B, ldb, nk, (T*)C, ldc, accumulate, s);
    if (need <= 8) return launch_auto<T, VT, P, 8>(ctx, A, (const T*)B, ldb, nk, (T*)C, ldc, accumulate, s);
    if (need <= 16) return launch_auto<T, VT, P, 16>(ctx, A, (const T*)B, ldb, nk, (T*)C, ldc, accumulate, s);
    return launch_auto<T, VT, P, 32>(ctx, A, (const T*)B, ldb, nk, (T*)C, ldc, accumulate, s);
  };
  return A->ptr_t == FGB_I32 ? go(int32_t(0)) : go(int64_t(0));
}

int spmm_auto(fgb_ctx* ctx, const fgb_sparse* A, const void* B, int64_t ldb, int64_t nk, void* C, int64_t ldc,
              int dtype, int accumulate, cudaStream_t s) {
  if (A->nrows == 0 || nk == 0) return FGB_OK;
  if (dtype == FGB_F64) return auto_typed<double, double>(ctx, A, B, ldb, nk, C, ldc, accumulate, s);
  if (A->val_t == FGB_BF16) return auto_typed<float, __nv_bfloat16>(ctx, A, B, ldb, nk, C, ldc, accumulate, s);
  return auto_typed<float, float>(ctx, A, B, ldb, nk, C, ldc, accumulate, s);
}

}  // namespace fgb
