// CSR SpMM of aligned operands with no schedule given: blocks of equal work.
//
// Row r sits at step r + ptr[r] of the walk over rows and stored entries, and
// a block owns the rows that begin in its share of the steps; it searches ptr
// for the first of them.  A group of G lanes (V columns a lane) folds a row of
// at most SA_ROW entries, with up to 8 gathers of B in flight; the groups of a
// warp are never made to meet.  Longer rows are listed and taken when the
// block's others are done: where there are a few of them, one a warp, an equal
// part per group of it (rows up to SA_WARP entries); else, and longer ones, by
// the whole block one after another, an equal part per group of the block, the
// parts added in a fixed order.
//
// A row of more entries than two shares hold steps is cut at the shares, but in
// a small product (SA_CUT_BYTES): the block in whose share it begins writes its
// part to C, the others leave theirs as carries, and spmm_auto_fixup adds a
// row's carries in the order of the blocks.  Results are the same run to run.
//
// A lane keeps 4 sums a column in FP32 (8 for up to 16 columns; FP64, whose
// pipe waits for the adds, 32 / G, at most 4): at least as many as sub-groups
// of a warp shared a row in the merge path, so that FP32 rounds no more.
//
// Bound: latency of the B-row gathers (8 a lane in flight, 3 blocks of 80
// registers an SM; with 2 blocks of 96 a fifth slower), FP64 also by its pipe.
// GB300, per call behind a cold L2, against the merge-path items that were the
// default before (the warp's sub-groups met at every row end, and carries were
// fixed up afterwards): 150,000 rows of 12, 120,000 columns, k = 64: F32 Zipf
// 204 -> 103 us, uniform 157 -> 69; F64 396 -> 286, 412 -> 245.  20,000 Zipf
// rows 98 -> 40; 100,000 rows of 30, k = 128, 252 -> 140.  Rows of 100 (50,000),
// k = 16 / 64 / 128, F32 96 -> 106, 236 -> 158, 344 -> 224; of 400 (20,000) 114
// -> 125, 325 -> 214, 488 -> 306 (one row after another by the block, at 2
// blocks an SM, 336 / 284 / 364 and 151 / 272 / 356).  One row of a million
// entries beside 200,000 of 8: k = 16 F32 1,294 -> 93, k = 64 F64 2,661 -> 351
// (whole, in one block, 21,126).
#include <algorithm>
#include <type_traits>

#include "spmm_common.cuh"

namespace fgb {

constexpr int SA_THREADS = 256;
constexpr int SA_ROW = 64;
constexpr int SA_LIST = 64;  // a share of SA_MAX_STEPS holds the beginnings of at most 32 rows over SA_ROW entries
// A block's share: an equal one of all steps while that keeps every block in
// the first wave, at most SA_MAX_STEPS (with 4096, 150,000 rows of 12, k = 64,
// 79 us in place of 66, 300,000 rows of 4 97 for 80).
constexpr int64_t SA_MIN_STEPS = 256, SA_MAX_STEPS = 2048;
// Rows are cut from as many gathered bytes (rows and entries times a row of B):
// below, the scratch and the second launch cost a call whose host side takes
// as long as its kernel 3 us (10,000 rows of 5, k = 64, 11.8 -> 14.6; through
// lazy tensors 22,828 rows of 5, k = 32, FP64, 34 -> 38), and a row that had
// all of the entries keeps one SM for 1.1 ms at most, in FP64 2.6.
constexpr double SA_CUT_BYTES = 64.0 * 1024 * 1024;
// Rows up to this length may be a warp's: 128 entries a group of it, at most
// 512; none in FP64 where a warp is one group with one sum a lane.
template <class T, int G>
constexpr int SA_WARP = G <= 8 ? 512 : sizeof(T) == 8 && G == 32 ? 0 : 4096 / G;
// Running sums a lane keeps for each column.
template <class T, int G>
__host__ __device__ constexpr int sa_sums() {
  return sizeof(T) == 4 ? (G == 4 ? 8 : 4) : G == 4 ? 4 : 32 / G;
}

// The sum that a batch's u-th entry goes to.  Eight entries are spread evenly
// over the sums.  What is left of a row goes in pairs, three in one: a row of
// up to 4 has its products fused into its sums, which rounds less there than
// sums of one product each (4 entries, FP32: relative error 3.6e-8 for 3.8e-8;
// 24 entries: 3.9e-8 by 4 or 8 sums, 7.4e-8 by one).
template <int N>
using Int = std::integral_constant<int, N>;
enum SaBatch { SA_EIGHT, SA_LOW4, SA_HIGH4, SA_FOUR, SA_REST };
template <SaBatch K>
using Kind = std::integral_constant<SaBatch, K>;
template <int U, SaBatch K>
__device__ constexpr int sa_sum(int u) {
  return K == SA_EIGHT ? u * U / 8 : K == SA_LOW4 ? u : K == SA_HIGH4 ? 4 + u : (K == SA_FOUR ? u / 2 : 2) % U;
}

// NB entries of a row from the t-th of the group's current ones; lane l of the
// group holds entries l, l + G, ...
template <class T, int G, int V, int U, int E, int NB, SaBatch K>
__device__ __forceinline__ void sa_batch(VecT<T, V> (&acc)[U], int t, const int (&my_j)[E], const T (&my_a)[E],
                                         const T* __restrict__ Bc, int64_t ldb, unsigned gmask, uint64_t pol) {
  VecT<T, V> b[NB];
#pragma unroll
  for (int u = 0; u < NB; ++u) {
    const int j = __shfl_sync(gmask, E == 1 || t + u < G ? my_j[0] : my_j[E - 1], t + u, G);
    b[u] = gather<T, V>(Bc + (int64_t)j * ldb, pol);
  }
#pragma unroll
  for (int u = 0; u < NB; ++u) {
    const T a = __shfl_sync(gmask, E == 1 || t + u < G ? my_a[0] : my_a[E - 1], t + u, G);
    acc_step<T, V>(acc[sa_sum<U, K>(u)], a, b[u], FM_FMA);
  }
}

template <class T, class VT, class PtrT, int G, int V>
__global__ void __launch_bounds__(SA_THREADS, 3) spmm_csr_auto(
    int64_t nrows, const PtrT* __restrict__ ptr, const int* __restrict__ idx, const VT* __restrict__ val,
    const T* __restrict__ B, int64_t ldb, T* __restrict__ C, int64_t ldc, int64_t c0, int64_t nk, int base,
    int accumulate, int64_t* __restrict__ carry_row, T* __restrict__ carry) {
  using IT = typename std::conditional<sizeof(PtrT) == 4, uint32_t, int64_t>::type;  // an entry's position
  constexpr int P = 32 / G, E = G < 8 ? 8 / G : 1;
  constexpr int U = sa_sums<T, G>();
  constexpr int NG = SA_THREADS / G, WARPS = SA_THREADS / 32;
  __shared__ int64_t s_long[SA_LIST];
  __shared__ int s_n;
  __shared__ VecT<T, V> s_part[2][WARPS][G];
  const int tid = threadIdx.x, lane = tid % G, g = tid / G;
  const unsigned gmask = group_mask<G>();
  const int64_t col = c0 + (int64_t)lane * V;
  const bool active = col < nk;  // V divides nk - c0
  const T* Bc = B + (active ? col : c0);  // lanes past nk gather what the group's first does, and store nothing
  const uint64_t pol_stream = policy_evict_first();
  const uint64_t pol_keep = policy_evict_last();
  const int64_t f0 = ld_ptr(ptr, 0);
  const int64_t steps = ld_ptr(ptr, nrows) - f0 + nrows;
  const int64_t per = (steps + gridDim.x - 1) / gridDim.x;
  const int64_t first = blockIdx.x * per, end = first + per;
  const int64_t whole = carry ? 2 * per : INT64_MAX;  // longer rows are cut at the shares
  pdl_allow_next();  // spmm_auto_fixup may be set up beside this launch
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

  // The sum of entries [p, p1) of a row by the group.
  auto fold = [&](IT p, IT p1) -> VecT<T, V> {
    VecT<T, V> acc[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
#pragma unroll
      for (int q = 0; q < V; ++q) acc[u].v[q] = T(0);
    for (IT pb = p; pb < p1; pb += G * E) {
      int my_j[E];
      T my_a[E];
#pragma unroll
      for (int e = 0; e < E; ++e) {
        const IT pe = pb + lane + e * G;
        my_j[e] = 0;
        my_a[e] = T(0);
        if (pe < p1) {
          my_j[e] = ld_stream_i32(idx + pe, pol_stream) - base;
          my_a[e] = load_val<T, VT>(val, pe, pol_stream);
        }
      }
      const int cnt = p1 - pb < (IT)(G * E) ? (int)(p1 - pb) : G * E;
      auto batch = [&](auto nb, auto kind, int t) {
        sa_batch<T, G, V, U, E, decltype(nb)::value, decltype(kind)::value>(acc, t, my_j, my_a, Bc, ldb, gmask,
                                                                            pol_keep);
      };
      int t = 0;
      if constexpr (U == 8) {  // 4 gathers ahead: 8 sums of 4 columns take the registers
        if (cnt == 8) {
          batch(Int<4>{}, Kind<SA_LOW4>{}, 0);
          batch(Int<4>{}, Kind<SA_HIGH4>{}, 4);
          t = 8;
        }
      } else {
        for (; t + 8 <= cnt; t += 8) batch(Int<8>{}, Kind<SA_EIGHT>{}, t);
      }
      if (t + 4 <= cnt) {
        batch(Int<4>{}, Kind<SA_FOUR>{}, t);
        t += 4;
      }
      if (t + 2 <= cnt) {
        batch(Int<2>{}, Kind<SA_REST>{}, t);
        t += 2;
      }
      if (t < cnt) batch(Int<1>{}, Kind<SA_REST>{}, t);
    }
#pragma unroll
    for (int h = U / 2; h >= 1; h >>= 1)
#pragma unroll
      for (int u = 0; u < h; ++u)
#pragma unroll
        for (int q = 0; q < V; ++q) acc[u].v[q] += acc[u + h].v[q];
    return acc[0];
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
    if (p1 - p0 > SA_ROW) {
      int kept = 0;
      if (lane == 0) {
        const int at = atomicAdd(&s_n, 1);
        if (at < SA_LIST) s_long[at] = row;
        kept = at < SA_LIST;  // always, if ptr ends where the host was told
      }
      if (__shfl_sync(gmask, kept, 0, G)) continue;
    }
    const VecT<T, V> acc = fold((IT)(p0 - base), (IT)(p1 - base));
    if (active) store(row, acc);
  }
  __syncthreads();
  const int nlong = s_n < SA_LIST ? s_n : SA_LIST;
  // Rows up to this length by the warps: from 4 of them that is sooner than a
  // barrier a row.
  const int by_warp = nlong >= 4 ? SA_WARP<T, G> : 0;
  // The part of a row that began in another share.
  const int64_t cut = lo > 0 ? lo - 1 : 0;
  int64_t c_first = 0, c_end = 0;
  if (carry && lo > 0) {
    const int64_t p0 = ld_ptr(ptr, cut) - f0, p1 = ld_ptr(ptr, cut + 1) - f0;
    if (p1 - p0 > whole) {
      c_first = first - cut;
      c_end = p1 < end - cut ? p1 : end - cut;
    }
  }
  const bool head = c_first < c_end;
  if (carry && c0 == 0 && tid == 0) carry_row[blockIdx.x] = head ? cut : -1;
  int turn = 0;
#pragma unroll 1
  for (int block = by_warp ? 0 : 1; block < 2; ++block) {  // the warps' rows, then the block's
    const int step = block ? 1 : WARPS;
#pragma unroll 1
    for (int l = block ? (head ? -1 : 0) : tid >> 5; l < nlong; l += step) {  // block- or warp-uniform
      int64_t row = cut, p0 = c_first + f0, p1 = c_end + f0;
      if (l >= 0) {
        row = s_long[l];
        p0 = ld_ptr(ptr, row);
        p1 = ld_ptr(ptr, row + 1);
        const bool cutting = p1 - p0 > whole;
        if ((p1 - p0 <= by_warp && !cutting) == (block != 0)) continue;
        if (cutting && p1 > f0 + end - row) p1 = f0 + end - row;  // the rest is the next blocks'
      }
      const int quantum = sizeof(T) == 4 ? 8 : block ? 16 : 1;
      const int parts = block ? NG : P, mine = block ? g : g % P;  // P groups a warp
      const int64_t part = ((p1 - p0 + parts - 1) / parts + quantum - 1) / quantum * quantum;
      const int64_t q0 = p0 + mine * part, q1 = q0 + part < p1 ? q0 + part : p1;
      VecT<T, V> acc;
#pragma unroll
      for (int q = 0; q < V; ++q) acc.v[q] = T(0);
      if (__any_sync(0xffffffffu, q0 < p1)) {  // warps with nothing to add leave the FP64 pipe to the others
        acc = fold((IT)(q0 < p1 ? q0 - base : 0), (IT)(q0 < p1 ? q1 - base : 0));
        __syncwarp();
#pragma unroll
        for (int m = G; m < 32; m <<= 1)
#pragma unroll
          for (int q = 0; q < V; ++q) acc.v[q] += __shfl_xor_sync(0xffffffffu, acc.v[q], m);
      }
      if (block) {
        turn ^= 1;  // the other half of s_part: one barrier a row
        if ((tid & 31) < G) s_part[turn][tid >> 5][lane] = acc;
        __syncthreads();
        if (tid < G) {
#pragma unroll
          for (int w = 1; w < WARPS; ++w)
#pragma unroll
            for (int q = 0; q < V; ++q) acc.v[q] += s_part[turn][w][lane].v[q];
        }
      }
      if (block ? tid >= G : (tid & 31) >= G) continue;
      if (!active) continue;
      if (l >= 0) {
        store(row, acc);
      } else {
#pragma unroll
        for (int q = 0; q < V; ++q) carry[blockIdx.x * nk + col + q] = acc.v[q];
      }
    }
  }
}

// Adds the carries of every row that was cut to it: a block per row, its
// carries in S consecutive runs, the runs in order.
template <class T, class PtrT>
__global__ void __launch_bounds__(SA_THREADS) spmm_auto_fixup(int64_t nrows, const PtrT* __restrict__ ptr,
                                                             int64_t nblocks, int64_t nk,
                                                             const int64_t* __restrict__ carry_row,
                                                             const T* __restrict__ carry, T* __restrict__ C,
                                                             int64_t ldc) {
  __shared__ T s_sum[SA_THREADS];
  pdl_wait_prev();
  int width = 4;  // columns at a time, a power of two
  while (width < nk && width < SA_THREADS) width *= 2;
  const int runs = SA_THREADS / width, run = threadIdx.x / width;
  for (int64_t w = blockIdx.x; w < nblocks; w += gridDim.x) {  // block-uniform
    const int64_t r = carry_row[w];
    if (r < 0 || (w > 0 && carry_row[w - 1] == r)) continue;
    const int64_t f0 = ld_ptr(ptr, 0);
    const int64_t per = (ld_ptr(ptr, nrows) - f0 + nrows + nblocks - 1) / nblocks;
    const int64_t n = (ld_ptr(ptr, r + 1) - f0 - 1 + r) / per - w + 1;  // its carries, up to its last entry's block
    const int64_t len = (n + runs - 1) / runs;
    const int64_t a = w + run * len, b = a + len < w + n ? a + len : w + n;
    for (int64_t c0 = 0; c0 < nk; c0 += width) {
      const int64_t c = c0 + threadIdx.x % width;
      T sum = T(0);
      if (c < nk) {
#pragma unroll 8
        for (int64_t k = a; k < b; ++k) sum += carry[k * nk + c];
      }
      s_sum[threadIdx.x] = sum;
      __syncthreads();
      if (run == 0 && c < nk) {
        for (int q = 1; q < runs; ++q) sum += s_sum[q * width + threadIdx.x];
        C[r * ldc + c] += sum;
      }
      __syncthreads();
    }
  }
}

// `need` given: only the scratch that the call takes.
template <class T, class VT, class PtrT, int G>
static int launch_auto(fgb_ctx* ctx, const fgb_sparse* A, const T* B, int64_t ldb, int64_t nk, T* C, int64_t ldc,
                       int accumulate, char* scratch, size_t* need, cudaStream_t s) {
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
  const size_t rows_bytes = (sizeof(int64_t) * grid + 255) & ~size_t(255);
  if (need) {
    // no row is as long where the matrix is no wider
    const bool cut = (double)steps * (double)nk * sizeof(T) >= SA_CUT_BYTES && A->ncols > 2 * share;
    *need = cut ? rows_bytes + sizeof(T) * grid * nk : 0;
    return FGB_OK;
  }
  int64_t* carry_row = (int64_t*)scratch;
  T* carry = scratch ? (T*)(scratch + rows_bytes) : nullptr;
  for (int64_t c0 = 0; c0 < nk; c0 += G * V) {
    kern<<<grid, SA_THREADS, 0, s>>>(A->nrows, (const PtrT*)A->ptr, (const int*)A->idx, (const VT*)A->val, B, ldb, C,
                                     ldc, c0, nk, A->index_base, accumulate, carry_row, carry);
    const int rc = check_launch("spmm_csr_auto");
    if (rc) return rc;
  }
  if (!carry) return FGB_OK;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::min<int64_t>(grid, 8 * ctx->num_sms));
  cfg.blockDim = dim3(SA_THREADS);
  cfg.stream = s;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, spmm_auto_fixup<T, PtrT>, A->nrows, (const PtrT*)A->ptr, (int64_t)grid, nk,
                     (const int64_t*)carry_row, (const T*)carry, C, ldc);
  return check_launch("spmm_auto_fixup");
}

template <class T, class VT>
static int auto_typed(fgb_ctx* ctx, const fgb_sparse* A, const void* B, int64_t ldb, int64_t nk, void* C, int64_t ldc,
                      int accumulate, char* scratch, size_t* need, cudaStream_t s) {
  constexpr int V = sizeof(T) == 4 ? 4 : 2;
  const int64_t lanes = (nk + V - 1) / V;  // that cover a row of B, at most a warp
  auto go = [&](auto ptr_t) -> int {
    using P = decltype(ptr_t);
    auto run = [&](auto g) {
      return launch_auto<T, VT, P, decltype(g)::value>(ctx, A, (const T*)B, ldb, nk, (T*)C, ldc, accumulate, scratch,
                                                       need, s);
    };
    if (lanes <= 4) return run(Int<4>{});
    if (lanes <= 8) return run(Int<8>{});
    if (lanes <= 16) return run(Int<16>{});
    return run(Int<32>{});
  };
  return A->ptr_t == FGB_I32 ? go(int32_t(0)) : go(int64_t(0));
}

static int auto_any(fgb_ctx* ctx, const fgb_sparse* A, const void* B, int64_t ldb, int64_t nk, void* C, int64_t ldc,
                    int dtype, int accumulate, char* scratch, size_t* need, cudaStream_t s) {
  if (dtype == FGB_F64)
    return auto_typed<double, double>(ctx, A, B, ldb, nk, C, ldc, accumulate, scratch, need, s);
  if (A->val_t == FGB_BF16)
    return auto_typed<float, __nv_bfloat16>(ctx, A, B, ldb, nk, C, ldc, accumulate, scratch, need, s);
  return auto_typed<float, float>(ctx, A, B, ldb, nk, C, ldc, accumulate, scratch, need, s);
}

size_t spmm_auto_scratch_bytes(fgb_ctx* ctx, const fgb_sparse* A, int64_t nk, int dtype) {
  size_t need = 0;
  if (A->nrows > 0 && nk > 0) auto_any(ctx, A, nullptr, 0, nk, nullptr, 0, dtype, 0, nullptr, &need, nullptr);
  return need;
}

int spmm_auto(fgb_ctx* ctx, const fgb_sparse* A, const void* B, int64_t ldb, int64_t nk, void* C, int64_t ldc,
              int dtype, int accumulate, void* scratch, size_t scratch_bytes, cudaStream_t s) {
  if (A->nrows == 0 || nk == 0) return FGB_OK;
  const size_t need = spmm_auto_scratch_bytes(ctx, A, nk, dtype);
  char* buf = need ? (char*)scratch : nullptr;
  if (buf && scratch_bytes < need)
    return set_error(FGB_EINVAL, "spmm: scratch of %zu bytes is below the %zu needed", scratch_bytes, need);
  if (need && !buf) FGB_CUDA_TRY(cudaMallocAsync((void**)&buf, need, s));
  const int rc = auto_any(ctx, A, B, ldb, nk, C, ldc, dtype, accumulate, buf, nullptr, s);
  if (buf && !scratch) cudaFreeAsync(buf, s);
  return rc;
}

}  // namespace fgb
