// Semiring SpMV over SparseList fibers.
//
// CSR (pull): a group of G lanes owns one row i and folds
//   acc = (+)_{j ascending} A[i,j] (*) x[j]
// lane-strided over the row's stored entries, then combines the G partials
// with xor-shuffles.  G = 1 is Finch's serial order: one running value per
// output, updated j ascending, exactly the update
//   y[i] = x[j] * A[i,j] + y[i]
// of Finch's CSC nest (test/reference64/typical/typical_spmv_csc.txt:61-79),
// so FGB_FINCH_ORDER results equal Finch's bit for bit.
//
// CSC (push): a group of G lanes owns one column j, reads x[j] once and
// applies y[i] <<(+)>>= A[i,j] (*) x[j] for every stored i with an atomic
// update.  For exact semirings (integer +, min, max, |) the atomics commute,
// so results are exact; float sums are exact up to summation order.
//
// OR-AND works on Bool (0 or 1) bytes, where `true` absorbs under | and
// `false` annihilates under &: the push skips the columns whose x[j] is
// false and the pull stops a lane's scan at its first true product.  The
// result is the full nest's, bit for bit; a sparse frontier touches only its
// own columns' entries.
#include <algorithm>
#include <type_traits>

#include "fgb_internal.cuh"
#include "semiring.cuh"

namespace fgb {

template <int SR, class VT, class A, class PtrT, int G, bool PATTERN, int FM>
__global__ void __launch_bounds__(256) spmv_csr_pull(int64_t nrows, const PtrT* __restrict__ ptr,
                                                     const int* __restrict__ idx,
                                                     const VT* __restrict__ val,
                                                     const A* __restrict__ x, A* __restrict__ y,
                                                     int base, int accumulate) {
  using S = Semi<SR, A>;
  const int lane = threadIdx.x & (G - 1);
  const int64_t group = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
  const int64_t ngroups = ((int64_t)gridDim.x * blockDim.x) / G;
  for (int64_t row = group; row < nrows; row += ngroups) {
    const int64_t p0 = ld_ptr(ptr, row) - base;
    const int64_t p1 = ld_ptr(ptr, row + 1) - base;
    A acc = (G == 1 && accumulate) ? y[row] : S::identity();
#pragma unroll 4
    for (int64_t p = p0 + lane; p < p1; p += G) {
      const int j = __ldg(idx + p) - base;
      const A a = PATTERN ? S::one() : to_acc<A>(val[p]);
      acc = S::step(acc, a, __ldg(x + j), FM);
      if (SR == SR_OA && acc) break;  // Bool: true absorbs every later product
    }
    if (G > 1) {
#pragma unroll
      for (int m = G / 2; m >= 1; m >>= 1) acc = S::add(acc, shfl_xor(group_mask<G>(), acc, m, G));
      if (lane == 0) y[row] = accumulate ? S::add(y[row], acc) : acc;
    } else {
      y[row] = acc;
    }
  }
}

// CSR pull that suits its schedule to the row lengths it finds, with no
// statistics from the host.  Every block reads the same 32 windows of 32
// consecutive rows, spread over the matrix (two coalesced loads a warp each).
//
// No sampled row longer than `cut`: `lanes` lanes per row, grid-strided, as
// spmv_csr_pull.  The groups of a warp are never made to meet (a ballot per
// row would have them wait for the longest of their rows: 171 against 140 us
// on the 4M-node graph), so a row of more than `limit` entries, which the
// sample missed, goes to a list.  Groups of 8 keep four sums a lane where rows
// average over 24 entries: a row's 32 sums, and its bits, are those of 32
// lanes, at fewer FP64 instructions (FP64, 400,000 rows of 100: 195 us, by
// equal shares with a warp a row 310).
//
// A longer row among them, or rows long on average (`cut` -1): the walk over
// rows and stored entries (row r sits at step r + ptr[r]) is cut into equal
// shares, one a warp, and a warp owns the rows that begin in its share: no row
// is split, no partial sums leave a warp, and a warp that meets long rows has
// fewer others.  It searches ptr for its first row and takes the rows 32 at a
// time: one of at most SPMV_LONG entries by its own lane, or, where the 32
// rows hold `fill4` entries, by 4 lanes (a lane's loads are uncoalesced: long
// enough rows pay for the two shuffles); a longer row by the whole warp, one
// of more than SPMV_BLOCK entries by way of the list.  Where the 32 rows
// average fewer than SPMV_SPARSE entries of 8 bytes, rows over
// SPMV_SPARSE_LONG count as long: the few lanes that had one kept the warp,
// and FP64 its pipe, busy for as many steps (Zipf 1M x 16, FP64, 153 -> 139
// us; 4M x 2 118 -> 103).  For 4-byte values it gains 2-7 % there, but the
// 4-byte builds spill as it is (28 to 40 bytes at the 32 registers that keep
// 64 warps an SM), more with the rule, and the 4M-node graph loses 5 %.
//
// When a block's warps are done they share its list, the longest rows by the
// whole block.  Which rows the list takes, and so a row's order of summation,
// depends on the matrix alone: lane groups that leave more than it holds have
// it filled again, run by run, and a warp lists the first of its own rows.
// `ordered` (FGB_FINCH_ORDER) folds every row as one running value, j
// ascending: a long row's entries are loaded 32 at a time and folded in order
// by every lane, in FP64 32 times a lane's own work for the pipe; so evenly
// long rows stay with their lanes where there are rows enough to fill the
// device (FP64, 400,000 rows of 50: 167 against 1,160 us by their warps).
//
// Bound: the gathers of x (one L1 tag a clock per SM), FP64 folds also by the
// FP64 pipe.  GB300, per call behind a cold L2, against fixed groups of 8 or
// 32 lanes or, over 311,296 rows, one lane for rows up to 32 entries and a
// warp for longer ones, with the contraction chosen at run time: Zipf 1M x 16
// FP64 281 -> 136 us, FP32 165 -> 103; uniform 4M x 8 FP64 365 -> 184, FP32
// 166 -> 144, Int32 min-plus 166 -> 144; rows of 4,000, 2,000 of them, FP64
// 82 -> 53, FP32 73 -> 46; 64 rows of 100,000, FP32, 1,205 -> 124.  The sample
// costs a uniform matrix about 1 us: 20,000 rows of 16, FP32, 3.2 -> 4.3 us in
// a graph.  Staging tiles of entries in shared memory (coalesced, every row
// folded from there) measured 298 (FP64) and 184 (FP32) on the uniform 4M
// rows, and equal shares alone 194 and 162.
constexpr int SPMV_LONG = 32, SPMV_SPARSE_LONG = 16, SPMV_SPARSE = 6;
constexpr int SPMV_BLOCK = 2048;  // a warp alone takes 8 us for one
constexpr int SPMV_LIST = 64;  // rows a block can leave to the end (a longer list costs L1)
constexpr int SPMV_MEAN4 = 14;

// First row whose step ptr[r] - f0 + r is at least `target` (nrows if none),
// by the warp: 32 probes a round.
template <class PtrT>
__device__ __forceinline__ int64_t spmv_step_row(int64_t nrows, const PtrT* __restrict__ ptr, int64_t f0,
                                                 int64_t entries, int64_t target, int lane) {
  int64_t lo = target > entries ? target - entries : 0;
  int64_t hi = target < nrows ? target : nrows;
  if (lo > hi) lo = hi;
  while (lo < hi) {  // warp-uniform; the span shrinks to at most span / 32 a round
    const int64_t step = (hi - lo + 31) / 32;
    const int64_t q = lo + lane * step;
    const bool before = q < hi && ld_ptr(ptr, q) - f0 + q < target;
    const int n = __popc(__ballot_sync(0xffffffffu, before));
    if (n == 0) {
      hi = lo;
    } else {
      const int64_t next = lo + n * step;
      lo += (n - 1) * step + 1;
      if (next < hi) hi = next;
    }
  }
  return lo;
}

template <int SR, class VT, class A, class PtrT, int FM>
__global__ void __launch_bounds__(256, sizeof(A) == 8 ? 6 : 8) spmv_csr_auto(int64_t nrows, const PtrT* __restrict__ ptr,
                                                        const int* __restrict__ idx,
                                                        const VT* __restrict__ val,
                                                        const A* __restrict__ x, A* __restrict__ y,
                                                        int base, int accumulate, int ordered, int lanes, int sums,
                                                        int64_t cut, int limit, int fill4) {
  using S = Semi<SR, A>;
  using IT = typename std::conditional<sizeof(PtrT) == 4, uint32_t, int64_t>::type;  // an entry's position
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int WARPS = 8;
  __shared__ A s_red[WARPS];
  __shared__ int64_t s_row[SPMV_LIST];  // rows left until the others are done
  __shared__ int s_n;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t warp = (int64_t)blockIdx.x * WARPS + w;
  const int64_t nwarps = (int64_t)gridDim.x * WARPS;
  // the thread's first row by lane groups, read beside the sample
  const int64_t first = (blockIdx.x * 256u + threadIdx.x) / (unsigned)lanes;
  IT p0 = 0, p1 = 0;
  bool over = false;
#pragma unroll
  for (int u = 0; u < 32 / WARPS; ++u) {
    const int64_t r = (int64_t)(w * (32 / WARPS) + u) * nrows / 32 + lane;
    if (r < nrows) over |= ld_ptr(ptr, r + 1) - ld_ptr(ptr, r) > cut;
  }
  if (threadIdx.x == 0) s_n = 0;
  const bool skewed = __syncthreads_or(over);

  constexpr std::integral_constant<bool, sizeof(A) == 8> wide{};
  auto term = [&](A acc, IT p) { return S::step(acc, to_acc<A>(val[p]), __ldg(x + (__ldg(idx + p) - base)), FM); };
  // Entries p, p + stride, ... below p1, added to `acc` in that order, four
  // of them loaded at once.  AHEAD: their values before the gathers of x, not
  // behind them (a choice of registers in flight, by measurement).
  auto fold = [&](A acc, IT p, IT p1, int stride, auto ahead) -> A {
    constexpr bool AHEAD = decltype(ahead)::value;
    for (; p + 3 * stride < p1; p += 4 * stride) {
      A a[4], xv[4];
      int j[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        j[u] = __ldg(idx + p + u * stride);
        if (AHEAD) a[u] = to_acc<A>(val[p + u * stride]);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) xv[u] = __ldg(x + (j[u] - base));
      if (!AHEAD)
#pragma unroll
        for (int u = 0; u < 4; ++u) a[u] = to_acc<A>(val[p + u * stride]);
#pragma unroll
      for (int u = 0; u < 4; ++u) acc = S::step(acc, a[u], xv[u], FM);
    }
#pragma unroll
    for (int u = 0; u < 3; ++u)
      if (p + u * stride < p1) acc = term(acc, p + u * stride);
    return acc;
  };
  auto fold_long = [&](int64_t row, IT q0, IT q1) {  // one row by the warp
    A acc;
    if (ordered) {
      acc = accumulate ? y[row] : S::identity();
      for (IT q = q0; q < q1; q += 32) {
        A a = A(0), xv = A(0);
        if (q + lane < q1) {
          a = to_acc<A>(val[q + lane]);
          xv = __ldg(x + (__ldg(idx + q + lane) - base));
        }
        const int n = q1 - q < 32 ? (int)(q1 - q) : 32;
#pragma unroll 4
        for (int u = 0; u < n; ++u)
          acc = S::step(acc, __shfl_sync(FULL, a, u), __shfl_sync(FULL, xv, u), FM);
      }
    } else {
      acc = fold(S::identity(), q0 + lane, q1, 32, wide);
#pragma unroll
      for (int m = 16; m >= 1; m >>= 1) acc = S::add(acc, shfl_xor(FULL, acc, m, 32));
      if (accumulate) acc = S::add(y[row], acc);
    }
    if (lane == 0) y[row] = acc;
  };

  // G lanes a row, U running sums a lane: entry p of a row is added to the
  // row's sum p mod G * U, and the sums are folded as a tree.
  auto by_lanes = [&](auto lanes_c, auto sums_c) {
    constexpr int G = decltype(lanes_c)::value, U = decltype(sums_c)::value;
    const int sub = lane % G;
    const int64_t ngroups = nwarps * 32 / G;
    for (int64_t row = first; row < nrows; row += ngroups) {
      p0 = (IT)(ld_ptr(ptr, row) - base);
      p1 = (IT)(ld_ptr(ptr, row + 1) - base);
      if (p1 - p0 > (IT)limit) {  // not sampled: the warps of the block fold it afterwards
        if (sub == 0) {
          const int at = atomicAdd(&s_n, 1);
          if (at < SPMV_LIST) s_row[at] = row;
        }
        continue;
      }
      A acc[U];
      acc[0] = G == 1 && accumulate ? y[row] : S::identity();
#pragma unroll
      for (int u = 1; u < U; ++u) acc[u] = S::identity();
      if constexpr (U == 1) {
        acc[0] = fold(acc[0], p0 + sub, p1, G, std::true_type{});
      } else {
        for (IT p = p0 + sub; p < p1; p += G * U) {
#pragma unroll
          for (int u = 0; u < U; ++u)
            if (p + u * G < p1) acc[u] = term(acc[u], p + u * G);
        }
#pragma unroll
        for (int h = U / 2; h >= 1; h >>= 1)
#pragma unroll
          for (int u = 0; u < h; ++u) acc[u] = S::add(acc[u], acc[u + h]);
      }
      if (G > 1) {
#pragma unroll
        for (int m = G / 2; m >= 1; m >>= 1) acc[0] = S::add(acc[0], shfl_xor(group_mask<G>(), acc[0], m, G));
        if (sub == 0) y[row] = accumulate ? S::add(y[row], acc[0]) : acc[0];
      } else {
        y[row] = acc[0];
      }
    }
  };
  if (!skewed) {
    using std::integral_constant;
    if (lanes == 1) by_lanes(integral_constant<int, 1>{}, integral_constant<int, 1>{});
    else if (lanes == 4) by_lanes(integral_constant<int, 4>{}, integral_constant<int, 1>{});
    else if (lanes == 32) by_lanes(integral_constant<int, 32>{}, integral_constant<int, 1>{});
    else if (sums == 1) by_lanes(integral_constant<int, 8>{}, integral_constant<int, 1>{});
    else by_lanes(integral_constant<int, 8>{}, integral_constant<int, 4>{});
  } else {
    const int64_t f0 = ld_ptr(ptr, 0);
    const int64_t entries = ld_ptr(ptr, nrows) - f0;
    const int64_t per = (entries + nrows + nwarps - 1) / nwarps;
    const int64_t end = (warp + 1) * per;
    int64_t r0 = spmv_step_row(nrows, ptr, f0, entries, warp * per, lane);
    int listed = 0;
    while (true) {  // warp-uniform
      const int64_t row = r0 + lane;
      p0 = p1 = 0;
      bool mine = false;
      if (row < nrows) {
        const int64_t at = ld_ptr(ptr, row), to = ld_ptr(ptr, row + 1);
        mine = at - f0 + row < end;
        p0 = (IT)(at - base);
        p1 = mine ? (IT)(to - base) : p0;
      }
      const IT n = p1 - p0;
      const int filled = sizeof(A) == 8 || !ordered  // entries in rows of at most SPMV_LONG
                             ? __reduce_add_sync(FULL, n <= SPMV_LONG ? (int)n : 0) : 0;
      const bool is_long = n > (IT)(ordered ? limit : sizeof(A) == 8 && filled < 32 * SPMV_SPARSE ? SPMV_SPARSE_LONG : SPMV_LONG);
      const int sn = is_long || !mine ? -1 : (int)n;  // a short row's entries
      if (!ordered && filled >= fill4) {
        const int sub = lane & 3;
#pragma unroll 1
        for (int b = lane >> 2; b < 32; b += 8) {
          const IT q0 = __shfl_sync(FULL, p0, b);
          const int bn = __shfl_sync(FULL, sn, b);
          A acc = S::identity();
          if (bn > 0) acc = fold(acc, q0 + sub, q0 + bn, 4, wide);
          acc = S::add(acc, shfl_xor(FULL, acc, 2, 32));
          acc = S::add(acc, shfl_xor(FULL, acc, 1, 32));
          if (sub == 0 && bn >= 0) y[r0 + b] = accumulate ? S::add(y[r0 + b], acc) : acc;
        }
      } else if (sn >= 0) {
        A acc = accumulate ? y[row] : S::identity();
        const int* ix = idx + p0;
        const VT* vx = val + p0;
#pragma unroll 4
        for (int k = 0; k < sn; ++k) acc = S::step(acc, to_acc<A>(vx[k]), __ldg(x + (__ldg(ix + k) - base)), FM);
        y[row] = acc;
      }
      unsigned longs = __ballot_sync(FULL, is_long);
      while (longs) {
        const int l = __ffs(longs) - 1;
        longs &= longs - 1;
        const IT q0 = __shfl_sync(FULL, p0, l), m = __shfl_sync(FULL, n, l);
        if (m > SPMV_BLOCK && !ordered && listed < SPMV_LIST / WARPS) {  // never more than the list holds
          if (lane == 0) s_row[atomicAdd(&s_n, 1)] = r0 + l;
          ++listed;
          continue;
        }
        fold_long(r0 + l, q0, q0 + m);
      }
      if (!__shfl_sync(FULL, (int)mine, 31)) break;  // the warp's rows end here
      r0 += 32;
    }
  }

  __syncthreads();
  // Lane groups may leave more than the list holds: it is then filled again
  // from SPMV_LIST of the block's rows at a time, so which rows the warps fold
  // does not depend on who came first.
  const bool again = s_n > SPMV_LIST;
  const int round = 256 / lanes;  // rows the block's groups take at once
  int64_t rb = (int64_t)blockIdx.x * round, part = 0;
  do {  // block-uniform
    if (again) {
      __syncthreads();
      if (threadIdx.x == 0) s_n = 0;
      __syncthreads();
      const int64_t row = rb + part + threadIdx.x;
      if (threadIdx.x < SPMV_LIST && part + threadIdx.x < round && row < nrows &&
          ld_ptr(ptr, row + 1) - ld_ptr(ptr, row) > limit)
        s_row[atomicAdd(&s_n, 1)] = row;
      __syncthreads();
      part += SPMV_LIST;
      if (part >= round) {
        part = 0;
        rb += (int64_t)gridDim.x * round;
      }
    }
    const int left = s_n;
    for (int l = w; l < left; l += WARPS) {
      const int64_t row = s_row[l];
      const IT q0 = (IT)(ld_ptr(ptr, row) - base), q1 = (IT)(ld_ptr(ptr, row + 1) - base);
      if (ordered || q1 - q0 <= SPMV_BLOCK) fold_long(row, q0, q1);
    }
    for (int l = 0; l < left && !ordered; ++l) {  // block-uniform: the longest by the whole block
      const int64_t row = s_row[l];
      const IT q0 = (IT)(ld_ptr(ptr, row) - base), q1 = (IT)(ld_ptr(ptr, row + 1) - base);
      if (q1 - q0 <= SPMV_BLOCK) continue;
      A acc = fold(S::identity(), q0 + threadIdx.x, q1, 32 * WARPS, wide);
#pragma unroll
      for (int m = 16; m >= 1; m >>= 1) acc = S::add(acc, shfl_xor(FULL, acc, m, 32));
      if (lane == 0) s_red[w] = acc;
      __syncthreads();
      if (threadIdx.x == 0) {
        for (int v = 1; v < WARPS; ++v) acc = S::add(acc, s_red[v]);
        y[row] = accumulate ? S::add(y[row], acc) : acc;
      }
      __syncthreads();
    }
  } while (again && rb < nrows);
}

template <int SR, class VT, class A, class PtrT, int G, bool PATTERN>
__global__ void __launch_bounds__(256) spmv_csc_push(int64_t ncols, const PtrT* __restrict__ ptr,
                                                     const int* __restrict__ idx,
                                                     const VT* __restrict__ val,
                                                     const A* __restrict__ x, A* __restrict__ y,
                                                     int base) {
  using S = Semi<SR, A>;
  const int lane = threadIdx.x & (G - 1);
  const int64_t group = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
  const int64_t ngroups = ((int64_t)gridDim.x * blockDim.x) / G;
  for (int64_t col = group; col < ncols; col += ngroups) {
    const A xj = __ldg(x + col);
    if (SR == SR_OA && !xj) continue;  // Bool: a & false adds nothing to any y[i]
    const int64_t p0 = ld_ptr(ptr, col) - base;
    const int64_t p1 = ld_ptr(ptr, col + 1) - base;
    if (p0 >= p1) continue;
    for (int64_t p = p0 + lane; p < p1; p += G) {
      const int i = __ldg(idx + p) - base;
      const A a = PATTERN ? S::one() : to_acc<A>(val[p]);
      AtomicAdd<SR, A>::apply(y + i, S::mul(a, xj));
    }
  }
}

// OR-AND push, warp-cooperative.  Each lane reads x for one column of a
// 32-column tile (four tiles in flight per lane); the warp takes an exclusive
// scan of the true columns' entry counts and spreads those entries over its
// 32 lanes, each finding its column by a binary search of the scan held in
// registers.  A false column costs one byte of x; the warp's lanes stay busy
// whatever the frontier's density.
template <class VT, class PtrT, bool PATTERN>
__global__ void __launch_bounds__(256) spmv_csc_push_oa(int64_t ncols, const PtrT* __restrict__ ptr,
                                                        const int* __restrict__ idx,
                                                        const VT* __restrict__ val,
                                                        const uint8_t* __restrict__ x,
                                                        uint8_t* __restrict__ y, int base) {
  constexpr unsigned FULL = 0xffffffffu;
  constexpr int U = 4;
  const int lane = threadIdx.x & 31;
  const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t c0 = warp * 32 * U; c0 < ncols; c0 += nwarps * 32 * U) {
    uint8_t xv[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int64_t col = c0 + 32 * u + lane;
      xv[u] = col < ncols ? __ldg(x + col) : uint8_t(0);
    }
#pragma unroll 1
    for (int u = 0; u < U; ++u) {
      const int64_t col = c0 + 32 * u + lane;
      if (!__any_sync(FULL, xv[u] != 0)) continue;
      int64_t p0 = 0, deg = 0;
      if (xv[u]) {
        p0 = ld_ptr(ptr, col) - base;
        deg = ld_ptr(ptr, col + 1) - base - p0;
      }
      int64_t incl = deg;  // inclusive scan of the entry counts over the warp
#pragma unroll
      for (int m = 1; m < 32; m <<= 1) {
        const int64_t t = __shfl_up_sync(FULL, incl, m);
        if (lane >= m) incl += t;
      }
      const int64_t excl = incl - deg;
      const int64_t total = __shfl_sync(FULL, incl, 31);
      for (int64_t k = 0; k < total; k += 32) {
        const int64_t e = k + lane;
        // owner: the largest lane whose scan start is <= e (it has entries)
        int l = 0;
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
          const int64_t s = __shfl_sync(FULL, excl, l + step);
          if (s <= e) l += step;
        }
        const int64_t pp = __shfl_sync(FULL, p0, l) + (e - __shfl_sync(FULL, excl, l));
        const uint8_t xj = __shfl_sync(FULL, xv[u], l);
        if (e < total) {
          const int i = __ldg(idx + pp) - base;
          const uint8_t a = PATTERN ? uint8_t(1) : val[pp];
          if (a & xj) *(volatile uint8_t*)(y + i) = 1;
        }
      }
    }
  }
}

template <int SR, class A>
__global__ void fill_identity(A* __restrict__ y, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    y[i] = Semi<SR, A>::identity();
}

// Lanes per fiber chosen by the plan autotuner for the calls it times and
// captures (0 = the heuristic below, 2 = spmv_csr_auto); set only around
// those calls.
static thread_local int t_group_override = 0;
constexpr int SPMV_AUTO = 2;
// Rows + entries from which a call without a plan takes spmv_csr_auto: below,
// its sample and its list cost about what a skewed matrix gains (10,000 rows
// of 2, FP32: 6.2 us uniform and 8.3 Zipf, against 4.2 and 16.5 by lanes).
constexpr int64_t SPMV_AUTO_STEPS = 1 << 16;

static int pick_group(double avg) {
  if (avg <= 2.0) return 1;
  if (avg <= 8.0) return 4;
  if (avg <= 24.0) return 8;
  return 32;
}

template <int SR, class VT, class A, class PtrT, bool PATTERN>
static int launch_typed(fgb_ctx* ctx, const fgb_sparse* A_, const void* x, void* y, unsigned flags,
                        cudaStream_t s) {
  const int base = A_->index_base;
  const int64_t nf = n_fibers(A_);
  const PtrT* ptr = (const PtrT*)A_->ptr;
  const int* idx = (const int*)A_->idx;
  const VT* val = (const VT*)A_->val;
  const double avg = nf ? (double)A_->nnz / (double)nf : 0.0;
  const int threads = 256;
  if (A_->orient == FGB_CSR) {
    const int accumulate = (flags & FGB_ACCUMULATE) ? 1 : 0;
    int fm = FM_DEFAULT;
    if (flags & FGB_NO_FMA) fm = FM_NOFMA;
    if (flags & FGB_FMA) fm = FM_FMA;
    if (nf == 0) return FGB_OK;
    const bool ordered = flags & FGB_FINCH_ORDER;
    int G = t_group_override > 0 ? t_group_override : ordered ? 1 : pick_group(avg);
    if constexpr (SR != SR_OA) {
      const int64_t steps = nf + A_->nnz;
      if (t_group_override > 0 ? G == SPMV_AUTO : steps >= SPMV_AUTO_STEPS) {
        // Lanes per row where no long row is sampled.  With rows enough to
        // fill the device, one, and 4 from 14 entries a row (8-byte values:
        // 1M x 8 rows 52 against 64 us, x 24 rows 176 against 131) or from 6
        // (4-byte: 4M x 2 rows 41 against 74, x 8 rows 148 against 142); with
        // fewer rows more lanes, so that more of the device works.  Over 24
        // entries a row (32 with many rows) 8 lanes with four sums each; 32
        // lanes where 8 a row leave 4-byte rows over 64 entries short of
        // warps (8,192 x 400, FP32: 14.4 us, by 8 27).  Equal shares, a warp
        // a row, from 160 entries a row (FP64 8,192 x 400 25 us, by 8 lanes
        // 51; 8,192 x 100 16.6 against 12.8; FP32 400,000 x 200 314 against
        // 329, x 100 187 against 176), few 4-byte rows from 640 (70,000 x 200
        // 67 against 44 by 8 lanes, 2,000 x 4,000 46 against 73).
        const bool many = nf >= (int64_t)ctx->num_sms * 2048;
        const bool wide = sizeof(A) == 8;
        int lanes = avg <= 2.0 ? 1 : avg <= 8.0 || wide ? 4 : 8, sums = 1;
        bool shares = false;
        if (ordered) lanes = 1;
        else if (avg > (many ? 32 : 24)) {
          shares = avg > (wide || many ? 160 : 640);
          lanes = avg > 64 && nf * 8 < (int64_t)ctx->num_sms * 2048 && !wide ? 32 : 8;
          sums = lanes == 32 ? 1 : 4;
        } else if (many) lanes = avg < (wide ? SPMV_MEAN4 : 6) ? 1 : 4;
        const int64_t spread = std::max<int64_t>(SPMV_LONG, (int64_t)(4.0 * avg));
        // A row that the sample would accept is not one that it missed.  In
        // Finch's order long rows go to their warps where they are fewer than
        // about the resident warps, which is where a lane's chain is longer
        // (FP64: 1,000 x 1,000 103 us by warps, 462 by lanes; 70,000 x 50 214
        // against 37; FP32, whose pipe is wider, 8,192 x 400 44 against 111).
        int64_t cut = spread, limit = std::max<int64_t>(32 * lanes, avg > 24 ? spread : 0);
        if (ordered) limit = avg > 24 && nf > (int64_t)ctx->num_sms * (wide ? 48 : 160) ? spread : SPMV_LONG;
        if (avg > 24 || !ordered) cut = std::min(cut, limit);
        limit = std::min<int64_t>(limit, 1 << 30);
        if (shares) cut = -1;
        // Rows that 4 or 8 lanes folded before lanes were sampled keep 4 sums
        // in FP32 (rows of 5 to 32 entries, 100,000 x 12 Zipf: relative error
        // 4.0e-8, with one sum 7.2e-8).
        const int fill4 = !many && avg > 2 && !wide ? 0 : 32 * SPMV_MEAN4;
        auto go = [&](auto fmc) {
          auto kern = spmv_csr_auto<SR, VT, A, PtrT, decltype(fmc)::value>;
          static const int occ = [&] {  // once per process (one device model); thread-safe
            int o = 0;
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&o, kern, threads, 0);
            return o > 0 ? o : 1;
          }();
          const int64_t need = (steps + 8 * 64 - 1) / (8 * 64);  // at least 64 steps a warp
          const int grid = (int)std::min<int64_t>(need, (int64_t)occ * ctx->num_sms);
          kern<<<grid, threads, 0, s>>>(nf, ptr, idx, val, (const A*)x, (A*)y, base, accumulate, ordered ? 1 : 0,
                                        lanes, sums, cut, (int)limit, fill4);
        };
        bool unfused = false;
        if constexpr (SR == SR_PT && std::is_floating_point<A>::value) {
          unfused = fm == FM_NOFMA;
          if (unfused) go(std::integral_constant<int, FM_NOFMA>{});
        }
        if (!unfused) go(std::integral_constant<int, FM_FMA>{});
        return check_launch("spmv_csr_auto");
      }
    }
    int grid = grid_for(nf * G, threads, ctx->num_sms, 8);
#define FGB_PULL_FM(GG, FMC)                                              \
  spmv_csr_pull<SR, VT, A, PtrT, GG, PATTERN, FMC><<<grid, threads, 0, s>>>( \
      nf, ptr, idx, val, (const A*)x, (A*)y, base, accumulate)
#define FGB_PULL(GG)                                                           \
  do {                                                                         \
    if constexpr (SR == SR_PT && std::is_floating_point<A>::value) {           \
      if (fm == FM_NOFMA) {                                                    \
        FGB_PULL_FM(GG, FM_NOFMA);                                             \
        break;                                                                 \
      }                                                                        \
    }                                                                          \
    FGB_PULL_FM(GG, FM_FMA);                                                   \
  } while (0)
    switch (G) {
      case 1: FGB_PULL(1); break;
      case 4: FGB_PULL(4); break;
      case 8: FGB_PULL(8); break;
      default: FGB_PULL(32); break;
    }
#undef FGB_PULL
#undef FGB_PULL_FM
    return check_launch("spmv_csr_pull");
  }
  // CSC push
  const int64_t m = A_->nrows;
  if (!(flags & FGB_ACCUMULATE) && m > 0) {
    fill_identity<SR, A><<<grid_for(m, threads, ctx->num_sms, 4), threads, 0, s>>>((A*)y, m);
    int rc = check_launch("fill_identity");
    if (rc) return rc;
  }
  if (nf == 0) return FGB_OK;
  if constexpr (SR == SR_OA) {
    if (t_group_override <= 0) {  // the plan may still time the lane-group kernels
      const int grid = grid_for((nf + 127) / 128 * 32, threads, ctx->num_sms, 8);
      spmv_csc_push_oa<VT, PtrT, PATTERN><<<grid, threads, 0, s>>>(nf, ptr, idx, val, (const uint8_t*)x,
                                                                  (uint8_t*)y, base);
      return check_launch("spmv_csc_push_oa");
    }
  }
  int G = t_group_override > 0 ? (t_group_override <= 1 ? 1 : t_group_override <= 8 ? 8 : 32)
                               : (avg <= 4.0 ? 1 : (avg <= 16.0 ? 8 : 32));
  int grid = grid_for(nf * G, threads, ctx->num_sms, 8);
#define FGB_PUSH(GG)                                                                    \
  spmv_csc_push<SR, VT, A, PtrT, GG, PATTERN><<<grid, threads, 0, s>>>(nf, ptr, idx, val, \
                                                                      (const A*)x, (A*)y, base)
  switch (G) {
    case 1: FGB_PUSH(1); break;
    case 8: FGB_PUSH(8); break;
    default: FGB_PUSH(32); break;
  }
#undef FGB_PUSH
  return check_launch("spmv_csc_push");
}

template <int SR, class VT, class A, bool PATTERN = false>
static int launch_ptr(fgb_ctx* ctx, const fgb_sparse* A_, const void* x, void* y, unsigned flags,
                      cudaStream_t s) {
  if (A_->ptr_t == FGB_I32)
    return launch_typed<SR, VT, A, int32_t, PATTERN>(ctx, A_, x, y, flags, s);
  return launch_typed<SR, VT, A, int64_t, PATTERN>(ctx, A_, x, y, flags, s);
}

template <int SR>
static int dispatch_numeric(fgb_ctx* ctx, const fgb_sparse* A_, const void* x, int x_t, void* y,
                            int y_t, unsigned flags, cudaStream_t s) {
  const int v = A_->val_t;
  if (x_t != y_t) return set_error(FGB_EUNSUPPORTED, "fgb_spmv: x and y dtypes differ");
  switch (y_t) {
    case FGB_F64:
      if (v == FGB_F64) return launch_ptr<SR, double, double>(ctx, A_, x, y, flags, s);
      break;
    case FGB_F32:
      if (v == FGB_F32) return launch_ptr<SR, float, float>(ctx, A_, x, y, flags, s);
      if (v == FGB_BF16 && SR == SR_PT)
        return launch_ptr<SR_PT, __nv_bfloat16, float>(ctx, A_, x, y, flags, s);
      break;
    case FGB_I32:
      if (v == FGB_I32) return launch_ptr<SR, int32_t, int32_t>(ctx, A_, x, y, flags, s);
      break;
    case FGB_I64:
      if (v == FGB_I64) return launch_ptr<SR, int64_t, int64_t>(ctx, A_, x, y, flags, s);
      break;
    default: break;
  }
  return set_error(FGB_EUNSUPPORTED, "fgb_spmv: no kernel for semiring %d with val %d, x/y %d", SR,
                   v, y_t);
}

}  // namespace fgb

using namespace fgb;

extern "C" int fgb_spmv(fgb_ctx* ctx, int semiring, const fgb_sparse* A, const void* x, int x_t,
                        void* y, int y_t, unsigned flags, void* stream) {
  if (!ctx) return set_error(FGB_EINVAL, "fgb_spmv: null ctx");
  int rc = check_sparse(A, "fgb_spmv: A", true);
  if (rc) return rc;
  const int64_t n_in = A->ncols, n_out = A->nrows;
  if ((n_in > 0 && !x) || (n_out > 0 && !y)) return set_error(FGB_EINVAL, "fgb_spmv: null x or y");
  if ((flags & FGB_FINCH_ORDER) && A->orient != FGB_CSR)
    return set_error(FGB_EUNSUPPORTED,
                     "fgb_spmv: FGB_FINCH_ORDER needs a CSR matrix (transpose once with "
                     "fgb_transpose)");
  cudaStream_t s = pick_stream(ctx, stream);
  switch (semiring) {
    case FGB_PLUS_TIMES: return dispatch_numeric<SR_PT>(ctx, A, x, x_t, y, y_t, flags, s);
    case FGB_MIN_PLUS: return dispatch_numeric<SR_MINP>(ctx, A, x, x_t, y, y_t, flags, s);
    case FGB_MAX_PLUS: return dispatch_numeric<SR_MAXP>(ctx, A, x, x_t, y, y_t, flags, s);
    case FGB_OR_AND:
      if (x_t != FGB_BOOL || y_t != FGB_BOOL)
        return set_error(FGB_EUNSUPPORTED, "fgb_spmv: OR_AND needs Bool x and y");
      if (A->val_t == FGB_NONE)
        return launch_ptr<SR_OA, uint8_t, uint8_t, true>(ctx, A, x, y, flags, s);
      if (A->val_t == FGB_BOOL)
        return launch_ptr<SR_OA, uint8_t, uint8_t, false>(ctx, A, x, y, flags, s);
      return set_error(FGB_EUNSUPPORTED, "fgb_spmv: OR_AND needs Bool or Pattern values");
    default: return set_error(FGB_EINVAL, "fgb_spmv: unknown semiring %d", semiring);
  }
}

namespace fgb {
// fgb_spmv with the lanes per fiber fixed to `group` (1, 4, 8 or 32).
int spmv_with_group(fgb_ctx* ctx, int semiring, const fgb_sparse* A, const void* x, int x_t,
                    void* y, int y_t, unsigned flags, int group, void* stream) {
  t_group_override = group;
  const int rc = fgb_spmv(ctx, semiring, A, x, x_t, y, y_t, flags, stream);
  t_group_override = 0;
  return rc;
}
}  // namespace fgb
