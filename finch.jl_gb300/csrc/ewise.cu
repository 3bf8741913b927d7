// Elementwise ops of two SparseList matrices and the fused
// elementwise-multiply + reduction.
//
// Two sparse operands (C = A .* B, C = A .+ B, sum(A .* B; dims)): a block
// takes consecutive fibers, whose coordinates are two contiguous runs, and
// merges each pair of sorted lists as Finch's two-finger merge does
// (test/reference64/typical/typical_merge_twofinger.txt: advance the smaller
// coordinate, emit on a match); see ew_tile_k.  Pass 1 of a sparse result
// counts each output fiber and a scan turns the counts into out_ptr; pass 2
// merges again and writes idx/val.
//
// sum(A .* B; dims) with a dense B: every fiber is reduced by a group of
// lanes.  Reductions along the compressed coordinate scatter into y with
// atomics; the all-dims reduction writes one partial per fiber and folds them
// in a fixed order, so it is deterministic.
#include <algorithm>
#include <climits>
#include <cub/cub.cuh>

#include "fgb_internal.cuh"
#include "semiring.cuh"

namespace fgb {

template <class PtrT>
struct Fiber {
  const PtrT* ptr;
  const int* idx;
  int base;
  __device__ int64_t lo(int64_t f) const { return ld_ptr(ptr, f) - base; }
  __device__ int64_t hi(int64_t f) const { return ld_ptr(ptr, f + 1) - base; }
  __device__ int at(int64_t p) const { return __ldg(idx + p) - base; }
};

// ---- merges of two sparse operands

enum { EW_COUNT = 0, EW_FILL = 1, EW_REDUCE = 2, EW_SCATTER = 3 };
constexpr int EW_THREADS = 128;
constexpr int EW_CAP = 2304;   // coordinates of a tile staged in shared memory
constexpr int EW_MEAN = 2048;  // coordinates a tile is sized for
constexpr int EW_LONG = 64;    // a pair of lists up to this length is merged by one thread
constexpr int EW_HUGE = 512;     // beyond this length the whole block merges a pair
constexpr unsigned EW_NONE = 0xffff;
static_assert(EW_CAP < EW_NONE, "a tile position fits 16 bits");

// For every element i of the ascending list ai[0, na) (stored from abase), by a warp: calls
// f(i, c, lb, match, before) in chunks of 32 (f is called by all lanes, with
// i < na where the lane has an element): lb is the number of elements of bi
// below c = ai[i], match whether bi[lb] == c, before the matches of elements
// below i.  bi is read once, a window of 32 at a time and two windows ahead;
// ranks are found by shuffles.
template <class F>
__device__ __forceinline__ void ew_warp_ranks(const int* ai, int abase, int na, const int* bi, int bbase, int nb,
                                              F&& f) {
  constexpr unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int b0 = 0, before = 0;
  int win = lane < nb ? bi[lane] - bbase : INT_MAX;
  int nxt = 32 + lane < nb ? bi[32 + lane] - bbase : INT_MAX;
  int nxt2 = 64 + lane < nb ? bi[64 + lane] - bbase : INT_MAX;
  int ahead = lane < na ? ai[lane] - abase : INT_MAX;
  for (int i0 = 0; i0 < na; i0 += 32) {
    const int i = i0 + lane;
    const int c = ahead;
    ahead = i + 32 < na ? ai[i + 32] - abase : INT_MAX;
    int lb = i < na ? -1 : 0;
    bool match = false;
    while (true) {
      int r = 0;  // elements of the window below c
#pragma unroll
      for (int step = 16; step >= 1; step >>= 1)
        if (__shfl_sync(FULL, win, r + step - 1) < c) r += step;
      const int at = __shfl_sync(FULL, win, r);
      if (lb < 0 && at >= c) {
        lb = b0 + r;
        match = at == c && lb < nb;
      }
      if (!__any_sync(FULL, lb < 0)) break;
      b0 += 32;  // ends at the latest with a window of INT_MAX
      win = nxt;
      nxt = nxt2;
      nxt2 = b0 + 64 + lane < nb ? bi[b0 + 64 + lane] - bbase : INT_MAX;
    }
    const unsigned m = __ballot_sync(FULL, match);
    f(i, c, lb, match, before + __popc(m & ((1u << lane) - 1)));
    before += __popc(m);
  }
}

// Number of elements of the ascending list bi[0, nb) below c, by a warp.
__device__ __forceinline__ int ew_warp_below(const int* bi, int bbase, int nb, int c) {
  const int lane = threadIdx.x & 31;
  int lo = 0, hi = nb;
  while (lo < hi) {
    const int step = (hi - lo + 31) / 32;
    const int q = lo + lane * step;
    const int n = __popc(__ballot_sync(0xffffffffu, q < hi && bi[q] - bbase < c));
    if (n == 0) {
      hi = lo;
    } else {
      const int next = lo + n * step;
      lo += (n - 1) * step + 1;
      if (next < hi) hi = next;
    }
  }
  return lo;
}

// One block: fibers [f0, f0 + R).  Their coordinates are staged in shared
// memory by coalesced loads when they fit; a pair of lists of at most EW_LONG
// coordinates is merged by its thread, a longer one by a warp, and one of more
// than EW_HUGE by the block, the first list cut into a slice per warp (a
// single warp walks 2,330 + 2,330 coordinates in about 50 us).
//   EW_COUNT    cnt[f] = coordinates of the result
//   EW_FILL     idx/val of the result: a staged tile's merge leaves, per
//               output, where its operands lie, and the block then reads the
//               values and writes C with consecutive threads on consecutive
//               outputs
//   EW_REDUCE   y[f] = sum of the products
//   EW_SCATTER  y[c] += product
// Bound: HBM and issue for short fibers, the warps' walk for long ones.
// GB300, whole calls, against one thread per fiber for everything (a thread
// that wrote its own fiber reached L2 with one partial sector per value, and
// a long pair was one thread's serial merge): A .+ B of 2M fibers of 8 + 8,
// F64, 632 -> 344 us (fill 520 -> 210); row sums of A .* B, 500,009 Zipf rows
// of 16 + 16, F32, 1258 -> 155; the same rows' A .+ B, F64, 2815 -> 565;
// uniform rows of 16 + 16 69 -> 66.  Not staging where only coordinates are
// read measured 83 there, 64 warps an SM against 48 66 against 75, and one
// warp for the longest pairs 322 in place of 155.
// One thread per fiber and no more stays up to 10 % faster on uniform rows of 2
// to 8 entries a pair where nothing is written but sums (21.8 us against 24.4
// at 5, F64): its warps never wait for a neighbour.  It is 5 to 8 times slower
// on Zipf rows of the same mean; without the block's barrier those took 84 us
// in place of 71, and a long pair's merge in a function of its own, out of the
// others' registers, gained nothing.
// STAGE: false for short fibers, see EW_STAGE_MEAN.
template <int MODE, bool STAGE, class T, class PA, class PB>
__global__ void __launch_bounds__(EW_THREADS, MODE == EW_FILL ? 10 : 16) ew_tile_k(int64_t nf, int R, Fiber<PA> a, const T* __restrict__ va,
                                                        Fiber<PB> b, const T* __restrict__ vb, int op,
                                                        int64_t* __restrict__ cnt, const int64_t* __restrict__ optr,
                                                        int32_t* __restrict__ oidx, T* __restrict__ out) {
  constexpr unsigned FULL = 0xffffffffu;
  __shared__ int s_idx[STAGE ? EW_CAP : 1];
  __shared__ unsigned s_src[MODE == EW_FILL && STAGE ? EW_CAP : 1];
  __shared__ int s_long[EW_THREADS];
  __shared__ int s_nlong;
  __shared__ int s_hits[EW_THREADS / 32];
  __shared__ T s_acc[EW_THREADS / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t f0 = (int64_t)blockIdx.x * R;
  const int rows = nf - f0 < R ? (int)(nf - f0) : R;
  const int64_t a0 = STAGE ? a.lo(f0) : 0, b0 = STAGE ? b.lo(f0) : 0;
  const int64_t na = STAGE ? a.lo(f0 + rows) - a0 : 0, nb = STAGE ? b.lo(f0 + rows) - b0 : 0;
  const bool staged = STAGE && na + nb <= EW_CAP;
  if (tid == 0) s_nlong = 0;
  int64_t pa = 0, pb = 0;  // the thread's fiber, from the tile's first entries
  int64_t la = 0, lb = 0;
  if (tid < rows) {
    pa = a.lo(f0 + tid) - a0;
    pb = b.lo(f0 + tid) - b0;
    la = a.hi(f0 + tid) - a0 - pa;
    lb = b.hi(f0 + tid) - b0 - pb;
  }
  if (staged) {
#pragma unroll 4
    for (int k = tid; k < (int)na; k += EW_THREADS) s_idx[k] = a.at(a0 + k);
#pragma unroll 4
    for (int k = tid; k < (int)nb; k += EW_THREADS) s_idx[(int)na + k] = b.at(b0 + k);
  }
  const int64_t o0 = MODE == EW_FILL ? optr[f0] : 0;
  const int total = MODE == EW_FILL && staged ? (int)min(optr[f0 + rows] - o0, (int64_t)EW_CAP) : 0;
  for (int k = tid; k < total; k += EW_THREADS) s_src[k] = EW_NONE | EW_NONE << 16;
  if (STAGE) __syncthreads();

  // Output n of fiber f0 + r (its o-th of `most`), from entries ka / kb of the tile (-1: none).
  auto emit = [&](int64_t at, int64_t most, int64_t o, int c, int64_t ka, int64_t kb) {
    if (o >= most) return;  // only where a list is not ascending
    if (staged) {
      if (at + o < EW_CAP) s_src[at + o] = (ka < 0 ? EW_NONE : (unsigned)ka) | (kb < 0 ? EW_NONE : (unsigned)kb) << 16;
      return;
    }
    oidx[o0 + at + o] = c;
    if (ka >= 0 && kb >= 0) out[o0 + at + o] = op == FGB_EW_MUL ? wmul(va[a0 + ka], vb[b0 + kb]) : wadd(va[a0 + ka], vb[b0 + kb]);
    else out[o0 + at + o] = ka >= 0 ? va[a0 + ka] : vb[b0 + kb];
  };

  // The thread's own fiber: two fingers over short lists.
  auto merge = [&](const int* ai, int abase, const int* bi, int bbase) {
    const int ea = (int)la, eb = (int)lb;
    int i = 0, j = 0, n = 0;
    T acc = T(0);
    int64_t at = 0, most = 0;
    if (MODE == EW_FILL) {
      at = optr[f0 + tid] - o0;
      most = optr[f0 + tid + 1] - o0 - at;
    }
    int ca = ea > 0 ? ai[0] - abase : INT_MAX, cb = eb > 0 ? bi[0] - bbase : INT_MAX;
    const bool all = MODE == EW_FILL && op == FGB_EW_ADD;
    while (all ? i < ea || j < eb : i < ea && j < eb) {
      const bool ma = ca <= cb, mb = cb <= ca;
      if (ma && mb) {
        if constexpr (MODE == EW_REDUCE) acc = fused(va[a0 + pa + i], vb[b0 + pb + j], acc);
        if constexpr (MODE == EW_SCATTER) atomicAdd(out + ca, wmul(va[a0 + pa + i], vb[b0 + pb + j]));
      }
      if (MODE == EW_FILL && (all || (ma && mb))) emit(at, most, n, min(ca, cb), ma ? pa + i : -1, mb ? pb + j : -1);
      n += all || (ma && mb);
      if (ma) ca = ++i < ea ? ai[i] - abase : INT_MAX;
      if (mb) cb = ++j < eb ? bi[j] - bbase : INT_MAX;
    }
    if (MODE == EW_COUNT) cnt[f0 + tid] = op == FGB_EW_ADD ? la + lb - n : n;
    if (MODE == EW_REDUCE) out[f0 + tid] = acc;
  };
  if (tid < rows) {
    if (la + lb > EW_LONG) {
      if (STAGE) s_long[atomicAdd(&s_nlong, 1)] = tid;
    } else if constexpr (!STAGE) {
      const int *ai = a.idx + pa, *bi = b.idx + pb;
      const int ea = (int)la, eb = (int)lb, shift = a.base - b.base;
      int i = 0, j = 0, n = 0;
      T acc = T(0);
      const int64_t at = MODE == EW_FILL ? optr[f0 + tid] : 0;
      while (i < ea && j < eb) {
        const int ca = __ldg(ai + i), cb = __ldg(bi + j) + shift;
        if (ca == cb) {
          if constexpr (MODE == EW_FILL) {
            oidx[at + n] = ca - a.base;
            out[at + n] = wmul(va[pa + i], vb[pb + j]);
          }
          if constexpr (MODE == EW_REDUCE) acc = fused(va[pa + i], vb[pb + j], acc);
          if constexpr (MODE == EW_SCATTER) atomicAdd(out + (ca - a.base), wmul(va[pa + i], vb[pb + j]));
          ++n;
        }
        i += ca <= cb;
        j += cb <= ca;
      }
      if (MODE == EW_COUNT) cnt[f0 + tid] = op == FGB_EW_ADD ? la + lb - n : n;
      if (MODE == EW_REDUCE) out[f0 + tid] = acc;
    } else if (staged) {
      merge(s_idx + pa, 0, s_idx + na + pb, 0);
    } else {
      merge(a.idx + a0 + pa, a.base, b.idx + b0 + pb, b.base);
    }
  }
  if (STAGE) {
    __syncthreads();
  } else {  // one barrier where no pair is long
    const bool is_long = tid < rows && la + lb > EW_LONG;
    if (!__syncthreads_or(is_long)) return;
    if (is_long) s_long[atomicAdd(&s_nlong, 1)] = tid;
    __syncthreads();
  }

  // Lists ai[0, ea) and bi[0, eb) -- entries qa.. and qb.. of the tile -- by a
  // warp, their outputs from `ofs` on: the lane's matches, and its sum.
  struct Part {
    int n;
    T acc;
  };
  auto merge_warp = [&](const int* ai, int abase, int ea, int64_t qa, const int* bi, int bbase, int eb, int64_t qb,
                        int64_t at, int64_t most, int64_t ofs, bool counting) -> Part {
    Part p{0, T(0)};
    ew_warp_ranks(ai, abase, ea, bi, bbase, eb, [&](int i, int c, int lbi, bool match, int before) {
      p.n += match;
      if constexpr (MODE == EW_REDUCE)
        if (match) p.acc = fused(va[a0 + qa + i], vb[b0 + qb + lbi], p.acc);
      if constexpr (MODE == EW_SCATTER)
        if (match) atomicAdd(out + c, wmul(va[a0 + qa + i], vb[b0 + qb + lbi]));
      if (MODE == EW_FILL && !counting && i < ea) {
        if (op == FGB_EW_ADD) emit(at, most, ofs + i + lbi - before, c, qa + i, match ? qb + lbi : -1);
        else if (match) emit(at, most, ofs + before, c, qa + i, qb + lbi);
      }
    });
    if (MODE == EW_FILL && op == FGB_EW_ADD && !counting)
      ew_warp_ranks(bi, bbase, eb, ai, abase, ea, [&](int j, int c, int lai, bool match, int before) {
        if (j < eb && !match) emit(at, most, ofs + j + lai - before, c, -1, qb + j);
      });
    return p;
  };
  const int nlong = s_nlong;
  auto pair = [&](int r, int64_t& qa, int64_t& qb, int& ea, int& eb, int64_t& at, int64_t& most) {
    qa = a.lo(f0 + r) - a0;
    qb = b.lo(f0 + r) - b0;
    ea = (int)(a.hi(f0 + r) - a0 - qa);
    eb = (int)(b.hi(f0 + r) - b0 - qb);
    at = most = 0;
    if (MODE == EW_FILL) {
      at = optr[f0 + r] - o0;
      most = optr[f0 + r + 1] - o0 - at;
    }
  };
  const int* const la_ = staged ? s_idx : a.idx + a0;
  const int* const lb_ = staged ? s_idx + na : b.idx + b0;
  const int abase = staged ? 0 : a.base, bbase = staged ? 0 : b.base;
  bool huge = false;
  for (int l = warp; l < nlong; l += EW_THREADS / 32) {
    const int r = s_long[l];
    int64_t qa, qb, at, most;
    int ea, eb;
    pair(r, qa, qb, ea, eb, at, most);
    if (ea + (int64_t)eb > EW_HUGE) {
      huge = true;
      continue;
    }
    Part p = merge_warp(la_ + qa, abase, ea, qa, lb_ + qb, bbase, eb, qb, at, most, 0, false);
    if (MODE == EW_COUNT) {
      const int n = __reduce_add_sync(FULL, p.n);
      if (lane == 0) cnt[f0 + r] = op == FGB_EW_ADD ? (int64_t)ea + eb - n : n;
    }
    if (MODE == EW_REDUCE) {
#pragma unroll
      for (int m = 16; m >= 1; m >>= 1) p.acc += shfl_xor(FULL, p.acc, m, 32);
      if (lane == 0) out[f0 + r] = p.acc;
    }
  }
  if (nlong > 0 && __syncthreads_or(huge)) {  // block-uniform
    constexpr int W = EW_THREADS / 32;
    for (int l = 0; l < nlong; ++l) {  // block-uniform
      const int r = s_long[l];
      int64_t qa, qb, at, most;
      int ea, eb;
      pair(r, qa, qb, ea, eb, at, most);
      if (ea + (int64_t)eb <= EW_HUGE) continue;
      // this warp's slice of the first list, and the second list's part beside it
      const int per = (ea + W - 1) / W;
      const int i0 = min(warp * per, ea), i1 = min(i0 + per, ea);
      const int* ai = la_ + qa;
      const int* bi = lb_ + qb;
      const int j0 = warp == 0 ? 0 : i0 < ea ? ew_warp_below(bi, bbase, eb, ai[i0] - abase) : eb;
      const int j1 = warp == W - 1 || i1 >= ea ? eb : ew_warp_below(bi, bbase, eb, ai[i1] - abase);
      const int je = max(j1, j0);  // lists that are not ascending
      Part p = merge_warp(ai + i0, abase, i1 - i0, qa + i0, bi + j0, bbase, je - j0, qb + j0, 0, 0, 0, true);
      p.n = __reduce_add_sync(FULL, p.n);
      if (MODE == EW_REDUCE) {
#pragma unroll
        for (int m = 16; m >= 1; m >>= 1) p.acc += shfl_xor(FULL, p.acc, m, 32);
      }
      if (lane == 0) {
        s_hits[warp] = p.n;
        s_acc[warp] = p.acc;
      }
      __syncthreads();
      if (MODE == EW_FILL) {
        int64_t ofs = op == FGB_EW_ADD ? (int64_t)i0 + j0 : 0;
        for (int w = 0; w < warp; ++w) ofs += op == FGB_EW_ADD ? -s_hits[w] : s_hits[w];
        merge_warp(ai + i0, abase, i1 - i0, qa + i0, bi + j0, bbase, je - j0, qb + j0, at, most, ofs, false);
      }
      if (tid == 0 && (MODE == EW_COUNT || MODE == EW_REDUCE)) {
        int64_t n = 0;
        T acc = s_acc[0];
        for (int w = 0; w < W; ++w) n += s_hits[w];
        for (int w = 1; w < W; ++w) acc += s_acc[w];
        if (MODE == EW_COUNT) cnt[f0 + r] = op == FGB_EW_ADD ? (int64_t)ea + eb - n : n;
        if (MODE == EW_REDUCE) out[f0 + r] = acc;
      }
      __syncthreads();
    }
  }
  if (MODE == EW_FILL && staged) {
    __syncthreads();
#pragma unroll 2
    for (int k = tid; k < total; k += EW_THREADS) {
      const unsigned src = s_src[k];
      const unsigned ka = src & 0xffff, kb = src >> 16;
      T v;
      if (src == (EW_NONE | EW_NONE << 16)) continue;  // only where a list is not ascending
      if (ka == EW_NONE) v = vb[b0 + kb];
      else if (kb == EW_NONE) v = va[a0 + ka];
      else v = op == FGB_EW_MUL ? wmul(va[a0 + ka], vb[b0 + kb]) : wadd(va[a0 + ka], vb[b0 + kb]);
      oidx[o0 + k] = ka == EW_NONE ? s_idx[na + kb] : s_idx[ka];
      out[o0 + k] = v;
    }
  }
}

// ---- fused elementwise multiply + reduce

// Per-fiber sums, dense B, G lanes per fiber.
template <int G, class T, class PA>
__global__ void reduce_fiber_dense(int64_t nf, Fiber<PA> a, const T* __restrict__ va,
                                   const T* __restrict__ D, int64_t ld, int csr, T* __restrict__ y) {
  const int lane = threadIdx.x & (G - 1);
  const int64_t group = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / G;
  const int64_t ngroups = ((int64_t)gridDim.x * blockDim.x) / G;
  for (int64_t f = group; f < nf; f += ngroups) {
    T acc = T(0);
    for (int64_t p = a.lo(f) + lane; p < a.hi(f); p += G) {
      const int64_t c = a.at(p);
      const T d = !D ? T(1) : csr ? __ldg(D + f * ld + c) : __ldg(D + c * ld + f);
      acc = fused(va[p], d, acc);
    }
#pragma unroll
    for (int m = G / 2; m >= 1; m >>= 1) acc += __shfl_xor_sync(group_mask<G>(), acc, m, G);
    if (lane == 0) y[f] = acc;
  }
}

// Scatter sums along the compressed coordinate: y[c] += A[f,c] * B[f,c].
template <class T, class PA>
__global__ void reduce_scatter_dense(int64_t nf, Fiber<PA> a, const T* __restrict__ va,
                                     const T* __restrict__ D, int64_t ld, int csr, T* __restrict__ y) {
  const int lane = threadIdx.x & 31;
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t f = w; f < nf; f += nw)
    for (int64_t p = a.lo(f) + lane; p < a.hi(f); p += 32) {
      const int64_t c = a.at(p);
      const T d = !D ? T(1) : csr ? __ldg(D + f * ld + c) : __ldg(D + c * ld + f);
      atomicAdd(y + c, wmul(va[p], d));
    }
}

// Deterministic fold of n partials: block b folds its consecutive share into
// out[b].
template <class T>
__global__ void fold_partials(const T* __restrict__ part, int64_t n, T* __restrict__ out) {
  __shared__ T sh[1024];
  const int64_t per = (n + gridDim.x - 1) / gridDim.x;
  const int64_t lo = blockIdx.x * per, hi = lo + per < n ? lo + per : n;
  T acc = T(0);
#pragma unroll 4
  for (int64_t i = lo + threadIdx.x; i < hi; i += blockDim.x) acc += part[i];
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int s = blockDim.x / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.x] = sh[0];
}

// part[0, n) (with room for EW_FOLD more behind) folded into out[0]: by one
// block up to 24 partials a thread (one SM reads about 100 GB/s: 2M partials
// took it 160 us; 20,000 6 us less than two launches), else in EW_FOLD
// consecutive shares first.
constexpr int EW_FOLD = 256;
template <class T>
static int fold_all(T* part, int64_t n, T* out, cudaStream_t s) {
  if (n > 24 * 1024) {
    fold_partials<T><<<EW_FOLD, 1024, 0, s>>>(part, n, part + n);
    part += n;
    n = EW_FOLD;
  }
  fold_partials<T><<<1, 1024, 0, s>>>(part, n, out);
  return check_launch("fold_partials");
}

template <class T>
__global__ void zero_vec(T* y, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
       i += (int64_t)gridDim.x * blockDim.x)
    y[i] = T(0);
}

// Counts for reduce(+, A; dims) of a Pattern (every stored entry is true)
// or Bool matrix: Julia sums Bools into Int64.  v NULL for a Pattern.
template <class P>
__global__ void count_fiber_k(int64_t nf, Fiber<P> a, const unsigned char* __restrict__ v,
                              long long* __restrict__ out) {
  for (int64_t f = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; f < nf;
       f += (int64_t)gridDim.x * blockDim.x) {
    const int64_t lo = a.lo(f), hi = a.hi(f);
    long long c = 0;
    if (!v) c = hi - lo;
    else
      for (int64_t p = lo; p < hi; ++p) c += v[p] ? 1 : 0;
    out[f] = c;
  }
}

template <class P>
__global__ void count_scatter_k(int64_t nnz, Fiber<P> a, const unsigned char* __restrict__ v,
                                unsigned long long* __restrict__ out) {
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < nnz;
       p += (int64_t)gridDim.x * blockDim.x)
    if (!v || v[p]) atomicAdd(out + a.at(p), 1ull);
}

template <class P>
static Fiber<P> fiber_of(const fgb_sparse* A) {
  return Fiber<P>{(const P*)A->ptr, (const int*)A->idx, A->index_base};
}

// Calls fn(Fiber<PA>, Fiber<PB>) with both ptr widths resolved.
template <class F>
static int with_fibers(const fgb_sparse* A, const fgb_sparse* B, F&& fn) {
  if (A->ptr_t == FGB_I32) {
    if (!B || B->ptr_t == FGB_I32) return fn(fiber_of<int32_t>(A), B ? fiber_of<int32_t>(B) : Fiber<int32_t>{});
    return fn(fiber_of<int32_t>(A), fiber_of<int64_t>(B));
  }
  if (!B || B->ptr_t == FGB_I32) return fn(fiber_of<int64_t>(A), B ? fiber_of<int32_t>(B) : Fiber<int32_t>{});
  return fn(fiber_of<int64_t>(A), fiber_of<int64_t>(B));
}

// Fibers per block of ew_tile_k: as many as its staging array is sized for
// on average, fewer where the blocks would not fill the device twice.
static int ew_rows(const fgb_ctx* ctx, const fgb_sparse* A, const fgb_sparse* B) {
  const int64_t nf = n_fibers(A);
  const double mean = (double)(A->nnz + B->nnz) / (double)nf;
  int64_t r = mean > 0 ? (int64_t)std::min(EW_MEAN / mean, (double)EW_THREADS) : EW_THREADS;
  r = std::min(r, (nf + 2 * ctx->num_sms - 1) / (2 * ctx->num_sms));
  return (int)std::max<int64_t>(r, 1);
}

// Below this many entries a pair of fibers on average, coordinates are read
// where they lie unless a sum's list is written: the copy into shared memory
// costs a chain of loads and a barrier, and short lists come out of L1.  Row
// sums of A .* B, F64, 873,496 uniform rows, staged against not: 5 a pair 31.2
// / 25.1 us, 8 37.0 / 35.2, 12 52.4 / 48.4, 16 63.9 / 65.2, 24 104 / 119; sums
// over rows 35.4 / 29.2, 41.6 / 39.5, 59.4 / 56.7, 72.2 / 76.5; Zipf rows
// 73.8 / 71.4 to 158 / 155 at 16; the list of A .* B 96 / 85 at 5, 109 / 99 at
// 8 (a thread writes the few places that two fibers share itself).
constexpr double EW_STAGE_MEAN = 14;
template <int MODE, class T>
static int ew_tile(fgb_ctx* ctx, const fgb_sparse* A, const fgb_sparse* B, int op, int64_t* cnt, const int64_t* optr,
                   int32_t* oidx, T* out, cudaStream_t s) {
  const int64_t nf = n_fibers(A);
  const int R = ew_rows(ctx, A, B);
  const unsigned blocks = (unsigned)((nf + R - 1) / R);
  return with_fibers(A, B, [&](auto fa, auto fb) {
    if ((MODE != EW_FILL || op == FGB_EW_MUL) && (double)A->nnz + (double)B->nnz < EW_STAGE_MEAN * (double)nf) {
      ew_tile_k<MODE, false><<<blocks, EW_THREADS, 0, s>>>(nf, R, fa, (const T*)A->val, fb, (const T*)B->val, op, cnt,
                                                           optr, oidx, out);
      return check_launch("ew_tile_k");
    }
    ew_tile_k<MODE, true><<<blocks, EW_THREADS, 0, s>>>(nf, R, fa, (const T*)A->val, fb, (const T*)B->val, op, cnt,
                                                        optr, oidx, out);
    return check_launch("ew_tile_k");
  });
}

static int check_pair(const fgb_sparse* A, const fgb_sparse* B, const char* who) {
  int rc = check_sparse(A, who, true);
  if (rc) return rc;
  rc = check_sparse(B, who, true);
  if (rc) return rc;
  if (A->nrows != B->nrows || A->ncols != B->ncols)
    return set_error(FGB_EINVAL, "%s: shape mismatch (%lld x %lld vs %lld x %lld)", who,
                     (long long)A->nrows, (long long)A->ncols, (long long)B->nrows,
                     (long long)B->ncols);
  if (A->orient != B->orient) return set_error(FGB_EINVAL, "%s: operands differ in orientation", who);
  if (A->val_t != B->val_t) return set_error(FGB_EUNSUPPORTED, "%s: operands differ in dtype", who);
  return FGB_OK;
}

}  // namespace fgb

using namespace fgb;

extern "C" {

int fgb_ewise_count(fgb_ctx* ctx, int op, const fgb_sparse* A, const fgb_sparse* B,
                    int64_t* out_ptr, int64_t* out_nnz, void* stream) {
  if (!ctx) return set_error(FGB_EINVAL, "fgb_ewise_count: null ctx");
  if (op != FGB_EW_MUL && op != FGB_EW_ADD) return set_error(FGB_EINVAL, "fgb_ewise_count: bad op");
  int rc = check_pair(A, B, "fgb_ewise_count");
  if (rc) return rc;
  if (!out_ptr || !out_nnz) return set_error(FGB_EINVAL, "fgb_ewise_count: null output");
  cudaStream_t s = pick_stream(ctx, stream);
  const int64_t nf = n_fibers(A);
  FGB_CUDA_TRY(cudaMemsetAsync(out_ptr, 0, sizeof(int64_t), s));
  if (nf > 0) {
    size_t tmp_bytes = 0;
    int64_t* counts = nullptr;
    cub::DeviceScan::InclusiveSum(nullptr, tmp_bytes, counts, out_ptr + 1, nf, s);
    void* tmp = nullptr;
    FGB_CUDA_TRY(cudaMallocAsync((void**)&counts, sizeof(int64_t) * nf + tmp_bytes, s));
    tmp = counts + nf;
    rc = ew_tile<EW_COUNT, float>(ctx, A, B, op, counts, nullptr, nullptr, nullptr, s);
    if (rc == FGB_OK) {
      cub::DeviceScan::InclusiveSum(tmp, tmp_bytes, counts, out_ptr + 1, nf, s);
      rc = check_launch("DeviceScan");
    }
    cudaFreeAsync(counts, s);
    if (rc) return rc;
  }
  FGB_CUDA_TRY(cudaMemcpyAsync(out_nnz, out_ptr + nf, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  FGB_CUDA_TRY(cudaStreamSynchronize(s));
  return FGB_OK;
}

int fgb_ewise_fill(fgb_ctx* ctx, int op, const fgb_sparse* A, const fgb_sparse* B,
                   const int64_t* out_ptr, int32_t* out_idx, void* out_val, void* stream) {
  if (!ctx) return set_error(FGB_EINVAL, "fgb_ewise_fill: null ctx");
  if (op != FGB_EW_MUL && op != FGB_EW_ADD) return set_error(FGB_EINVAL, "fgb_ewise_fill: bad op");
  int rc = check_pair(A, B, "fgb_ewise_fill");
  if (rc) return rc;
  const int64_t nf = n_fibers(A);
  if (nf == 0) return FGB_OK;
  if (!out_ptr) return set_error(FGB_EINVAL, "fgb_ewise_fill: null out_ptr");
  cudaStream_t s = pick_stream(ctx, stream);
  switch (A->val_t) {
    case FGB_F64: return ew_tile<EW_FILL>(ctx, A, B, op, nullptr, out_ptr, out_idx, (double*)out_val, s);
    case FGB_F32: return ew_tile<EW_FILL>(ctx, A, B, op, nullptr, out_ptr, out_idx, (float*)out_val, s);
    case FGB_I32: return ew_tile<EW_FILL>(ctx, A, B, op, nullptr, out_ptr, out_idx, (int32_t*)out_val, s);
    case FGB_I64: return ew_tile<EW_FILL>(ctx, A, B, op, nullptr, out_ptr, out_idx, (int64_t*)out_val, s);
    default: return set_error(FGB_EUNSUPPORTED, "fgb_ewise_fill: dtype %d", A->val_t);
  }
}

int fgb_ewise_reduce(fgb_ctx* ctx, int dims, const fgb_sparse* A, const fgb_sparse* B,
                     const void* B_dense, int64_t ldb, void* y, int dtype, unsigned flags,
                     void* stream) {
  if (!ctx) return set_error(FGB_EINVAL, "fgb_ewise_reduce: null ctx");
  if (dims < 0 || dims > 2) return set_error(FGB_EINVAL, "fgb_ewise_reduce: dims must be 0, 1 or 2");
  int rc = B ? check_pair(A, B, "fgb_ewise_reduce") : check_sparse(A, "fgb_ewise_reduce: A", true);
  if (rc) return rc;
  if (!B && B_dense && ldb < A->ncols) return set_error(FGB_EINVAL, "fgb_ewise_reduce: ldb < ncols");
  if (!B && !B_dense && (A->val_t == FGB_NONE || A->val_t == FGB_BOOL) && dtype == FGB_I64) {
    // reduce(+, A; dims) of a Pattern or Bool matrix: Int64 counts
    if (!y) return set_error(FGB_EINVAL, "fgb_ewise_reduce: null y");
    cudaStream_t s = pick_stream(ctx, stream);
    const int64_t nf = n_fibers(A);
    const bool per_fiber = dims == 0 || (A->orient == FGB_CSR ? dims == 2 : dims == 1);
    const int64_t out_len = dims == 0 ? 1 : (dims == 2 ? A->nrows : A->ncols);
    const unsigned char* v = A->val_t == FGB_BOOL ? (const unsigned char*)A->val : nullptr;
    if (!per_fiber || nf == 0)
      FGB_CUDA_TRY(cudaMemsetAsync(y, 0, sizeof(long long) * out_len, s));
    if (!per_fiber)
      return with_fibers(A, nullptr, [&](auto fa, auto) {
        count_scatter_k<<<grid_for(A->nnz, 256, ctx->num_sms, 8), 256, 0, s>>>(A->nnz, fa, v,
                                                                                 (unsigned long long*)y);
        return check_launch("count_scatter");
      });
    if (nf == 0) return FGB_OK;
    long long* target = (long long*)y;
    if (dims == 0) FGB_CUDA_TRY(cudaMallocAsync((void**)&target, sizeof(long long) * (nf + EW_FOLD), s));
    rc = with_fibers(A, nullptr, [&](auto fa, auto) {
      count_fiber_k<<<grid_for(nf, 256, ctx->num_sms, 8), 256, 0, s>>>(nf, fa, v, target);
      return check_launch("count_fiber");
    });
    if (rc == FGB_OK && dims == 0) rc = fold_all<long long>(target, nf, (long long*)y, s);
    if (target != (long long*)y) cudaFreeAsync(target, s);
    return rc;
  }
  if (A->val_t != dtype) return set_error(FGB_EUNSUPPORTED, "fgb_ewise_reduce: A dtype != dtype");
  if (dtype != FGB_F32 && dtype != FGB_F64)
    return set_error(FGB_EUNSUPPORTED, "fgb_ewise_reduce: dtype %d", dtype);
  if (!y) return set_error(FGB_EINVAL, "fgb_ewise_reduce: null y");
  cudaStream_t s = pick_stream(ctx, stream);
  const int64_t nf = n_fibers(A);
  const bool csr = A->orient == FGB_CSR;
  // per-fiber reduction when the reduced dimension is the uncompressed one
  const bool per_fiber = dims == 0 || (csr ? dims == 2 : dims == 1);
  const int64_t out_len = dims == 0 ? 1 : (dims == 2 ? A->nrows : A->ncols);
  const size_t esz = dtype == FGB_F64 ? 8 : 4;
  void* target = y;
  if (dims == 0 && nf > 0) FGB_CUDA_TRY(cudaMallocAsync(&target, (nf + EW_FOLD) * esz, s));
  const int grid = grid_for(nf * 8, 256, ctx->num_sms, 8);
  auto body = [&](auto tag) -> int {
    using T = decltype(tag);
    const T* va = (const T*)A->val;
    if (!per_fiber) {
      zero_vec<T><<<grid_for(out_len, 256, ctx->num_sms, 4), 256, 0, s>>>((T*)y, out_len);
      if (B) return nf ? ew_tile<EW_SCATTER, T>(ctx, A, B, FGB_EW_MUL, nullptr, nullptr, nullptr, (T*)y, s) : FGB_OK;
      return with_fibers(A, nullptr, [&](auto fa, auto) {
        reduce_scatter_dense<<<grid_for(nf * 32, 256, ctx->num_sms, 8), 256, 0, s>>>(
            nf, fa, va, (const T*)B_dense, ldb, csr ? 1 : 0, (T*)y);
        return check_launch("reduce_scatter");
      });
    }
    if (nf == 0) {
      zero_vec<T><<<1, 32, 0, s>>>((T*)y, out_len);
      return check_launch("zero_vec");
    }
    int r = B ? ew_tile<EW_REDUCE, T>(ctx, A, B, FGB_EW_MUL, nullptr, nullptr, nullptr, (T*)target, s)
              : with_fibers(A, nullptr, [&](auto fa, auto) {
                  reduce_fiber_dense<8><<<grid, 256, 0, s>>>(nf, fa, va, (const T*)B_dense, ldb, csr ? 1 : 0,
                                                             (T*)target);
                  return check_launch("reduce_fiber");
                });
    if (r) return r;
    return dims == 0 ? fold_all<T>((T*)target, nf, (T*)y, s) : FGB_OK;
  };
  rc = dtype == FGB_F64 ? body(double(0)) : body(float(0));
  if (target != y) cudaFreeAsync(target, s);
  (void)flags;
  return rc;
}

}  // extern "C"
