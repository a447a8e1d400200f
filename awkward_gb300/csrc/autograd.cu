// autograd.cu -- backward kernels for differentiable jagged operations.
//
// awkward has no CUDA backward kernels (its differentiation goes through JAX,
// src/awkward/_connect/jax/reducers.py:51-200); these entry points back the
// torch.autograd.Function classes of awkward_gb300/autograd.py:
//   segmented sum      d x_j = g_{list(j)}                      (broadcast by offsets)
//   segmented max      d x_{argmax(l)} = g_l, 0 elsewhere        (argmax-routed scatter)
//   jagged softmax     y_j = exp(x_j - m_l) / sum_k exp(x_k - m_l)
//                      d x_j = y_j (g_j - sum_k g_k y_k)         (fused Jacobian product)
// The forward sum and max use the segmented reducers of this library.
//
// The sum's and float softmax kernels work in rounds of 32 lists per warp, without
// block barriers.
#include <math.h>

#include "list_tile.cuh"

using namespace gb;

namespace {

template <class T>
__device__ __forceinline__ T exp_t(T v);
template <>
__device__ __forceinline__ float exp_t<float>(float v) { return __expf(v); }
template <>
__device__ __forceinline__ double exp_t<double>(double v) { return exp(v); }

template <class T>
__device__ __forceinline__ T max_t(T a, T b) { return a > b ? a : b; }

// Zero a[j] for j outside [offsets[0], offsets[nlists]) within [0, nvalues): the
// elements no list covers, by threads t of `stride`.  Only those elements are
// touched (none when the offsets span the whole array).
template <class T>
__device__ __forceinline__ void zero_outside(T* __restrict__ a, const int64_t* __restrict__ offsets,
                                             long long nlists, long long nvalues, long long t,
                                             long long stride) {
  long long lo = __ldg(offsets), hi = __ldg(offsets + nlists);
  lo = lo < 0 ? 0 : (lo > nvalues ? nvalues : lo);
  hi = hi < lo ? lo : (hi > nvalues ? nvalues : hi);
  for (long long j = t; j < lo; j += stride) a[j] = T(0);
  for (long long j = hi + t; j < nvalues; j += stride) a[j] = T(0);
}

// ---------------------------------------------------------------- sum backward
// Warp rounds of 32 lists (one lane per list, list ends loaded coalesced,
// starts from the lane below): each lane writes its list's gradient value
// over its elements in a per-warp stage in shared memory, then the warp copies
// the round's span out with consecutive lanes on consecutive elements
// (coalesced stores).  A round whose span exceeds the stage (long lists)
// writes straight from its lanes.  No block barriers: warps run independently.
constexpr int kBcastStage = 1024;  // elements staged per warp and round

template <class T>
__global__ void __launch_bounds__(256)
    sum_backward_rounds_kernel(T* __restrict__ gx, const T* __restrict__ gout,
                               const int64_t* __restrict__ offsets, long long nlists,
                               long long nvalues) {
  zero_outside(gx, offsets, nlists, nvalues, blockIdx.x * (long long)blockDim.x + threadIdx.x,
               (long long)gridDim.x * blockDim.x);
  __shared__ T stage[256 / 32][kBcastStage];
  T* sw = stage[threadIdx.x >> 5];
  const int lane = threadIdx.x & 31;
  const long long nrounds = (nlists + 31) / 32;
  const long long stride = (long long)gridDim.x * (blockDim.x >> 5);
  for (long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5; r < nrounds;
       r += stride) {
    const long long base = r * 32, li = base + lane;
    const bool act = li < nlists;
    const long long en = __ldg(offsets + (act ? li : nlists - 1) + 1);
    long long st = __shfl_up_sync(0xffffffffu, en, 1);
    if (lane == 0) st = __ldg(offsets + base);
    const unsigned acts = __ballot_sync(0xffffffffu, act);
    const long long lo = __shfl_sync(0xffffffffu, st, 0);
    const long long hi = __shfl_sync(0xffffffffu, en, 31 - __clz(acts));
    const T g = act ? __ldg(gout + li) : T(0);
    const bool sorted = __all_sync(0xffffffffu, !act || st <= en);
    if (sorted && hi - lo <= kBcastStage) {
      if (act)
        for (long long j = st; j < en; j++) sw[j - lo] = g;
      __syncwarp();
      const int span = (int)(hi - lo);
      for (int j = lane; j < span; j += 32) gx[lo + j] = sw[j];
      __syncwarp();
    } else if (act) {
      for (long long j = st; j < en; j++) gx[j] = g;
    }
  }
}

// ---------------------------------------------------------------- max backward
// argmax holds global element indices (-1 for an empty list); indices outside
// [0, nelements) are ignored.
template <class T>
__global__ void max_backward_kernel(T* __restrict__ gx, const T* __restrict__ gout,
                                    const int64_t* __restrict__ argmax, long long nelements,
                                    long long nlists) {
  for (long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x; l < nlists;
       l += (long long)gridDim.x * blockDim.x) {
    const long long j = argmax[l];
    if (j >= 0 && j < nelements) gx[j] = gout[l];
  }
}

// ---------------------------------------------------------------- softmax
// Floats go by rounds of 32 lists, one per warp, a list's bounds on each lane.  The round's
// longest list chooses how many lanes share a list, 4 to 32, and how many elements
// a lane has, 6 at most; these are loaded once, kept in registers, reduced with
// shuffles among the list's lanes and stored, the loads of several steps in flight.
// Lists of more than kSoftLongest elements go one by one, a warp on each, in three
// passes.  Where the mean is above that, or few lists leave most of the chip idle, a
// warp has fewer lists, and those of more than kSoftWarp elements are taken by the
// whole CTA.  (Only there: the barrier that the CTA's lists need cost rounds of short
// lists 10 to 15 %.)  Bound by the instructions of places past the lists' ends at
// first, by HBM from mean 16 on: 1M lists, us (forward, backward with y kept): mean 4
// 44, 43 -> 21, 22; mean 16 61, 68 -> 36, 47 (128 and 192 MB, 19 and 28 us); 20000
// lists of mean 500 188, 425 -> 42, 68; 32 lists of 100000 20000, 19100 -> 392, 347.
// Before, tiles of 64 lists were staged in shared memory, one thread reducing each
// list; 32 lists to every warp, a long one making all 32 go one by one, had taken
// 45700 and 39200 us for the last.
constexpr int kSoftThreads = 128;
constexpr int kSoftLongest = 32 * 6;
constexpr int kSoftWarp = 1024;  // longest list of a CTA of few lists taken by one warp
constexpr int kSoftFlight = 24;  // 4-byte words a lane has in flight

template <class T, class F>
__device__ __forceinline__ T lanes_reduce(T v, int lanes, F f) {
  for (int d = 1; d < lanes; d <<= 1) v = f(v, __shfl_xor_sync(0xffffffffu, v, d));
  return v;
}
template <class T>
__device__ __forceinline__ T lanes_max(T v, int lanes) {
  return lanes_reduce(v, lanes, [](T a, T b) { return max_t(a, b); });
}
template <class T>
__device__ __forceinline__ T lanes_sum(T v, int lanes) {
  return lanes_reduce(v, lanes, [](T a, T b) { return a + b; });
}

// The threads that take one long list between them: a warp, or the CTA.
struct TeamWarp {
  static constexpr int kLanes = 32;
  int lane;
  template <class T>
  __device__ __forceinline__ T max(T v) const { return lanes_max(v, 32); }
  template <class T>
  __device__ __forceinline__ T sum(T v) const { return lanes_sum(v, 32); }
};
struct TeamBlock {
  static constexpr int kLanes = kSoftThreads;
  int lane;
  float* part;  // a place for each warp
  template <class F>
  __device__ __forceinline__ float join(float v, F f) const {
    __syncthreads();  // (the places may still be read)
    if ((lane & 31) == 0) part[lane >> 5] = v;
    __syncthreads();
    v = part[0];
#pragma unroll
    for (int w = 1; w < kLanes / 32; w++) v = f(v, part[w]);
    return v;
  }
  __device__ __forceinline__ float max(float v) const {
    return join(lanes_max(v, 32), [](float a, float b) { return max_t(a, b); });
  }
  __device__ __forceinline__ float sum(float v) const {
    return join(lanes_sum(v, 32), [](float a, float b) { return a + b; });
  }
};

// What becomes of a list whose elements a lane group holds: in[0] = x (forward), or
// in[0] = gy and in[1] = the saved y or x (backward).
struct SoftForward {
  static constexpr int kArrays = 1;
  static constexpr bool kZeroPad = false;
  template <class T, int N>
  __device__ __forceinline__ static void apply(const T (&in)[1][N], T (&out)[N], int lanes) {
    T m = -INFINITY;
#pragma unroll
    for (int k = 0; k < N; k++) m = max_t(m, in[0][k]);
    m = lanes_max(m, lanes);
    T sum = 0;
#pragma unroll
    for (int k = 0; k < N; k++) {
      out[k] = exp_t(in[0][k] - m);
      sum += out[k];
    }
    const T inv = T(1) / lanes_sum(sum, lanes);  // one division per list; elements multiply by it
#pragma unroll
    for (int k = 0; k < N; k++) out[k] *= inv;
  }
  // one list, x[0 .. n), by a team (TeamWarp or TeamBlock)
  template <class T, class Team>
  __device__ __forceinline__ static void list(T* out, const T* const (&in)[1], long long n, Team team) {
    T m = -INFINITY, sum = 0;
    for (long long q = team.lane; q < n; q += Team::kLanes) m = max_t(m, in[0][q]);
    m = team.max(m);
    for (long long q = team.lane; q < n; q += Team::kLanes) sum += out[q] = exp_t(in[0][q] - m);
    const T inv = T(1) / team.sum(sum);
    for (long long q = team.lane; q < n; q += Team::kLanes) out[q] *= inv;
  }
};
// d x_j = y_j (g_j - sum_k g_k y_k)
struct SoftBackwardSaved {
  static constexpr int kArrays = 2;
  static constexpr bool kZeroPad = true;
  template <class T, int N>
  __device__ __forceinline__ static void apply(const T (&in)[2][N], T (&out)[N], int lanes) {
    T dot = 0;
#pragma unroll
    for (int k = 0; k < N; k++) dot += in[0][k] * in[1][k];
    dot = lanes_sum(dot, lanes);
#pragma unroll
    for (int k = 0; k < N; k++) out[k] = in[1][k] * (in[0][k] - dot);
  }
  template <class T, class Team>
  __device__ __forceinline__ static void list(T* out, const T* const (&in)[2], long long n, Team team) {
    T dot = 0;
    for (long long q = team.lane; q < n; q += Team::kLanes) dot += in[0][q] * in[1][q];
    dot = team.sum(dot);
    for (long long q = team.lane; q < n; q += Team::kLanes) out[q] = in[1][q] * (in[0][q] - dot);
  }
};
// The same with y computed again from x.
struct SoftBackward {
  static constexpr int kArrays = 2;
  static constexpr bool kZeroPad = false;
  template <class T, int N>
  __device__ __forceinline__ static void apply(const T (&in)[2][N], T (&out)[N], int lanes) {
    T m = -INFINITY;
#pragma unroll
    for (int k = 0; k < N; k++) m = max_t(m, in[1][k]);
    m = lanes_max(m, lanes);
    T sum = 0, gsum = 0;
#pragma unroll
    for (int k = 0; k < N; k++) {
      out[k] = exp_t(in[1][k] - m);
      sum += out[k];
      gsum += in[0][k] * out[k];
    }
    const T inv = T(1) / lanes_sum(sum, lanes);
    const T dot = lanes_sum(gsum, lanes) * inv;
#pragma unroll
    for (int k = 0; k < N; k++) out[k] = out[k] * inv * (in[0][k] - dot);
  }
  template <class T, class Team>
  __device__ __forceinline__ static void list(T* out, const T* const (&in)[2], long long n, Team team) {
    T m = -INFINITY, sum = 0, gsum = 0;
    for (long long q = team.lane; q < n; q += Team::kLanes) m = max_t(m, in[1][q]);
    m = team.max(m);
    for (long long q = team.lane; q < n; q += Team::kLanes) {
      const T e = out[q] = exp_t(in[1][q] - m);
      sum += e;
      gsum += in[0][q] * e;
    }
    const T inv = T(1) / team.sum(sum);
    const T dot = team.sum(gsum) * inv;
    for (long long q = team.lane; q < n; q += Team::kLanes)
      out[q] = out[q] * inv * (in[0][q] - dot);
  }
};

// One round of `lists` lists (32 when SHARE is) with at most LANES * ITEMS elements:
// lane l holds list l's first element (relative to the pointers) and length.
template <int LANES, int ITEMS, int SHARE, class Op, class T>
__device__ __forceinline__ void soft_round(Op, T* __restrict__ out, const T* const (&in)[Op::kArrays],
                                           int first, int len, int lists, int lane) {
  constexpr int kMost = kSoftFlight / ((int)sizeof(T) / 4 * ITEMS * Op::kArrays);
  constexpr int kSteps = kMost >= 4 ? 4 : kMost >= 2 ? 2 : 1;  // steps in flight
  const int i0 = lane % LANES;
#pragma unroll 1
  for (int s0 = 0; SHARE == 32 ? s0 < LANES : s0 * (32 / LANES) < lists; s0 += kSteps) {
    T v[kSteps][Op::kArrays][ITEMS];
    int at[kSteps], left[kSteps];  // the lane's first element, the elements from there on
#pragma unroll
    for (int s = 0; s < kSteps; s++) {
      const int from = (s0 + s) * (32 / LANES) + lane / LANES;
      at[s] = __shfl_sync(0xffffffffu, first, from) + i0;
      left[s] = __shfl_sync(0xffffffffu, len, from) - i0;
#pragma unroll
      for (int k = 0; k < ITEMS; k++)
#pragma unroll
        for (int a = 0; a < Op::kArrays; a++)
          v[s][a][k] = k * LANES < left[s] ? __ldg(in[a] + at[s] + k * LANES)
                       : a == Op::kArrays - 1 && !Op::kZeroPad ? T(-INFINITY) : T(0);
    }
#pragma unroll
    for (int s = 0; s < kSteps; s++) {
      T r[ITEMS];
      Op::apply(v[s], r, LANES);
#pragma unroll
      for (int k = 0; k < ITEMS; k++)
        if (k * LANES < left[s]) out[at[s] + k * LANES] = r[k];
    }
  }
}

// A warp takes SHARE lists, or (0) a quarter of the CTA's `lists`.
template <class Op, int SHARE>
__global__ void __launch_bounds__(kSoftThreads)
    softmax_kernel(float* __restrict__ out, const float* __restrict__ in0, const float* __restrict__ in1,
                   const int64_t* __restrict__ offsets, long long nlists, long long nvalues,
                   int lists, unsigned rounds_blocks) {
  if (blockIdx.x >= rounds_blocks) {  // the elements no list covers
    zero_outside(out, offsets, nlists, nvalues,
                 (blockIdx.x - rounds_blocks) * (long long)kSoftThreads + threadIdx.x,
                 (long long)(gridDim.x - rounds_blocks) * kSoftThreads);
    return;
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int share = SHARE ? SHARE : (lists + 3) / 4;
  const long long l0 = blockIdx.x * (long long)lists;
  const long long l = l0 + warp * share + lane;
  const long long stop = l0 + lists < nlists ? l0 + lists : nlists;
  const bool act = lane < share && l < stop;
  const long long begin = __ldg(offsets + (act ? l : stop));
  const long long end = __ldg(offsets + (act ? l + 1 : stop));
  const long long base = __shfl_sync(0xffffffffu, begin, 0);
  const long long n = end - begin;
  const float* const in[2] = {in0, in1};
  int len = (int)n;
  if (__any_sync(0xffffffffu, n < 0 || n > kSoftLongest)) {
    // the long ones by the warp (with SHARE 0 up to kSoftWarp elements); all of them
    // where the round cannot reach its lists by 32-bit places from its first
    const int most = __shfl_sync(0xffffffffu, end, 31) - base < 1ll << 30 ? kSoftLongest : 0;
    for (unsigned m = __ballot_sync(0xffffffffu, n > most && (SHARE || n <= kSoftWarp)); m; m &= m - 1) {
      const int j = __ffs(m) - 1;
      const long long b = __shfl_sync(0xffffffffu, begin, j);
      const float* p[Op::kArrays];
#pragma unroll
      for (int a = 0; a < Op::kArrays; a++) p[a] = in[a] + b;
      Op::list(out + b, p, __shfl_sync(0xffffffffu, n, j), TeamWarp{lane});
    }
    if (n < 0 || n > most) len = 0;
  }
  const int longest = __reduce_max_sync(0xffffffffu, len);
  if (longest > 0) {
    const float* p[Op::kArrays];
#pragma unroll
    for (int a = 0; a < Op::kArrays; a++) p[a] = in[a] + base;
    const int first = (int)(begin - base);
    float* o = out + base;
    if (longest <= 8) soft_round<4, 2, SHARE>(Op(), o, p, first, len, share, lane);
    else if (longest <= 16) soft_round<4, 4, SHARE>(Op(), o, p, first, len, share, lane);
    else if (longest <= 24) soft_round<4, 6, SHARE>(Op(), o, p, first, len, share, lane);
    else if (longest <= 32) soft_round<8, 4, SHARE>(Op(), o, p, first, len, share, lane);
    else if (longest <= 48) soft_round<8, 6, SHARE>(Op(), o, p, first, len, share, lane);
    else if (longest <= 96) soft_round<16, 6, SHARE>(Op(), o, p, first, len, share, lane);
    else soft_round<32, 6, SHARE>(Op(), o, p, first, len, share, lane);
  }
  if constexpr (SHARE == 0) {  // the CTA's lists of more than kSoftWarp elements
    __shared__ long long s_long[kSoftThreads];
    __shared__ int s_longs;
    __shared__ float s_part[kSoftThreads / 32];
    if (!__syncthreads_or(n > kSoftWarp)) return;
    if (threadIdx.x == 0) s_longs = 0;
    __syncthreads();
    if (n > kSoftWarp) s_long[atomicAdd(&s_longs, 1)] = l;
    __syncthreads();
    const int longs = s_longs;
    for (int j = 0; j < longs; j++) {
      const long long b = __ldg(offsets + s_long[j]);
      const float* p[Op::kArrays];
#pragma unroll
      for (int a = 0; a < Op::kArrays; a++) p[a] = in[a] + b;
      Op::list(out + b, p, __ldg(offsets + s_long[j] + 1) - b, TeamBlock{(int)threadIdx.x, s_part});
    }
  }
}

// Doubles, whose exponentials and sums fill the narrow 64-bit unit, go by tiles of
// kTileSoft lists per CTA instead, where no lane works for a place past a list's
// end: the tile's elements are staged in shared memory with a map from elements to
// lists, the list's threads reduce it, and all threads take the elements, one
// exponential each.  A tile of more elements goes list by list.
// 1M lists, us (forward, backward with y kept, with y computed again): mean 4
// 502, 64, 498 -> 220, 54, 265; mean 16 1390, 149, 1475 -> 689, 146, 826; mean 24,
// whose tiles of 64 lists did not fit, 1987, 234, 2103 -> 969, 193, 1152 (the kernel
// for floats: 590, 93, 674; 1275, 203, 1459; 1975, 306, 2265).
constexpr int kTileSoft = 64;
constexpr int kTileElems = 1024;

struct SoftTile {
  long long loc[kTileSoft + 1];  // offsets of the tile's lists, relative to its first element
  unsigned char owner[kTileElems];  // list of each element
  long long base;                 // first element of the tile
  int count;                      // lists in this tile
  int mapped;                     // the elements fit
};

// One element global -> shared memory without a register round trip
// (cp.async, completed by cp_async_wait_all).
template <class T>
__device__ __forceinline__ void cp_async_elem(T* dst, const T* src) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(src), "n"(sizeof(T))
               : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Stage a tile of `lists` lists: offsets[l0 .. l0+count] and, if it has at most
// kTileElems elements, its elements of src0 (and src1 when given) into dst0 (dst1) and
// the element -> list map (all threads; ends with __syncthreads).  The
// element copies are issued first, from the tile's two end offsets alone, so
// they are in flight together with the offsets loads.
template <class T>
__device__ __forceinline__ void stage_soft_tile(SoftTile& t, const int64_t* __restrict__ offsets,
                                                long long l0, long long nlists, int lists, T* dst0, const T* __restrict__ src0, T* dst1,
                                                const T* __restrict__ src1) {
  const long long rem = nlists - l0;
  const int count = (int)(rem < lists ? rem : lists);
  const long long base = __ldg(offsets + l0);
  const long long total = __ldg(offsets + l0 + count) - base;
  const bool mapped = total <= kTileElems;
  if (mapped) {
    for (long long q = threadIdx.x; q < total; q += blockDim.x) {
      cp_async_elem(dst0 + q, src0 + base + q);
      if (src1) cp_async_elem(dst1 + q, src1 + base + q);
    }
  }
  for (int i = threadIdx.x; i <= kTileSoft; i += blockDim.x) {
    const int k = i < count ? i : count;
    t.loc[i] = __ldg(offsets + l0 + k) - base;
  }
  if (threadIdx.x == 0) {
    t.base = base;
    t.count = count;
    t.mapped = mapped ? 1 : 0;
  }
  __syncthreads();
  if (mapped && (int)threadIdx.x < count) {
    const int a = (int)t.loc[threadIdx.x], b = (int)t.loc[threadIdx.x + 1];
    for (int q = a; q < b; q++) t.owner[q] = (unsigned char)threadIdx.x;
  }
  cp_async_wait_all();
  __syncthreads();
}

// A thread's share of its list: kSoftThreads / lists threads, of one warp, for each.
struct SoftShare {
  int list, begin, end, step;
};
__device__ __forceinline__ SoftShare soft_share(const SoftTile& t, int lists) {
  const int step = kSoftThreads / lists, r = threadIdx.x / step;
  if (r >= t.count) return {r, 0, 0, step};
  return {r, (int)t.loc[r] + (int)threadIdx.x % step, (int)t.loc[r + 1], step};
}

// s_list[] and s_dot[] have a place for each list of the tile, also past its last.
__device__ __forceinline__ void soft_tile(SoftForward, const SoftTile& t, int lists, double* s0,
                                          const double*, double* s_list, double*,
                                          double* __restrict__ out) {
  const SoftShare h = soft_share(t, lists);
  const int total = (int)t.loc[t.count];
  double m = -INFINITY;
  for (int q = h.begin; q < h.end; q += h.step) m = max_t(m, s0[q]);
  s_list[h.list] = lanes_max(m, h.step);
  __syncthreads();
  for (int q = threadIdx.x; q < total; q += kSoftThreads) s0[q] = exp_t(s0[q] - s_list[t.owner[q]]);
  __syncthreads();
  double sum = 0;
  for (int q = h.begin; q < h.end; q += h.step) sum += s0[q];
  s_list[h.list] = 1.0 / lanes_sum(sum, h.step);
  __syncthreads();
  for (int q = threadIdx.x; q < total; q += kSoftThreads) out[q] = s0[q] * s_list[t.owner[q]];
}
__device__ __forceinline__ void soft_tile(SoftBackwardSaved, const SoftTile& t, int lists, double* sg,
                                          const double* sy, double* s_list, double*,
                                          double* __restrict__ out) {
  const SoftShare h = soft_share(t, lists);
  const int total = (int)t.loc[t.count];
  double d = 0;
  for (int q = h.begin; q < h.end; q += h.step) d += sg[q] * sy[q];
  s_list[h.list] = lanes_sum(d, h.step);
  __syncthreads();
  for (int q = threadIdx.x; q < total; q += kSoftThreads)
    out[q] = sy[q] * (sg[q] - s_list[t.owner[q]]);
}
__device__ __forceinline__ void soft_tile(SoftBackward, const SoftTile& t, int lists, double* sg,
                                          double* sx, double* s_list, double* s_dot,
                                          double* __restrict__ out) {
  const SoftShare h = soft_share(t, lists);
  const int total = (int)t.loc[t.count];
  double m = -INFINITY;
  for (int q = h.begin; q < h.end; q += h.step) m = max_t(m, sx[q]);
  s_list[h.list] = lanes_max(m, h.step);
  __syncthreads();
  for (int q = threadIdx.x; q < total; q += kSoftThreads) sx[q] = exp_t(sx[q] - s_list[t.owner[q]]);
  __syncthreads();
  double sum = 0, gsum = 0;
  for (int q = h.begin; q < h.end; q += h.step) {
    sum += sx[q];
    gsum += sg[q] * sx[q];
  }
  const double inv = 1.0 / lanes_sum(sum, h.step);
  s_list[h.list] = inv;
  s_dot[h.list] = lanes_sum(gsum, h.step) * inv;
  __syncthreads();
  for (int q = threadIdx.x; q < total; q += kSoftThreads) {
    const int l = t.owner[q];
    out[q] = sx[q] * s_list[l] * (sg[q] - s_dot[l]);
  }
}

template <class Op>
__global__ void __launch_bounds__(kSoftThreads)
    softmax_tile_kernel(double* __restrict__ out, const double* __restrict__ in0,
                        const double* __restrict__ in1, const int64_t* __restrict__ offsets,
                        long long nlists, long long nvalues, int lists, unsigned tiles) {
  __shared__ SoftTile t;
  __shared__ double s0[kTileElems], s1[Op::kArrays == 2 ? kTileElems : 1];
  __shared__ double s_list[kTileSoft], s_dot[kTileSoft];
  if (blockIdx.x >= tiles) {
    zero_outside(out, offsets, nlists, nvalues,
                 (blockIdx.x - tiles) * (long long)kSoftThreads + threadIdx.x,
                 (long long)(gridDim.x - tiles) * kSoftThreads);
    return;
  }
  stage_soft_tile(t, offsets, (long long)blockIdx.x * lists, nlists, lists, s0, in0,
                  Op::kArrays == 2 ? s1 : nullptr, Op::kArrays == 2 ? in1 : nullptr);
  if (t.mapped) {
    soft_tile(Op(), t, lists, s0, s1, s_list, s_dot, out + t.base);
    return;
  }
  const double* const in[2] = {in0, in1};
  for (int r = threadIdx.x >> 5; r < t.count; r += kSoftThreads / 32) {
    const double* p[Op::kArrays];
#pragma unroll
    for (int a = 0; a < Op::kArrays; a++) p[a] = in[a] + t.base + t.loc[r];
    Op::list(out + t.base + t.loc[r], p, t.loc[r + 1] - t.loc[r], TeamWarp{(int)threadIdx.x & 31});
  }
}

template <class Op, class T>
cudaError_t softmax(T* out, const T* in0, const T* in1, const int64_t* offsets, long long nlists,
                    long long nvalues, cudaStream_t s) {
  const long long mean = nvalues / nlists;
  int lists = sizeof(T) == 8 ? kTileSoft : kSoftThreads;
  if (sizeof(T) == 8) {
    // doubles: the most lists, 8 to kTileSoft, of which a tile's elements fit with a
    // quarter to spare (by the mean length)
    while (lists > 8 && mean * lists > kTileElems / 5 * 4) lists /= 2;
  } else {
    // floats: a round of 32 lists per warp where they are short, 8 where few or long
    // ones would leave most of the chip idle, fewer when a CTA would then take more than
    // 16384 elements.  With 32 and so, us, forward: 1000 lists of mean 500 103 and 33,
    // 1000 heavy-tailed lists of mean 60 48 and 17, 60000 of mean 250 81 and 52.
    while (lists > 32 && (nlists / lists < 2 * device_sm_count() || mean > 192)) lists /= 2;
    while (lists > 1 && mean * lists > kSoftWarp * 16) lists /= 2;
  }
  const unsigned blocks = (unsigned)((nlists + lists - 1) / lists);
  const unsigned rest = nvalues > 0 ? 2 * device_sm_count() : 0;
  if constexpr (sizeof(T) == 8)
    softmax_tile_kernel<Op><<<blocks + rest, kSoftThreads, 0, s>>>(out, in0, in1, offsets, nlists,
                                                                   nvalues, lists, blocks);
  else
    (lists == kSoftThreads ? softmax_kernel<Op, 32> : softmax_kernel<Op, 0>)<<<
        blocks + rest, kSoftThreads, 0, s>>>(out, in0, in1, offsets, nlists, nvalues, lists, blocks);
  return cudaGetLastError();
}

}  // namespace

// ================================================================== entry points
#define GB_AUTOGRAD(SUFFIX, T)                                                                  \
  GB_EXPORT int awkward_gb300_segment_sum_backward_##SUFFIX(                                    \
      T* grad_x, const T* grad_out, const int64_t* offsets, int64_t nlists, int64_t nvalues,   \
      void* stream) {                                                                           \
    cudaStream_t s = (cudaStream_t)stream;                                                      \
    if (nlists <= 0) return (int)(nvalues > 0 ? cudaMemsetAsync(grad_x, 0, sizeof(T) * (size_t)nvalues, s) : cudaSuccess); \
    sum_backward_rounds_kernel<T><<<device_sm_count() * 8, 256, 0, s>>>(                        \
        grad_x, grad_out, offsets, nlists, nvalues);                                            \
    return (int)cudaGetLastError();                                                             \
  }                                                                                             \
  GB_EXPORT int awkward_gb300_segment_max_backward_##SUFFIX(                                    \
      T* grad_x, const T* grad_out, const int64_t* argmax, int64_t nelements, int64_t nlists,  \
      void* stream) {                                                                           \
    cudaStream_t s = (cudaStream_t)stream;                                                      \
    if (nelements > 0) {                                                                        \
      cudaError_t e = cudaMemsetAsync(grad_x, 0, sizeof(T) * (size_t)nelements, s);             \
      if (e != cudaSuccess) return (int)e;                                                      \
    }                                                                                           \
    if (nlists <= 0) return 0;                                                                  \
    long long g = (nlists + 255) / 256;                                                         \
    const long long cap = (long long)device_sm_count() * 16;                                    \
    max_backward_kernel<T><<<(unsigned)(g < cap ? g : cap), 256, 0, s>>>(                      \
        grad_x, grad_out, argmax, nelements, nlists);                                           \
    return (int)cudaGetLastError();                                                             \
  }                                                                                             \
  GB_EXPORT int awkward_gb300_jagged_softmax_forward_##SUFFIX(                                  \
      T* y, const T* x, const int64_t* offsets, int64_t nlists, int64_t nvalues, void* stream) { \
    cudaStream_t s = (cudaStream_t)stream;                                                      \
    if (nlists <= 0) return (int)(nvalues > 0 ? cudaMemsetAsync(y, 0, sizeof(T) * (size_t)nvalues, s) : cudaSuccess); \
    return (int)softmax<SoftForward, T>(y, x, (const T*)nullptr, offsets, nlists, nvalues, s);  \
  }                                                                                             \
  GB_EXPORT int awkward_gb300_jagged_softmax_backward_##SUFFIX(                                 \
      T* grad_x, const T* grad_y, const T* x, const T* y_saved, const int64_t* offsets,        \
      int64_t nlists, int64_t nvalues, void* stream) {                                          \
    cudaStream_t s = (cudaStream_t)stream;                                                      \
    if (nlists <= 0) return (int)(nvalues > 0 ? cudaMemsetAsync(grad_x, 0, sizeof(T) * (size_t)nvalues, s) : cudaSuccess); \
    return (int)(y_saved ? softmax<SoftBackwardSaved, T>(grad_x, grad_y, y_saved, offsets,      \
                                                         nlists, nvalues, s)                    \
                         : softmax<SoftBackward, T>(grad_x, grad_y, x, offsets, nlists,         \
                                                    nvalues, s));                               \
  }

GB_AUTOGRAD(float32, float)
GB_AUTOGRAD(float64, double)
