// sort_impl.cuh -- segmented sort and argsort (the entry points are in
// sort_argsort_*.cu and sort_values*.cu, split only to compile in parallel).
//
//   awkward_argsort  awkward_argsort.cpp:62-108
//   awkward_sort     awkward_sort.cpp:62-117
//
// Every element becomes an unsigned order key (32 bits for values of up to 4
// bytes, else 64) whose ascending order is the requested order (descending
// keys are complemented), with awkward's comparator rules: integers and bool
// compare directly; floating point puts NaN before every number in both
// directions, and -0.0 equals +0.0.  Equal keys keep their input order -- the
// stable order (std::stable_sort's; it is also a valid answer when `stable`
// is false).  Segments by length:
//   <= 32      a warp takes 32 segments: keys staged in its shared memory, and
//              every lane sorts its segment in registers by a network;
//   <= 2048    tiles of whole segments (up to 4095 elements) sorted by one CTA
//              with a radix sort in shared memory, the segment as last digit;
//   longer     runs of 16384 sorted by one CTA each with the same radix sort,
//              then merged pass by pass (4096 outputs per CTA); the pass that
//              completes a segment writes its output.
// The radix sort and the merges work on 32-bit keys.  A 64-bit key is reduced
// to (key - smallest) >> s, the smallest shift that fits 32 bits; that keeps
// the order except for ties of the kept bits, which are resolved by the full
// keys where they occur (few: 16384 normal doubles have about 50 tied pairs).
// One pass over the segments sorts the short ones and lists the others; the
// long class's count, total and longest length are read back once, while the
// CTA class runs, and only when `length` admits a long segment.  Offsets are
// taken to be non-decreasing, as awkward builds them.
#pragma once

#include <limits.h>

#include <type_traits>

#include "gb_common.cuh"
#include "radix_sort.cuh"

using namespace gb;

namespace {

constexpr int kSortBlock = 256;
constexpr int kShortMax = 32;                  // longest segment sorted by a lane
constexpr int kMidMax = 2048;                  // ... in a tile of whole segments
constexpr int kMidWindow = 2048;               // a tile: the segments that start in a window
constexpr int kMidItems = 16;                  // 256 x 16 = 4096 slots >= kMidWindow - 1 + kMidMax
constexpr int kRunBlock = 1024;                // CTA of a run
constexpr int kRunItems = 16;
constexpr int kRun = kRunBlock * kRunItems;    // run length of long segments
static_assert(kSortBlock * kMidItems >= kMidWindow - 1 + kMidMax, "a tile fits its CTA");

// Counter words (device; set to -1 per call, so an add returns one less than
// the count before it).  kCntLong counts the long segments in its low
// kLongBits bits and, above them, the pairs of those of several runs by
// sixteens (whole 128-byte lines of pairs).
enum { kCntMidTotal = 0, kCntLong = 1, kCntLongTotal = 2, kCntLongMax = 3, kCntLimit = 4,
       kCntWords = 8 };
constexpr int kLongBits = 28;  // (segments of more than kMidMax elements)
static_assert(kCntWords <= Readback::kWords, "the counters are read back in one piece");

// ------------------------------------------------------------ order keys
template <class T>
using okey_t = typename std::conditional<(sizeof(T) <= 4), unsigned, unsigned long long>::type;

template <class T>
__device__ __forceinline__ okey_t<T> order_key(T v, bool asc) {
  okey_t<T> k;
  if constexpr (std::is_same<T, float>::value) {
    unsigned b = __float_as_uint(v);
    if ((b & 0x7fffffffu) > 0x7f800000u) return 0u;  // NaN: first in both directions
    if ((b << 1) == 0) b = 0;                        // -0.0 == +0.0
    k = (b >> 31) ? ~b : (b | 0x80000000u);
  } else if constexpr (std::is_same<T, double>::value) {
    unsigned long long b = (unsigned long long)__double_as_longlong(v);
    if ((b & 0x7fffffffffffffffull) > 0x7ff0000000000000ull) return 0ull;
    if ((b << 1) == 0) b = 0;
    k = (b >> 63) ? ~b : (b | 0x8000000000000000ull);
  } else if constexpr (sizeof(T) <= 4) {
    k = std::is_signed<T>::value ? (unsigned)(int)v ^ 0x80000000u : (unsigned)v;
  } else {
    k = (unsigned long long)v ^ (std::is_signed<T>::value ? 0x8000000000000000ull : 0ull);
  }
  return asc ? k : ~k;
}

// The value of a 32-bit order key, except where several values share it (NaN,
// the two zeros): then `at` is read.
template <class T>
__device__ __forceinline__ T key_value(unsigned key, bool asc, const T* at) {
  if constexpr (std::is_same<T, float>::value) {
    if (key == 0u) return *at;
    const unsigned k = asc ? key : ~key;
    if (k == 0x80000000u) return *at;
    return __uint_as_float((k >> 31) ? (k & 0x7fffffffu) : ~k);
  } else {
    const unsigned k = asc ? key : ~key;
    return (T)(std::is_signed<T>::value ? (int)(k ^ 0x80000000u) : (int)k);
  }
}

// Segment bounds clamped to [0, length] (the CPU clamps against `length`;
// a negative offset, undefined there, stays inside the buffers here).
template <class U>
__device__ __forceinline__ void seg_bounds(const U* offsets, long long i, long long length,
                                           long long* st, long long* sp) {
  long long a = (long long)offsets[i], b = (long long)offsets[i + 1];
  if (a > length) a = length;
  if (b > length) b = length;
  if (a < 0) a = 0;
  if (b < 0) b = 0;
  *st = a;
  *sp = b;
}

// Position p = st + j of a segment receives its j-th element in order, the
// segment-local index `local`: argsort writes it, sort gathers its value
// (only the first `limit` = min(offsets[last], length) positions).
template <class T, bool ARG>
__device__ __forceinline__ void emit(void* out, const T* x, long long st, long long j,
                                     long long local, long long limit) {
  if (ARG) static_cast<int64_t*>(out)[st + j] = local;
  else if (st + j < limit) static_cast<T*>(out)[st + j] = x[st + local];
}
// The same with the element's exact 32-bit order key at hand: a sort needs no
// gather.
template <class T, bool ARG>
__device__ __forceinline__ void emit_key(void* out, const T* x, long long st, long long j,
                                         long long local, long long limit, unsigned key, bool asc) {
  if constexpr (ARG || sizeof(T) > 4) emit<T, ARG>(out, x, st, j, local, limit);
  else if (st + j < limit) static_cast<T*>(out)[st + j] = key_value<T>(key, asc, x + st + local);
}

// The CPU's sort copies min(offsets[last], length) values (argsort: all of
// them).
template <class U, bool ARG>
__device__ __forceinline__ long long sort_limit(const U* offsets, long long olen,
                                                long long length) {
  if (ARG) return length;
  if (olen <= 0) return 0;
  const long long last = (long long)offsets[olen - 1];
  return last < length ? last : length;
}

// Positions outside [offsets[0], offsets[last]): argsort keeps the iota, sort
// copies through (below `limit`).
template <class T, class U, bool ARG>
__device__ __forceinline__ void sort_gaps(void* out, const T* __restrict__ x, long long length,
                                          const U* offsets, long long nseg, long long limit) {
  long long first = 0, last = 0;
  if (nseg >= 0) {
    first = (long long)offsets[0];
    last = (long long)offsets[nseg];
    first = first < 0 ? 0 : first > length ? length : first;
    last = last < first ? first : last > length ? length : last;
  }
  const long long gap = first + (length - last);
  for (long long g = blockIdx.x * (long long)kSortBlock + threadIdx.x; g < gap;
       g += (long long)gridDim.x * kSortBlock) {
    const long long i = g < first ? g : last + (g - first);
    if (ARG) static_cast<int64_t*>(out)[i] = i;
    else if (i < limit) static_cast<T*>(out)[i] = x[i];
  }
}
template <class T, class U, bool ARG>
__global__ void __launch_bounds__(kSortBlock)
    sort_gaps_kernel(void* out, const T* __restrict__ x, long long length, const U* offsets,
                     long long nseg) {
  sort_gaps<T, U, ARG>(out, x, length, offsets, nseg, sort_limit<U, ARG>(offsets, nseg + 1, length));
}

// ------------------------------------------------------------ short segments
// Sort the segments of <= kShortMax elements and list the others.  A warp
// takes 32 consecutive segments and stages their keys in its shared memory
// (coalesced loads, nothing to look up while the segments are contiguous and
// short); a lane then sorts its segment in registers.  A compare-exchange is
// one min and one max: the words are 27 bits of key above 5 of position (the
// top bits of a floating-point key; otherwise the keys less the segment's
// smallest, shifted to fit), and the network is as wide as the warp's longest
// segment needs (Batcher's for 8, 16, 24 or 32).  A segment with neighbours
// that tie in the kept bits while others were dropped is finished by an
// insertion sort on its whole keys; a warp that meets many of them takes the words
// of its next segments by their own range.  The order goes back through the stage,
// for coalesced stores.
//
// Bound by instructions (ALU 73 %; DRAM traffic is the input and output once).
// argsort of 2M float64 lists of mean 8: 80 us, against 166 us for counting
// ranks over keys staged by a CTA with barriers, and 147-192 us for counting
// them in a warp; the whole call 117 us against 229 us.  Eight CTAs a SM leave
// the widest network too few registers.
//
// The mid class is listed by the elements before it: every listed segment is
// longer than kShortMax, so slot (base / (kShortMax + 1)) is its own and one
// atomic gives it its place.
constexpr int kShortStage = 4096;  // bytes of a warp's stage: 16 segments always fit
constexpr int kSmallBlocks = 4;    // resident CTAs per SM (32 registers hold the widest network)
constexpr int kListStep = kShortMax + 1;
// Lanes of a warp with ties from which the warp looks at the range of its segments'
// floating-point keys before the next networks, and the bits that the range has to
// gain (or it is not looked at again).  Lists of float64 whose values are within 2^-20
// of each other, 2M of mean 4, 8, 1M of 16, 600000 of 25: 113, 170, 222, 361 us, with
// the fixed bits alone 198, 402, 530, 644 (normal values 89, 110, 130, 208).
constexpr int kCloserLanes = 8;
constexpr int kCloserBits = 4;

// The staged word of a value: its order key, for double the high word of it.
template <class T>
using stage_t = typename std::conditional<std::is_same<T, double>::value, unsigned, okey_t<T>>::type;
// (A double's is never above a larger double's: the values next to the zeros
// with a negative sign share the zeros' word, and are told apart as ties.)
template <class T>
__device__ __forceinline__ stage_t<T> stage_word(T v, bool asc) {
  if constexpr (std::is_same<T, double>::value) {
    const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
    const unsigned mag = hi & 0x7fffffffu;
    unsigned k = hi ^ ((unsigned)((int)hi >> 31) | 0x80000000u);
    if (hi == 0x80000000u) k = hi;
    k = asc ? k : ~k;
    return mag > 0x7ff00000u || (mag == 0x7ff00000u && lo != 0u) ? 0u : k;  // NaN first
  } else {
    return order_key<T>(v, asc);
  }
}

// Batcher's odd-even merge sort of N registers.
template <int N>
__device__ __forceinline__ void sort_network(unsigned (&c)[N]) {
#pragma unroll
  for (int p = 1; p < N; p <<= 1) {
#pragma unroll
    for (int k = p; k >= 1; k >>= 1) {
#pragma unroll
      for (int a = 0; a < N; a++) {
        const int b = a + k, off = a - k % p;
        if (off >= 0 && (off / k) % 2 == 0 && b < N && a / (2 * p) == b / (2 * p)) {
          const unsigned lo = min(c[a], c[b]), hi = max(c[a], c[b]);
          c[a] = lo;
          c[b] = hi;
        }
      }
    }
  }
}

// Floating-point words by the range [min, max] of the words staged: a key less the
// smallest possible one, aligned to the largest difference, which has `width` bits.
// (A double next to the zeros may have its key a word beside its stage word.)
template <class T>
struct StageRange {
  okey_t<T> lo = 0;
  int width = 8 * (int)sizeof(T);
  __device__ __forceinline__ void set(unsigned min, unsigned max) {
    if constexpr (sizeof(T) == 8) {
      lo = (unsigned long long)(min ? min - 1u : 0u) << 32;
      width = 64 - __clzll((long long)(((unsigned long long)(~max ? max + 1u : max) << 32 | 0xffffffffull) - lo));
    } else {
      lo = min;
      width = 32 - __clz((int)(max - min));
    }
  }
  __device__ __forceinline__ unsigned word(T v, bool asc) const {
    const unsigned long long d = (unsigned long long)(order_key<T>(v, asc) - lo);
    return width > 32 ? (unsigned)(d >> (width - 32)) : width > 0 ? (unsigned)d << (32 - width) : 0u;
  }
};

// The lane's segment (n <= N staged words from slot loc; its values at xs):
// leaves its order in the stage as 32-bit words, position + `base`.  Whole warp.
// Floating-point words are of keys of `kept_of` bits.  Returns whether the lane had ties
// to put in order.
template <int N, class T>
__device__ __forceinline__ bool short_order(unsigned char* stage, int loc, int n,
                                            const T* __restrict__ xs, bool asc, int base, int kept_of) {
  using W = stage_t<T>;
  const W* word = reinterpret_cast<const W*>(stage) + loc;
  unsigned c[N];
  bool dropped = kept_of > 27;
  if constexpr (std::is_floating_point<T>::value) {
#pragma unroll
    for (int j = 0; j < N; j++) {
      c[j] = ~0u;
      if (j < n) c[j] = (word[j] & ~31u) | j;
    }
  } else if constexpr (sizeof(T) <= 2) {
    // 16 bits above the smallest key of the type (the same in both directions
    // for the signed ones)
    const unsigned lo = std::is_signed<T>::value ? 0x7fff8000u : asc ? 0u : 0xffff0000u;
    dropped = false;
#pragma unroll
    for (int j = 0; j < N; j++) {
      c[j] = ~0u;
      if (j < n) c[j] = (word[j] - lo) << 5 | j;
    }
  } else {
    W lo = ~W(0), hi = 0;
#pragma unroll
    for (int j = 0; j < N; j++)
      if (j < n) {
        const W k = word[j];
        if constexpr (sizeof(W) == 4) c[j] = k;
        lo = k < lo ? k : lo;
        hi = k > hi ? k : hi;
      }
    const int width = 64 - __clzll((long long)(hi - lo));
    const int shift = n > 0 && width > 27 ? width - 27 : 0;
    dropped = shift > 0;
#pragma unroll
    for (int j = 0; j < N; j++) {
      unsigned k = ~0u;
      if (j < n) {
        if constexpr (sizeof(W) == 4) k = (c[j] - lo) >> shift;
        else k = (unsigned)((word[j] - lo) >> shift);
        k = k << 5 | j;
      }
      c[j] = k;
    }
  }
  sort_network(c);
  __syncwarp();  // every lane has read its words
  unsigned* order = reinterpret_cast<unsigned*>(stage) + loc;
  bool tie = false;
#pragma unroll
  for (int j = 0; j < N; j++) {
    if (j < n) order[j] = (c[j] & 31u) + base;
    if (j > 0) tie |= (c[j] ^ c[j - 1]) < 32u && j < n;
  }
  tie = tie && dropped;
  if (tie) {
    for (int j = 1; j < n; j++) {
      const unsigned e = order[j];
      const okey_t<T> k = order_key<T>(xs[e - base], asc);
      int i = j;
      for (; i > 0; i--) {
        const unsigned o = order[i - 1];
        const okey_t<T> ko = order_key<T>(xs[o - base], asc);
        if (ko < k || (ko == k && o < e)) break;
        order[i] = o;
      }
      order[i] = e;
    }
  }
  __syncwarp();
  return tie;
}

struct SortLists {
  unsigned long long* counters;
  long long* mid_st;   // by slot: first element, or -1
  long long* mid_len;  // by slot: base * kMidMax + (length - 1)
  long long mid_slots;
  long long* long_st;  // by order of arrival
  long long* long_len;
  long long* long_base;  // place in the pair buffers (segments of several runs)
  long long long_cap;
};

template <class T, class U, bool ARG>
__global__ void __launch_bounds__(kSortBlock, kSmallBlocks)
    sort_small_kernel(void* out, const T* __restrict__ x, long long length,
                      const U* __restrict__ offsets, long long nseg, bool asc, SortLists ls) {
  using W = stage_t<T>;
  __shared__ __align__(16) unsigned char s_stage[kSortBlock / 32][kShortStage];
  const long long limit = sort_limit<U, ARG>(offsets, nseg + 1, length);
  sort_gaps<T, U, ARG>(out, x, length, offsets, nseg, limit);
  if (blockIdx.x == 0 && threadIdx.x == 0) ls.counters[kCntLimit] = (unsigned long long)limit;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  W* word = reinterpret_cast<W*>(s_stage[w]);
  const unsigned* order = reinterpret_cast<const unsigned*>(s_stage[w]);
  const long long nbatch = (nseg + 31) / 32;
  int ranged = 0;  // 1: many ties so far, by fixed bits; 2: the range gains nothing
  for (long long b = (blockIdx.x * (long long)kSortBlock + threadIdx.x) >> 5; b < nbatch;
       b += ((long long)gridDim.x * kSortBlock) >> 5) {
    const long long s = b * 32 + lane;
    long long st = 0, sp = 0;
    if (s < nseg) seg_bounds(offsets, s, length, &st, &sp);
    const long long L = sp - st;
    const bool mid = L > kShortMax && L <= kMidMax;
    if (__any_sync(0xffffffffu, mid)) {
      const int n = mid ? (int)L : 0;
      int incl = n;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
      }
      unsigned long long base = 0;
      if (lane == 31) base = atomicAdd(ls.counters + kCntMidTotal, (unsigned long long)incl) + 1ull;
      base = __shfl_sync(0xffffffffu, base, 31) + (unsigned long long)(incl - n);
      const long long slot = (long long)(base / kListStep);
      if (mid && slot < ls.mid_slots) {  // beyond them only with overlapping segments
        ls.mid_st[slot] = st;
        ls.mid_len[slot] = (long long)base * kMidMax + (L - 1);
      }
    }
    if (L > kMidMax) {
      const unsigned long long pairs = L > kRun ? (unsigned long long)(L + 15) / 16 : 0ull;
      const unsigned long long before = atomicAdd(ls.counters + kCntLong, pairs << kLongBits | 1ull) + 1ull;
      const long long k = (long long)(before & ((1ull << kLongBits) - 1ull));
      if (k < ls.long_cap) {  // beyond it only with overlapping segments
        ls.long_st[k] = st;
        ls.long_len[k] = L;
        ls.long_base[k] = (long long)(before >> kLongBits) * 16;
        atomicAdd(ls.counters + kCntLongTotal, (unsigned long long)L);
        atomicMax(reinterpret_cast<long long*>(ls.counters + kCntLongMax), L);
      }
    }
    const int n = L > 0 && L <= kShortMax ? (int)L : 0;
    int incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += o;
    }
    const int all = __shfl_sync(0xffffffffu, incl, 31);
    if (all == 0) continue;
    const int longest = __reduce_max_sync(0xffffffffu, n);
    const long long prev = __shfl_up_sync(0xffffffffu, sp, 1);
    const bool chain = __all_sync(0xffffffffu, L == n && (lane == 0 || st == prev || s >= nseg));
    const int parts = all <= (int)(kShortStage / sizeof(W)) ? 1 : 2;
    for (int part = 0; part < parts; part++) {
      const int half = __shfl_sync(0xffffffffu, incl, 15);
      const int from = part == 0 ? 0 : half;
      const int cnt = (part == 0 && parts == 2 ? half : all) - from;
      const long long st0 = __shfl_sync(0xffffffffu, st, 16 * part);
      const int loc = incl - n - from;
      const int mine = parts == 1 || (lane >> 4) == part ? n : 0;
      if (chain) {
        for (int e0 = 0; e0 < cnt; e0 += 256) {
          T v[8];  // eight loads in flight
#pragma unroll
          for (int u = 0; u < 8; u++) {
            const int e = e0 + 32 * u + lane;
            v[u] = T(0);
            if (e < cnt) v[u] = x[st0 + e];
          }
#pragma unroll
          for (int u = 0; u < 8; u++) {
            const int e = e0 + 32 * u + lane;
            if (e < cnt) word[e] = stage_word<T>(v[u], asc);
          }
        }
      } else {
        for (unsigned m = __ballot_sync(0xffffffffu, mine > 0); m; m &= m - 1) {
          const int r = __ffs(m) - 1;
          const long long rs = __shfl_sync(0xffffffffu, st, r);
          const int rl = __shfl_sync(0xffffffffu, loc, r), rn = __shfl_sync(0xffffffffu, mine, r);
          if (lane < rn) word[rl + lane] = stage_word<T>(x[rs + lane], asc);
        }
      }
      __syncwarp();
      // (a sort's order holds places in the stage while the segments are
      // contiguous there and in memory: the values follow without a look-up)
      const int base = !ARG && chain ? loc : 0;
      StageRange<T> range;
      if constexpr (std::is_floating_point<T>::value) {
        if (ranged == 1) {
          unsigned min = ~0u, max = 0u;
          for (int e = lane; e < cnt; e += 32) {
            min = word[e] < min ? word[e] : min;
            max = word[e] > max ? word[e] : max;
          }
          range.set(__reduce_min_sync(0xffffffffu, min), __reduce_max_sync(0xffffffffu, max));
          if (range.width + kCloserBits > (int)(8 * sizeof(T))) {
            range = StageRange<T>();
            ranged = 2;
          } else if (chain) {
#pragma unroll 4
            for (int e = lane; e < cnt; e += 32) word[e] = range.word(x[st0 + e], asc);
          } else {
            for (unsigned m = __ballot_sync(0xffffffffu, mine > 0); m; m &= m - 1) {
              const int r = __ffs(m) - 1;
              const long long rs = __shfl_sync(0xffffffffu, st, r);
              const int rl = __shfl_sync(0xffffffffu, loc, r), rn = __shfl_sync(0xffffffffu, mine, r);
              if (lane < rn) word[rl + lane] = range.word(x[rs + lane], asc);
            }
          }
          __syncwarp();
        }
      }
      bool tie;
      if (longest <= 8) tie = short_order<8>(s_stage[w], loc, mine, x + st, asc, base, range.width);
      else if (longest <= 16) tie = short_order<16>(s_stage[w], loc, mine, x + st, asc, base, range.width);
      else if (longest <= 24) tie = short_order<24>(s_stage[w], loc, mine, x + st, asc, base, range.width);
      else tie = short_order<32>(s_stage[w], loc, mine, x + st, asc, base, range.width);
      if constexpr (std::is_floating_point<T>::value)
        if (ranged < 2 && __popc(__ballot_sync(0xffffffffu, tie)) >= kCloserLanes) ranged++;
      if (chain) {
#pragma unroll 4
        for (int e = lane; e < cnt; e += 32) {
          if (ARG) static_cast<int64_t*>(out)[st0 + e] = order[e];
          else if (st0 + e < limit) static_cast<T*>(out)[st0 + e] = x[st0 + order[e]];
        }
      } else {
        for (unsigned m = __ballot_sync(0xffffffffu, mine > 0); m; m &= m - 1) {
          const int r = __ffs(m) - 1;
          const long long rs = __shfl_sync(0xffffffffu, st, r);
          const int rl = __shfl_sync(0xffffffffu, loc, r), rn = __shfl_sync(0xffffffffu, mine, r);
          if (lane < rn) emit<T, ARG>(out, x, rs, lane, order[rl + lane], limit);
        }
      }
      __syncwarp();
    }
  }
}

// ------------------------------------------------------------ radix sort of a CTA's tile
// key[slot] / idx[slot]: the 32-bit keys and where they came from.  The slots
// of a warp are consecutive (32 * nitems), item j of lane l at 32 * j + l, so
// a pass that ranks equal digits by (warp, item, lane) is stable.
template <int THREADS, int ITEMS, bool SEGMENTS>
struct RadixTile {
  static constexpr int kThreads = THREADS, kItems = ITEMS;
  static constexpr int kWarps = THREADS / 32;
  unsigned key[THREADS * ITEMS];
  unsigned short idx[THREADS * ITEMS];
  unsigned match[kWarps][256];        // lanes of a warp that hold each digit (0 between steps)
  unsigned short count[kWarps][256];  // digits of each warp, then their first slots
  unsigned scan[kWarps + 1];
  unsigned long long lo, hi;          // block min / max
  unsigned char of[SEGMENTS ? THREADS * ITEMS : 1];  // segment of each element
};
// The tile is the start of the CTA's dynamic shared memory (a function that is
// not inlined then still addresses it as shared).
template <class Tile>
__device__ __forceinline__ Tile& radix_tile() {
  extern __shared__ __align__(16) unsigned char radix_smem[];
  return *reinterpret_cast<Tile*>(radix_smem);
}

// Smallest and largest of the threads' values (all threads; ends with a barrier).
template <class Tile, class K>
__device__ __forceinline__ void tile_minmax(Tile& s, K lo, K hi) {
  if (threadIdx.x == 0) {
    s.lo = ~0ull;
    s.hi = 0ull;
  }
  __syncthreads();
  if constexpr (sizeof(K) == 4) {
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
  } else {
#pragma unroll
    for (int d = 16; d > 0; d >>= 1) {
      const K a = __shfl_xor_sync(0xffffffffu, lo, d), b = __shfl_xor_sync(0xffffffffu, hi, d);
      lo = a < lo ? a : lo;
      hi = b > hi ? b : hi;
    }
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(&s.lo, (unsigned long long)lo);
    atomicMax(&s.hi, (unsigned long long)hi);
  }
  __syncthreads();
}

// One stable counting pass over kThreads * nitems slots, by 8 bits of the key
// or, with shift < 0, by the element's segment.  Slots past the elements hold
// all ones (segment 255) and are last after every pass: 255 is the last digit,
// and they come last among its slots.
template <class Tile>
__device__ __noinline__ void radix_pass(int nitems, int shift) {
  Tile& s = radix_tile<Tile>();
  constexpr int THREADS = Tile::kThreads, ITEMS = Tile::kItems, kWarps = Tile::kWarps;
  auto digit = [&](unsigned k, unsigned i) {
    return shift < 0 ? (unsigned)s.of[i] : (k >> shift) & 255u;
  };
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const unsigned lt = (1u << lane) - 1u;
  for (int i = threadIdx.x; i < kWarps * 128; i += THREADS)
    reinterpret_cast<unsigned*>(&s.count[0][0])[i] = 0u;
  for (int i = threadIdx.x; i < kWarps * 256; i += THREADS) (&s.match[0][0])[i] = 0u;
  unsigned key[ITEMS];
  unsigned ri[ITEMS];  // rank << 16 | idx
  const int slot0 = w * 32 * nitems + lane;
#pragma unroll
  for (int j = 0; j < ITEMS; j++)
    if (j < nitems) {
      key[j] = s.key[slot0 + 32 * j];
      ri[j] = s.idx[slot0 + 32 * j];
    }
  __syncthreads();
  // lanes of equal digits find each other by an or into the digit's word: the
  // unit of the match instruction was 61 % busy at 326 us for the runs of 9M
  // floats, this takes 196 us (bound by shared-memory wavefronts, 67 %)
  unsigned short* cnt = s.count[w];
  unsigned* match = s.match[w];
#pragma unroll
  for (int j = 0; j < ITEMS; j++)
    if (j < nitems) {
      const unsigned d = digit(key[j], ri[j]);
      atomicOr(match + d, 1u << lane);
      __syncwarp();
      const unsigned peers = match[d];
      const unsigned r = cnt[d] + __popc(peers & lt);
      __syncwarp();
      if ((peers >> lane) == 1u) {  // the last of its peers
        cnt[d] = (unsigned short)(r + 1);
        match[d] = 0u;
      }
      __syncwarp();
      ri[j] |= r << 16;
    }
  __syncthreads();
  unsigned run = 0;
  if (threadIdx.x < 256) {
#pragma unroll 8
    for (int i = 0; i < kWarps; i++) {
      const unsigned c = s.count[i][threadIdx.x];
      s.count[i][threadIdx.x] = (unsigned short)run;
      run += c;
    }
  }
  unsigned total;
  auto add = [](unsigned a, unsigned b) { return a + b; };
  const unsigned first = block_exclusive_scan<THREADS>(run, add, 0u, s.scan, &total);
  if (threadIdx.x < 256) {
#pragma unroll 8
    for (int i = 0; i < kWarps; i++) s.count[i][threadIdx.x] += (unsigned short)first;
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < ITEMS; j++)
    if (j < nitems) {
      const unsigned i = ri[j] & 0xffffu;
      const unsigned d = digit(key[j], i);
      const unsigned at = cnt[d] + (ri[j] >> 16);
      s.key[at] = key[j];
      s.idx[at] = (unsigned short)i;
    }
  __syncthreads();
}

// Passes over the low `bits` bits of the keys.
template <class Tile>
__device__ __forceinline__ void radix_bits(int nitems, int bits) {
  for (int shift = 0; shift < bits; shift += 8) radix_pass<Tile>(nitems, shift);
}

__device__ __forceinline__ int bit_width(unsigned long long v) { return 64 - __clzll((long long)v); }

// Order the slots whose kept bits tie by the full keys full(idx), equal ones
// by idx, inside [seg_lo(q), seg_hi(q)) of slot q.  Slots that tie with their
// left neighbour and hold another full key are marked first: only runs with a
// mark are ordered (equal values, zeros above all, tie in long runs without
// one).  Returns false (on every thread) when a run of more than kTieRun slots has
// a mark: nothing is ordered then.
// (200000 float64 lists of mean 60, half their values within 2^-20 of each other: 782
// us, with runs of up to 32 ordered here 1030.)
constexpr int kTieRun = 16;
template <class Tile, class Full, class Lo, class Hi>
__device__ __forceinline__ bool fix_ties(Tile& s, int count, Full full, Lo seg_lo, Hi seg_hi) {
  constexpr int THREADS = Tile::kThreads, ITEMS = Tile::kItems;
  unsigned* marks = &s.match[0][0];  // a bit per slot (the passes clear it again)
  for (int i = threadIdx.x; i < THREADS * ITEMS / 32; i += THREADS) marks[i] = 0u;
  __syncthreads();
  bool any = false;
#pragma unroll 2
  for (int j = 0; j < ITEMS; j++) {
    const int q = threadIdx.x + j * THREADS;
    if (q >= count) break;
    if (q > seg_lo(q) && s.key[q - 1] == s.key[q] && full(s.idx[q - 1]) != full(s.idx[q])) {
      atomicOr(marks + (q >> 5), 1u << (q & 31));
      any = true;
    }
  }
  if (!__syncthreads_or(any)) return true;
  bool bad = false;  // (the slots are in order: a run of more than kTieRun from q on)
#pragma unroll 2
  for (int j = 0; j < ITEMS; j++) {
    const int q = threadIdx.x + j * THREADS;
    if (q + kTieRun >= count) break;
    if (s.key[q + kTieRun] != s.key[q] || q + kTieRun >= seg_hi(q)) continue;
    const int w = (q + 1) >> 5, sh = (q + 1) & 31;  // the marks of q + 1 .. q + kTieRun
    bad |= (__funnelshift_r(marks[w], sh ? marks[w + 1] : 0u, sh) & ((1u << kTieRun) - 1u)) != 0u;
  }
  if (__syncthreads_or(bad)) return false;
  int to[ITEMS];  // new slot << 16 | idx, or -1
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const int q = threadIdx.x + j * THREADS;
    to[j] = -1;
    if (q >= count) continue;
    const unsigned k = s.key[q];
    const int lo = seg_lo(q), hi = seg_hi(q);
    const bool left = q > lo && s.key[q - 1] == k, right = q + 1 < hi && s.key[q + 1] == k;
    if (!left && !right) continue;
    int a = q, b = q + 1;
    while (a > lo && q - a < kTieRun && s.key[a - 1] == k) a--;
    while (b < hi && b - q < kTieRun && s.key[b] == k) b++;
    unsigned marked = 0;  // slots a+1 .. b-1
    for (int i = a + 1; i < b; i++) marked |= marks[i >> 5] >> (i & 31) & 1u;
    if (!marked) continue;  // (else the run has kTieRun slots at most)
    const unsigned long long mine = full(s.idx[q]);
    int r = a;
    for (int i = a; i < b; i++) {
      if (i == q) continue;
      const unsigned long long o = full(s.idx[i]);
      r += (o < mine) || (o == mine && i < q) ? 1 : 0;
    }
    if (r != q) to[j] = r << 16 | s.idx[q];
  }
  __syncthreads();
#pragma unroll
  for (int j = 0; j < ITEMS; j++)
    if (to[j] >= 0) s.idx[to[j] >> 16] = (unsigned short)to[j];
  __syncthreads();
  return true;
}

// When that fails: the runs of ties numbered in order, and the slots sorted by that
// number and the next of the `left` dropped bits, as many as fit 32 bits with it.
// dropped(idx) are a slot's dropped bits.  Returns the bits still not looked at (0:
// slots with equal keys have equal full keys).
//
// Argsort of float64 lists, half their values within 2^-20 of each other, 20000 of mean
// 500, 1000 of 8000, 300 of 30000: 679, 594, 749 us; with a sort by the dropped bits and
// another by the kept ones 1322, 964, 1038 (normal values 358, 328, 373).
template <class Tile, class Dropped, class Lo>
__device__ __forceinline__ int split_ties(Tile& s, int count, int nitems, int left, Dropped dropped,
                                          Lo seg_lo) {
  constexpr int THREADS = Tile::kThreads, ITEMS = Tile::kItems;
  __syncthreads();
  const int q0 = threadIdx.x * ITEMS;
  unsigned first = 0, begins = 0;  // a bit per slot of the thread: a run begins there
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const int q = q0 + j;
    if (q < count && (q == seg_lo(q) || s.key[q] != s.key[q - 1])) begins |= 1u << j;
  }
  unsigned total;
  auto add = [](unsigned a, unsigned b) { return a + b; };
  first = block_exclusive_scan<THREADS>((unsigned)__popc(begins), add, 0u, s.scan, &total);
  const int bits = total > 1 ? 32 - __clz((int)(total - 1)) : 0;
  const int take = left < 32 - bits ? left : 32 - bits;
  left -= take;
  const unsigned long long mask = (1ull << take) - 1ull;
  __syncthreads();  // (every key has been compared)
#pragma unroll
  for (int j = 0; j < ITEMS; j++) {
    const int q = q0 + j;
    if (q >= nitems * THREADS) break;
    unsigned k = ~0u;
    if (q < count) {
      const unsigned run = first + __popc(begins & ((2u << j) - 1u)) - 1u;
      k = (unsigned)((unsigned long long)run << take | (dropped(s.idx[q]) >> left & mask));
    }
    s.key[q] = k;
  }
  __syncthreads();
  radix_bits<Tile>(nitems, bits + take);
  return left;
}

// ------------------------------------------------------------ tiles of whole segments
// The listed segments of kShortMax+1 .. kMidMax elements.  A tile is the
// segments whose base (the elements listed before them) lies in a window of
// kMidWindow: their slots are the window's, at most 63.
using MidTile = RadixTile<kSortBlock, kMidItems, true>;
template <class T, bool ARG>
__global__ void __launch_bounds__(kSortBlock, 4)
    sort_mid_kernel(void* out, const T* __restrict__ x, bool asc, SortLists ls) {
  using K = okey_t<T>;
  using Tile = MidTile;
  Tile& s = radix_tile<Tile>();
  unsigned char* s_of = s.of;
  __shared__ long long s_st[64];
  __shared__ int s_loc[65];
  __shared__ int s_n[2];
  const long long limit = (long long)ls.counters[kCntLimit];
  const long long total = (long long)(ls.counters[kCntMidTotal] + 1ull);
  const int lane = threadIdx.x & 31;
  for (long long w0 = (long long)blockIdx.x * kMidWindow; w0 < total;
       w0 += (long long)gridDim.x * kMidWindow) {
    const long long slot0 = w0 / kListStep;
    long long st = -1, base = 0;
    int len = 0;
    if (threadIdx.x < 64) {
      const long long slot = slot0 + threadIdx.x;
      if (slot < ls.mid_slots) st = ls.mid_st[slot];
      if (st >= 0) {
        const long long v = ls.mid_len[slot];
        base = v / kMidMax;
        len = (int)(v % kMidMax) + 1;
        if (base < w0 || base >= w0 + kMidWindow) st = -1;
      }
      const unsigned m = __ballot_sync(0xffffffffu, st >= 0);
      if (lane == 0) s_n[threadIdx.x >> 5] = __popc(m);
      len = st >= 0 ? len : 0;
      base = __popc(m & ((1u << lane) - 1u));  // rank among the warp's
    }
    __syncthreads();
    const int nseg = s_n[0] + s_n[1];
    if (threadIdx.x < 64 && st >= 0) {
      const int r = (int)base + (threadIdx.x >= 32 ? s_n[0] : 0);
      s_st[r] = st;
      s_loc[r + 1] = len;
    }
    __syncthreads();
    if (threadIdx.x < 32) {  // lengths to first slots
      int a = 2 * lane < nseg ? s_loc[2 * lane + 1] : 0;
      const int b = 2 * lane + 1 < nseg ? s_loc[2 * lane + 2] : 0;
      int incl = a + b;
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const int o = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += o;
      }
      a = incl - b;
      __syncwarp();
      s_loc[2 * lane + 1] = a;
      s_loc[2 * lane + 2] = incl;
      if (lane == 0) s_loc[0] = 0;
    }
    __syncthreads();
    const int count = s_loc[nseg];
    const int nitems = (count + kSortBlock - 1) / kSortBlock;
    for (int g = threadIdx.x >> 5; g < nseg; g += kSortBlock / 32)
      for (int q = s_loc[g] + lane; q < s_loc[g + 1]; q += 32) s_of[q] = (unsigned char)g;
    for (int q = count + threadIdx.x; q < nitems * kSortBlock; q += kSortBlock)
      s_of[q] = 255;  // padding: last in every pass
    __syncthreads();
    auto full = [&](int q) -> K {
      const int g = s_of[q];
      return order_key<T>(x[s_st[g] + (q - s_loc[g])], asc);
    };
    K lo = ~K(0), hi = 0;
    for (int q = threadIdx.x; q < count; q += kSortBlock) {
      const K k = full(q);
      if constexpr (sizeof(T) <= 4) s.key[q] = k;
      lo = k < lo ? k : lo;
      hi = k > hi ? k : hi;
    }
    tile_minmax(s, lo, hi);
    lo = (K)s.lo;
    hi = (K)s.hi;
    const int width = bit_width(hi - lo), shift = width > 32 ? width - 32 : 0;
    for (int q = threadIdx.x; q < nitems * kSortBlock; q += kSortBlock) {
      unsigned k = ~0u;
      if (q < count) {
        if constexpr (sizeof(T) <= 4) k = s.key[q] - lo;
        else k = (unsigned)((full(q) - lo) >> shift);
      }
      s.key[q] = k;
      s.idx[q] = (unsigned short)q;
    }
    __syncthreads();
    radix_bits<Tile>(nitems, width - shift);
    if (nseg > 1) radix_pass<Tile>(nitems, -1);
    if constexpr (sizeof(T) > 4) {
      auto seg_lo = [&](int q) { return s_loc[s_of[q]]; };
      auto seg_hi = [&](int q) { return s_loc[s_of[q] + 1]; };
      auto whole = [&](int i) { return (unsigned long long)full(i); };
      auto dropped = [&](int i) { return (unsigned long long)(full(i) - lo); };
      for (int left = shift; left > 0 && !fix_ties(s, count, whole, seg_lo, seg_hi);)
        left = split_ties(s, count, nitems, left, dropped, seg_lo);
    }
    for (int q = threadIdx.x; q < count; q += kSortBlock) {
      const int g = s_of[q], b = s_loc[g];
      const int local = (int)s.idx[q] - b;
      if constexpr (sizeof(T) <= 4)
        emit_key<T, ARG>(out, x, s_st[g], q - b, local, limit, s.key[q] + (unsigned)lo, asc);
      else
        emit<T, ARG>(out, x, s_st[g], q - b, local, limit);
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------ long segments
__global__ void long_runs_kernel(const long long* __restrict__ lens, long long nlong,
                                 long long* __restrict__ runs) {
  for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < nlong;
       k += (long long)gridDim.x * blockDim.x)
    runs[k] = (lens[k] + kRun - 1) / kRun;
}

// Last k with first[k] <= r (first[0] = 0 <= r), 32 probes at a time (whole warp).
__device__ __forceinline__ long long warp_find(const long long* __restrict__ first, long long n,
                                               long long r) {
  const int lane = threadIdx.x & 31;
  long long lo = 0, hi = n;
  while (hi - lo > 1) {
    const long long step = (hi - lo + 31) >> 5;
    const long long k = lo + lane * step;
    const int cnt = __popc(__ballot_sync(0xffffffffu, k < hi && first[k] <= r));
    lo += (cnt - 1) * step;
    hi = lo + step < hi ? lo + step : hi;
  }
  return lo;
}

struct LongSegs {
  const long long* st;     // first element
  const long long* len;
  const long long* base;   // place in the pair buffers, which hold the segments of several runs
  const long long* run0;   // runs of the segments before it
  const long long* total;  // device word: all runs
  long long n;
  unsigned long long* lo;  // smallest and largest order key (64-bit keys)
  unsigned long long* hi;
};

// The run of CTA `r` (all threads; false past the last): its segment, first
// element and the segment's place in the pair buffers.
struct LongRun {
  long long seg, st, len, r0, base;
};
__device__ __forceinline__ bool long_run(LongRun& v, const LongSegs& g, long long r) {
  __shared__ long long s_seg;
  if (r >= *g.total) return false;
  if (threadIdx.x < 32) {
    const long long k = warp_find(g.run0, g.n, r);
    if (threadIdx.x == 0) s_seg = k;
  }
  __syncthreads();
  v.seg = s_seg;
  v.st = g.st[v.seg];
  v.len = g.len[v.seg];
  v.r0 = (r - g.run0[v.seg]) * kRun;
  v.base = g.base[v.seg];
  return true;
}

__device__ __forceinline__ int key_shift(unsigned long long lo, unsigned long long hi) {
  const int width = bit_width(hi - lo);
  return width > 32 ? width - 32 : 0;
}

// Smallest and largest 64-bit order key of the segments of several runs.
template <class T>
__global__ void __launch_bounds__(kRunBlock)
    long_minmax_kernel(const T* __restrict__ x, LongSegs g, bool asc) {
  LongRun v;
  if (!long_run(v, g, blockIdx.x) || v.len <= kRun) return;
  const int n = (int)(v.len - v.r0 < kRun ? v.len - v.r0 : kRun);
  unsigned long long lo = ~0ull, hi = 0ull;
  for (int i = threadIdx.x; i < n; i += kRunBlock) {
    const unsigned long long k = order_key<T>(x[v.st + v.r0 + i], asc);
    lo = k < lo ? k : lo;
    hi = k > hi ? k : hi;
  }
#pragma unroll
  for (int d = 16; d > 0; d >>= 1) {
    const unsigned long long a = __shfl_xor_sync(0xffffffffu, lo, d), b = __shfl_xor_sync(0xffffffffu, hi, d);
    lo = a < lo ? a : lo;
    hi = b > hi ? b : hi;
  }
  if ((threadIdx.x & 31) == 0) {
    atomicMin(g.lo + v.seg, lo);
    atomicMax(g.hi + v.seg, hi);
  }
}

// Pairs of a run on their way through the merges: kept key bits and
// segment-local index in one word (unique, and ordered as (key, index)), or,
// for segments of 2^32 elements or more, the full key and a 64-bit index.
struct WidePair {
  unsigned long long key, idx;
};
__device__ __forceinline__ unsigned long long pair_index(unsigned long long p) { return p & 0xffffffffull; }
__device__ __forceinline__ unsigned long long pair_index(const WidePair& p) { return p.idx; }

using RunTile = RadixTile<kRunBlock, kRunItems, false>;

// Sort one run in shared memory.  A segment of one run is written out; the
// others' runs go to the pair buffer.
template <class T, bool ARG>
__global__ void __launch_bounds__(kRunBlock)
    sort_runs_kernel(void* out, const T* __restrict__ x, LongSegs g, bool asc, bool wide,
                     const unsigned long long* __restrict__ counters, void* __restrict__ dst) {
  using K = okey_t<T>;
  using Tile = RunTile;
  Tile& s = radix_tile<Tile>();
  LongRun v;
  if (!long_run(v, g, blockIdx.x)) return;
  const bool whole = v.len <= kRun;
  const int n = (int)(v.len - v.r0 < kRun ? v.len - v.r0 : kRun);
  const int nitems = (n + kRunBlock - 1) / kRunBlock;
  const T* xr = x + v.st + v.r0;
  // kept bits: (key - lo) >> shift, lo and shift of the segment when its runs
  // are merged by them, else of the run
  K lo = ~K(0), hi = 0;
#pragma unroll
  for (int j = 0; j < kRunItems; j++) {
    const int q = threadIdx.x + j * kRunBlock;
    if (q < n) {
      const K k = order_key<T>(xr[q], asc);
      if constexpr (sizeof(T) <= 4) s.key[q] = k;
      lo = k < lo ? k : lo;
      hi = k > hi ? k : hi;
    }
  }
  tile_minmax(s, lo, hi);
  lo = (K)s.lo;
  hi = (K)s.hi;
  if constexpr (sizeof(T) > 4)
    if (!whole && !wide) {
      lo = g.lo[v.seg];
      hi = g.hi[v.seg];
    }
  const int shift = key_shift(lo, hi);
  const int width = bit_width(hi - lo);
#pragma unroll
  for (int j = 0; j < kRunItems; j++) {
    const int q = threadIdx.x + j * kRunBlock;
    if (j < nitems) {
      unsigned k = ~0u;
      if (q < n) {
        if constexpr (sizeof(T) <= 4) k = s.key[q] - lo;
        else k = (unsigned)((order_key<T>(xr[q], asc) - lo) >> shift);
      }
      s.key[q] = k;
      s.idx[q] = (unsigned short)q;
    }
  }
  __syncthreads();
  radix_bits<Tile>(nitems, width - shift);
  if constexpr (sizeof(T) > 4) {
    auto full = [&](int i) { return (unsigned long long)order_key<T>(xr[i], asc); };
    auto dropped = [&](int i) { return full(i) - lo; };
    auto seg_lo = [](int) { return 0; };
    bool split = false;
    for (int left = shift; left > 0 && !fix_ties(s, n, full, seg_lo, [n](int) { return n; });) {
      left = split_ties(s, n, nitems, left, dropped, seg_lo);
      split = true;
    }
    if (split && !whole) {  // the merges go by the kept bits
      for (int q = threadIdx.x; q < n; q += kRunBlock) s.key[q] = (unsigned)(dropped(s.idx[q]) >> shift);
      __syncthreads();
    }
  }
  if (whole) {
    const long long limit = (long long)counters[kCntLimit];
    for (int q = threadIdx.x; q < n; q += kRunBlock) {
      if constexpr (sizeof(T) <= 4)
        emit_key<T, ARG>(out, x, v.st, q, s.idx[q], limit, s.key[q] + (unsigned)lo, asc);
      else
        emit<T, ARG>(out, x, v.st, q, s.idx[q], limit);
    }
    return;
  }
  for (int q = threadIdx.x; q < n; q += kRunBlock) {
    const unsigned i = s.idx[q];
    const long long at = v.base + v.r0 + q;
    if (!wide) {
      const unsigned k = sizeof(T) <= 4 ? s.key[q] + (unsigned)lo : s.key[q];
      static_cast<unsigned long long*>(dst)[at] =
          (unsigned long long)k << 32 | (unsigned long long)(v.r0 + i);
    } else {
      static_cast<WidePair*>(dst)[at] =
          WidePair{(unsigned long long)order_key<T>(xr[i], asc), (unsigned long long)(v.r0 + i)};
    }
  }
}

// a before b, a's run being the earlier one (so ties of key go to a).  Words
// whose kept bits tie are compared by the full keys when bits were dropped.
template <class T>
__device__ __forceinline__ bool before(unsigned long long a, unsigned long long b, const T* xs,
                                       bool asc, bool dropped) {
  if constexpr (sizeof(T) > 4) {
    if (dropped && (a >> 32) == (b >> 32)) {
      const okey_t<T> ka = order_key<T>(xs[pair_index(a)], asc);
      const okey_t<T> kb = order_key<T>(xs[pair_index(b)], asc);
      return ka <= kb;
    }
  }
  return a < b;
}
template <class T>
__device__ __forceinline__ bool before(const WidePair& a, const WidePair& b, const T*, bool, bool) {
  return a.key <= b.key;
}

// Outputs merged per thread and per CTA (a tile never straddles two runs).
template <class P>
struct MergeTile {
  static constexpr int kPer = sizeof(P) == 8 ? 16 : 4;
  static constexpr int kTile = kSortBlock * kPer;
  static_assert(kRun % kTile == 0, "merge tiles do not straddle runs");
};
__device__ __forceinline__ int mslot(int p) { return p + (p >> 4); }

// One merge pass at run width w: runs [lo, lo+w) and [lo+w, lo+2w) of each
// segment longer than w merge into 2w; a segment no longer than 2w is then
// complete and written out.  A CTA produces a tile of outputs: two of its
// warps find the inputs by 32-way searches, and they are staged in shared
// memory (padded one slot per 16: threads merge 16 consecutive outputs each).
template <class T, bool ARG, class P>
__global__ void __launch_bounds__(kSortBlock)
    sort_merge_kernel(void* out, const T* __restrict__ x, LongSegs g, bool asc, long long w,
                      const unsigned long long* __restrict__ counters, const P* __restrict__ src,
                      P* __restrict__ dst) {
  constexpr int kMergePer = MergeTile<P>::kPer, kMergeTile = MergeTile<P>::kTile;
  __shared__ P s_p[kMergeTile + kMergeTile / 16];
  __shared__ long long s_split[2];
  LongRun v;
  constexpr int kSub = kRun / kMergeTile;
  if (!long_run(v, g, blockIdx.x / kSub)) return;
  const long long o0 = v.r0 + (long long)(blockIdx.x % kSub) * kMergeTile;
  if (v.len <= w || o0 >= v.len) return;
  const T* xs = x + v.st;
  bool dropped = false;
  if constexpr (sizeof(T) > 4 && std::is_same<P, unsigned long long>::value)
    dropped = key_shift(g.lo[v.seg], g.hi[v.seg]) > 0;
  const long long lo = o0 / (2 * w) * (2 * w);
  const long long mid = lo + w < v.len ? lo + w : v.len;
  const long long hi = lo + 2 * w < v.len ? lo + 2 * w : v.len;
  const long long na = mid - lo, nb = hi - mid;
  const long long o1 = o0 + kMergeTile < hi ? o0 + kMergeTile : hi;
  const P* pa = src + v.base + lo;
  const P* pb = src + v.base + mid;
  if (threadIdx.x < 64) {
    // pairs of run a among the first d outputs: first i with !(a[i] before
    // b[d - i - 1]), 32 probes at a time
    const int lane = threadIdx.x & 31;
    const long long d = (threadIdx.x < 32 ? o0 : o1) - lo;
    long long from = d - nb > 0 ? d - nb : 0, to = d < na ? d : na;
    while (from < to) {
      const long long step = (to - from + 31) >> 5;
      const long long i = from + lane * step;
      const bool in = i < to && before<T>(pa[i], pb[d - i - 1], xs, asc, dropped);
      const int cnt = __popc(__ballot_sync(0xffffffffu, in));
      if (cnt == 0) break;
      const long long last = from + (cnt - 1) * step;  // before: the answer is past it
      to = last + step < to ? last + step : to;
      from = last + 1;
    }
    if (lane == 0) s_split[threadIdx.x >> 5] = from;
  }
  __syncthreads();
  const long long a0 = s_split[0], b0 = (o0 - lo) - a0;
  const int ca = (int)(s_split[1] - a0), cnt = (int)(o1 - o0), cb = cnt - ca;
  for (int i = threadIdx.x; i < cnt; i += kSortBlock)
    s_p[mslot(i)] = i < ca ? pa[a0 + i] : pb[b0 + (i - ca)];
  __syncthreads();
  const int d = threadIdx.x * kMergePer;
  P o[kMergePer];
  if (d < cnt) {
    int from = d - cb > 0 ? d - cb : 0, to = d < ca ? d : ca;
    while (from < to) {
      const int i = (from + to) >> 1;
      if (before<T>(s_p[mslot(i)], s_p[mslot(ca + d - i - 1)], xs, asc, dropped)) from = i + 1;
      else to = i;
    }
    int i = from, j = ca + d - from;
    P va = s_p[mslot(i < ca ? i : 0)], vb = s_p[mslot(j < cnt ? j : 0)];
#pragma unroll
    for (int k = 0; k < kMergePer; k++) {
      const bool take_a = i < ca && (j >= cnt || before<T>(va, vb, xs, asc, dropped));
      o[k] = take_a ? va : vb;
      if (take_a) {
        i++;
        va = s_p[mslot(i < ca ? i : 0)];
      } else {
        j++;
        vb = s_p[mslot(j < cnt ? j : 0)];
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kMergePer; k++)
    if (d + k < cnt) s_p[mslot(d + k)] = o[k];
  __syncthreads();
  if (v.len > 2 * w) {
    for (int i = threadIdx.x; i < cnt; i += kSortBlock) dst[v.base + o0 + i] = s_p[mslot(i)];
    return;
  }
  const long long limit = (long long)counters[kCntLimit];
  for (int i = threadIdx.x; i < cnt; i += kSortBlock) {
    const P p = s_p[mslot(i)];
    if constexpr (sizeof(T) <= 4 && std::is_same<P, unsigned long long>::value)
      emit_key<T, ARG>(out, x, v.st, o0 + i, (long long)pair_index(p), limit, (unsigned)(p >> 32), asc);
    else
      emit<T, ARG>(out, x, v.st, o0 + i, (long long)pair_index(p), limit);
  }
}

template <class T, bool ARG, class P>
cudaError_t sort_long(void* toptr, const T* x, const SortLists& ls, long long nlong, long long total,
                      long long merged, long long maxl, bool asc, uint64_t inv, uint64_t* err,
                      cudaStream_t s) {
  const long long bound = total / kRun + nlong;  // runs, at most
  const bool merges = maxl > kRun;
  // two pair buffers for the `merged` elements of segments of several runs
  const size_t pair_bytes = sizeof(P) * (size_t)merged;
  void* mem = nullptr;
  cudaError_t e = scratch_alloc(&mem, 2 * pair_bytes + sizeof(long long) * (size_t)(3 * nlong + 1), s);
  if (e != cudaSuccess) return e;
  P* a = static_cast<P*>(mem);
  P* b = a + merged;
  long long* run0 = reinterpret_cast<long long*>(b + merged);
  long long* ntotal = run0 + nlong;
  LongSegs g;
  g.st = ls.long_st;
  g.len = ls.long_len;
  g.base = ls.long_base;
  g.run0 = run0;
  g.total = ntotal;
  g.n = nlong;
  g.lo = reinterpret_cast<unsigned long long*>(ntotal + 1);
  g.hi = g.lo + nlong;
  long_runs_kernel<<<(unsigned)((nlong + 255) / 256 < 1024 ? (nlong + 255) / 256 : 1024), 256, 0, s>>>(
      ls.long_len, nlong, run0);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = exclusive_scan_i64(run0, run0, nlong, ntotal, inv, err, s);
  if (e == cudaSuccess && merges && sizeof(T) > 4) {
    e = cudaMemsetAsync(g.lo, 0xff, sizeof(long long) * (size_t)nlong, s);
    if (e == cudaSuccess) e = cudaMemsetAsync(g.hi, 0, sizeof(long long) * (size_t)nlong, s);
    if (e == cudaSuccess) {
      if constexpr (sizeof(T) > 4)
        long_minmax_kernel<T><<<(unsigned)bound, kRunBlock, 0, s>>>(x, g, asc);
      e = cudaGetLastError();
    }
  }
  if (e == cudaSuccess) {
    constexpr int bytes = (int)sizeof(RunTile);
    e = cudaFuncSetAttribute(sort_runs_kernel<T, ARG>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (e == cudaSuccess) {
      sort_runs_kernel<T, ARG><<<(unsigned)bound, kRunBlock, bytes, s>>>(
          toptr, x, g, asc, sizeof(P) > 8, ls.counters, a);
      e = cudaGetLastError();
    }
  }
  for (long long w = kRun; w < maxl && e == cudaSuccess; w <<= 1) {
    sort_merge_kernel<T, ARG, P><<<(unsigned)(bound * (kRun / MergeTile<P>::kTile)), kSortBlock, 0, s>>>(
        toptr, x, g, asc, w, ls.counters, a, b);
    e = cudaGetLastError();
    P* t = a;
    a = b;
    b = t;
  }
  cudaError_t f = scratch_free(mem, s);
  return e != cudaSuccess ? e : f;
}

template <class T, class U, bool ARG>
cudaError_t launch_sort(void* toptr, const T* x, long long length, const U* offsets,
                        long long offsetslength, bool ascending, uint64_t inv, uint64_t* err,
                        cudaStream_t s) {
  if (length <= 0) return cudaSuccess;
  const long long nseg = offsetslength - 1;
  const long long cap = (long long)device_sm_count() * 16;
  auto grid = [cap](long long want) { return (unsigned)(want < 1 ? 1 : want < cap ? want : cap); };
  if (nseg <= 0) {
    sort_gaps_kernel<T, U, ARG><<<grid((length + kSortBlock - 1) / kSortBlock), kSortBlock, 0, s>>>(
        toptr, x, length, offsets, nseg < 0 ? -1 : nseg);
    return cudaGetLastError();
  }
  SortLists ls;
  ls.mid_slots = length > kShortMax ? length / kListStep + 2 : 0;
  ls.long_cap = length / (kMidMax + 1) + 1 < nseg ? length / (kMidMax + 1) + 1 : nseg;
  void* scratch = nullptr;
  cudaError_t e = scratch_alloc(
      &scratch, sizeof(long long) * (size_t)(kCntWords + 2 * ls.mid_slots + 3 * ls.long_cap), s);
  if (e != cudaSuccess) return e;
  ls.counters = static_cast<unsigned long long*>(scratch);
  ls.mid_st = reinterpret_cast<long long*>(ls.counters + kCntWords);
  ls.mid_len = ls.mid_st + ls.mid_slots;
  ls.long_st = ls.mid_len + ls.mid_slots;
  ls.long_len = ls.long_st + ls.long_cap;
  ls.long_base = ls.long_len + ls.long_cap;
  e = cudaMemsetAsync(scratch, 0xff, sizeof(long long) * (size_t)(kCntWords + ls.mid_slots), s);
  if (e == cudaSuccess) {
    const long long tiles = (nseg + kSortBlock - 1) / kSortBlock;  // 32 segments a warp
    const long long most = (long long)device_sm_count() * kSmallBlocks;
    sort_small_kernel<T, U, ARG><<<(unsigned)(tiles < most ? tiles : most), kSortBlock, 0, s>>>(
        toptr, x, length, offsets, nseg, ascending, ls);
    e = cudaGetLastError();
  }
  Readback rb;
  if (e == cudaSuccess && length > kMidMax) {
    e = rb.queue(ls.counters, kCntWords, s);
    if (e == cudaSuccess) e = rb.mark(s);
  }
  if (e == cudaSuccess && length > kShortMax) {
    const long long tiles = (length + kMidWindow - 1) / kMidWindow;
    const long long most = (long long)device_sm_count() * 8;
    sort_mid_kernel<T, ARG><<<(unsigned)(tiles < most ? tiles : most), kSortBlock, sizeof(MidTile), s>>>(
        toptr, x, ascending, ls);
    e = cudaGetLastError();
  }
  if (rb.used()) {  // (whatever failed since: the buffer goes back when its copy is done)
    const cudaError_t w = rb.wait();
    if (e == cudaSuccess) e = w;
    const unsigned long long* words = rb.words();
    const long long found = (long long)((words[kCntLong] + 1ull) & ((1ull << kLongBits) - 1ull));
    const long long nlong = found < ls.long_cap ? found : ls.long_cap;
    const long long total = (long long)(words[kCntLongTotal] + 1ull);
    const long long merged = (long long)((words[kCntLong] + 1ull) >> kLongBits) * 16;
    const long long maxl = (long long)words[kCntLongMax];
    if (e == cudaSuccess && nlong > 0) {
      // a pair's index is 32 bits unless a segment needs more
      if (maxl <= (1ll << 32))
        e = sort_long<T, ARG, unsigned long long>(toptr, x, ls, nlong, total, merged, maxl, ascending,
                                                  inv, err, s);
      else
        e = sort_long<T, ARG, WidePair>(toptr, x, ls, nlong, total, merged, maxl, ascending, inv,
                                        err, s);
    }
  }
  cudaError_t f = scratch_free(scratch, s);
  return e != cudaSuccess ? e : f;
}

}  // namespace

#define GB_ARGSORT(SUF, T, USUF, U)                                                            \
  GB_EXPORT int awkward_argsort_##SUF##_##USUF(int64_t* toptr, const T* fromptr, int64_t length, \
                                               const U* offsets, int64_t offsetslength,       \
                                               bool ascending, bool stable,                   \
                                               uint64_t invocation_index, uint64_t* err_code, \
                                               void* stream) {                                \
    (void)stable;                                                                             \
    return (int)launch_sort<T, U, true>(toptr, fromptr, length, offsets, offsetslength,        \
                                        ascending, invocation_index, err_code,                \
                                        (cudaStream_t)stream);                                \
  }
#define GB_ARGSORT_ALL(SUF, T)                                                                 \
  GB_ARGSORT(SUF, T, int32, int32_t)                                                           \
  GB_ARGSORT(SUF, T, uint32, uint32_t)                                                         \
  GB_ARGSORT(SUF, T, uint64, uint64_t)                                                         \
  GB_ARGSORT(SUF, T, int64, int64_t)
#define GB_SORT(SUF, T)                                                                        \
  GB_EXPORT int awkward_sort_##SUF(T* toptr, const T* fromptr, int64_t length,                 \
                                   const int64_t* offsets, int64_t offsetslength,             \
                                   bool ascending, bool stable, uint64_t invocation_index,    \
                                   uint64_t* err_code, void* stream) {                        \
    (void)stable;                                                                             \
    return (int)launch_sort<T, int64_t, false>(toptr, fromptr, length, offsets, offsetslength, \
                                               ascending, invocation_index, err_code,         \
                                               (cudaStream_t)stream);                         \
  }
