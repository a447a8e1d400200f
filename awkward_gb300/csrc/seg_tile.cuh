// seg_tile.cuh -- the range walk of the segmented reducers over 4- and 8-byte
// elements (sum, max, min, argmax, argmin).
//
// A warp takes its range's lists in rounds: as many of the next 32 lists as
// hold at most kSpan elements (288 of 8 bytes, 544 of 4) together.  The round's
// elements are one span of the content; it is copied to shared memory with
// asynchronous 16-byte copies while the round before is reduced, so an element
// passes L1 once and global loads are whole lines.  Then, by the round's lists:
//   all of at most 16    a lane per list (lane_results);
//   up to a mean of 96   element-parallel (round_results): lane l reduces the K
//                        consecutive elements from l * K on -- K odd, so that
//                        the lanes' reads never meet in a bank -- and where a
//                        list ends, a bit in a bitmap of the span, the running
//                        result is put away; what a lane has left after its
//                        last end is joined to the first result of a later lane
//                        by shuffles.  Every lane has the same work whatever
//                        the lengths;
//   longer               the warp on one list after the other, or on a few at once
//                        (warp_results).
// Lane i then holds the result of list i of the round (coalesced stores).  A
// list longer than kSpan is reduced by the whole warp from global memory, and so,
// four lists at a time, is a range of lists of 96 to kSpan elements of which a round
// would hold few (direct_results).
//
// The walk before had a lane per list reading from global memory: about 16 cache
// lines a load, and as many steps as the warp's longest list.  Bound now by the
// ALU (75-80 %), the earlier one by load latency.  10M lists of Poisson(8),
// float64: max 174 -> 148 us, argmax 177 -> 153, sum 240 -> 223 (and the sum is
// exact now).  16M elements in lists of mean 35: sum 95 -> 60 us, max 86 -> 42;
// heavy-tailed lists of mean 60: max 128 -> 55.  The sum of lists of 100 to 288
// doubles is the exception (mean 100 62 -> 70 us, 220 57 -> 65).  The lines: with the
// lanes up to 24 elements the sum at mean 16 (24M elements) took 91 us, with 16
// 83; with 8, lists of mean 5 took up to 40 % longer.  Element-parallel at a
// mean of 100 the sum took 117 us (16M elements), the warp on each list 74.
//
// Included by reduce_ops.cuh, between the reducers and their launcher.
#pragma once

namespace gb {

// Elements of a round, at most (9 or 17 per lane: 2.2 KB).
template <class T>
constexpr int kSpan = sizeof(T) == 8 ? 288 : 544;
constexpr int kLaneList = 16;  // longest list of a round reduced by a lane per list
constexpr int kWarpList = 96;  // mean length from which the warp takes lists one by one

// ---------------------------------------------------------------- element operations
// Extrema compare signed integer keys: integers themselves (unsigned ones with
// the top bit flipped), floating point the raw key of f64_raw_key, whose
// winner is exact unless it is a zero or a NaN; ~key for a minimum.
template <class T>
using tile_key_t = typename std::conditional<sizeof(T) == 4, int, long long>::type;

template <class T, bool MAX>
__device__ __forceinline__ tile_key_t<T> tile_key(T v) {
  tile_key_t<T> k;
  if constexpr (std::is_same<T, double>::value) {
    const int h = __double2hiint(v), s = h >> 31;
    const unsigned hi = (unsigned)h ^ ((unsigned)s >> 1), lo = (unsigned)__double2loint(v) ^ (unsigned)s;
    k = (long long)((unsigned long long)hi << 32 | lo);
  } else if constexpr (std::is_same<T, float>::value) {
    const int b = __float_as_int(v);
    k = b ^ (int)((unsigned)(b >> 31) >> 1);
  } else if constexpr (std::is_signed<T>::value) {
    k = (tile_key_t<T>)v;
  } else {
    k = (tile_key_t<T>)(v ^ (T(1) << (8 * sizeof(T) - 1)));
  }
  return MAX ? k : ~k;
}
// The value of a key (every key is a bijection of the value's bits).
template <class T, bool MAX>
__device__ __forceinline__ T tile_value(tile_key_t<T> k) {
  if (!MAX) k = ~k;
  if constexpr (std::is_same<T, double>::value) return __longlong_as_double(f64_raw_key(k));
  else if constexpr (std::is_same<T, float>::value) return __int_as_float(k ^ (int)((unsigned)(k >> 31) >> 1));
  else if constexpr (std::is_signed<T>::value) return (T)k;
  else return (T)k ^ (T(1) << (8 * sizeof(T) - 1));
}
// Neither a zero nor a NaN (every integer is exact).
template <class T>
__device__ __forceinline__ bool winner_exact(T v) {
  if constexpr (std::is_same<T, double>::value) {
    return raw_winner_exact(__double_as_longlong(v));
  } else if constexpr (std::is_same<T, float>::value) {
    return (unsigned)((__float_as_int(v) & 0x7fffffff) - 1) < 0x7f800000u;
  } else {
    return true;
  }
}

// How a reducer is walked: not at all here (Walk::kNone), as an extremum, a
// plain running sum, or the exact sum of doubles.
enum class Walk { kNone, kExtremum, kArg, kPlainSum, kExactSum };
template <class T>
constexpr bool tile_type() {
  return std::is_same<T, double>::value || std::is_same<T, float>::value ||
         (std::is_integral<T>::value && sizeof(T) >= 4);
}
template <class Op>
struct WalkOf {
  static constexpr Walk value = Walk::kNone;
};
template <class T, bool MAX>
struct WalkOf<ExtremumOp<T, MAX>> {
  static constexpr Walk value = tile_type<T>() ? Walk::kExtremum : Walk::kNone;
  static constexpr bool kMax = MAX;
};
template <class T, bool MAX>
struct WalkOf<ArgExtremumOp<T, MAX>> {
  static constexpr Walk value = tile_type<T>() ? Walk::kArg : Walk::kNone;
  static constexpr bool kMax = MAX;
};
template <class OUT, class IN>
struct WalkOf<SumOp<OUT, IN>> {
  static constexpr Walk value =
      tile_type<IN>() && tile_type<OUT>() && sizeof(OUT) == sizeof(IN) && !std::is_same<OUT, double>::value
          ? Walk::kPlainSum
          : Walk::kNone;
};
template <>
struct WalkOf<FixedSumOp<double>> {
  static constexpr Walk value = Walk::kExactSum;
};

// ---------------------------------------------------------------- exact sums
// A double of exponent field e is m * 2^(e - 1075), m its 53-bit significand:
// with w = e - low in 0..24, m * 2^w is added as its upper 27 and lower 26 bits
// times +-2^w to two 64-bit integers (one wide multiply-add each; 4096 addends
// stay below 2^63), so no bit is lost, and the sum is rounded once.  Running
// sums are subtracted at the lists' ends: integers lose nothing.  Exact results
// do not depend on `low`, on the lanes or on the range split.  A round with an
// element outside the window takes the window below its own largest element,
// and if that does not hold it (more than 24 binades, subnormals, infinities,
// NaN) each list is summed by its lane: in its own window if that holds the
// list, else by the general accumulator.
struct Wide {
  long long hi, lo;  // hi * 2^26 + lo
};
__device__ __forceinline__ Wide operator+(Wide a, Wide b) { return {a.hi + b.hi, a.lo + b.lo}; }
__device__ __forceinline__ Wide operator-(Wide a, Wide b) { return {a.hi - b.hi, a.lo - b.lo}; }
constexpr unsigned kWindow = 24;

// Add one double; one that is not 0 and outside the window sets bits of `bad`
// (what it adds then is not defined).
__device__ __forceinline__ void wide_add(Wide& a, double v, unsigned low, unsigned& bad) {
  const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v);
  asm("{\n\t.reg .pred out;\n\t.reg .b32 u, w, f, h, l;\n\t"
      "add.u32 u, %3, %3;\n\t"
      "shr.u32 w, u, 21;\n\t"
      "sub.u32 w, w, %5;\n\t"
      "shr.s32 f, %3, 31;\n\t"
      "or.b32 f, f, 1;\n\t"
      "shl.b32 f, f, w;\n\t"  // 0 for w > 31, and so for a zero
      "shf.l.wrap.b32 h, %4, %3, 6;\n\t"
      "lop3.b32 h, h, 0x3ffffff, 0x4000000, 0xea;\n\t"  // h & a | b
      "and.b32 l, %4, 0x3ffffff;\n\t"
      "mad.wide.s32 %0, h, f, %0;\n\t"
      "mad.wide.s32 %1, l, f, %1;\n\t"
      "setp.gt.u32 out, w, %6;\n\t"
      "@out lop3.b32 %2, %2, u, %4, 0xfe;\n\t}"  // all three or'ed
      : "+l"(a.hi), "+l"(a.lo), "+r"(bad)
      : "r"(hi), "r"(lo), "r"(low), "n"(kWindow));
}
// Windows for which every sum is a normal double or 0: a round's, and the
// larger range of a list's own (so a list has the same result by either).
constexpr unsigned kRoundLow = 100, kRoundHigh = 1970;
constexpr unsigned kListLow = 64, kListHigh = 2000;

// a * 2^(low - 1075), rounded to nearest-even.
__device__ __forceinline__ double wide_value(Wide a, unsigned low) {
  // both parts exact as doubles (nearly always): one rounding in the
  // multiply-add, and the scale added to the exponent
  if ((unsigned long long)(a.hi + (1ll << 53)) <= 1ull << 54 &&
      (unsigned long long)(a.lo + (1ll << 53)) <= 1ull << 54) {
    const double d = __fma_rn(__ll2double_rn(a.hi), 67108864.0, __ll2double_rn(a.lo));
    const long long b = __double_as_longlong(d);
    return __longlong_as_double((b << 1) == 0 ? 0ll : b + ((long long)((int)low - 1075) << 52));
  }
  // hi * 2^26 + lo as a 96-bit integer h * 2^32 + l
  const long long part = a.lo + ((a.hi & 63) << 26);
  long long h = (a.hi >> 6) + (part >> 32);
  unsigned l = (unsigned)part;
  const bool neg = h < 0;
  if (neg) {
    h = ~h + (l == 0u);
    l = 0u - l;
  }
  unsigned long long m = l;
  int e = (int)low - 1075;
  if (h) {
    const int z = __clzll(h);
    const unsigned long long t = (unsigned long long)l << 32;  // the 32 bits below h
    m = z ? ((unsigned long long)h << z) | (t >> (64 - z)) : (unsigned long long)h;
    if (t << z) m |= 1ull;  // (far below the rounding position)
    e += 32 - z;
  }
  if (m == 0) return 0.0;
  const long long b = __double_as_longlong(__ull2double_rn(m)) + ((long long)e << 52);
  return __longlong_as_double(b | (neg ? (long long)0x8000000000000000ull : 0ll));
}

// One list of staged doubles by its lane.
__device__ __forceinline__ double lane_sum(const double* p, int n) {
  unsigned top = 0, bottom = 0xffffffffu;
  for (int i = 0; i < n; i++) {
    const unsigned hi = (unsigned)__double2hiint(p[i]), lo = (unsigned)__double2loint(p[i]);
    const unsigned e = (hi + hi) >> 21;
    if ((hi + hi) | lo) {
      top = e > top ? e : top;
      bottom = e < bottom ? e : bottom;
    }
  }
  if (bottom == 0xffffffffu) return 0.0;  // no element but zeros
  if (bottom >= kListLow && top <= kListHigh && top - bottom <= kWindow) {
    Wide a{0, 0};
    unsigned bad = 0;
    for (int i = 0; i < n; i++) wide_add(a, p[i], bottom, bad);
    return wide_value(a, bottom);
  }
  FxAcc a{0, 1, 0, 0.0};
  for (int i = 0; i < n; i++) a = fx_add_f64(a, p[i]);
  return fx_finalize(a);
}

// ---------------------------------------------------------------- a round
// Shared memory of one warp.
template <class Op>
struct alignas(16) TileSpan {
  using T = store_t<typename Op::In>;
  static constexpr Walk W = WalkOf<Op>::value;
  static constexpr int kVec = 16 / (int)sizeof(T);
  T buf[2][kSpan<T> + kVec];        // spans, from their 16-byte line on
  unsigned bits[kSpan<T> / 32 + 2];    // bit p: a list ends after element p
  unsigned char first[32];          // sums: rank of the first list that ends in a lane
  union {
    Wide sums[W == Walk::kExactSum ? 32 : 1];            // by rank
    unsigned short at[W == Walk::kArg ? kSpan<T> : 1];      // winner of the list that ends here
  } r;
};

// Copy elements x[0 .. n) to dst, x[0] at dst[shift], where shift is x's place
// in its 16-byte line (whole warp; completed by the copy group).
template <class T>
__device__ __forceinline__ int span_copy(T* dst, const T* x, int n, int lane) {
  constexpr int kVec = 16 / (int)sizeof(T);
  const int shift = (int)((reinterpret_cast<uintptr_t>(x) & 15) / sizeof(T));
  int head = (kVec - shift) & (kVec - 1);  // elements before the first whole line
  if (head > n) head = n;
  const int lines = (n - head) / kVec, rest = n - head - lines * kVec;
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst + shift);
  const T* src = x + head + kVec * lane;
  const unsigned to = d + (unsigned)(head * sizeof(T)) + 16u * lane;
#pragma unroll
  for (int i = 0; i < (kSpan<T> / kVec + 31) / 32; i++)
    if (lane + 32 * i < lines)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(to + 512u * i), "l"(src + 32 * kVec * i)
                   : "memory");
  if (lane < head)
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d + (unsigned)(lane * sizeof(T))),
                 "l"(x + lane), "n"(sizeof(T))
                 : "memory");
  const int tail = n - rest + lane;
  if (lane < rest)
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d + (unsigned)(tail * sizeof(T))),
                 "l"(x + tail), "n"(sizeof(T))
                 : "memory");
  return shift;
}

// Stores of a lane for which `yes` is not 0 (predicated, where the compiler would branch
// around each).
__device__ __forceinline__ void store_if(unsigned yes, unsigned at, unsigned v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.b32 [%1], %2;\n\t}" ::"r"(yes),
               "r"(at), "r"(v)
               : "memory");
}
__device__ __forceinline__ void store_if(unsigned yes, unsigned at, unsigned short v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.b16 [%1], %2;\n\t}" ::"r"(yes),
               "r"(at), "h"(v)
               : "memory");
}
__device__ __forceinline__ void store_if(unsigned yes, unsigned at, unsigned long long v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %0, 0;\n\t@p st.shared.b64 [%1], %2;\n\t}" ::"r"(yes),
               "r"(at), "l"(v)
               : "memory");
}
__device__ __forceinline__ void push_if(unsigned yes, unsigned& at, Wide v) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\t@p st.shared.v2.b64 [%0], {%2, %3};\n\t"
               "@p add.u32 %0, %0, 16;\n\t}"
               : "+r"(at)
               : "r"(yes), "l"(v.hi), "l"(v.lo));
}
template <class V>
__device__ __forceinline__ auto word_of(V v) {
  if constexpr (sizeof(V) == 8) {
    unsigned long long w;
    memcpy(&w, &v, 8);
    return w;
  } else {
    unsigned w;
    memcpy(&w, &v, 4);
    return w;
  }
}

// What a warp keeps from round to round: the sums' window, or the key of an
// extremum's identity (nothing beats a NaN identity).
template <class Op>
struct WalkState {
  // 2^-16 to 2^9 to begin with (never so low that a zero's exponent is in it)
  unsigned low = 1023 - 16;
};
template <class T, bool MAX>
struct WalkState<ExtremumOp<T, MAX>> {
  tile_key_t<T> ident;
  const T* x;
};

template <class T, bool MAX>
__device__ __forceinline__ tile_key_t<T> ident_key(const ExtremumOp<T, MAX>& op) {
  using Key = tile_key_t<T>;
  return is_nan(op.ident) ? (Key)~((Key)1 << (8 * sizeof(Key) - 1)) : tile_key<T, MAX>(op.ident);
}

// The window below the largest element `top` of a round (hi words doubled, all
// lanes'), one binade to spare; false when there is none.
__device__ __forceinline__ bool move_window(unsigned& low, unsigned top) {
  top = (__reduce_max_sync(0xffffffffu, top) >> 21) + 1u;
  if (top < kRoundLow + kWindow || top > kRoundHigh) return false;
  low = top - kWindow;
  return true;
}

// The results of a round whose longest list has `longest` elements, a lane per
// list: `p` is the span in shared memory, the lane's list its n elements from a
// on.
template <class Op>
__device__ __forceinline__ typename Op::Out lane_results(const Op& op,
                                                         const store_t<typename Op::In>* p, int n,
                                                         int longest, int a, WalkState<Op>& state,
                                                         bool& done) {
  using T = store_t<typename Op::In>;
  constexpr Walk W = WalkOf<Op>::value;
  const T* q = p + a;
  if constexpr (W == Walk::kExactSum) {
    for (int attempt = 0;; attempt++) {
      Wide w{0, 0};
      unsigned bad = 0;
      for (int i = 0; i < longest; i += 4) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
          double v = 0.0;
          if (i + u < n) v = q[i + u];
          wide_add(w, v, state.low, bad);
        }
      }
      done = !__any_sync(0xffffffffu, bad != 0u);
      if (done) return wide_value(w, state.low);
      unsigned top = 0;
      for (int i = 0; i < n; i++) {
        const unsigned u = 2u * (unsigned)__double2hiint(q[i]);
        top = u > top ? u : top;
      }
      if (attempt == 1 || !move_window(state.low, top)) return 0.0;
    }
  } else if constexpr (W == Walk::kPlainSum) {
    using V = typename Op::Out;
    V acc = V(0);
    for (int i = 0; i < longest; i += 4) {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        V v = V(0);
        if (i + u < n) v = static_cast<V>(q[i + u]);
        acc = acc + v;
      }
    }
    return acc;
  } else {
    constexpr bool MAX = WalkOf<Op>::kMax;
    using Key = tile_key_t<T>;
    // (past its end a lane reads its last element again, which beats nothing)
    const int last = n > 0 ? n - 1 : 0;
    Key best = tile_key<T, MAX>(q[0]);
    int at = 0;
    for (int i = 1; i < longest; i += 4) {
#pragma unroll
      for (int u = 0; u < 4; u++) {
        const int j = i + u < last ? i + u : last;
        const Key k = tile_key<T, MAX>(q[j]);
        const bool take = k > best;
        best = take ? k : best;
        if (W == Walk::kArg) at = take ? j : at;
      }
    }
    const T v = tile_value<T, MAX>(best);
    bool exact = n <= 0 || winner_exact(v);
    if constexpr (W == Walk::kArg) {
      if (std::is_floating_point<T>::value) exact = exact && !(n > 0 && is_nan(q[0]));
      if (exact) return n > 0 ? a + at : -1;
    } else {
      if (exact) return n > 0 && best > state.ident ? v : op.ident;
    }
    typename Op::Acc acc = op.identity();  // a zero or a NaN won: the exact rules
    for (int i = 0; i < n; i++) acc = op.step(acc, q[i], a + i, i == 0, 0);
    return op.finalize(acc, 0);
  }
}

// The results of a round of a few long lists, the whole warp on one after the
// other: `p` is the span in shared memory, the lane's list its n elements from a
// on, `lists` of them.
template <class Op>
__device__ __forceinline__ typename Op::Out warp_each_results(const Op& op,
                                                         const store_t<typename Op::In>* p, int lists,
                                                         int n, int a, int lane, WalkState<Op>& state,
                                                         bool& done) {
  using T = store_t<typename Op::In>;
  constexpr Walk W = WalkOf<Op>::value;
  constexpr unsigned kFull = 0xffffffffu;
  typename Op::Out mine{};
  for (int l = 0; l < lists; l++) {
    const T* q = p + __shfl_sync(kFull, a, l);
    const int m = __shfl_sync(kFull, n, l);
    typename Op::Out v;
    if constexpr (W == Walk::kExactSum) {
      for (int attempt = 0;; attempt++) {
        Wide w{0, 0};
        unsigned bad = 0;
#pragma unroll 3
        for (int i = lane; i < m; i += 32) wide_add(w, q[i], state.low, bad);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
          w = w + Wide{__shfl_xor_sync(kFull, w.hi, d), __shfl_xor_sync(kFull, w.lo, d)};
        v = wide_value(w, state.low);
        if (!__any_sync(kFull, bad != 0u)) break;
        unsigned top = 0;
        for (int i = lane; i < m; i += 32) {
          const unsigned u = 2u * (unsigned)__double2hiint(q[i]);
          top = u > top ? u : top;
        }
        if (attempt == 1 || !move_window(state.low, top)) {
          done = false;
          break;
        }
      }
      if (!done) return mine;
    } else if constexpr (W == Walk::kPlainSum) {
      using V = typename Op::Out;
      V acc = V(0);
      for (int i = lane; i < m; i += 32) acc = acc + static_cast<V>(q[i]);
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) acc = acc + __shfl_xor_sync(kFull, acc, d);
      v = acc;
    } else {
      constexpr bool MAX = WalkOf<Op>::kMax;
      using Key = tile_key_t<T>;
      // (m > 0, and a lane past the end takes the last element)
      int at = lane < m ? lane : m - 1;
      Key best = tile_key<T, MAX>(q[at]);
      for (int i = lane + 32; i < m; i += 32) {
        const Key k = tile_key<T, MAX>(q[i]);
        if (k > best) {
          best = k;
          at = i;
        }
      }
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) {
        const Key o = __shfl_xor_sync(kFull, best, d);
        const int oa = __shfl_xor_sync(kFull, at, d);
        if (o > best || (o == best && oa < at)) {
          best = o;
          at = oa;
        }
      }
      const T x = tile_value<T, MAX>(best);
      bool exact = winner_exact(x);
      if constexpr (W == Walk::kArg) {
        if (std::is_floating_point<T>::value) exact = exact && !is_nan(q[0]);
        v = (int)(q - p) + at;
      } else {
        v = best > state.ident ? x : op.ident;
      }
      if (!exact) {  // a zero or a NaN won: the exact rules
        typename Op::Acc acc = op.identity();
        for (int i = lane; i < m; i += 32) acc = op.step(acc, q[i], (int)(q - p) + i, i == 0, 0);
        v = op.finalize(warp_allreduce(op, acc), 0);
      }
    }
    if (lane == l) mine = v;
  }
  return mine;
}

// The same for the extrema of 4-byte elements: two or four lists at once, with 16 or 8
// lanes on each (float32 lists of mean 100 to 220, 16M elements: max 34-42 -> 30-34 us;
// the others' kernels have no registers left for it).
template <class Op>
__device__ __forceinline__ typename Op::Out group_results(const Op& op,
                                                          const store_t<typename Op::In>* p, int lists,
                                                          int n, int a, int lane,
                                                          const WalkState<Op>& state) {
  using T = store_t<typename Op::In>;
  constexpr unsigned kFull = 0xffffffffu;
  typename Op::Out mine{};
  constexpr bool MAX = WalkOf<Op>::kMax;
  using Key = tile_key_t<T>;
  const int lanes = lists > 2 ? 8 : lists > 1 ? 16 : 32;
  const int group = lane / lanes, sub = lane & (lanes - 1);
  for (int l = 0; l < lists; l += 32 / lanes) {
    const int few = lists - l < 32 / lanes ? lists - l : 32 / lanes;
    const int of = l + (group < few ? group : 0);  // the lane's list
    const int first = __shfl_sync(kFull, a, of);
    const int m = __shfl_sync(kFull, n, of);
    const T* q = p + first;
    // (a lane past the end takes the last element)
    Key best = tile_key<T, MAX>(q[sub < m ? sub : m - 1]);
    for (int i = sub + lanes; i < m; i += lanes) {
      const Key k = tile_key<T, MAX>(q[i]);
      best = k > best ? k : best;
    }
    for (int d = lanes >> 1; d > 0; d >>= 1) {
      const Key o = __shfl_xor_sync(kFull, best, d);
      best = o > best ? o : best;
    }
    const T x = tile_value<T, MAX>(best);
    const bool exact = winner_exact(x);
    typename Op::Out v = best > state.ident ? x : op.ident;
    // a zero or a NaN won: the exact rules, by the whole warp
    for (unsigned rest = __ballot_sync(kFull, !exact); rest;) {
      const int from = __ffs(rest) - 1;
      const int f = __shfl_sync(kFull, first, from), c = __shfl_sync(kFull, m, from);
      typename Op::Acc acc = op.identity();
      for (int i = lane; i < c; i += 32) acc = op.step(acc, p[f + i], f + i, i == 0, 0);
      const typename Op::Out w = op.finalize(warp_allreduce(op, acc), 0);
      if (first == f) v = w;
      rest &= ~__ballot_sync(kFull, first == f);
    }
    const typename Op::Out w = __shfl_sync(kFull, v, (lane - l) * lanes & 31);
    if (lane >= l && lane < l + few) mine = w;
  }
  return mine;
}
template <class Op>
__device__ __forceinline__ typename Op::Out warp_results(const Op& op,
                                                         const store_t<typename Op::In>* p, int lists,
                                                         int n, int a, int lane, WalkState<Op>& state,
                                                         bool& done) {
  if constexpr (WalkOf<Op>::value == Walk::kExtremum && sizeof(store_t<typename Op::In>) == 4)
    return group_results(op, p, lists, n, a, lane, state);
  else
    return warp_each_results(op, p, lists, n, a, lane, state, done);
}

// A range whose lists of 8-byte elements have a mean of kWarpList and more, and none
// of which is longer than a round holds, is taken 32 lists at a time without a copy:
// a round would hold one to three of them.  Four at once, eight lanes on each, straight
// from memory.  16M elements in lists of mean 100, 150 and 220: argmax of doubles 57,
// 57, 47 -> 46, 43, 44 us, max of int64 49, 48, 40 -> 41, 40, 42, argmax 50, 50, 41 ->
// 43, 41, 42.  The sums and the maxima of doubles stay with the rounds: their kernels
// have no registers left, and every length paid for it (max at mean 8 44 -> 53 us; sums
// of lists of 290 to 400 51 -> 62, of mean 100 73 -> 58).
template <class Op>
constexpr bool kDirect =
    sizeof(store_t<typename Op::In>) == 8 &&
    (WalkOf<Op>::value == Walk::kArg ||
     (WalkOf<Op>::value == Walk::kExtremum && std::is_integral<typename Op::In>::value));

// The results of such lists: x is the first one's first element, the lane's list its n
// elements from a on, `lists` of them.
template <class Op>
__device__ __forceinline__ typename Op::Out direct_results(const Op& op,
                                                           const store_t<typename Op::In>* x, int lists,
                                                           int n, int a, int lane,
                                                           const WalkState<Op>& state) {
  using T = store_t<typename Op::In>;
  using Out = typename Op::Out;
  constexpr Walk W = WalkOf<Op>::value;
  constexpr unsigned kFull = 0xffffffffu;
  constexpr int kFlight = 8;
  const int sub = lane & 7;
  tile_key_t<T> top = 0;  // of the lane's list: its winner
  int place = 0;
  for (int l = 0; l < lists; l += 4) {
    const int of = l + (lane >> 3);
    const T* q = x + __shfl_sync(kFull, a, of & 31);
    int m = __shfl_sync(kFull, n, of & 31);
    if (of >= lists) m = 0;
    const int longest = __reduce_max_sync(kFull, m);
    const int from = (lane - l) * 8 & 31;  // the lane with its list's result, if it is one of the four
    const bool mine = lane >= l && lane < l + 4;
    constexpr bool MAX = WalkOf<Op>::kMax;
    using Key = tile_key_t<T>;
    constexpr Key kLowest = (Key)((unsigned long long)1 << (8 * sizeof(Key) - 1));
    Key best = kLowest;
    int at = 0x7fffffff;  // (none)
    for (int i = sub; i < longest; i += 8 * kFlight) {
      T v[kFlight];
#pragma unroll
      for (int u = 0; u < kFlight; u++) v[u] = i + 8 * u < m ? __ldg(q + i + 8 * u) : T(0);
#pragma unroll
      for (int u = 0; u < kFlight; u++) {
        const Key k = tile_key<T, MAX>(v[u]);
        const bool take = i + 8 * u < m && (k > best || at == 0x7fffffff);
        best = take ? k : best;
        at = take ? i + 8 * u : at;
      }
    }
#pragma unroll
    for (int d = 4; d > 0; d >>= 1) {
      const Key o = __shfl_xor_sync(kFull, best, d);
      const int oa = __shfl_xor_sync(kFull, at, d);
      if (o > best || (o == best && oa < at)) {
        best = o;
        at = oa;
      }
    }
    best = __shfl_sync(kFull, best, from);
    at = __shfl_sync(kFull, at, from);
    if (mine) {
      top = best;
      place = at;
    }
  }
  const T winner = tile_value<T, WalkOf<Op>::kMax>(top);
  bool exact = n <= 0 || winner_exact(winner);
  Out v;
  if constexpr (W == Walk::kArg) {
    if (std::is_floating_point<T>::value) exact = exact && !(n > 0 && is_nan(__ldg(x + a)));
    v = n > 0 ? a + place : -1;
  } else {
    v = n > 0 && top > state.ident ? winner : op.ident;
  }
  // a zero or a NaN won: the exact rules, by the whole warp
  for (unsigned rest = __ballot_sync(kFull, !exact); rest; rest &= rest - 1) {
    const int of = __ffs(rest) - 1;
    const int first = __shfl_sync(kFull, a, of), m = __shfl_sync(kFull, n, of);
    typename Op::Acc acc = op.identity();
    for (int i = lane; i < m; i += 32) acc = op.step(acc, __ldg(x + first + i), first + i, i == 0, 0);
    const Out w = op.finalize(warp_allreduce(op, acc), 0);
    if (lane == of) v = w;
  }
  return v;
}

// The results of a round's lists, element-parallel: `p` is the span in shared
// memory, n its elements, [a, b) the lane's list in it (a == b without one),
// `begin` its place in the range.  K elements per lane, 32 * K >= n.
template <int K, class Op>
__device__ __forceinline__ typename Op::Out round_results(const Op& op, TileSpan<Op>& s,
                                                          store_t<typename Op::In>* p, int n,
                                                          int a, int b, int begin, int lane,
                                                          WalkState<Op>& state,
                                                          bool& done) {
  using T = store_t<typename Op::In>;
  constexpr Walk W = WalkOf<Op>::value;
  constexpr unsigned kFull = 0xffffffffu;
  const unsigned lt = (1u << lane) - 1u;
  // the ends, and the lane's K of them; the lane of the span's end reads zeros past it
  static_assert(K <= 32);
  if (lane <= K) s.bits[lane] = 0u;
  if constexpr (W == Walk::kExactSum)
    if (n + lane < 32 * K) p[n + lane] = 0.0;
  __syncwarp();
  const bool some = b > a;
  if (some) atomicOr(s.bits + ((b - 1) >> 5), 1u << ((b - 1) & 31));
  int rank = 0, owner = 0;
  if constexpr (W == Walk::kExactSum) {
    rank = __popc(__ballot_sync(kFull, some) & (lt | (1u << lane))) - 1;
    owner = b > 0 ? (int)((unsigned)(b - 1) / (unsigned)K) : -1;  // the lane of the list's end
    const int prev = __shfl_up_sync(kFull, owner, 1);
    if (some && (lane == 0 || owner != prev)) s.first[owner] = (unsigned char)rank;
  }
  __syncwarp();
  const int q0 = lane * K;
  const unsigned ends =
      __funnelshift_r(s.bits[q0 >> 5], s.bits[(q0 >> 5) + 1], q0 & 31) & ((1u << K) - 1u);
  T* q = p + q0;
  T e[K];  // (loaded before any result is stored among them)
  if constexpr (W != Walk::kExactSum) {
#pragma unroll
    for (int k = 0; k < K; k++) e[k] = q[k];
  }

  if constexpr (W == Walk::kExactSum) {
    Wide w;
    unsigned bad;
    const int r0 = s.first[lane];
    for (int attempt = 0;; attempt++) {
      bad = 0;
      w = Wide{0, 0};
      unsigned r = (unsigned)__cvta_generic_to_shared(s.r.sums + r0);
      if (q0 < n) {
#pragma unroll
        for (int k = 0; k < K; k++) {
          wide_add(w, q[k], state.low, bad);
          push_if(ends & 1u << k, r, w);
        }
      }
      if (!__any_sync(kFull, bad != 0u) || attempt == 1) break;
      unsigned top = 0;  // the window below this round's largest element, one binade to spare
      if (q0 < n) {
#pragma unroll
        for (int k = 0; k < K; k++) {
          const unsigned u = 2u * (unsigned)__double2hiint(q[k]);
          top = u > top ? u : top;
        }
      }
      if (!move_window(state.low, top)) break;
    }
    done = !__any_sync(kFull, bad != 0u);
    if (!done) return 0.0;
    Wide before = w;  // all the elements of the lanes up to this one
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const Wide o{__shfl_up_sync(kFull, before.hi, d), __shfl_up_sync(kFull, before.lo, d)};
      if (lane >= d) before = before + o;
    }
    before = before - w;
    __syncwarp();
    // the running sum at the list's end and at its beginning
    const int from = owner < 0 ? 0 : owner;
    Wide end{__shfl_sync(kFull, before.hi, from), __shfl_sync(kFull, before.lo, from)};
    end = rank < 0 ? Wide{0, 0} : end + s.r.sums[rank];
    Wide begin{__shfl_up_sync(kFull, end.hi, 1), __shfl_up_sync(kFull, end.lo, 1)};
    if (lane == 0) begin = Wide{0, 0};
    return wide_value(end - begin, state.low);
  } else {
    // Where a list ends, its result (an extremum's key) takes the place of its
    // last element; an arg-result, the winner's element, goes to r.at and the
    // elements stay.
    const unsigned qa = (unsigned)__cvta_generic_to_shared(q);
    const int back = [&] {  // lanes back to the nearest one below with an end
      const unsigned prev = ~__ballot_sync(kFull, ends == 0u) & lt;
      return prev ? lane - (31 - __clz(prev)) : lane;
    }();
    const int steps = __reduce_max_sync(kFull, ends ? back : 0);
    const int e0 = __ffs(ends) - 1;  // the first end
    if constexpr (W == Walk::kPlainSum) {
      using V = typename Op::Out;
      static_assert(sizeof(V) == sizeof(T), "results fit the elements' places");
      // In a long chain a float keeps its roundings' errors beside the sum, and
      // the lane's part is rounded once (the multiply-add units are idle here;
      // a mean of 35 elements lost more than the walk by groups of 8 lanes did).
      constexpr bool kKeep = std::is_floating_point<V>::value && K > 9;
      V acc = V(0), lost = V(0);
#pragma unroll
      for (int k = 0; k < K; k++) {
        const V v = static_cast<V>(e[k]), sum = acc + v;
        V full = sum;
        if constexpr (kKeep) {
          const V got = sum - acc;
          lost = lost + ((acc - (sum - got)) + (v - got));
          // (an infinite or NaN sum has no error to add)
          if (fabsf(sum) <= 3.402823466e38f) full = sum + lost;
          lost = ends & 1u << k ? V(0) : lost;
        }
        store_if(ends & 1u << k, qa + (unsigned)(k * sizeof(V)), word_of(full));
        acc = ends & 1u << k ? V(0) : sum;
      }
      if constexpr (kKeep)
        if (fabsf(acc) <= 3.402823466e38f) acc = acc + lost;
      // what the lanes from the last one with an end on have left over, by
      // doubling steps (few roundings in a row)
      const int reach = ends ? 0 : back;
      for (int d = 1; d <= steps; d <<= 1) {
        const V o = __shfl_up_sync(kFull, acc, d);
        if (d <= reach) acc = o + acc;
      }
      const V carry = __shfl_up_sync(kFull, acc, 1);
      if (ends && lane > 0) {
        V* r = reinterpret_cast<V*>(q + e0);
        *r = carry + *r;
      }
      __syncwarp();
      return some ? *reinterpret_cast<const V*>(p + b - 1) : V(0);
    } else {
      constexpr bool MAX = WalkOf<Op>::kMax;
      constexpr bool ARG = W == Walk::kArg;
      using Key = tile_key_t<T>;
      constexpr Key kLowest = (Key)((unsigned long long)1 << (8 * sizeof(Key) - 1));
      Key* qk = reinterpret_cast<Key*>(q);
      const unsigned ra = ARG ? (unsigned)__cvta_generic_to_shared(s.r.at + q0) : 0u;
      Key best = tile_key<T, MAX>(e[0]);
      int at = q0;
#pragma unroll
      for (int k = 0; k < K; k++) {
        if (k > 0) {
          const Key v = tile_key<T, MAX>(e[k]);
          const bool take = (ends & 1u << (k - 1)) != 0 || v > best;
          best = take ? v : best;
          if (ARG) at = take ? q0 + k : at;
        }
        if constexpr (ARG) store_if(ends & 1u << k, ra + 2u * k, (unsigned short)at);
        else store_if(ends & 1u << k, qa + (unsigned)(k * sizeof(T)), word_of(best));
      }
      if (ends >> (K - 1) & 1u) {  // nothing left over
        best = kLowest;
        at = -1;
      }
      Key carry = kLowest;
      int cat = -1;
      const int reach = ends ? 0 : back;
      for (int d = 1; d <= steps; d <<= 1) {  // (the earlier of equals wins)
        const Key o = __shfl_up_sync(kFull, best, d);
        if constexpr (ARG) {
          const int oa = __shfl_up_sync(kFull, at, d);
          if (d <= reach && oa >= 0 && (at < 0 || o >= best)) {
            best = o;
            at = oa;
          }
        } else {
          if (d <= reach && o > best) best = o;
        }
      }
      carry = __shfl_up_sync(kFull, best, 1);
      if constexpr (ARG) cat = __shfl_up_sync(kFull, at, 1);
      if (lane == 0) {
        carry = kLowest;
        cat = -1;
      }
      if constexpr (ARG) {
        if (cat >= 0 && ends && carry >= tile_key<T, MAX>(p[s.r.at[q0 + e0]]))
          s.r.at[q0 + e0] = (unsigned short)cat;
      } else {
        if (ends && carry > qk[e0]) qk[e0] = carry;
      }
      __syncwarp();
      typename Op::Acc acc = op.identity();
      if constexpr (ARG) {
        const int w = some ? s.r.at[b - 1] : 0;
        bool exact = !some || winner_exact(p[w]);
        if (some && std::is_floating_point<T>::value) exact = exact && !is_nan(p[a]);
        if (exact) return some ? w : -1;
        for (int i = a; i < b; i++) acc = op.step(acc, p[i], i, i == a, 0);
      } else {
        const Key best = some ? reinterpret_cast<const Key*>(p)[b - 1] : kLowest;
        const T v = tile_value<T, MAX>(best);
        if (!some || winner_exact(v)) return some && best > state.ident ? v : op.ident;
        // a zero or a NaN won: the exact rules, over the elements in memory
        // (results stand in some of their places here)
        for (int i = a; i < b; i++) acc = op.step(acc, __ldg(state.x + begin + i), i, i == a, 0);
      }
      return op.finalize(acc, 0);
    }
  }
}

// ---------------------------------------------------------------- long runs
// fn(element, its index) for the lane's of the n > 0 elements at x, strided, in
// order; eight loads in flight.
template <class T, class F>
__device__ __forceinline__ void strided(const T* x, int n, int lane, F fn) {
  for (int i = lane; i < n; i += 8 * 32) {
    T v[8];
#pragma unroll
    for (int u = 0; u < 8; u++) v[u] = __ldg(x + (i + 32 * u < n ? i + 32 * u : i));
#pragma unroll
    for (int u = 0; u < 8; u++)
      if (i + 32 * u < n) fn(v[u], i + 32 * u);
  }
}

// Elements [s, e) of list `li` (first element st) by the whole warp, strided.
template <class Op>
__device__ __forceinline__ typename Op::Acc long_run(const Op& op, const store_t<typename Op::In>* x,
                                                     long long s, long long e, long long st,
                                                     long long li) {
  using T = store_t<typename Op::In>;
  constexpr Walk W = WalkOf<Op>::value;
  const int lane = threadIdx.x & 31, n = (int)(e - s);
  if constexpr (W == Walk::kPlainSum) {
    if (e > s && e - s < (1ll << 30)) {
      typename Op::Acc a = op.identity();
      if constexpr (std::is_floating_point<T>::value) {
        // eight elements among themselves first: the rounding errors grow with an
        // eighth of them (20000 floats, relative: 2.7e-7 element by element, 1.3e-7 so)
        for (int i = lane; i < n; i += 8 * 32) {
          T v[8];
#pragma unroll
          for (int u = 0; u < 8; u++) v[u] = i + 32 * u < n ? __ldg(x + s + i + 32 * u) : T(0);
          a += ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        }
      } else {
        strided(x + s, n, lane, [&](T v, int) { a = a + static_cast<typename Op::Out>(v); });
      }
      return warp_allreduce(op, a);
    }
  } else if constexpr ((W == Walk::kExtremum || W == Walk::kArg) && !std::is_same<T, double>::value) {
    constexpr bool MAX = WalkOf<Op>::kMax;
    using Key = tile_key_t<T>;
    if (e > s && e - s < (1ll << 30)) {
      Key best = 0;
      int at = -1;
      strided(x + s, n, lane, [&](T v, int j) {
        const Key k = tile_key<T, MAX>(v);
        if (at < 0 || k > best) {
          best = k;
          at = j;
        }
      });
#pragma unroll
      for (int d = 16; d > 0; d >>= 1) {
        const Key o = __shfl_xor_sync(0xffffffffu, best, d);
        const int oa = __shfl_xor_sync(0xffffffffu, at, d);
        if (oa >= 0 && (at < 0 || o > best || (o == best && oa < at))) {
          best = o;
          at = oa;
        }
      }
      const T v = tile_value<T, MAX>(best);
      bool exact = winner_exact(v);
      if (W == Walk::kArg && st >= s && st < e) exact = exact && !is_nan(__ldg(x + st));
      if (exact) return {v, s + at};
    }
  }
  return run_coop<32>(op, x, s, e, st, li);
}

// The sum of a list of up to kAbsorb doubles, exact when one window holds it
// (its own, as in lane_sum); false otherwise.
__device__ __forceinline__ bool long_sum(const double* x, int n, unsigned& low, double* v) {
  const int lane = threadIdx.x & 31;
  unsigned use = low;
  for (int attempt = 0; attempt < 2; attempt++) {
    Wide w{0, 0};
    unsigned bad = 0;
    strided(x, n, lane, [&](double v, int) { wide_add(w, v, use, bad); });
    if (!__any_sync(0xffffffffu, bad != 0u)) {
#pragma unroll
      for (int d = 16; d > 0; d >>= 1)
        w = w + Wide{__shfl_xor_sync(0xffffffffu, w.hi, d), __shfl_xor_sync(0xffffffffu, w.lo, d)};
      *v = wide_value(w, use);
      return true;
    }
    unsigned top = 0;
    for (int i = lane; i < n; i += 32) {
      const unsigned u = 2u * (unsigned)__double2hiint(__ldg(x + i));
      top = u > top ? u : top;
    }
    move_window(low, top);  // (for the lists that follow)
    top = __reduce_max_sync(0xffffffffu, top) >> 21;
    if (top < kListLow + kWindow || top > kListHigh) return false;
    use = top - kWindow;
  }
  return false;
}

// ---------------------------------------------------------------- a range
// Reduce the lists of merge-path diagonal range [d0, d1) of one array (whole
// warp), as seg_reduce_range does: each list that ends in the range to
// out[list], the partials of the giant lists crossing its ends to `rec`.
template <class Op>
__device__ __forceinline__ void seg_tile_range(const Op& op,
                                               const store_t<typename Op::In>* __restrict__ x,
                                               const int64_t* __restrict__ offsets,
                                               long long nlists, long long e0, long long E,
                                               long long d0, long long d1,
                                               typename Op::Out* __restrict__ out,
                                               RangeRecord<typename Op::Acc>& rec, TileSpan<Op>& s) {
  constexpr unsigned kFull = 0xffffffffu;
  int lane;
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));  // (kept, not read again each round)
  const bool upper = lane >= 16;
  const long long split = mp_search_half(offsets, nlists, e0, E, upper ? d1 : d0,
                                         upper ? 0xffff0000u : 0x0000ffffu);
  const long long I0 = __shfl_sync(kFull, split, 0), I1 = __shfl_sync(kFull, split, 16);
  const long long J0 = e0 + (d0 - I0), J1 = e0 + (d1 - I1);
  long long base = I0, lo = __ldg(offsets + I0);
  // the giant lists crossing the range's ends
  if (I0 < I1 && lo < J0) {
    const long long en = __ldg(offsets + I0 + 1);
    if (en - lo > kAbsorb) {
      const typename Op::Acc a = long_run(op, x, J0, en, lo, I0);
      if (lane == 0) rec.head_acc = a;
      base = I0 + 1;
      lo = en;
    }
  }
  if (I1 < nlists) {
    const long long st = __ldg(offsets + I1), en = __ldg(offsets + I1 + 1);
    if (en - st > kAbsorb) {
      const typename Op::Acc a = long_run(op, x, st < J0 ? J0 : st, J1, st, I1);
      if (lane == 0) rec.tail_acc = a;
    }
  }
  if (lane == 0) seg_range_records(op, offsets, nlists, I0, I1, J0, rec);
  if (base >= I1) return;

  // From here on lists and elements count from the first of the range, in 32
  // bits (a range holds fewer than 2^31 of both; the offsets' low words, unsigned,
  // give the differences).
  using T = store_t<typename Op::In>;
  const T* xr = x + lo;
  const unsigned* ends = reinterpret_cast<const unsigned*>(offsets + base + 1);
  typename Op::Out* to = out + base;
  const int lists = (int)(I1 - base);
  const unsigned first = (unsigned)lo;
  auto load_end = [&](int l) {
    l = l < lists ? l : lists - 1;
    return __ldg(ends + 2 * (long long)l);  // (nothing waits for it here)
  };
  if constexpr (kDirect<Op>) {
    const int n = (int)(__ldg(ends + 2 * (long long)(lists - 1)) - first);
    bool direct = n >= (long long)lists * kWarpList;
    for (int b = 0; b < lists && direct; b += 32) {
      const unsigned en = load_end(b + lane), up = __shfl_up_sync(kFull, en, 1);
      const unsigned st = lane ? up : b ? load_end(b - 1) : first;
      direct = __all_sync(kFull, en - st <= (unsigned)kSpan<T>);
    }
    if (direct) {
      WalkState<Op> state;
      if constexpr (WalkOf<Op>::value == Walk::kExtremum) state.ident = ident_key(op);
      for (int b = 0; b < lists; b += 32) {
        const int c = lists - b < 32 ? lists - b : 32;
        const unsigned en = load_end(b + lane), up = __shfl_up_sync(kFull, en, 1);
        const unsigned st = lane ? up : b ? load_end(b - 1) : first;
        typename Op::Out v = direct_results(op, xr, c, lane < c ? (int)(en - st) : 0, (int)(st - first),
                                            lane, state);
        if constexpr (WalkOf<Op>::value == Walk::kArg) v = v < 0 ? v : v + lo;
        if (lane < c) to[b + lane] = v;
      }
      return;
    }
  }
  // the round from list b, element l on, with the lanes' loaded ends: its
  // lists (0 when the first is too long for one), their ends relative to l,
  // its elements and where it ends
  struct Round {
    int nl, rel, n, hi, shift;
  };
  auto plan = [&](int b, int l, unsigned en, int buf) {
    Round r;
    r.rel = (int)(en - (first + (unsigned)l));
    const unsigned m = __ballot_sync(kFull, (unsigned)r.rel > (unsigned)kSpan<T> || lane >= lists - b);
    r.nl = m ? __ffs(m) - 1 : 32;
    r.n = __shfl_sync(kFull, r.rel, r.nl ? r.nl - 1 : 0);
    r.hi = l + r.n;
    r.shift = 0;
    if (r.nl) r.shift = span_copy(s.buf[buf], xr + l, r.n, lane);
    asm volatile("cp.async.commit_group;" ::: "memory");
    return r;
  };
  WalkState<Op> state;
  if constexpr (WalkOf<Op>::value == Walk::kExtremum) {
    state.ident = ident_key(op);
    state.x = xr;
  }
  // list ends are loaded two rounds ahead, elements copied one ahead
  int at = 0, begin = 0, which = 0;
  Round now = plan(0, 0, load_end(lane), 0);
  int next = now.nl ? now.nl : 1;
  unsigned en = load_end(next + lane);
  while (true) {
    Round ahead{0, 0, 0, 0, 0};
    if (next < lists) {
      ahead = plan(next, now.hi, en, which ^ 1);
      en = load_end(next + (ahead.nl ? ahead.nl : 1) + lane);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_all;" ::: "memory");
    }
    if (now.nl) {
      T* p = s.buf[which] + now.shift;
      const bool act = lane < now.nl;
      const int n = now.n, b = act ? now.rel : n;
      int a = __shfl_up_sync(kFull, b, 1);
      if (lane == 0) a = 0;
      if (a > b) a = b;
      typename Op::Out v;
      bool done = true;  // false: an exact sum needs a window per list
      __syncwarp();
      const int longest = __reduce_max_sync(kFull, b - a);
      if (longest <= kLaneList) v = lane_results(op, p, b - a, longest, a, state, done);
      else if (n >= now.nl * kWarpList &&
               __all_sync(kFull, !act || b > a))
        v = warp_results(op, p, now.nl, b - a, a, lane, state, done);
      else if (n <= 32 * 5) v = round_results<5>(op, s, p, n, a, b, begin, lane, state, done);
      else if (sizeof(T) == 8 || n <= 32 * 9)
        v = round_results<9>(op, s, p, n, a, b, begin, lane, state, done);
      else v = round_results<sizeof(T) == 8 ? 9 : 17>(op, s, p, n, a, b, begin, lane, state, done);
      if constexpr (WalkOf<Op>::value == Walk::kExactSum)
        if (!done) v = lane_sum(p + a, b - a);
      // (arg-results are relative to the round)
      if constexpr (WalkOf<Op>::value == Walk::kArg) v = v < 0 ? v : v + (lo + begin);
      if (act) to[at + lane] = v;
      __syncwarp();
    } else {
      const long long e = lo + (now.hi < begin ? begin : now.hi), li = (I1 - lists) + at;
      bool whole = false;
      if constexpr (WalkOf<Op>::value == Walk::kExactSum) {
        double v;
        if (e - (lo + begin) <= kAbsorb) whole = long_sum(xr + begin, (int)(e - (lo + begin)), state.low, &v);
        if (whole && lane == 0) to[at] = v;
      }
      if (!whole) {
        const typename Op::Acc a = long_run(op, x, lo + begin, e, lo + begin, li);
        if (lane == 0) to[at] = op.finalize(a, li);
      }
    }
    if (next >= lists) break;
    at = next;
    begin = now.hi;
    now = ahead;
    next = at + (now.nl ? now.nl : 1);
    which ^= 1;
  }
}

// The range walk of a reducer: the element-parallel one where it has it.
template <class Op>
constexpr bool kTileWalk = WalkOf<Op>::value != Walk::kNone;
// Resident CTAs of kSegBlock threads per SM (the tile walk: 64 registers, and
// 19 to 42 KB of shared memory).
template <class Op>
constexpr int kWalkBlocks = kTileWalk<Op> ? 4 : kSegMinBlocks;
struct NoSpan {};
template <class Op>
using span_t = typename std::conditional<kTileWalk<Op>, TileSpan<Op>, NoSpan>::type;

template <class Op>
__device__ __forceinline__ void seg_walk(const Op& op, const store_t<typename Op::In>* __restrict__ x,
                                         const int64_t* __restrict__ offsets, long long nlists,
                                         long long e0, long long E, long long d0, long long d1,
                                         typename Op::Out* __restrict__ out,
                                         RangeRecord<typename Op::Acc>& rec, span_t<Op>& span) {
  if constexpr (kTileWalk<Op>) seg_tile_range(op, x, offsets, nlists, e0, E, d0, d1, out, rec, span);
  else seg_reduce_range(op, x, offsets, nlists, e0, E, d0, d1, out, rec);
}

}  // namespace gb
