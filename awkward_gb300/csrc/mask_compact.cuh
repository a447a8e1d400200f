// mask_compact.cuh -- array[mask] by a bitmap of the whole mask, in two streaming
// kernels that do not depend on the lists' lengths; shared by the per-array entry
// point (awkward_gb300_jagged_mask_select_sized) and the batched one:
//
//   mask bits   a CTA turns 32768 mask bytes into bits (two aligned 16-byte loads
//               per 32 bytes, eight in flight), gives each 32-bit word the true
//               entries of the tile before it and writes the tile's total; the
//               CTA that finishes last scans the totals;
//   mask apply  some CTAs copy: a warp takes 1024 elements, and for each of their
//               32 words a lane whose bit is set loads its element and stores it
//               at its rank, 16 words in flight, the next 32 words loaded
//               meanwhile; the others write the new offsets, the rank of each
//               list's end (three look-ups).
//
// mask_select_tile (mask_select.cuh) does it in one kernel, 1024 lists at a time,
// and waits at its barriers for the tile's offsets, mask, counts and look-back in
// turn; a tile whose mask outgrows its bitmap, lists of mean 16 and more, it counts
// with a thread per list.  Bound by HBM: 4M lists, 32M float64 elements, 40 % kept
// (420 MB, 62 us): the bits take 15 us and the rest 74, the one kernel 124; batched
// over ten arrays of 28M elements 15 + 53 and 162 us.
#pragma once

#include "list_tile.cuh"
#include "mask_select.cuh"

namespace gb {

constexpr int kChunk = 1024;                                    // elements a warp copies at once
constexpr int kMaskChunks = 4;                                  // chunks per warp of a bits tile
constexpr int kMaskTile = kChunk * kMaskChunks * (kTileBlock / 32);  // elements of a bits tile
constexpr int kMaskFlight = 16;  // 8 words in flight: 87 us instead of 79

// Below kCompactMin elements one launch (mask_select_tile) is the shorter way as long
// as its tiles' masks fit their bitmaps.  One kernel and two, us, at lists of mean 4:
// 2^16 uint8 elements 19 and 23, float64 21 and 19; 2^19 21 and 25, 23 and 21; 2^20
// 25 and 27, 25 and 22; 2^22 38 and 31, 41 and 31.  At mean 30: 2^16 71 and 23, 2^25
// 225 and 91; at mean 1000: 2^16 887 and 23, 2^25 2954 and 86.
constexpr long long kCompactMin = 1 << 20;
inline bool mask_compact(long long nelements, long long nlists) {
  return nelements >= kCompactMin ||
         (nelements > kMaskBits && nelements / (kMaskBits / kTileLists) > nlists);
}

// The tables of a run of tiles: bit p of an array's bitmap is its element
// first + p - shift, shift the place of the first element's byte in its 16-byte
// line, so an array of n elements has tiles for n + 15 bits and one more word.
struct MaskBits {
  long long* tile_before;          // per tile: its total, then the total before it
  unsigned long long* finished;    // tiles done (zero before the launch)
  unsigned* words;                 // kMaskTile / 32 per tile
  unsigned short* before;          // per word: true entries of its tile before it
};
inline long long mask_tiles(long long nelements) {
  return (nelements + 15) / kMaskTile + 1;
}
inline size_t mask_bits_bytes(long long tiles) {
  return (size_t)(tiles + 1) * 8 + (size_t)tiles * (kMaskTile / 32) * 6;
}
inline MaskBits mask_bits_at(void* p, long long tiles) {
  MaskBits b;
  b.finished = static_cast<unsigned long long*>(p);
  b.tile_before = static_cast<long long*>(p) + 1;
  b.words = reinterpret_cast<unsigned*>(b.tile_before + tiles);
  b.before = reinterpret_cast<unsigned short*>(b.words + tiles * (kMaskTile / 32));
  return b;
}

struct MaskSpan {
  long long first;  // offsets[0]
  int shift;
  long long nbits;  // shift + elements of the lists' span (no more than the tables hold)
};
// The span of lists whose mask has `masklen` entries; *inside is false when these are
// known and it reaches past them or holds more than `nelements`.
__device__ __forceinline__ MaskSpan mask_span(const uint8_t* mask, long long masklen,
                                              const int64_t* offsets, long long nlists,
                                              long long nelements, bool* inside = nullptr) {
  MaskSpan s;
  s.first = __ldg(offsets);
  long long last = __ldg(offsets + nlists);
  if (inside) *inside = true;
  if (masklen != kAnyLength) {
    if (inside) *inside = s.first >= 0 && last <= masklen && last - s.first <= nelements;
    s.first = s.first < 0 ? 0 : s.first > masklen ? masklen : s.first;
    last = last > masklen ? masklen : last;
  }
  long long n = last - s.first;
  n = n < 0 ? 0 : n > nelements ? nelements : n;
  s.shift = (int)(reinterpret_cast<uintptr_t>(mask + s.first) & 15);
  s.nbits = s.shift + n;
  return s;
}

struct MaskBitsSmem {
  int total[kMaskTile / kChunk];
  long long scan[kTileBlock / 32 + 1];
  bool last;
};

// Tile `t` of the tables, tile `local` of its array, by the whole CTA; the last of
// the launch's gridDim.x tiles scans the totals.
__device__ __forceinline__ void mask_bits_tile(MaskBitsSmem& sm, const MaskBits& b, long long t,
                                               long long local, const uint8_t* mask,
                                               const MaskSpan& span) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const long long at = local * kMaskTile + warp * (kMaskChunks * kChunk);  // first bit
  const uint8_t* line = mask + span.first - span.shift + at + lane * 32;
  unsigned word[kMaskChunks];
  if (at >= span.shift && at + kMaskChunks * kChunk <= span.nbits) {
    uint4 v[kMaskChunks][2];
#pragma unroll
    for (int c = 0; c < kMaskChunks; c++) {
      v[c][0] = __ldg(reinterpret_cast<const uint4*>(line + c * kChunk));
      v[c][1] = __ldg(reinterpret_cast<const uint4*>(line + c * kChunk) + 1);
    }
#pragma unroll
    for (int c = 0; c < kMaskChunks; c++)
      word[c] = nonzero_bits16(v[c][0]) | nonzero_bits16(v[c][1]) << 16;
  } else {
#pragma unroll
    for (int c = 0; c < kMaskChunks; c++) {
      const long long lo = at + c * kChunk + lane * 32, hi = lo + 32;
      word[c] = 0;
      if (lo >= span.shift && hi <= span.nbits) {
        const uint4* p = reinterpret_cast<const uint4*>(line + c * kChunk);
        word[c] = nonzero_bits16(__ldg(p)) | nonzero_bits16(__ldg(p + 1)) << 16;
        continue;
      }
      const int j0 = lo < span.shift ? (int)(span.shift - lo < 32 ? span.shift - lo : 32) : 0;
      const int j1 = hi > span.nbits ? (int)(span.nbits > lo ? span.nbits - lo : 0) : 32;
      for (int j = j0; j < j1; j++) word[c] |= (unsigned)(line[c * kChunk + j] != 0) << j;
    }
  }
  int excl[kMaskChunks];
#pragma unroll
  for (int c = 0; c < kMaskChunks; c++) {
    int incl = __popc(word[c]);
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += o;
    }
    excl[c] = incl - __popc(word[c]);
    if (lane == 31) sm.total[warp * kMaskChunks + c] = incl;
  }
  __syncthreads();
  if (warp == 0) {  // a chunk per lane
    const int n = sm.total[lane];
    int incl = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int o = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += o;
    }
    sm.total[lane] = incl - n;
    if (lane == 31) {
      b.tile_before[t] = incl;
      __threadfence();
      sm.last = atomicAdd(b.finished, 1ull) == gridDim.x - 1;
    }
  }
  __syncthreads();
  const long long w0 = t * (kMaskTile / 32) + warp * (kMaskChunks * 32) + lane;
#pragma unroll
  for (int c = 0; c < kMaskChunks; c++) {
    b.words[w0 + c * 32] = word[c];
    b.before[w0 + c * 32] = (unsigned short)(sm.total[warp * kMaskChunks + c] + excl[c]);
  }
  if (!sm.last) return;
  __threadfence();
  constexpr int kPer = 8;
  auto add = [](long long x, long long y) { return x + y; };
  long long carry = 0;
  for (long long base = 0; base < gridDim.x; base += kTileBlock * kPer) {
    const long long i0 = base + threadIdx.x * kPer;
    long long n[kPer], sum = 0;
#pragma unroll
    for (int i = 0; i < kPer; i++) {
      n[i] = i0 + i < gridDim.x ? __ldcg(b.tile_before + i0 + i) : 0;
      sum += n[i];
    }
    long long all;
    long long run = carry + block_exclusive_scan<kTileBlock>(sum, add, 0ll, sm.scan, &all);
#pragma unroll
    for (int i = 0; i < kPer; i++) {
      if (i0 + i < gridDim.x) b.tile_before[i0 + i] = run;
      run += n[i];
    }
    carry += all;
    __syncthreads();
  }
}
static_assert(kMaskTile / kChunk == 32, "one lane per chunk in the tile's scan");
static_assert(kMaskTile <= 65536, "ranks in a tile are 16 bits");

// What a warp holds of a chunk: lane w its word w, the ranks before it.
struct MaskChunk {
  unsigned word;
  int before;
  long long tile_before;
};
__device__ __forceinline__ MaskChunk mask_chunk(const MaskBits& b, long long c) {
  const int lane = threadIdx.x & 31;
  return {b.words[c * 32 + lane], b.before[c * 32 + lane],
          b.tile_before[c / (kMaskTile / kChunk)]};
}

// Copy a chunk's selected elements (whole warp): `from` is the element of its bit 0
// plus the lane, `out` the output of its tile's first rank.
template <class W, bool CARRY>
__device__ __forceinline__ void mask_copy(const MaskChunk& ch, const W* __restrict__ from, W* out,
                                          int64_t* carry, long long e0) {
  constexpr unsigned kFull = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1u;
#pragma unroll
  for (int g = 0; g < 32; g += kMaskFlight) {
    W v[kMaskFlight];
#pragma unroll
    for (int u = 0; u < kMaskFlight; u++)
      v[u] = __shfl_sync(kFull, ch.word, g + u) >> lane & 1u ? __ldg(from + 32 * (g + u)) : W(0);
#pragma unroll
    for (int u = 0; u < kMaskFlight; u++) {
      const unsigned w = __shfl_sync(kFull, ch.word, g + u);
      const int r = __shfl_sync(kFull, ch.before, g + u) + __popc(w & below);
      if (w >> lane & 1u) {
        out[r] = v[u];
        if constexpr (CARRY) carry[r] = e0 + 32 * (g + u);
      }
    }
  }
}

// The rank of list end `o` in its array, whose tiles begin at tile t0.
__device__ __forceinline__ long long mask_rank(long long o, const MaskBits& b, long long t0,
                                               const MaskSpan& span) {
  long long p = o - span.first + span.shift;
  p = p < 0 ? 0 : p > span.nbits ? span.nbits : p;
  const long long w = t0 * (kMaskTile / 32) + (p >> 5);
  return b.tile_before[w / (kMaskTile / 32)] + b.before[w] +
         __popc(b.words[w] & ((1u << (p & 31)) - 1u));
}

}  // namespace gb
