#pragma once
// Building blocks of the column-group kernels (mr_fused.cu): one warp works on
// C adjacent columns at once in a shared row space.
//
// The rows that any of the columns touches are marked in one bitmap over a
// window of rows; a row's rank -- its place among the marked rows -- is the
// prefix count of its 32-row word plus a population count, two shared-memory
// reads without any probing.  Values live in dense arrays indexed by rank, C
// values side by side, so one lookup serves all C columns, and a walk over
// ranks is a walk over rows in ascending order.  A column that lacks a row
// holds 0 there, which adds nothing to its sums.
//
// Why C columns: adjacent columns of a grid operator share most of their rows
// (four columns of the 7-point 40^3 operator with 16 entries each: 205 product
// rows together, 445 one by one), and what a warp does once per column -- the
// sequential sums in row order above all -- runs side by side for all of them.

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "colkit.cuh"
#include "device.cuh"

namespace spai {

// (aligned to 16 bytes at most: the arrays are placed at multiples of 16)
template <class T, int C>
struct alignas(sizeof(T) * C < 16 ? sizeof(T) * C : 16) GroupValues {
  T v[C];
};

// A bitmap over `words` 32-row words from row `lo` (which may be negative),
// with a summary bit per word and the rank of each word's first marked row.
struct RowWindow {
  uint32_t* bits;
  uint32_t* summary;
  uint8_t* prefix;
  int32_t lo;
  int words;

  __device__ __forceinline__ bool Holds(int32_t row) const {
    return static_cast<uint32_t>(row - lo) < static_cast<uint32_t>(words) * 32u;
  }
  // row must be held by the window
  __device__ __forceinline__ void Mark(int32_t row) {
    const int off = row - lo;
    atomicOr(&bits[off >> 5], 1u << (off & 31));
    atomicOr(&summary[off >> 10], 1u << ((off >> 5) & 31));
  }
  // The same where most rows are marked already (three in four rows of A Z): a read is cheaper than an atomic.
  __device__ __forceinline__ void MarkNew(int32_t row) {
    const int off = row - lo;
    if ((bits[off >> 5] & (1u << (off & 31))) == 0u) Mark(row);
  }
  // rank of a row that was marked
  __device__ __forceinline__ int Rank(int32_t row) const {
    const int off = row - lo;
    return prefix[off >> 5] + __popc(bits[off >> 5] & ((1u << (off & 31)) - 1u));
  }
  // rank of a row, or `absent` when it is not marked
  __device__ __forceinline__ int FindOr(int32_t row, int absent) const {
    const bool held = Holds(row);
    const int off = held ? row - lo : 0;
    const uint32_t b = bits[off >> 5];
    const uint32_t bit = 1u << (off & 31);
    const int rank = prefix[off >> 5] + __popc(b & (bit - 1u));
    return held && (b & bit) != 0u ? rank : absent;
  }
};

__host__ __device__ inline int GroupSummaryWords(int words) { return (words + 31) / 32; }

// Shared memory of one window (prefix included).
__host__ __device__ inline size_t WindowBytes(int words) {
  return Round16(static_cast<size_t>(words) * 4) + Round16(static_cast<size_t>(GroupSummaryWords(words)) * 4) +
         Round16(static_cast<size_t>(words));
}

inline __device__ RowWindow WindowAt(unsigned char*& base, int words, int32_t lo) {
  RowWindow w;
  w.bits = reinterpret_cast<uint32_t*>(base);
  base += Round16(static_cast<size_t>(words) * 4);
  w.summary = reinterpret_cast<uint32_t*>(base);
  base += Round16(static_cast<size_t>(GroupSummaryWords(words)) * 4);
  w.prefix = base;
  base += Round16(static_cast<size_t>(words));
  w.lo = lo;
  w.words = words;
  return w;
}

inline __device__ void ClearWindow(RowWindow& w, int lane) {
  __syncwarp();
  ClearWords(w.bits, w.words, lane);
  ClearWords(w.summary, GroupSummaryWords(w.words), lane);
  __syncwarp();
}

// Clears the words of the listed rows only (offsets from lo).
inline __device__ void ClearRows(RowWindow& w, const uint16_t* rows, int count, int lane) {
  __syncwarp();
#pragma unroll 1
  for (int r = lane; r < count; r += kWarp) w.bits[rows[r] >> 5] = 0u;
#pragma unroll 1
  for (int s = lane; s < GroupSummaryWords(w.words); s += kWarp) w.summary[s] = 0u;
  __syncwarp();
}

__device__ __forceinline__ int WarpInclusive(int v, int lane) {
#pragma unroll
  for (int o = 1; o < kWarp; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += y;
  }
  return v;
}

// Ranks the marked rows: fills the words' prefixes (kPrefix; meaningful while
// at most 256 rows are marked) and, when rows is given, lists the rows in
// ascending order as offsets from lo.  `list` is scratch for `cap` entries.
// Returns the number of marked rows, or cap + 1 when there are more than cap
// (then nothing usable is written).  Ends with __syncwarp.
template <bool kPrefix>
inline __device__ int RankRows(RowWindow& w, uint16_t* rows, uint16_t* list, int cap, int lane) {
  __syncwarp();
  const int summaries = GroupSummaryWords(w.words);
  int nonempty = 0;
#pragma unroll 1
  for (int s0 = 0; s0 < summaries; s0 += kWarp) {
    const int s = s0 + lane;
    uint32_t left = s < summaries ? w.summary[s] : 0u;
    const int own = __popc(left);
    const int inclusive = WarpInclusive(own, lane);
    int at = nonempty + inclusive - own;
    nonempty += __shfl_sync(0xffffffffu, inclusive, 31);
    if (nonempty > cap) return cap + 1;
#pragma unroll 1
    for (; left != 0u; left &= left - 1u) list[at++] = static_cast<uint16_t>(s * 32 + (__ffs(left) - 1));
  }
  __syncwarp();
  int total = 0;
#pragma unroll 1
  for (int w0 = 0; w0 < nonempty; w0 += kWarp) {
    const bool have = w0 + lane < nonempty;
    const int word = have ? list[w0 + lane] : 0;
    uint32_t b = have ? w.bits[word] : 0u;
    const int own = __popc(b);
    const int inclusive = WarpInclusive(own, lane);
    int at = total + inclusive - own;
    total += __shfl_sync(0xffffffffu, inclusive, 31);
    if (total > cap) return cap + 1;
    if (kPrefix && have) w.prefix[word] = static_cast<uint8_t>(at);
    if (rows != nullptr) {
#pragma unroll 1
      for (; b != 0u; b &= b - 1u) rows[at++] = static_cast<uint16_t>(word * 32 + (__ffs(b) - 1));
    }
  }
  __syncwarp();
  return total;
}

// Magnitudes as integers of the same order (NaN above infinity).
__device__ __forceinline__ uint32_t MagnitudeBits(float v) {
  return static_cast<uint32_t>(__float_as_int(v)) & 0x7FFFFFFFu;
}
__device__ __forceinline__ unsigned long long MagnitudeBits(double v) {
  return static_cast<unsigned long long>(__double_as_longlong(v)) & 0x7FFFFFFFFFFFFFFFull;
}
// The magnitude with these bits (the second argument selects the type).
__device__ __forceinline__ float MagnitudeFrom(uint32_t key, float) { return __int_as_float(static_cast<int>(key)); }
__device__ __forceinline__ double MagnitudeFrom(unsigned long long key, double) {
  return __longlong_as_double(static_cast<long long>(key));
}
template <class T>
struct MagnitudeOf;
template <>
struct MagnitudeOf<float> {
  using Key = uint32_t;
};
template <>
struct MagnitudeOf<double> {
  using Key = unsigned long long;
};

// The warp's largest and smallest key: exact for float, from the upper words
// for double (an upper bound whose lower word is all ones, a lower bound whose
// lower word is 0).
__device__ __forceinline__ uint32_t LargestKey(uint32_t key) { return __reduce_max_sync(0xffffffffu, key); }
__device__ __forceinline__ uint32_t SmallestKey(uint32_t key) { return __reduce_min_sync(0xffffffffu, key); }
__device__ __forceinline__ unsigned long long LargestKey(unsigned long long key) {
  const uint32_t top = __reduce_max_sync(0xffffffffu, static_cast<uint32_t>(key >> 32));
  return (static_cast<unsigned long long>(top) << 32) | 0xFFFFFFFFull;
}
__device__ __forceinline__ unsigned long long SmallestKey(unsigned long long key) {
  return static_cast<unsigned long long>(__reduce_min_sync(0xffffffffu, static_cast<uint32_t>(key >> 32))) << 32;
}
__device__ __forceinline__ double MagnitudeValue(uint32_t key) {
  return static_cast<double>(__int_as_float(static_cast<int>(key)));
}
__device__ __forceinline__ double MagnitudeValue(unsigned long long key) {
  return __longlong_as_double(static_cast<long long>(key));
}

}  // namespace spai
