// Sums in the reference's order on sm_100a: every column batch is one
// sequential chain of additions (AccSquares / AccDot of a batch,
// methods_common.cpp:112-122), evaluated piecewise in parallel with the same
// bits (ordered_sum.cuh).
//
// One block per batch.  A tile of 8 terms per thread is staged in shared
// memory (the next tile's loads are in flight meanwhile); every warp
// summarises its 256 terms for the running sum's binade, one warp scans the
// warps' maps, applies all that stay inside the binade and adds the first
// piece that does not term by term.  The chain's own cost, about 8 cycles a
// term on one thread, is paid only for those pieces (a few dozen per sum).
// What bounds it: the latency of the block's summary-and-scan rounds; a sum
// is still one block, because its rounds depend on the running sum.  Measured
// on one batch of 98,304 entries: 146 us (squares) and 126 us (dots), where
// one thread walking the batch took 3,970 us and 23,200 us (every entry waited
// for its loads); 64 batches of 6,600 entries: 67 and 56 us against 1,080 and
// 18,600 us.

#include <cuda_runtime.h>

#include <cstdint>

#include "device.cuh"
#include "ops.cuh"
#include "ordered_sum.cuh"

namespace spai {

namespace {

constexpr int kTermsPerThread = 8;
constexpr int kPiece = kWarp * kTermsPerThread;  // terms of one warp
constexpr int kMaxSumWarps = 32;

// Shared-memory place of term i: two doubles of padding after every eight, so
// that lanes reading their own eight terms hit different banks.
__device__ __forceinline__ int TermAt(int i) { return i + 2 * (i >> 3); }

__device__ __forceinline__ SumMap ShuffleMap(const SumMap& m, int delta, bool up) {
  SumMap o;
#pragma unroll
  for (int p = 0; p < 2; ++p) {
    o.inc[p] = up ? __shfl_up_sync(0xffffffffu, m.inc[p], delta) : __shfl_down_sync(0xffffffffu, m.inc[p], delta);
  }
  o.lo = up ? __shfl_up_sync(0xffffffffu, m.lo, delta) : __shfl_down_sync(0xffffffffu, m.lo, delta);
  o.hi = up ? __shfl_up_sync(0xffffffffu, m.hi, delta) : __shfl_down_sync(0xffffffffu, m.hi, delta);
  o.bad = up ? __shfl_up_sync(0xffffffffu, m.bad, delta) : __shfl_down_sync(0xffffffffu, m.bad, delta);
  return o;
}

// The map of this warp's piece (every lane's eight terms in order), on lane 0.
__device__ __forceinline__ SumMap PieceMap(const double* own, double scale, SumState state, int lane) {
  double t[kTermsPerThread];
#pragma unroll
  for (int i = 0; i < kTermsPerThread / 2; ++i) {
    const double2 v = reinterpret_cast<const double2*>(own)[i];
    t[2 * i] = v.x;
    t[2 * i + 1] = v.y;
  }
  if (state != kSumNormal) {
    bool zero = state == kSumZero;
#pragma unroll
    for (int i = 0; i < kTermsPerThread; ++i) zero = zero && t[i] == 0.0;
    SumMap m = EmptyMap();
    m.bad = __all_sync(0xffffffffu, zero) ? 0 : 1;
    return m;
  }
  TermRun run;
#pragma unroll
  for (int i = 0; i < kTermsPerThread; ++i) run.Add(t[i], scale);
  SumMap mine = run.Map();
#pragma unroll
  for (int o = 1; o < kWarp; o <<= 1) {
    const SumMap later = ShuffleMap(mine, o, false);
    if ((lane & (2 * o - 1)) == 0) mine = Then(mine, later);
  }
  return mine;
}

// The maps of pieces 0..lane, one after another, on every lane.
__device__ __forceinline__ SumMap ScanMaps(const SumMap& own, int lane) {
  SumMap prefix = own;
#pragma unroll
  for (int o = 1; o < kWarp; o <<= 1) {
    const SumMap before = ShuffleMap(prefix, o, true);
    if (lane >= o) prefix = Then(before, prefix);
  }
  return prefix;
}

// out[b] = the sequential sum over entries [ptr[first[b]], ptr[first[b + 1]])
// of val[p]^2 (kSquares) or val[p].
template <class T, bool kSquares>
__global__ void __launch_bounds__(1024) OrderedSumKernel(const T* __restrict__ val, const int64_t* __restrict__ ptr,
                                                         const int64_t* __restrict__ first, int64_t batches,
                                                         double* __restrict__ out) {
  extern __shared__ __align__(16) double ordered_terms[];
  __shared__ SumMap maps[kMaxSumWarps];
  __shared__ double running;
  __shared__ int next_piece;
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int warps = blockDim.x >> 5;
  const int tile = blockDim.x * kTermsPerThread;
  auto term = [&](int64_t p, int64_t end) {
    if (p >= end) return 0.0;  // padding after the last term changes nothing
    const double v = static_cast<double>(val[p]);
    return kSquares ? Mul(v, v) : v;
  };
  for (int64_t b = blockIdx.x; b < batches; b += gridDim.x) {
    const int64_t begin = ptr[first[b]];
    const int64_t end = ptr[first[b + 1]];
    double ahead[kTermsPerThread];
#pragma unroll
    for (int i = 0; i < kTermsPerThread; ++i) ahead[i] = term(begin + i * blockDim.x + tid, end);
    if (tid == 0) running = 0.0;
    for (int64_t base = begin; base < end; base += tile) {
#pragma unroll
      for (int i = 0; i < kTermsPerThread; ++i) ordered_terms[TermAt(i * blockDim.x + tid)] = ahead[i];
      __syncthreads();
#pragma unroll
      for (int i = 0; i < kTermsPerThread; ++i) ahead[i] = term(base + tile + i * blockDim.x + tid, end);
      const int pieces = end - base < tile ? static_cast<int>((end - base + kPiece - 1) / kPiece) : warps;
      int start = 0;
      while (start < pieces) {
        const double s = running;
        double scale;
        const SumState state = Classify(s, &scale);
        if (warp >= start && warp < pieces) {
          const SumMap mine = PieceMap(ordered_terms + TermAt(tid * kTermsPerThread), scale, state, lane);
          if (lane == 0) maps[warp] = mine;
        }
        __syncthreads();
        if (warp == 0) {
          const SumMap prefix = ScanMaps(lane >= start && lane < pieces ? maps[lane] : EmptyMap(), lane);
          double moved = s;
          const bool kept = ApplyMap(prefix, s, state, &moved);
          const unsigned failed = __ballot_sync(0xffffffffu, !kept && lane >= start && lane < pieces);
          const int stop = failed != 0u ? __ffs(failed) - 1 : pieces;  // first piece that leaves the binade
          double now = __shfl_sync(0xffffffffu, moved, stop > 0 ? stop - 1 : 0);
          if (stop <= start) now = s;
          if (lane == 0) {
            if (stop < pieces) {
              const double2* t2 = reinterpret_cast<const double2*>(ordered_terms + TermAt(stop * kPiece));
              for (int g = 0; g < kWarp; ++g) {  // eight terms, two doubles of padding
#pragma unroll
                for (int i = 0; i < kTermsPerThread / 2; ++i) {
                  const double2 v = t2[i];
                  now = Add(now, v.x);
                  now = Add(now, v.y);
                }
                t2 += (kTermsPerThread + 2) / 2;
              }
            }
            running = now;
            next_piece = stop < pieces ? stop + 1 : pieces;
          }
        }
        __syncthreads();
        start = next_piece;
      }
    }
    __syncthreads();
    if (tid == 0) out[b] = running;
    __syncthreads();
  }
}

// terms[p] = x[p] * y at x's row (0 where y's column has no such row), for
// every entry p of x.  Warp per column; a row is first looked for at the same
// place of y's column (equal patterns, e.g. R and Pr R), then by binary search.
template <class T>
__global__ void DotTermsKernel(CscView<T> x, CscView<T> y, double* __restrict__ terms) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  for (int64_t j = warp; j < x.cols; j += warps) {
    const int64_t xs = x.ptr[j];
    const int64_t xe = x.ptr[j + 1];
    const int64_t ys = y.ptr[j];
    const int64_t ye = y.ptr[j + 1];
    for (int64_t p = xs + lane; p < xe; p += kWarp) {
      const int32_t row = x.idx[p];
      int64_t q = ys + (p - xs);
      if (q >= ye || y.idx[q] != row) {
        int64_t lo = ys;
        int64_t hi = ye;
        while (lo < hi) {
          const int64_t mid = lo + ((hi - lo) >> 1);
          if (y.idx[mid] < row) {
            lo = mid + 1;
          } else {
            hi = mid;
          }
        }
        q = lo;
      }
      const bool hit = q < ye && y.idx[q] == row;
      terms[p] = hit ? Mul(static_cast<double>(x.val[p]), static_cast<double>(y.val[q])) : 0.0;
    }
  }
}

// Threads of a batch's block.  Long batches take the largest tile (8,192
// terms a round); short ones a smaller block, so that a round is not padding.
int SumThreads(int64_t entries, int64_t batches) {
  const int64_t average = entries / (batches > 0 ? batches : 1);
  if (average >= 16384) return 1024;
  return average >= 512 ? 256 : kWarp;
}

template <class T, bool kSquares>
void LaunchOrderedSum(Ctx& ctx, const T* val, const int64_t* ptr, int64_t entries, const int64_t* first,
                      int64_t batches, double* out) {
  const int threads = SumThreads(entries, batches);
  const size_t smem = sizeof(double) * static_cast<size_t>(threads) * (kTermsPerThread + 2);
  SPAI_CUDA(cudaFuncSetAttribute(OrderedSumKernel<T, kSquares>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(sizeof(double) * 1024 * (kTermsPerThread + 2))));
  const int64_t cap = static_cast<int64_t>(ctx.sm_count) * 16;
  const int grid = static_cast<int>(batches < cap ? batches : cap);
  OrderedSumKernel<T, kSquares><<<grid, threads, smem, ctx.stream>>>(val, ptr, first, batches, out);
  SPAI_LAUNCH_CHECK();
}

}  // namespace

template <class T>
void OrderedSquares(Ctx& ctx, const DevCsc<T>& x, const int64_t* first, int64_t batches, double* out) {
  LaunchOrderedSum<T, true>(ctx, x.val.data(), x.ptr.data(), x.nnz, first, batches, out);
}

template <class T>
void OrderedDots(Ctx& ctx, const DevCsc<T>& x, const DevCsc<T>& y, const int64_t* first, int64_t batches,
                 double* out) {
  // the common rows in ascending order from either side: take the shorter one
  const DevCsc<T>& from = x.nnz <= y.nnz ? x : y;
  const DevCsc<T>& other = x.nnz <= y.nnz ? y : x;
  ctx.dot_terms.Reserve(static_cast<size_t>(from.nnz > 0 ? from.nnz : 1), ctx.stream);
  DotTermsKernel<T><<<GridFor(from.cols * kWarp, 256), 256, 0, ctx.stream>>>(View(from), View(other),
                                                                            ctx.dot_terms.data());
  SPAI_LAUNCH_CHECK();
  LaunchOrderedSum<double, false>(ctx, ctx.dot_terms.data(), from.ptr.data(), from.nnz, first, batches, out);
}

template void OrderedSquares<double>(Ctx&, const DevCsc<double>&, const int64_t*, int64_t, double*);
template void OrderedSquares<float>(Ctx&, const DevCsc<float>&, const int64_t*, int64_t, double*);
template void OrderedDots<double>(Ctx&, const DevCsc<double>&, const DevCsc<double>&, const int64_t*, int64_t, double*);
template void OrderedDots<float>(Ctx&, const DevCsc<float>&, const DevCsc<float>&, const int64_t*, int64_t, double*);

}  // namespace spai
