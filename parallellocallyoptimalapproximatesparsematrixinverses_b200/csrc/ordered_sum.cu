// Sums in the reference's order on sm_100a: every column batch is one
// sequential chain of additions (AccSquares / AccDot of a batch,
// methods_common.cpp:112-122), evaluated piecewise in parallel with the same
// bits (ordered_sum.cuh).
//
// One block (or cluster) per batch.  A tile of 8 terms per thread is staged in shared
// memory (the next tile's loads are in flight meanwhile); every warp
// summarises its 256 terms for the running sum's binade, one warp scans the
// warps' maps, applies all that stay inside the binade and adds the first
// piece that does not term by term.  The chain's own cost, about 8 cycles a
// term on one thread, is paid only for those pieces (a few dozen per sum).
// What bounds it: the latency of the rounds, because each depends on the
// running sum, and the issue of the maps' arithmetic within a block; long
// batches are therefore spread over a cluster of eight blocks.  Measured on
// one batch of 98,304 entries: 113 us (squares) and 100 us (dots), where one
// thread walking the batch took 3,970 us and 23,200 us (every entry waited for
// its loads); 64 batches of 6,600 entries: 67 and 55 us against 1,080 and
// 18,600 us.

#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <cstdint>

#include "device.cuh"
#include "ops.cuh"
#include "ordered_sum.cuh"

namespace spai {

namespace {

namespace cg = cooperative_groups;

constexpr int kTermsPerThread = 8;
constexpr int kPiece = kWarp * kTermsPerThread;  // terms of one warp
constexpr int kMaxSumWarps = 8;

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

__device__ __forceinline__ SumMap ShuffleFrom(const SumMap& m, int lane) {
  SumMap o;
#pragma unroll
  for (int p = 0; p < 2; ++p) o.inc[p] = __shfl_sync(0xffffffffu, m.inc[p], lane);
  o.lo = __shfl_sync(0xffffffffu, m.lo, lane);
  o.hi = __shfl_sync(0xffffffffu, m.hi, lane);
  o.bad = __shfl_sync(0xffffffffu, m.bad, lane);
  return o;
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
__global__ void __launch_bounds__(256) OrderedSumKernel(const T* __restrict__ val, const int64_t* __restrict__ ptr,
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

// The same with a cluster of eight blocks of 256 threads per batch, for long
// batches: block r stages terms [2048 r, 2048 r + 2048) of a tile of 16,384.
// A round composes the blocks' maps in every block (each receives all eight
// over distributed shared memory); where one fails, its block adds the piece
// that does not fit and hands the sum on.
constexpr int kSumBlocks = 8;
constexpr int kSumBlockThreads = 256;
constexpr int kSumBlockPieces = kSumBlockThreads / kWarp;

template <class T, bool kSquares>
__global__ void __cluster_dims__(kSumBlocks, 1, 1) __launch_bounds__(kSumBlockThreads)
    OrderedSumClusterKernel(const T* __restrict__ val, const int64_t* __restrict__ ptr,
                            const int64_t* __restrict__ first, int64_t batches, double* __restrict__ out) {
  __shared__ __align__(16) double terms[kSumBlockThreads * (kTermsPerThread + 2)];
  __shared__ SumMap prefixes[kSumBlockPieces];      // maps of this block's pieces up to each
  __shared__ SumMap blocks[2][kSumBlocks];          // [round parity] every block's map
  __shared__ SumMap maps[kSumBlockPieces];
  __shared__ double running;
  __shared__ int next_piece;
  __shared__ int settled;  // every piece of the tile is in the sum
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank());
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  constexpr int kBlockTile = kSumBlockThreads * kTermsPerThread;
  constexpr int64_t kTile = static_cast<int64_t>(kSumBlocks) * kBlockTile;
  int round = 0;
  auto term = [&](int64_t p, int64_t end) {
    if (p >= end) return 0.0;  // padding after the last term changes nothing
    const double v = static_cast<double>(val[p]);
    return kSquares ? Mul(v, v) : v;
  };
  // A block's shared memory may be written from outside only once that block runs; each later round's stores
  // follow a cluster barrier of the round before.
  cluster.sync();
  for (int64_t b = blockIdx.x / kSumBlocks; b < batches; b += gridDim.x / kSumBlocks) {
    const int64_t begin = ptr[first[b]];
    const int64_t end = ptr[first[b + 1]];
    const int64_t mine = static_cast<int64_t>(rank) * kBlockTile;
    double ahead[kTermsPerThread];
#pragma unroll
    for (int i = 0; i < kTermsPerThread; ++i) ahead[i] = term(begin + mine + i * kSumBlockThreads + tid, end);
    if (tid == 0) running = 0.0;
    for (int64_t base = begin; base < end; base += kTile) {
#pragma unroll
      for (int i = 0; i < kTermsPerThread; ++i) terms[TermAt(i * kSumBlockThreads + tid)] = ahead[i];
      __syncthreads();
#pragma unroll
      for (int i = 0; i < kTermsPerThread; ++i) {
        ahead[i] = term(base + kTile + mine + i * kSumBlockThreads + tid, end);
      }
      const int pieces = end - base < kTile ? static_cast<int>((end - base + kPiece - 1) / kPiece)
                                            : kSumBlocks * kSumBlockPieces;
      int start = 0;  // first piece of the tile that is not in the sum yet
      while (start < pieces) {
        const double s = running;
        double scale;
        const SumState state = Classify(s, &scale);
        const int parity = round++ & 1;
        const int own = rank * kSumBlockPieces + warp;
        SumMap map = EmptyMap();
        if (own >= start && own < pieces) map = PieceMap(terms + TermAt(tid * kTermsPerThread), scale, state, lane);
        if (lane == 0) maps[warp] = map;
        __syncthreads();
        if (warp == 0) {
          const SumMap prefix = ScanMaps(lane < kSumBlockPieces ? maps[lane] : EmptyMap(), lane);
          if (lane < kSumBlockPieces) prefixes[lane] = prefix;
          const SumMap all = ShuffleFrom(prefix, kSumBlockPieces - 1);
          if (lane < kSumBlocks) *cluster.map_shared_rank(&blocks[parity][rank], lane) = all;
        }
        cluster.sync();
        // the first block whose pieces leave the binade, by every warp 0 alike
        if (warp == 0) {
          const SumMap prefix = ScanMaps(lane < kSumBlocks ? blocks[parity][lane] : EmptyMap(), lane);
          double moved = s;
          const bool kept = ApplyMap(prefix, s, state, &moved);
          const bool has = lane < kSumBlocks && (lane + 1) * kSumBlockPieces > start && lane * kSumBlockPieces < pieces;
          const unsigned failed = __ballot_sync(0xffffffffu, has && !kept);
          const int stop = failed != 0u ? __ffs(failed) - 1 : kSumBlocks;
          // the sum after the blocks before it (those without pieces leave it as it is)
          const double after = __shfl_sync(0xffffffffu, moved, stop > 0 ? stop - 1 : 0);
          const bool any_before = stop > 0 && stop * kSumBlockPieces > start;
          double now = any_before ? after : s;
          if (stop == kSumBlocks) {
            if (lane == 0) {
              running = now;
              next_piece = pieces;
            }
          } else if (stop == rank) {
            SumState here;
            double unused;
            here = Classify(now, &unused);
            double within = now;
            const int piece = rank * kSumBlockPieces + lane;
            const bool mine_has = lane < kSumBlockPieces && piece >= start && piece < pieces;
            const bool fits = lane < kSumBlockPieces && here == state && ApplyMap(prefixes[lane], now, here, &within);
            const unsigned bad = __ballot_sync(0xffffffffu, mine_has && !fits);
            // the first piece that does not fit; none when only the composed bounds were too wide
            const int at = bad != 0u ? __ffs(bad) - 1 : kSumBlockPieces;
            const double before = __shfl_sync(0xffffffffu, within, at > 0 ? at - 1 : 0);
            if (at > 0 && rank * kSumBlockPieces + at > start) now = before;
            if (lane == 0 && at < kSumBlockPieces) {
              const double2* t2 = reinterpret_cast<const double2*>(terms + TermAt(at * kPiece));
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
            now = __shfl_sync(0xffffffffu, now, 0);
            if (lane < kSumBlocks) {
              *cluster.map_shared_rank(&running, lane) = now;
              const int next = rank * kSumBlockPieces + (at < kSumBlockPieces ? at + 1 : at);
              *cluster.map_shared_rank(&next_piece, lane) = next < pieces ? next : pieces;
            }
          }
          if (lane == 0) settled = stop == kSumBlocks ? 1 : 0;
        }
        __syncthreads();
        if (settled == 0) cluster.sync();
        start = next_piece;
        __syncthreads();
      }
    }
    __syncthreads();
    if (rank == 0 && tid == 0) out[b] = running;
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

// From this many entries a batch on average, a cluster per batch: 98,304
// entries take 113 us against 162 us with one block of 1,024 threads, but
// batches of 6,600 entries 91 us against 67 us with one block of 256 (their
// rounds are changes of binade, and a round in a cluster costs two barriers).
constexpr int64_t kClusterEntries = 16384;

template <class T, bool kSquares>
void LaunchOrderedSum(Ctx& ctx, const T* val, const int64_t* ptr, int64_t entries, const int64_t* first,
                      int64_t batches, double* out) {
  const int64_t average = entries / (batches > 0 ? batches : 1);
  const int64_t cap = static_cast<int64_t>(ctx.sm_count) * 16;
  if (average >= kClusterEntries) {
    const int64_t clusters = batches < cap / kSumBlocks ? batches : cap / kSumBlocks;
    OrderedSumClusterKernel<T, kSquares><<<static_cast<unsigned>(clusters * kSumBlocks), kSumBlockThreads, 0,
                                           ctx.stream>>>(val, ptr, first, batches, out);
    SPAI_LAUNCH_CHECK();
    return;
  }
  // short batches: a block each, small enough that a round is not padding.  With 32 and 256 threads: 8.3 and 13.6 us
  // for batches of 128 squares, 11.9 and 11.9 for 256, 18.9 and 17.7 for 512, 31.8 and 25.8 for 1,024 (140,000 in all).
  const int threads = average >= 512 ? 256 : kWarp;
  const size_t smem = sizeof(double) * static_cast<size_t>(threads) * (kTermsPerThread + 2);
  OrderedSumKernel<T, kSquares><<<static_cast<unsigned>(batches < cap ? batches : cap), threads, smem, ctx.stream>>>(
      val, ptr, first, batches, out);
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
