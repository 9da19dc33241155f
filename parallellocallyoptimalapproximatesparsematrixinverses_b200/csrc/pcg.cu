// PCG evaluator on sm_100a (reference methods_cython/backward_error.pyx:69-144).
//
// A whole solve is one cooperative kernel.  Its blocks form clusters of
// eight; a cluster owns whole 4096-row chunks of the canonical tree
// (tree.cuh), block k of it the chunk's tree lanes 32k .. 32k+31, and warp w
// of the block the w-th term of those lanes: every thread owns one row of a
// chunk.  An iteration has two grid-wide reductions and nothing else that
// waits:
//
//   1. p = z + beta p and ap = A p, the neighbours' p formed on the fly from
//      z and the previous p; the dot <p, ap>.
//   2. x += alpha p, r -= alpha ap and z = M r, the neighbours' r formed on
//      the fly from the previous r and ap; the dots <r, r> and <r, z>.
//
// (p and r alternate between two buffers, so that no thread overwrites what a
// neighbour still reads.)  A refresh -- at convergence or periodic -- adds
// r = b - A x with its dot and z = M r with its dot.  Recomputing a
// neighbour's value repeats the owner's operations on the same inputs, so it
// has the owner's bits; the dots keep the tree's order, and the CPU oracle
// reproduces every iterate bit for bit.
//
// A reduction: the 16 terms of a lane are added in order through shared
// memory; the lane sums travel to the cluster's first block as asynchronous
// remote stores counted by a barrier in its shared memory, whose warps fold
// them to the chunk's sum.  With one chunk (n <= 4096) every block receives
// and folds them, and a cluster barrier publishes the vectors.  Otherwise
// every block announces its vectors on one counter (after a fence; that takes
// about 1,200 cycles, so it runs beside the folding), the chunk sums go to
// global memory as 16-byte words that carry the reduction's number, and every
// block polls both and folds the tree's next level itself.  The polls are
// bounded, in seconds and by the longest row that one thread walks (a count of
// polls alone abandoned solves with rows of millions of entries): a block that
// gives up poisons the counter, every other block sees
// that at its next reduction, and the solve ends with an error.  Every block
// decides the recurrence's scalars from the totals; the history keeps ||r||^2
// until the end, so that no square root or division is on the way to the next
// iteration unless the stop test is close.
//
// What bounds it: while every cluster owns one chunk (61,440 rows on the 15
// clusters of a B200 that fit one block per SM) the
// latency of an iteration's two reductions and gathers; the rows of both
// matrices then stay in shared memory for the whole solve where they fit.
// Beyond, the L2 reads of the two matrices and the gathers; the matrices are
// re-laid out once per solve in slices of 32 rows (entry e of the 32 rows side
// by side), so that a warp reads full lines, and a slice whose longest row
// would waste more than half of it stays in CSR.
// Measured per iteration, against one graph node per product and per dot
// (thread-per-row CSR products, dots on one block per chunk): 5.8 us against
// 29 us at n = 3,969; 14 against 30 at 62,500; 17.4 against 39 at 90,000; 43
// against 61 at 262,144 (M in FP32, about 18 entries a row).

#include <cuda_runtime.h>

#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <map>
#include <mutex>
#include <stdexcept>
#include <type_traits>
#include <vector>

#include "device.cuh"
#include "ops.cuh"
#include "pcg.cuh"
#include "profile.cuh"
#include "tree.cuh"

namespace spai {

namespace {

namespace cg = cooperative_groups;

constexpr int kClusterBlocks = 8;   // kTreeLanes / kWarp: one warp-wide group of tree lanes per block
constexpr int kSolveThreads = kWarp * kTreeTerms;  // one warp per term of a lane
constexpr int kGroupRounds = 4;     // chunks of a cluster folded at a time
constexpr unsigned long long kWaitNs = 4'000'000'000ull;  // how long a block waits for other clusters
constexpr unsigned long long kOwnWaitNs = 4 * kWaitNs;    // and for its own, whose blocks may be waiting so long
// What the longest row adds to both: one thread walks a row, and an entry takes
// it up to 0.3 us (two dependent loads for four entries).  Rows up to
// kShortWalk entries are covered anyway.
constexpr unsigned long long kWaitNsPerEntry = 2000;
constexpr int64_t kShortWalk = 65536;
constexpr unsigned kFreePolls = 4096;  // polls before a wait looks at the clock
constexpr unsigned long long kPoison = 1ull << 63;  // set in a cluster's counter by a block that gave up
constexpr int kFlagStride = 16;                 // counters 128 bytes apart
static_assert(kClusterBlocks * kWarp == kTreeLanes, "a cluster covers a chunk's lanes");

// A row-compressed matrix and its sliced copy.
template <class TV>
struct SolveMatrix {
  const int64_t* ptr;
  const int32_t* idx;
  const TV* val;
  int64_t* slice;      // per slice of 32 rows: offset in the sliced copy, or -1 (rows stay in CSR)
  int32_t* slice_idx;  // null: no room for a copy, all rows stay in CSR
  TV* slice_val;
  unsigned long long* used;  // entries of the sliced copy taken so far
};

// A chunk sum on its way between clusters: the value and the reduction it belongs to, in one 16-byte word.
struct alignas(16) TaggedSum {
  double sum;
  unsigned long long tag;
};

struct SolveOutcome {
  int64_t count;
  int64_t status;
  int32_t aborted;  // a poll ran into its limit
  int32_t pad;
};

template <class TM>
struct SolveArgs {
  SolveMatrix<double> a;
  SolveMatrix<TM> m;
  const double* b;
  double* x;
  double* r[2];
  double* p[2];
  double* z;
  double* ap;
  double* history;
  TaggedSum* partial;  // chunk sums: 2 alternating sets of 2 * chunks (tags zero at the start)
  unsigned long long* arrived;  // per cluster (kFlagStride apart): blocks whose vectors are visible, over all reductions
  SolveOutcome* outcome;
  int64_t n;
  int64_t chunks;
  unsigned long long* longest;  // entries that one thread walks per reduction, at most; 0 up to kShortWalk
  unsigned long long wait_ns;   // a block's patience with other clusters
  unsigned free_polls;          // polls before it looks at the clock
  int64_t max_iterations;
  int64_t refresh_period;
  double tolerance;
  int room;            // bytes of dynamic shared memory after SolveShared
};

// One row of a matrix: entry e at idx[e * stride], val[e * stride].
template <class TV>
struct RowRef {
  const int32_t* idx;
  const TV* val;
  int stride;
  int len;
  int width;  // the longest row of its slice
};

// Entries of a slice's rows: the longest row, and whether slicing wastes at most half.
template <class TV>
__device__ __forceinline__ int SliceWidth(const SolveMatrix<TV>& m, int64_t row, int64_t n, int64_t* first, int* len,
                                          bool* dense) {
  *first = row < n ? m.ptr[row] : 0;
  *len = row < n ? static_cast<int>(m.ptr[row + 1] - *first) : 0;
  const int width = __reduce_max_sync(0xffffffffu, *len);
  long long total = *len;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) total += __shfl_xor_sync(0xffffffffu, total, o);
  *dense = static_cast<long long>(width) * kWarp <= 2 * total + 2 * kWarp;
  return width;
}

// Copies the 32 rows of a slice, one per lane, into the sliced layout when
// that wastes at most half of it (the copy then never exceeds twice the
// entries plus two per row, what the host reserves).  Returns the lane's row's
// length.
template <class TV>
__device__ int SliceRows(const SolveMatrix<TV>& m, int64_t slice, int64_t n, int lane) {
  int64_t first;
  int len;
  bool dense;
  const int width = SliceWidth(m, slice * kWarp + lane, n, &first, &len, &dense);
  long long at = -1;
  if (dense && m.slice_idx != nullptr) {
    if (lane == 0) at = static_cast<long long>(atomicAdd(m.used, static_cast<unsigned long long>(width) * kWarp));
    at = __shfl_sync(0xffffffffu, at, 0);
    for (int e = 0; e < len; ++e) {
      m.slice_idx[at + static_cast<int64_t>(e) * kWarp + lane] = m.idx[first + e];
      m.slice_val[at + static_cast<int64_t>(e) * kWarp + lane] = m.val[first + e];
    }
  }
  if (lane == 0) m.slice[slice] = at;
  return len;
}

template <class TV>
__device__ __forceinline__ RowRef<TV> FindRow(const SolveMatrix<TV>& m, int64_t row) {
  const int64_t first = m.ptr[row];
  const int len = static_cast<int>(m.ptr[row + 1] - first);
  const int64_t at = m.slice[row >> 5];
  if (at >= 0) return RowRef<TV>{m.slice_idx + at + (row & 31), m.slice_val + at + (row & 31), kWarp, len, len};
  return RowRef<TV>{m.idx + first, m.val + first, 1, len, len};
}

__device__ __forceinline__ int32_t LoadStreamed(const int32_t* p) {
  int32_t v;
  asm volatile("ld.global.L1::no_allocate.s32 %0, [%1];" : "=r"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ float LoadStreamed(const float* p) {
  float v;
  asm volatile("ld.global.L1::no_allocate.f32 %0, [%1];" : "=f"(v) : "l"(p));
  return v;
}

__device__ __forceinline__ double LoadStreamed(const double* p) {
  double v;
  asm volatile("ld.global.L1::no_allocate.f64 %0, [%1];" : "=d"(v) : "l"(p));
  return v;
}

// The row times the vector that `in` yields, entries in storage order (the
// reference's _row_dot).  kResident (rows in shared memory): up to 16 gathers
// in flight, so that a row waits for one round trip; otherwise four, and the
// entries pass the L1, which keeps the gathered vectors.
template <bool kResident, class TV, class In>
__device__ __forceinline__ double RowDot(const RowRef<TV>& row, In in) {
  double sum = 0.0;
  if constexpr (kResident) {
    const auto group = [&](auto wide, int e0) {
      constexpr int kWide = decltype(wide)::value;
      double g[kWide];
#pragma unroll
      for (int e = 0; e < kWide; ++e) g[e] = e0 + e < row.len ? in(row.idx[(e0 + e) * row.stride]) : 0.0;
#pragma unroll
      for (int e = 0; e < kWide; ++e) {
        if (e0 + e < row.len) sum = Add(sum, Mul(static_cast<double>(row.val[(e0 + e) * row.stride]), g[e]));
      }
    };
    int e0 = 0;
    for (; row.width - e0 > 8; e0 += 16) group(std::integral_constant<int, 16>(), e0);
    if (e0 < row.width) group(std::integral_constant<int, 8>(), e0);
  } else {
    constexpr int kWide = 4;
    for (int e0 = 0; e0 < row.len; e0 += kWide) {
      int32_t c[kWide];
      TV v[kWide];
#pragma unroll
      for (int e = 0; e < kWide; ++e) {
        const bool have = e0 + e < row.len;
        const int64_t at = static_cast<int64_t>(e0 + e) * row.stride;
        c[e] = have ? LoadStreamed(row.idx + at) : 0;
        v[e] = have ? LoadStreamed(row.val + at) : TV(0);
      }
      double g[kWide];
#pragma unroll
      for (int e = 0; e < kWide; ++e) g[e] = e0 + e < row.len ? in(c[e]) : 0.0;
#pragma unroll
      for (int e = 0; e < kWide; ++e) {
        if (e0 + e < row.len) sum = Add(sum, Mul(static_cast<double>(v[e]), g[e]));
      }
    }
  }
  return sum;
}

// The tree's butterfly over 256 values, eight per lane: v[g] is value 32 g + lane.
__device__ __forceinline__ double FoldLanes(double (&v)[kClusterBlocks]) {
#pragma unroll
  for (int o = kClusterBlocks / 2; o > 0; o >>= 1) {
#pragma unroll
    for (int g = 0; g < o; ++g) v[g] = Add(v[g], v[g + o]);
  }
  double s = v[0];
#pragma unroll
  for (int o = kWarp / 2; o >= 1; o >>= 1) s = Add(s, __shfl_xor_sync(0xffffffffu, s, o));
  return s;
}

__device__ __forceinline__ unsigned long long LoadAcquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void StoreTagged(TaggedSum* p, double sum, unsigned long long tag) {
  asm volatile("{\n\t.reg .b128 w;\n\tmov.b128 w, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], w;\n\t}"
               :: "l"(p), "l"(__double_as_longlong(sum)), "l"(tag) : "memory");
}

__device__ __forceinline__ TaggedSum LoadTagged(const TaggedSum* p) {
  long long bits;
  TaggedSum t;
  asm volatile("{\n\t.reg .b128 w;\n\tld.relaxed.gpu.global.b128 w, [%2];\n\tmov.b128 {%0, %1}, w;\n\t}"
               : "=l"(bits), "=l"(t.tag) : "l"(p) : "memory");
  t.sum = __longlong_as_double(bits);
  return t;
}

__device__ __forceinline__ uint32_t SharedAddress(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// The address of this block's shared variable `local` in block `rank` of the cluster.
__device__ __forceinline__ uint32_t RemoteAddress(uint32_t local, int rank) {
  uint32_t remote;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"(rank));
  return remote;
}

// Stores v to a remote block's shared memory and counts its 8 bytes on that block's barrier.
__device__ __forceinline__ void StoreCounted(uint32_t remote, uint32_t remote_barrier, double v) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];"
               :: "r"(remote), "l"(__double_as_longlong(v)), "r"(remote_barrier) : "memory");
}

__device__ __forceinline__ void ExpectBytes(uint64_t* barrier, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" :: "r"(SharedAddress(barrier)), "r"(bytes)
               : "memory");
}

// Whether a wait that began at *start (0: now) has run out.  Out of line: a wait
// comes here only after thousands of polls, and the polls are on the way to the
// next iteration (inline, solves of one or a few chunks took 2 % longer).
__device__ __noinline__ bool WaitExpired(unsigned long long* start, unsigned long long limit_ns,
                                         const unsigned long long* longest) {
  unsigned long long now;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(now));
  if (*start == 0) *start = now;
  return now - *start >= limit_ns && now - *start >= limit_ns + kWaitNsPerEntry * LoadAcquire(longest);
}

__device__ __forceinline__ void StoreRemote(uint32_t remote, unsigned long long v) {
  asm volatile("st.shared::cluster.u64 [%0], %1;" :: "r"(remote), "l"(v) : "memory");
}

// False when the barrier's phase did not end within the limit.
__device__ __forceinline__ bool WaitPhase(uint64_t* barrier, unsigned parity, const unsigned long long* longest) {
  const uint32_t at = SharedAddress(barrier);
  unsigned long long start = 0;
  for (unsigned polls = 0;;) {
    unsigned ended;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}" : "=r"(ended) : "r"(at), "r"(parity) : "memory");
    if (ended) return true;
    if (++polls >= kFreePolls && WaitExpired(&start, kOwnWaitNs, longest)) return false;
  }
}

// Shared memory of a block.
struct alignas(16) SolveShared {
  double totals[2][2];                                         // [reduction parity][dot]
  uint64_t barrier[2];                                         // lane sums of a group have arrived
  // The reduction after which a block of the cluster first gave up (none: all
  // ones); that block writes it into every block of the cluster.
  volatile unsigned long long first_dead;
  int widths[kTreeTerms];
  int abort;  // this block gives up
  int leave;  // another one gave up a reduction ago
};

// A block's part in a reduction to which it adds nothing, without a wait for
// other clusters (see the end of the kernel): `group_count` groups of rounds
// have been folded before, and `reduction` is its number.
__device__ __noinline__ void Farewell(unsigned char* smem, unsigned long long* arrived, TaggedSum* partial,
                                      const unsigned long long* longest, int64_t chunks, int group_rounds,
                                      unsigned group_count, unsigned long long reduction, int dots) {
  SolveShared& sh = *reinterpret_cast<SolveShared*>(smem);
  double* lanes = reinterpret_cast<double*>(smem + sizeof(SolveShared));
  const int64_t clusters = gridDim.x / kClusterBlocks;
  const int64_t mine = blockIdx.x / kClusterBlocks;
  const int64_t rounds = (chunks - mine + clusters - 1) / clusters;
  const int rank = static_cast<int>(cg::this_cluster().block_rank());
  const bool solo = chunks == 1;
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int rq = dots == 2 ? warp >> 1 : warp;
  const int d = dots == 2 ? warp & 1 : 0;
  const int parity = static_cast<int>(reduction & 1);
  __syncthreads();
  for (int64_t round = 0; round < rounds; round += group_rounds, ++group_count) {
    const int q = static_cast<int>(rounds - round < group_rounds ? rounds - round : group_rounds);
    const bool last = round + q == rounds;
    const unsigned gp = group_count & 1;
    if (last && !solo && threadIdx.x == 0) {
      // after what thread 0 may have told the cluster's blocks
      __threadfence();
      atomicAdd(arrived + mine * kFlagStride, 1ull);
    }
    if (warp < q * dots) {
      const uint32_t slot =
          SharedAddress(lanes + ((gp * group_rounds + rq) * 2 + d) * kTreeLanes + kWarp * rank + lane);
      const uint32_t barrier = SharedAddress(&sh.barrier[gp]);
      for (int k = 0; k < (solo ? kClusterBlocks : 1); ++k) {
        StoreCounted(RemoteAddress(slot, k), RemoteAddress(barrier, k), 0.0);
      }
    }
    if (solo) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    if (solo || rank == 0) {
      if (threadIdx.x == 0) {
        ExpectBytes(&sh.barrier[gp], static_cast<unsigned>(sizeof(double) * kTreeLanes) * dots * q);
      }
      if (warp < q * dots) {
        WaitPhase(&sh.barrier[gp], (group_count >> 1) & 1, longest);
        if (lane == 0 && !solo) {
          StoreTagged(partial + (2 * parity + d) * chunks + mine + (round + rq) * clusters, 0.0, reduction);
        }
      }
    }
    if (solo) {
      asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    } else if (!last) {
      cg::this_cluster().sync();
    }
  }
}

// kOneRound: every cluster owns one chunk, one block per SM, and the matrices'
// rows stay in shared memory where they fit (latency counts); otherwise two
// blocks per SM (bytes in flight count; one block of 128 registers and eight
// entries in flight was 5 % slower at n = 262,144).
template <class TM, bool kOneRound>
__global__ void __launch_bounds__(kSolveThreads, kOneRound ? 1 : 2) PcgSolveKernel(const SolveArgs<TM> a) {
  extern __shared__ __align__(16) unsigned char pcg_smem[];
  SolveShared& sh = *reinterpret_cast<SolveShared*>(pcg_smem);
  constexpr int kRounds = kOneRound ? 1 : kGroupRounds;
  double* lanes = reinterpret_cast<double*>(pcg_smem + sizeof(SolveShared));  // [group parity][round][dot][tree lane]
  double* terms = lanes + 2 * kRounds * 2 * kTreeLanes;                       // [group parity][round][dot][warp][lane]
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank());
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  const int64_t clusters = gridDim.x / kClusterBlocks;
  const int64_t mine = blockIdx.x / kClusterBlocks;
  const bool solo = a.chunks == 1;
  const int64_t in_chunk = static_cast<int64_t>(kTreeLanes) * warp + kWarp * rank + lane;
  const int64_t n = a.n;
  const int64_t rounds = (a.chunks - mine + clusters - 1) / clusters;
  unsigned group_count = 0;        // groups of rounds folded so far
  unsigned long long reduction = 0;  // number of the running reduction, from 1
  bool aborted = false;
  int64_t walk = 0;  // entries this thread walks per reduction, at most

  if (threadIdx.x == 0) {
    for (int i = 0; i < 2; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(SharedAddress(&sh.barrier[i])) : "memory");
    }
    sh.first_dead = ~0ull;
    sh.abort = 0;
    sh.leave = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }

  // the rows this thread owns (kOneRound), or where to find them
  RowRef<double> row_a{nullptr, nullptr, 1, 0, 0};
  RowRef<TM> row_m{nullptr, nullptr, 1, 0, 0};
  if constexpr (kOneRound) {
    const int64_t row = mine * kTreeChunk + in_chunk;
    int64_t first_a;
    int64_t first_m;
    bool dense;
    const int wa = SliceWidth(a.a, row, n, &first_a, &row_a.len, &dense);
    const int wm = SliceWidth(a.m, row, n, &first_m, &row_m.len, &dense);
    walk = row_a.len > row_m.len ? row_a.len : row_m.len;
    constexpr int kEntryA = sizeof(double) + sizeof(int32_t);
    constexpr int kEntryM = sizeof(TM) + sizeof(int32_t);
    // bytes of the 16 warps' slices (saturated: long rows never fit)
    if (lane == 0) {
      const long long bytes = static_cast<long long>(kWarp) * (static_cast<long long>(wa) * kEntryA +
                                                               static_cast<long long>(wm) * kEntryM);
      sh.widths[warp] = static_cast<int>(bytes < (1 << 20) ? (bytes + 15) / 16 * 16 : (1 << 20));
    }
    __syncthreads();
    int before = 0;
    int total = 0;
    for (int w = 0; w < kTreeTerms; ++w) {
      before += w < warp ? sh.widths[w] : 0;
      total += sh.widths[w];
    }
    if (total <= a.room) {
      unsigned char* base = reinterpret_cast<unsigned char*>(terms + 2 * kRounds * 2 * kTreeTerms * kWarp) + before;
      double* va = reinterpret_cast<double*>(base);
      TM* vm = reinterpret_cast<TM*>(va + static_cast<size_t>(wa) * kWarp);
      int32_t* ia = reinterpret_cast<int32_t*>(vm + static_cast<size_t>(wm) * kWarp);
      int32_t* im = ia + static_cast<size_t>(wa) * kWarp;
      for (int e = 0; e < row_a.len; ++e) {
        ia[e * kWarp + lane] = a.a.idx[first_a + e];
        va[e * kWarp + lane] = a.a.val[first_a + e];
      }
      for (int e = 0; e < row_m.len; ++e) {
        im[e * kWarp + lane] = a.m.idx[first_m + e];
        vm[e * kWarp + lane] = a.m.val[first_m + e];
      }
      row_a = RowRef<double>{ia + lane, va + lane, kWarp, row_a.len, wa};
      row_m = RowRef<TM>{im + lane, vm + lane, kWarp, row_m.len, wm};
    } else {
      const int64_t slice = row >> 5;
      if (slice * kWarp < n) {
        SliceRows(a.a, slice, n, lane);
        SliceRows(a.m, slice, n, lane);
        __syncwarp();
        if (row < n) {
          row_a = FindRow(a.a, row);
          row_m = FindRow(a.m, row);
          row_a.width = wa;
          row_m.width = wm;
        }
      }
    }
  } else {
    int64_t walk_m = 0;
    for (int64_t c = mine; c < a.chunks; c += clusters) {
      const int64_t first = c * kTreeChunk + in_chunk - lane;
      if (first < n) {
        walk += SliceRows(a.a, first >> 5, n, lane);
        walk_m += SliceRows(a.m, first >> 5, n, lane);
      }
    }
    walk = walk > walk_m ? walk : walk_m;
    __syncwarp();
  }
  if (walk > kShortWalk) atomicMax(a.longest, static_cast<unsigned long long>(walk));
  const auto a_row = [&](int64_t row) {
    if constexpr (kOneRound) {
      return row_a;
    } else {
      return FindRow(a.a, row);
    }
  };
  const auto m_row = [&](int64_t row) {
    if constexpr (kOneRound) {
      return row_m;
    } else {
      return FindRow(a.m, row);
    }
  };
  cluster.sync();  // the barriers are initialised

  // Runs body(row, d0, d1) for every row this thread owns and reduces d0 (and
  // d1 when dots == 2) over all rows with the canonical tree into t0, t1; what
  // the bodies wrote is visible to every block afterwards.
  auto reduce = [&](int dots, auto body, double& t0, double& t1) {
    ++reduction;
    const int parity = static_cast<int>(reduction & 1);
    int q = 0;
    int64_t group_first = mine;
    for (int64_t round = 0; round < rounds; ++round) {
      const int64_t row = (mine + round * clusters) * kTreeChunk + in_chunk;
      double d0 = 0.0;  // a missing row adds +0.0 to a sum started at +0.0: no change
      double d1 = 0.0;
      if (row < n) body(row, d0, d1);
      const unsigned gp = group_count & 1;
      double* mine_at = terms + ((gp * kRounds + q) * 2 * kTreeTerms + warp) * kWarp + lane;
      mine_at[0] = d0;
      if (dots == 2) mine_at[kTreeTerms * kWarp] = d1;
      const bool last = round + 1 == rounds;
      if (++q == kRounds || last) {
        __syncthreads();
        if (last && !solo && threadIdx.x == kSolveThreads - 1) {
          // this block's vectors are written: announce them (beside the folding below)
          __threadfence();
          atomicAdd(a.arrived + mine * kFlagStride, 1ull);
        }
        if (warp < q * dots) {
          const int rq = dots == 2 ? warp >> 1 : warp;
          const int d = dots == 2 ? warp & 1 : 0;
          const double* from = terms + ((gp * kRounds + rq) * 2 + d) * kTreeTerms * kWarp + lane;
          double s = 0.0;
#pragma unroll
          for (int t = 0; t < kTreeTerms; ++t) s = Add(s, from[t * kWarp]);
          const uint32_t slot = SharedAddress(lanes + ((gp * kRounds + rq) * 2 + d) * kTreeLanes + kWarp * rank + lane);
          const uint32_t barrier = SharedAddress(&sh.barrier[gp]);
          if (solo) {
#pragma unroll
            for (int k = 0; k < kClusterBlocks; ++k) StoreCounted(RemoteAddress(slot, k), RemoteAddress(barrier, k), s);
          } else {
            StoreCounted(RemoteAddress(slot, 0), RemoteAddress(barrier, 0), s);
          }
        }
        if (solo) asm volatile("barrier.cluster.arrive.release;" ::: "memory");
        if (solo || rank == 0) {
          if (threadIdx.x == 0) {
            ExpectBytes(&sh.barrier[gp], static_cast<unsigned>(sizeof(double) * kTreeLanes) * dots * q);
          }
          if (warp < q * dots) {
            if (!WaitPhase(&sh.barrier[gp], (group_count >> 1) & 1, a.longest)) sh.abort = 1;
            const int rq = dots == 2 ? warp >> 1 : warp;
            const int d = dots == 2 ? warp & 1 : 0;
            const double* from = lanes + ((gp * kRounds + rq) * 2 + d) * kTreeLanes;
            double v[kClusterBlocks];
#pragma unroll
            for (int g = 0; g < kClusterBlocks; ++g) v[g] = from[kWarp * g + lane];
            const double s = FoldLanes(v);
            if (lane == 0) {
              if (solo) {
                sh.totals[parity][d] = s;
              } else {
                StoreTagged(a.partial + (2 * parity + d) * a.chunks + group_first + rq * clusters, s, reduction);
              }
            }
          }
        }
        ++group_count;
        group_first += clusters * q;
        q = 0;
        if (!last) cluster.sync();  // the next group but one reuses this group's lanes
      }
    }
    if (solo) {
      asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
      __syncthreads();
      t0 = sh.totals[parity][0];
      t1 = sh.totals[parity][1];
      aborted = sh.abort != 0 || sh.first_dead < reduction;
      return;
    }
    if (warp < dots) {
      const TaggedSum* sums = a.partial + (2 * parity + warp) * a.chunks;
      unsigned long long start = 0;
      double v[kClusterBlocks];
      bool lost = false;
#pragma unroll
      for (int g = 0; g < kClusterBlocks; ++g) {
        double s = 0.0;
        for (int64_t i = kWarp * g + lane; i < a.chunks; i += kTreeLanes) {
          TaggedSum t = LoadTagged(sums + i);
          for (unsigned polls = 0; t.tag != reduction && !lost; t = LoadTagged(sums + i)) {
            lost = ++polls >= a.free_polls && WaitExpired(&start, a.wait_ns, a.longest);
          }
          s = Add(s, t.sum);
        }
        v[g] = s;
      }
      if (lost) sh.abort = 1;
      __syncwarp();
      const double s = FoldLanes(v);
      if (lane == 0) sh.totals[parity][warp] = s;
    } else if (warp == 2) {
      for (int64_t c = lane; c < clusters; c += kWarp) {
        // The own cluster's blocks always arrive, dead or alive, and once they
        // have, what a dead one told this block is visible.
        const bool own = c == mine;
        unsigned long long start = 0;
        for (unsigned polls = 0;;) {
          const unsigned long long seen = LoadAcquire(a.arrived + c * kFlagStride);
          // a poisoned counter reads as full, but for the own cluster's
          if ((own ? seen & ~kPoison : seen) >= reduction * kClusterBlocks) {
            if (seen & kPoison) sh.abort = 1;
            break;
          }
          if (++polls >= (own ? kFreePolls : a.free_polls) &&
              WaitExpired(&start, own ? kOwnWaitNs : a.wait_ns, a.longest)) {
            sh.abort = 1;
            break;
          }
        }
        if (own && sh.first_dead < reduction) sh.leave = 1;
      }
    }
    __syncthreads();
    t0 = sh.totals[parity][0];
    t1 = sh.totals[parity][1];
    aborted = (sh.abort | sh.leave) != 0;
  };

  double t0 = 0.0;
  double t1 = 0.0;
  const bool writer = blockIdx.x == 0 && threadIdx.x == 0;
  // prologue: x = 0, r = b, z = M r, p = z
  reduce(2, [&](int64_t row, double& d0, double& d1) {
    const double ri = a.b[row];
    a.x[row] = 0.0;
    a.r[0][row] = ri;
    const double zi = RowDot<kOneRound>(m_row(row), [&](int32_t c) { return a.b[c]; });
    a.z[row] = zi;
    d0 = Mul(ri, ri);
    d1 = Mul(ri, zi);
  }, t0, t1);
  const double b_norm = __dsqrt_rn(t0);
  // The stop test error = sqrt(rr) / b_norm <= tolerance without the root and
  // the division while rr is clearly above: where nothing can over- or
  // underflow, both round within a few ulp, far less than the margin.
  const double tol = a.tolerance;
  const bool in_range = b_norm > 1e-100 && b_norm < 1e100 && (tol == 0.0 || (tol > 1e-40 && tol < 1e40));
  const double clear_above = Mul(Mul(Mul(tol, b_norm), Mul(tol, b_norm)), 1.000001);
  double r_z = t1;
  double beta = 0.0;
  double rr = t0;
  int64_t count = 1;
  int64_t status = 0;
  bool done = !(1 < a.max_iterations && 1.0 > tol);
  bool first = true;  // p = z on the first iteration, z + beta p afterwards
  int next_dots = 1;  // dots of the reduction that follows: two after step 1, where the recurrence may also break down
  int pb = 0;         // buffer that holds the current p (written in step 1)
  int rb = 0;         // buffer that holds the current r
  while (!done && !aborted) {
    // 1. the direction and A p
    const double* p_old = pb == 0 ? a.p[0] : a.p[1];
    double* p_new = pb == 0 ? a.p[1] : a.p[0];
    const auto direction = [&](int64_t i) {
      const double zi = a.z[i];
      return first ? zi : Add(zi, Mul(beta, p_old[i]));
    };
    reduce(1, [&](int64_t row, double& d0, double&) {
      // every load before the first store: a store would wait for its own row's loads
      const double z_own = a.z[row];
      const double p_own = first ? 0.0 : p_old[row];
      const double ap = RowDot<kOneRound>(a_row(row), [&](int32_t c) { return direction(c); });
      const double pi = first ? z_own : Add(z_own, Mul(beta, p_own));
      p_new[row] = pi;
      a.ap[row] = ap;
      d0 = Mul(pi, ap);
    }, t0, t1);
    next_dots = 2;
    if (aborted) break;
    pb ^= 1;
    first = false;
    const double den = t0;
    if (!isfinite(r_z) || !isfinite(den) || r_z == 0.0 || den == 0.0) {
      status = 2;
      break;
    }
    const double alpha = __ddiv_rn(r_z, den);
    if (!isfinite(alpha)) {
      status = 2;
      break;
    }
    // 2. the step, the residual and z = M r
    const double* r_old = rb == 0 ? a.r[0] : a.r[1];
    double* r_new = rb == 0 ? a.r[1] : a.r[0];
    const auto residual = [&](int64_t i) { return __dsub_rn(r_old[i], Mul(alpha, a.ap[i])); };
    reduce(2, [&](int64_t row, double& d0, double& d1) {
      const double x_own = a.x[row];
      const double p_own = p_new[row];
      const double r_own = r_old[row];
      const double ap_own = a.ap[row];
      const double zi = RowDot<kOneRound>(m_row(row), [&](int32_t c) { return residual(c); });
      const double ri = __dsub_rn(r_own, Mul(alpha, ap_own));
      a.x[row] = Add(x_own, Mul(alpha, p_own));
      r_new[row] = ri;
      a.z[row] = zi;
      d0 = Mul(ri, ri);
      d1 = Mul(ri, zi);
    }, t0, t1);
    next_dots = 1;
    if (aborted) break;
    rb ^= 1;
    rr = t0;
    double r_z_new = t1;
    bool finite = true;
    bool above = in_range && rr > clear_above && rr > 1e-200 && rr < 1e200;
    bool converged = false;
    if (!above) {
      const double error = __ddiv_rn(__dsqrt_rn(rr), b_norm);
      converged = error <= tol;
      finite = isfinite(error);
      above = error > tol;
    }
    const bool periodic = a.refresh_period > 0 && count % a.refresh_period == 0;
    if (converged || periodic) {
      // the true residual replaces the recurrence's
      reduce(1, [&](int64_t row, double& d0, double&) {
        const double ax = RowDot<kOneRound>(a_row(row), [&](int32_t c) { return a.x[c]; });
        const double ri = __dsub_rn(a.b[row], ax);
        r_new[row] = ri;
        d0 = Mul(ri, ri);
      }, t0, t1);
      if (aborted) break;
      rr = t0;
      const double error = __ddiv_rn(__dsqrt_rn(rr), b_norm);
      finite = isfinite(error);
      above = error > tol;
      reduce(1, [&](int64_t row, double& d0, double&) {
        const double zi = RowDot<kOneRound>(m_row(row), [&](int32_t c) { return r_new[c]; });
        a.z[row] = zi;
        d0 = Mul(r_new[row], zi);
      }, t0, t1);
      if (aborted) break;
      r_z_new = t0;
    }
    beta = converged ? 0.0 : __ddiv_rn(r_z_new, r_z);
    r_z = r_z_new;
    if (writer) a.history[count] = rr;
    ++count;
    if (!finite) {
      status = 3;
      done = true;
    } else if (!isfinite(beta)) {
      status = 2;
      done = true;
    } else {
      done = !(count < a.max_iterations && above);
    }
  }
  // epilogue: the true residual at exit
  if (!aborted) {
    reduce(next_dots, [&](int64_t row, double& d0, double&) {
      const double ax = RowDot<kOneRound>(a_row(row), [&](int32_t c) { return a.x[c]; });
      const double ri = __dsub_rn(a.b[row], ax);
      d0 = Mul(ri, ri);
    }, t0, t1);
    next_dots = 1;
  }
  if (blockIdx.x == 0) {
    __syncthreads();
    // the history's norms, from the squares the writer left
    for (int64_t i = 1 + threadIdx.x; i < count - 1; i += kSolveThreads) {
      a.history[i] = __ddiv_rn(__dsqrt_rn(a.history[i]), b_norm);
    }
    if (writer) {
      const double h = __ddiv_rn(__dsqrt_rn(t0), b_norm);
      if (count > 1) a.history[0] = 1.0;
      a.history[count - 1] = h;
      if (!isfinite(h)) {
        status = 3;
      } else if (h <= tol) {
        status = 1;
      }
      a.outcome->count = count;
      a.outcome->status = status;
      a.outcome->aborted = aborted ? 1 : 0;
    }
  }
  // No block leaves while a neighbour may still store to its shared memory.  All
  // blocks of a cluster take part in the same reductions, so that every block
  // that receives has waited for all that was sent to it.  A block that gives up
  // after reduction k tells its cluster and takes part in reduction k + 1 with
  // nothing to add (how many dots that one has follows from k); one that finds
  // itself told leaves after k + 1, where the whole cluster is by then, since
  // each block waits for its cluster's arrival.  A block that is done takes part
  // in one more reduction too, because another may have given up after the last
  // one.  Clusters leave one after another; the poisoned counter spares the
  // others their wait.
  if (!(solo ? sh.first_dead < reduction : sh.leave != 0)) {
    if (aborted && threadIdx.x == 0) {
      const uint32_t slot = SharedAddress(const_cast<unsigned long long*>(&sh.first_dead));
      for (int k = 0; k < kClusterBlocks; ++k) StoreRemote(RemoteAddress(slot, k), reduction);
      if (!solo) atomicOr(a.arrived + mine * kFlagStride, kPoison);
    }
    Farewell(pcg_smem, a.arrived, a.partial, a.longest, a.chunks, kRounds, group_count, reduction + 1, next_dots);
  }
  cluster.sync();
}

// Dynamic shared memory of a solve block: the double buffers of lane sums and terms follow SolveShared, then (one
// round) the matrices.
template <bool kOneRound>
constexpr size_t SolveBytes() {
  return sizeof(SolveShared) +
         sizeof(double) * 2 * (kOneRound ? 1 : kGroupRounds) * 2 * (kTreeLanes + kTreeTerms * kWarp);
}
constexpr size_t kBlockSharedBytes = 227 * 1024;  // what a block may use on sm_100

// Launch attributes of a solve: clusters of eight, all blocks resident at once.
struct SolveLaunch {
  cudaLaunchConfig_t config = {};
  cudaLaunchAttribute attributes[2] = {};

  SolveLaunch(cudaStream_t stream, size_t smem) {
    attributes[0].id = cudaLaunchAttributeClusterDimension;
    attributes[0].val.clusterDim.x = kClusterBlocks;
    attributes[0].val.clusterDim.y = 1;
    attributes[0].val.clusterDim.z = 1;
    attributes[1].id = cudaLaunchAttributeCooperative;
    attributes[1].val.cooperative = 1;
    config.attrs = attributes;
    config.numAttrs = 2;
    config.blockDim = dim3(kSolveThreads);
    config.gridDim = dim3(kClusterBlocks);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
  }
};

template <bool kOneRound>
constexpr size_t LaunchBytes() {
  return kOneRound ? kBlockSharedBytes : SolveBytes<false>();
}

std::atomic<int64_t> g_wait_ns{static_cast<int64_t>(kWaitNs)};  // the next solve's patience (SetNextPcgWait)

// Clusters of the solve kernel that fit on the current device at once (asked once per device).
template <class TM, bool kOneRound>
int64_t ResidentClusters(int device) {
  static std::mutex mutex;
  static std::map<int, int> known;
  std::lock_guard<std::mutex> lock(mutex);
  const auto it = known.find(device);
  if (it != known.end()) return it->second;
  const auto kernel = PcgSolveKernel<TM, kOneRound>;
  SPAI_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 static_cast<int>(LaunchBytes<kOneRound>())));
  SolveLaunch launch(nullptr, LaunchBytes<kOneRound>());
  launch.config.numAttrs = 1;  // the cluster shape alone decides residency
  int clusters = 0;
  SPAI_CUDA(cudaOccupancyMaxActiveClusters(&clusters, kernel, &launch.config));
  if (clusters < 1) throw CudaError("PCG: no cluster of the solve kernel fits on the device");
  known[device] = clusters;
  return clusters;
}

// One thread per row, entries in storage order (the reference's _row_dot).
template <class TM>
__global__ void SpmvKernel(CscView<TM> a, const double* __restrict__ x, double* __restrict__ y) {
  for (int64_t row = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; row < a.cols;
       row += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    double s = 0.0;
    for (int64_t k = a.ptr[row]; k < a.ptr[row + 1]; ++k) {
      s = Add(s, Mul(static_cast<double>(a.val[k]), x[a.idx[k]]));
    }
    y[row] = s;
  }
}

}  // namespace

void SetNextPcgWait(int64_t ns) { g_wait_ns.store(ns < 0 ? static_cast<int64_t>(kWaitNs) : ns); }

template <class TM>
void Spmv(Ctx& ctx, const DevCsc<TM>& a_rows, const double* x, double* y) {
  // algorithmic bytes: the matrix once, x once, y written once
  const double bytes = static_cast<double>(a_rows.nnz) * (sizeof(TM) + sizeof(int32_t)) +
                       static_cast<double>(a_rows.cols + 1) * sizeof(int64_t) + 16.0 * static_cast<double>(a_rows.cols);
  prof::Scope scope(ctx.stream, "pcg_spmv", bytes);
  SpmvKernel<TM><<<GridFor(a_rows.cols, 128), 128, 0, ctx.stream>>>(View(a_rows), x, y);
  SPAI_LAUNCH_CHECK();
}

template <class TM>
void RunPcg(Ctx& ctx, const DevCsc<double>& a, const DevCsc<TM>& m, const double* b, double* x,
            const PcgOptions& opt, PcgResult& result) {
  const int64_t n = a.cols;
  if (n <= 0) throw std::invalid_argument("PCG needs n > 0");
  if (n > kTreeChunk * kTreeChunk) throw std::invalid_argument("PCG supports at most 4096^2 rows");
  if (opt.max_iterations <= 0) throw std::invalid_argument("max_iterations must be positive");
  const int64_t chunks = CeilDiv(n, kTreeChunk);
  const int64_t slices = CeilDiv(n, kWarp);
  const cudaStream_t st = ctx.stream;
  // r, p (two of each), z, ap, the history and the chunk sums
  DevBuf<double> vectors, history;
  DevBuf<TaggedSum> partial;
  vectors.Reserve(static_cast<size_t>(6 * n), st);
  history.Reserve(static_cast<size_t>(opt.max_iterations), st);
  partial.Reserve(static_cast<size_t>(4 * chunks), st);
  // the sliced copies (at most twice the entries plus two per row, see SliceRows) and their slice offsets;
  // a matrix whose copy the device has no room for is read as it is
  DevBuf<int64_t> slice_at;
  DevBuf<int32_t> a_idx, m_idx;
  DevBuf<double> a_val;
  DevBuf<TM> m_val;
  slice_at.Reserve(static_cast<size_t>(2 * slices), st);
  const auto reserve_copy = [&](int64_t nnz, DevBuf<int32_t>& idx, auto& val) {
    const size_t room = static_cast<size_t>(2 * nnz + 2 * (n + kWarp));
    try {
      idx.Reserve(room, st);
      val.Reserve(room, st);
    } catch (const CudaError&) {
      cudaGetLastError();
      idx.Release();
      val.Release();
      CacheFlush(st);
    }
  };
  reserve_copy(a.nnz, a_idx, a_val);
  reserve_copy(m.nnz, m_idx, m_val);
  // two slice cursors, the longest walk and the outcome, zeroed
  struct Control {
    unsigned long long used[2];
    unsigned long long longest;
    SolveOutcome outcome;
  };
  DevBuf<Control> control;
  control.Reserve(1, st);
  SPAI_CUDA(cudaMemsetAsync(control.data(), 0, sizeof(Control), st));
  SPAI_CUDA(cudaMemsetAsync(partial.data(), 0, sizeof(TaggedSum) * static_cast<size_t>(4 * chunks), st));
  Control* c = control.data();
  SolveArgs<TM> args{};
  args.a = SolveMatrix<double>{a.ptr.data(), a.idx.data(), a.val.data(), slice_at.data(), a_idx.data(), a_val.data(),
                               &c->used[0]};
  args.m = SolveMatrix<TM>{m.ptr.data(), m.idx.data(), m.val.data(), slice_at.data() + slices, m_idx.data(),
                           m_val.data(), &c->used[1]};
  args.b = b;
  args.x = x;
  double* v = vectors.data();
  args.r[0] = v;
  args.r[1] = v + n;
  args.p[0] = v + 2 * n;
  args.p[1] = v + 3 * n;
  args.z = v + 4 * n;
  args.ap = v + 5 * n;
  args.history = history.data();
  args.partial = partial.data();
  args.outcome = &c->outcome;
  args.longest = &c->longest;
  args.wait_ns = static_cast<unsigned long long>(g_wait_ns.exchange(static_cast<int64_t>(kWaitNs)));
  args.free_polls = args.wait_ns == kWaitNs ? kFreePolls : 0;
  args.n = n;
  args.chunks = chunks;
  args.max_iterations = opt.max_iterations;
  args.refresh_period = opt.refresh_period;
  args.tolerance = opt.tolerance;
  // one chunk per cluster while the clusters that fit at once cover every chunk
  auto kernel = PcgSolveKernel<TM, true>;
  size_t smem = LaunchBytes<true>();
  int64_t clusters = ResidentClusters<TM, true>(ctx.device);
  if (clusters < chunks) {
    kernel = PcgSolveKernel<TM, false>;
    smem = LaunchBytes<false>();
    clusters = ResidentClusters<TM, false>(ctx.device);
  }
  args.room = static_cast<int>(kBlockSharedBytes - SolveBytes<true>());
  clusters = std::min(clusters, chunks);
  DevBuf<unsigned long long> arrived;
  const size_t flags = static_cast<size_t>(clusters * kFlagStride);
  arrived.Reserve(flags, st);
  SPAI_CUDA(cudaMemsetAsync(arrived.data(), 0, sizeof(unsigned long long) * flags, st));
  args.arrived = arrived.data();
  {
    prof::Scope scope(st, "pcg_solve", 0.0);
    SolveLaunch launch(st, smem);
    launch.config.gridDim = dim3(static_cast<unsigned>(clusters * kClusterBlocks));
    SPAI_CUDA(cudaLaunchKernelEx(&launch.config, kernel, args));
    SPAI_LAUNCH_CHECK();
  }
  static_assert(sizeof(SolveOutcome) <= 8 * sizeof(int64_t), "the outcome fits the pinned counts");
  SPAI_CUDA(cudaMemcpyAsync(ctx.host_counts, args.outcome, sizeof(SolveOutcome), cudaMemcpyDeviceToHost, st));
  result.history.assign(static_cast<size_t>(opt.max_iterations), 0.0);
  SPAI_CUDA(cudaMemcpyAsync(result.history.data(), history.data(), sizeof(double) * opt.max_iterations,
                            cudaMemcpyDeviceToHost, st));
  ctx.Sync();
  SolveOutcome outcome;
  std::memcpy(&outcome, ctx.host_counts, sizeof(outcome));
  if (outcome.aborted != 0) throw CudaError("PCG: the blocks of the solve stopped answering one another");
  const int64_t count = outcome.count;
  if (count < 1 || count > opt.max_iterations) throw CudaError("PCG returned an invalid iteration count");
  result.history.resize(static_cast<size_t>(count));
  result.status = outcome.status;
  // algorithmic bytes of the solve: per iteration A and M once plus the vector traffic (17 n doubles)
  const double per_iteration = static_cast<double>(a.nnz) * 12.0 + static_cast<double>(m.nnz) * (sizeof(TM) + 4) +
                               8.0 * 17.0 * static_cast<double>(n);
  prof::AddBytes("pcg_solve", per_iteration * static_cast<double>(count));
}

template void RunPcg<double>(Ctx&, const DevCsc<double>&, const DevCsc<double>&, const double*, double*,
                             const PcgOptions&, PcgResult&);
template void RunPcg<float>(Ctx&, const DevCsc<double>&, const DevCsc<float>&, const double*, double*,
                            const PcgOptions&, PcgResult&);
template void Spmv<double>(Ctx&, const DevCsc<double>&, const double*, double*);
template void Spmv<float>(Ctx&, const DevCsc<float>&, const double*, double*);

}  // namespace spai
