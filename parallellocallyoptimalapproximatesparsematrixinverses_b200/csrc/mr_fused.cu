// The fused, graph-captured Global MR iteration (mr_fused.cuh).
//
// Slot layouts (all in HBM, sized once per solver):
//   M    topk slots per column, rows ascending, count per column
//   M^T  two sets (the drop kernel reads one and writes the other), cap_mt
//        slots per row in arrival order, count per row
//   Z    cap_z slots per column, rows ascending (Z = Pr R keeps R's pattern)
// Z is never transposed: the drop kernel needs row j of Z only for column j,
// and forms it from the rows of M it has (M^T) and row j of A, with the same
// products in the same order as the residual kernel's column of R.  The
// residual kernel clears the M^T set the drop kernel has just read, so the
// next drop kernel fills it again from zero.

#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <memory>
#include <stdexcept>
#include <vector>

#include "colgroup.cuh"
#include "colkit.cuh"
#include "device.cuh"
#include "mr_fused.cuh"
#include "ops.cuh"
#include "profile.cuh"
#include "select.cuh"
#include "tree.cuh"

namespace spai {

void CountLaunches(int64_t count);

namespace {

constexpr int kGroupWarps = 2;      // warps per block of the drop and residual kernels on column groups
constexpr int kColumnWarps = 4;     // and of those that go column by column
constexpr int kDropWindowWords = 512;  // bitmap words of a drop column on its own: windows of 16,384 rows
constexpr int kDropWindowRows = kDropWindowWords * 32;
constexpr int kWindowWords = 1024;  // bitmap words of a residual column on its own: windows of 32,768 rows
constexpr int kWindowRows = kWindowWords * 32;
constexpr int kRowsCap = 1024;      // longest row list of one product column
constexpr int kMaxTopK = 32;
constexpr int kMaxGroupWords = 2048;  // windows of column groups: up to 65,536 rows (16-bit offsets)
constexpr int kDropRowsCap = 512;  // candidate rows of one drop column; also bounds Z's slots per column

// Overflow bits (FusedState::overflow).
constexpr int kOverflowMt = 1;      // a row of M^T exceeded cap_mt
constexpr int kOverflowRow = 2;     // row j of R had more entries than its hash takes
constexpr int kOverflowSide = 4;    // a drop column's merged rows exceeded kDropCap

// Stop codes (FusedState::stop).
constexpr int kRunning = 0;
constexpr int kConverged = 1;
constexpr int kBreakdown = 2;
constexpr int kIterationLimit = 3;
constexpr int kOverflowStop = 4;
constexpr int kScatteredStop = 5;  // too few column groups fit: the host goes on column by column

struct FusedRow {
  int64_t iteration;
  double residual_norm;
  double density_m;
  double density_direction;
};

// Device-resident loop state.
struct FusedState {
  double alpha;                 // step length of the next iteration
  int64_t iteration;            // last history row appended
  int64_t parity;               // M^T set the next drop kernel reads
  unsigned long long nnz_m;     // entries of M written by this iteration's drop kernel
  unsigned long long nnz_z;     // entries of Z written by this iteration's residual kernel
  unsigned long long nnz_dir;   // entries of the Z this iteration's step used (its history row's direction)
  unsigned long long last_nnz_m;  // the last iteration's counts (read by the host when profiling)
  unsigned long long last_nnz_z;
  int32_t overflow;
  int32_t stop;
  unsigned int arrive;          // blocks of the decide kernel that are done
  unsigned int unfit;           // groups of this iteration's two kernels that went column by column
  int64_t bodies;               // loop-body executions
  int64_t last_unfit;           // the last step's count (batched runs)
};

template <class T>
struct FusedArgs {
  int64_t n;
  int topk;
  int cap_z;
  int cap_mt;
  int ell;  // ELL slots of A (multiple of 4)
  int m_hash_slots;   // residual kernel: M(:, j)
  int z_hash_slots;   // residual kernel: Z(:, j)
  int d_mt_slots;     // drop kernel: M(j, :)
  int d_r_slots;      // drop kernel: R(j, :)
  int words;           // 32-row words of the column groups' windows (0: every column on its own)
  int64_t bandwidth;   // largest |i - k| over the entries of A
  int64_t unfit_limit;    // groups of an iteration's two kernels that may go column by column
  size_t drop_bytes;      // shared memory of a warp
  size_t residual_bytes;
  int64_t max_iterations;
  double tolerance;
  const int32_t* a_cols_ell;
  const int32_t* a_rows_ell;
  const T* a_rows_ell_val;
  const T* pr;
  int32_t* m_rows;
  T* m_vals;
  int32_t* m_cnt;
  int32_t* mt_cols[2];
  T* mt_vals[2];
  int32_t* mt_cnt[2];
  int32_t* z_rows;
  T* z_vals;
  int32_t* z_cnt;
  double* sq;          // per-column sum of squares of R
  double* tt;          // per-column ||Pr A Z(:, j)||^2
  double* bt;          // per-column <Z(:, j), Pr A Z(:, j)>
  double* chunk;       // 3 * chunks
  const double* alpha; // step length of every column (batched runs), or null: state->alpha
  FusedRow* history;   // max_iterations + 1 rows
  FusedState* state;
};

// ---------------------------------------------------------------------------
// Drop kernel: per column j, S = 0.5 (U(:, j) + U(j, :)^T) with U = M + alpha Z.
//
// M(:, j) and Z(:, j) are read from the column's sorted slots (binary
// searches); two small hashes in shared memory hold M(j, :) (row j of M, from
// M^T) and R(j, :).  Row j of R is formed
// here: for the entries k of row j of A in ascending order, every entry
// M(k, i) of row k of M adds A(j, k) M(k, i) to R(j, i) -- for each i the
// terms arrive in ascending k, exactly the sum the residual kernel forms for
// R(j, i) in column i.  The candidate rows i of S(:, j) (the rows of M(:, j)
// and Z(:, j), the keys of the two hashes, and j) are marked in a window
// bitmap and read back in ascending order; each one's U(i, j), U(j, i) and
// S(i, j) come from those lookups, with
// the union's and the symmetrisation's arithmetic (UnionPadded,
// SymmetrizeDropKernel).  Exact zeros of U are not pruned here: an entry that
// is zero on both sides gives S(i, j) = 0, which the drop rule removes, and a
// zero on one side gives the same half sum as an absent one, so the kept
// entries and their order are the unfused kernels'.

// Returns the slot of key (inserted when absent: *fresh), or -1 when the table is full.
__device__ __forceinline__ int FindOrInsert(int32_t* keys, int bits, int32_t key, bool* fresh) {
  const uint32_t mask = (1u << bits) - 1u;
  uint32_t h = (static_cast<uint32_t>(key) * 2654435761u) >> (32 - bits);
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    const int32_t old = atomicCAS(&keys[h], kEmpty, key);
    if (old == kEmpty) {
      *fresh = true;
      return static_cast<int>(h);
    }
    if (old == key) {
      *fresh = false;
      return static_cast<int>(h);
    }
    h = (h + 1u) & mask;
  }
  *fresh = false;
  return -1;
}

__device__ __forceinline__ int FindSlot(const int32_t* keys, int bits, int32_t key) {
  const uint32_t mask = (1u << bits) - 1u;
  uint32_t h = (static_cast<uint32_t>(key) * 2654435761u) >> (32 - bits);
  for (uint32_t probe = 0; probe <= mask; ++probe) {
    const int32_t k = keys[h];
    if (k == key) return static_cast<int>(h);
    if (k == kEmpty) return -1;
    h = (h + 1u) & mask;
  }
  return -1;
}

// Entries of one row of M^T a lane holds while row j of R is formed (cap_mt <= 4 * kMaxTopK).
constexpr int kMtPerLane = 4;
static_assert(4 * kMaxTopK <= kMtPerLane * kWarp, "a row of M^T must fit the lanes' registers");

// 32-row words of the bitmaps' summaries, in whole warps.
constexpr int kDropSummary = (kDropWindowWords + kWarp * kWarp - 1) / (kWarp * kWarp) * kWarp;
constexpr int kResidualSummary = (kWindowWords + kWarp * kWarp - 1) / (kWarp * kWarp) * kWarp;

template <class T>
__host__ __device__ size_t DropWarpBytes(int own, int mt, int r) {
  return Round16(static_cast<size_t>(kDropWindowWords) * 4) + Round16(static_cast<size_t>(kDropSummary) * 4) +
         Round16(static_cast<size_t>(kDropRowsCap) * 2) +
         Round16(static_cast<size_t>(mt + r) * 4) + Round16(static_cast<size_t>(mt + r) * sizeof(T)) +
         Round16(static_cast<size_t>(own) * 4) + Round16(static_cast<size_t>(own) * sizeof(T)) +
         Round16(kDropCap * sizeof(T)) + Round16(kDropCap * sizeof(int32_t));
}

// The drop decision of one column and its survivors: DecideDrops' rules
// (select.cuh) on `count` nonzero values vals[r] of rows row_of(r), NB
// entries per lane.  The relative threshold needs the sequential sum of
// squares only when the smallest magnitude could lie below it; the cut of the
// top-k is found by bisection on the magnitudes' bits, ties going to the
// larger row.
template <class T, int NB, class Row>
__device__ __forceinline__ int DropAndWriteIn(const FusedArgs<T>& a, Row row_of, const T* vals, int count, int64_t j,
                                              int64_t other, int lane, int* overflow) {
  using Key = typename MagnitudeOf<T>::Key;
  T val[NB];
  Key key[NB];  // 0: dropped or absent
  int32_t row[NB];
  unsigned diagonal = 0u;
  Key largest = 0;
  Key smallest = ~Key(0);
#pragma unroll
  for (int t = 0; t < NB; ++t) {
    const int r = t * kWarp + lane;
    val[t] = r < count ? vals[r] : T(0);
    row[t] = r < count ? row_of(r) : -1;
    key[t] = MagnitudeBits(val[t]);
    if (key[t] != 0) {
      largest = key[t] > largest ? key[t] : largest;
      smallest = key[t] < smallest ? key[t] : smallest;
    }
    if (static_cast<int64_t>(row[t]) == j) diagonal |= 1u << t;
  }
  // thr = eps sqrt(sum v^2) <= eps sqrt(256) max|v| (1 + rounding): below 17 eps max|v|
  const Key top = LargestKey(largest);
  const Key bottom = SmallestKey(smallest);
  const double hi = MagnitudeValue(top);
  const double lo = MagnitudeValue(bottom);
  int kept = count;
  if (!(hi < 1e150 && lo > 17.0 * kDblEps * hi)) {
    double thr = 0.0;
    if (lane == 0) {
      double sq = 0.0;
#pragma unroll 1
      for (int r = 0; r < count; ++r) {
        const double v = static_cast<double>(vals[r]);
        sq = Add(sq, Mul(v, v));
      }
      thr = Mul(kDblEps, sqrt(sq));
    }
    thr = __shfl_sync(0xffffffffu, thr, 0);
    kept = 0;
#pragma unroll
    for (int t = 0; t < NB; ++t) {
      const bool keep = ((diagonal >> t) & 1u) != 0u || fabs(static_cast<double>(val[t])) >= thr;
      if (!keep) key[t] = 0;
      kept += __popc(__ballot_sync(0xffffffffu, key[t] != 0));
    }
  }
  if (kept > a.topk) {
    // the diagonal stays; of the other candidates the `wanted` largest (|v|, row)
    const bool has_diagonal = __any_sync(0xffffffffu, diagonal != 0u);
    const int wanted = a.topk - (has_diagonal ? 1 : 0);
    Key cand[NB];
#pragma unroll
    for (int t = 0; t < NB; ++t) cand[t] = ((diagonal >> t) & 1u) != 0u ? Key(0) : key[t];
    Key below = bottom;   // at least `wanted` candidates are >= below
    Key above = top + 1;  // fewer than `wanted` are >= above
    int at_above = 0;
    if (wanted <= 0) below = ~Key(0);
#pragma unroll 1
    while (wanted > 0) {
      const Key mid = below + ((above - below) >> 1);
      int n = 0;
#pragma unroll
      for (int t = 0; t < NB; ++t) n += __popc(__ballot_sync(0xffffffffu, cand[t] >= mid));
      if (n == wanted) {
        below = mid;
        break;
      }
      if (n > wanted) {
        below = mid;
      } else {
        above = mid;
        at_above = n;
      }
      if (above - below <= 1) {
        // several candidates share the cut's magnitude: the larger rows win
        int need = wanted - at_above;
#pragma unroll
        for (int t = NB - 1; t >= 0; --t) {
          unsigned equal = __ballot_sync(0xffffffffu, cand[t] == below);
#pragma unroll 1
          for (int surplus = __popc(equal) - need; surplus > 0; --surplus) {
            if (lane == __ffs(equal) - 1) cand[t] = 0;
            equal &= equal - 1u;
          }
          need -= __popc(equal);
        }
        break;
      }
    }
#pragma unroll
    for (int t = 0; t < NB; ++t) {
      const bool keep = ((diagonal >> t) & 1u) != 0u || (cand[t] != 0 && cand[t] >= below);
      if (!keep) key[t] = 0;
    }
  }
  int32_t* out_rows = a.m_rows + j * a.topk;
  T* out_vals = a.m_vals + j * a.topk;
  int at = 0;
#pragma unroll
  for (int t = 0; t < NB; ++t) {
    const bool mine = key[t] != 0;
    const unsigned mask = __ballot_sync(0xffffffffu, mine);
    if (mine) {
      const int o = at + __popc(mask & LaneMaskBelow());
      out_rows[o] = row[t];
      out_vals[o] = val[t];
      const int slot = atomicAdd(&a.mt_cnt[other][row[t]], 1);
      if (slot < a.cap_mt) {
        a.mt_cols[other][static_cast<int64_t>(row[t]) * a.cap_mt + slot] = static_cast<int32_t>(j);
        a.mt_vals[other][static_cast<int64_t>(row[t]) * a.cap_mt + slot] = val[t];
      } else {
        *overflow |= kOverflowMt;
      }
    }
    at += __popc(mask);
  }
  if (lane == 0) a.m_cnt[j] = at;
  return at;
}

// The same for any count <= kDropCap.
template <class T, class Row>
__device__ __forceinline__ int DropAndWrite(const FusedArgs<T>& a, Row row_of, const T* vals, int count, int64_t j,
                                            int64_t other, int lane, int* overflow) {
  static_assert(kDropCap == 8 * kWarp, "eight entries per lane hold the longest column");
  if (count <= 2 * kWarp) return DropAndWriteIn<T, 2>(a, row_of, vals, count, j, other, lane, overflow);
  if (count <= 4 * kWarp) return DropAndWriteIn<T, 4>(a, row_of, vals, count, j, other, lane, overflow);
  return DropAndWriteIn<T, 8>(a, row_of, vals, count, j, other, lane, overflow);
}

// A warp's shared memory while it goes column by column, and what holds for all of its columns.
template <class T>
struct DropSlab {
  uint32_t* bm;
  uint32_t* summary;
  uint16_t* rows;
  int32_t* keys;  // the two tables, one after another
  T* vals;
  int32_t* mr;  // M(:, j) then Z(:, j): rows
  T* mv;        // and values
  T* s_vals;    // the nonzero entries of S(:, j)
  int32_t* s_rows;
  int b_mt;
  int b_r;
  int64_t parity;
  T alpha;

  // clear: whether the window has to be cleared.
  __device__ __forceinline__ DropSlab(const FusedArgs<T>& a, unsigned char* base, bool clear, int lane) {
    const int table = a.d_mt_slots + a.d_r_slots;
    const int own = a.topk + a.cap_z;
    bm = reinterpret_cast<uint32_t*>(base);
    base += Round16(static_cast<size_t>(kDropWindowWords) * 4);
    summary = reinterpret_cast<uint32_t*>(base);
    base += Round16(static_cast<size_t>(kDropSummary) * 4);
    rows = reinterpret_cast<uint16_t*>(base);
    base += Round16(static_cast<size_t>(kDropRowsCap) * 2);
    keys = reinterpret_cast<int32_t*>(base);
    base += Round16(static_cast<size_t>(table) * 4);
    vals = reinterpret_cast<T*>(base);
    base += Round16(static_cast<size_t>(table) * sizeof(T));
    mr = reinterpret_cast<int32_t*>(base);
    base += Round16(static_cast<size_t>(own) * 4);
    mv = reinterpret_cast<T*>(base);
    base += Round16(static_cast<size_t>(own) * sizeof(T));
    s_vals = reinterpret_cast<T*>(base);
    base += Round16(kDropCap * sizeof(T));
    s_rows = reinterpret_cast<int32_t*>(base);
    b_mt = Log2(a.d_mt_slots);
    b_r = Log2(a.d_r_slots);
    parity = a.state->parity;
    alpha = static_cast<T>(a.state->alpha);
    if (clear) {
      __syncwarp();
      ClearWords(bm, kDropWindowWords, lane);
      ClearWords(summary, kDropSummary, lane);
      __syncwarp();
    }
  }
};

// One column on its own; its window is clear before and after.  Returns the
// overflow bits; *written grows by the column's entries.  kUnroll: of the short
// loops; 1 inside the group kernels, whose registers they would raise.
template <class T, int kUnroll>
__device__ __forceinline__ int DropColumn(const FusedArgs<T>& a, const DropSlab<T>& slab, int64_t j,
                                          unsigned long long* written_out) {
  const int lane = threadIdx.x & 31;
  const int table = a.d_mt_slots + a.d_r_slots;
  uint32_t* bm = slab.bm;
  uint32_t* summary = slab.summary;
  uint16_t* rows = slab.rows;
  int32_t* keys = slab.keys;
  int32_t* mr = slab.mr;
  int32_t* zr = mr + a.topk;
  T* mv = slab.mv;
  T* zv = mv + a.topk;
  T* s_vals = slab.s_vals;
  int32_t* s_rows = slab.s_rows;
  int32_t* k_mt = keys;
  int32_t* k_r = k_mt + a.d_mt_slots;
  T* v_mt = slab.vals;
  T* v_r = v_mt + a.d_mt_slots;
  const int b_mt = slab.b_mt;
  const int b_r = slab.b_r;
  const int r_limit = a.d_r_slots / 2;  // distinct keys of R(j, :) the table takes
  const int64_t parity = slab.parity;
  const int64_t other = parity ^ 1;
  const T alpha = a.alpha != nullptr ? static_cast<T>(a.alpha[j]) : slab.alpha;
  int overflow = 0;
  {
    const int nm = a.m_cnt[j];
    const int nz = a.z_cnt[j];
    const int nmt = a.mt_cnt[parity][j];
    if (nmt > a.cap_mt) {
      return kOverflowMt;
    }
    ClearTable(keys, table, lane);
    // M(:, j) and Z(:, j) into shared memory (sorted by row), then M(j, :) into its hash
#pragma unroll kUnroll
    for (int e = lane; e < nm; e += kWarp) {
      mr[e] = a.m_rows[j * a.topk + e];
      mv[e] = a.m_vals[j * a.topk + e];
    }
#pragma unroll kUnroll
    for (int e = lane; e < nz; e += kWarp) {
      zr[e] = a.z_rows[j * a.cap_z + e];
      zv[e] = a.z_vals[j * a.cap_z + e];
    }
    __syncwarp();
    const int32_t* mtc = a.mt_cols[parity] + j * a.cap_mt;
    const T* mtv = a.mt_vals[parity] + j * a.cap_mt;
    int32_t lo = static_cast<int32_t>(j);
    int32_t hi = static_cast<int32_t>(j);
    bool fresh;
    // M(:, j) and Z(:, j) are sorted: their ends bound the window, and lookups are binary searches
    if (nm > 0) {
      lo = min(lo, mr[0]);
      hi = max(hi, mr[nm - 1]);
    }
    if (nz > 0) {
      lo = min(lo, zr[0]);
      hi = max(hi, zr[nz - 1]);
    }
#pragma unroll kUnroll
    for (int e = lane; e < nmt; e += kWarp) {
      const int at = FindOrInsert(k_mt, b_mt, mtc[e], &fresh);
      v_mt[at] = mtv[e];
      lo = min(lo, mtc[e]);
      hi = max(hi, mtc[e]);
    }
    // R(j, :) = e_j^T - A(j, :) M: terms in ascending k for every column i.  Lane u holds
    // entry u of row j of A and the length of row k_u of M^T; the rows of M^T are loaded
    // one step ahead of the step that adds them, so their loads overlap.
    int32_t k_lane = -1;
    T a_lane = T(0);
    int nk_lane = 0;
    if (lane < a.ell) {
      k_lane = a.a_rows_ell[j * a.ell + lane];
      if (k_lane >= 0) {
        a_lane = a.a_rows_ell_val[j * a.ell + lane];
        nk_lane = a.mt_cnt[parity][k_lane];
      }
    }
    int r_keys = 0;
    bool r_full = __any_sync(0xffffffffu, nk_lane > a.cap_mt);
    int32_t cur_i[kMtPerLane];
    T cur_v[kMtPerLane];
    int32_t next_i[kMtPerLane];
    T next_v[kMtPerLane];
    auto load_row = [&](int u, int32_t (&ii)[kMtPerLane], T (&vv)[kMtPerLane]) {
      const int32_t k = __shfl_sync(0xffffffffu, k_lane, u);
      const int nk = r_full ? 0 : __shfl_sync(0xffffffffu, nk_lane, u);
      const int32_t* kc = a.mt_cols[parity] + static_cast<int64_t>(k) * a.cap_mt;
      const T* kv = a.mt_vals[parity] + static_cast<int64_t>(k) * a.cap_mt;
#pragma unroll
      for (int q = 0; q < kMtPerLane; ++q) {
        const int e = q * kWarp + lane;
        ii[q] = -1;
        vv[q] = T(0);
        if (k >= 0 && e < nk) {
          ii[q] = kc[e];
          vv[q] = kv[e];
        }
      }
    };
    load_row(0, cur_i, cur_v);
#pragma unroll 1
    for (int u = 0; u < a.ell && !r_full; ++u) {
      const int32_t k = __shfl_sync(0xffffffffu, k_lane, u);
      const int nk = __shfl_sync(0xffffffffu, nk_lane, u);
      const T a_jk = __shfl_sync(0xffffffffu, a_lane, u);
      if (u + 1 < a.ell) load_row(u + 1, next_i, next_v);
      if (k >= 0) {  // warp-uniform
#pragma unroll
        for (int q = 0; q < kMtPerLane; ++q) {
          if (q * kWarp < nk) {  // warp-uniform
            const int e = q * kWarp + lane;
            bool is_new = false;
            bool lost = false;
            if (e < nk) {
              const int32_t i = cur_i[q];
              const T prod = Mul(a_jk, cur_v[q]);
              const int at = FindOrInsert(k_r, b_r, i, &is_new);
              if (at < 0) {
                lost = true;
              } else {
                // a column i appears once in row k of M: no two lanes share a slot here
                v_r[at] = is_new ? prod : Add(v_r[at], prod);
                lo = min(lo, i);
                hi = max(hi, i);
              }
            }
            r_keys += __popc(__ballot_sync(0xffffffffu, is_new));
            if (__any_sync(0xffffffffu, lost)) r_full = true;
          }
        }
        __syncwarp();
        if (r_keys > r_limit) r_full = true;
      }
#pragma unroll
      for (int q = 0; q < kMtPerLane; ++q) {
        cur_i[q] = next_i[q];
        cur_v[q] = next_v[q];
      }
    }
    if (r_full) {
      return kOverflowRow;
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    // S(:, j) in row order, one window of kDropWindowRows rows at a time
    int count = 0;
    bool too_long = false;
#pragma unroll 1
    for (int32_t seg_lo = lo; seg_lo <= hi; seg_lo += kDropWindowRows) {
      const int32_t seg_hi = hi - seg_lo < kDropWindowRows ? hi : seg_lo + (kDropWindowRows - 1);
      const int words = (seg_hi - seg_lo) / 32 + 1;
      if (lane == 0 && j >= seg_lo && j <= seg_hi) MarkRow(bm, summary, static_cast<int>(j - seg_lo));
#pragma unroll kUnroll
      for (int e = lane; e < nm; e += kWarp) {
        if (mr[e] >= seg_lo && mr[e] <= seg_hi) MarkRow(bm, summary, mr[e] - seg_lo);
      }
#pragma unroll kUnroll
      for (int e = lane; e < nz; e += kWarp) {
        if (zr[e] >= seg_lo && zr[e] <= seg_hi) MarkRow(bm, summary, zr[e] - seg_lo);
      }
#pragma unroll kUnroll
      for (int t = lane; t < table; t += kWarp) {
        const int32_t key = keys[t];
        if (key != kEmpty && key >= seg_lo && key <= seg_hi) MarkRow(bm, summary, key - seg_lo);
      }
      __syncwarp();
      const int found = DrainRows(bm, summary, SummaryWords(words), rows, lane);
      if (count + found > kDropCap || found > kDropRowsCap) {
        too_long = true;
        break;
      }
#pragma unroll 1
      for (int r0 = 0; r0 < found; r0 += kWarp) {
        const int r = r0 + lane;
        bool emit = false;
        int32_t i = 0;
        T v = T(0);
        if (r < found) {
          i = seg_lo + static_cast<int32_t>(rows[r]);
          // U(i, j) = M(i, j) (+) alpha Z(i, j)
          int pm = LowerBoundShared(mr, nm, i);
          int pz = LowerBoundShared(zr, nz, i);
          pm = pm < nm && mr[pm] == i ? pm : -1;
          pz = pz < nz && zr[pz] == i ? pz : -1;
          const bool own = pm >= 0 || pz >= 0;
          T u_own = T(0);
          if (pm >= 0 && pz >= 0) {
            u_own = Add(mv[pm], Mul(alpha, zv[pz]));
          } else if (pm >= 0) {
            u_own = Add(mv[pm], T(0));
          } else if (pz >= 0) {
            u_own = Add(T(0), Mul(alpha, zv[pz]));
          }
          // U(j, i) = M(j, i) (+) alpha Z(j, i), Z(j, i) = pr_j R(j, i) unless R(j, i) is an exact zero
          const int pmt = FindSlot(k_mt, b_mt, i);
          const int pr = FindSlot(k_r, b_r, i);
          bool z_row = false;
          T z_ji = T(0);
          if (pr >= 0 || static_cast<int64_t>(i) == j) {
            T rv = pr >= 0 ? -v_r[pr] : T(0);
            if (static_cast<int64_t>(i) == j) rv = Add(rv, T(1));
            if (!(rv == T(0))) {
              z_row = true;
              z_ji = Mul(a.pr[j], rv);
            }
          }
          const bool trans = pmt >= 0 || z_row;
          T u_tr = T(0);
          if (pmt >= 0 && z_row) {
            u_tr = Add(v_mt[pmt], Mul(alpha, z_ji));
          } else if (pmt >= 0) {
            u_tr = Add(v_mt[pmt], T(0));
          } else if (z_row) {
            u_tr = Add(T(0), Mul(alpha, z_ji));
          }
          // the half sum of the symmetrisation (dropping.cpp:106-120)
          if (own && trans) {
            v = Mul(T(0.5), Add(u_own, u_tr));
          } else if (own) {
            v = Mul(T(0.5), Add(u_own, T(0)));
          } else if (trans) {
            v = Mul(T(0.5), Add(T(0), u_tr));
          }
          emit = !(v == T(0));  // exact zeros are dropped
        }
        const unsigned mask = __ballot_sync(0xffffffffu, emit);
        if (emit) {
          const int o = count + __popc(mask & LaneMaskBelow());
          s_rows[o] = i;
          s_vals[o] = v;
        }
        count += __popc(mask);
      }
      __syncwarp();
    }
    if (too_long) {
      // leave the bitmap clear for the next column before skipping this one
#pragma unroll 1
      for (int32_t seg_lo = lo; seg_lo <= hi; seg_lo += kDropWindowRows) {
        const int32_t seg_hi = hi - seg_lo < kDropWindowRows ? hi : seg_lo + (kDropWindowRows - 1);
        ClearWords(bm, (seg_hi - seg_lo) / 32 + 1, lane);
        ClearWords(summary, SummaryWords((seg_hi - seg_lo) / 32 + 1), lane);
      }
      __syncwarp();
      return kOverflowSide;
    }
    __syncwarp();
    const int kept = DropAndWrite<T>(a, [&](int r) { return s_rows[r]; }, s_vals, count, j, other, lane, &overflow);
    *written_out += static_cast<unsigned long long>(kept);
    __syncwarp();
  }
  return overflow;
}

// ---------------------------------------------------------------------------
// The drop step of C adjacent columns (colgroup.cuh).  With absent entries
// held as 0 every case of the union and of the half sum is one expression:
//   U(i, j) = M(i, j) + alpha Z(i, j), U(j, i) = M(j, i) + alpha pr_j R(j, i),
//   S(i, j) = 0.5 (U(i, j) + U(j, i)),
// because x + 0 is x and an entry that is zero on both sides is dropped.
// 32 / C lanes walk the entries of one column; its terms of row j of R arrive
// in ascending k, one row of M^T after another.
//
// What bounds it: the latency of its dependent steps (loads of rows of M^T,
// shared-memory updates, the bisection) over the warps that its shared memory
// and registers allow (12 an SM); a third of the issue slots are used and 6 % of
// the memory bandwidth.  Measured at 64^3, 16 entries a column, FP32, four
// columns a warp: 0.91 ms and 1,170 warp instructions a column, against 2.41 ms
// and 5,000 with hashes and one column a warp; 47^3 FP64 0.52 against 0.86 ms.

constexpr int kGroupDropRows = 256;  // candidate rows of a group (ranks fit the window's byte prefixes)

template <class T, int C>
__host__ __device__ size_t DropGroupBytes(int words) {
  return WindowBytes(words) + Round16(static_cast<size_t>(kGroupDropRows) * 2) +
         2 * static_cast<size_t>(kGroupDropRows) * sizeof(GroupValues<T, C>);
}

// Entries s, s + kLanes, ... of a slot list: the first kHeld of them in
// registers (rows loaded once, values when asked for), the rest read where
// they are used.  (The group kernels' loops are otherwise kept rolled:
// unrolled throughout, the drop kernel's code outgrew the instruction caches
// and it ran 1.5 times as long.)
template <class T, int kLanes, int kHeld>
struct HeldSlots {
  const int32_t* rows;
  const T* vals;
  int n;
  int s;
  int32_t row[kHeld];
  T val[kHeld];

  __device__ __forceinline__ HeldSlots(const int32_t* r, const T* v, int count, int lane_in_column)
      : rows(r), vals(v), n(count), s(lane_in_column) {
#pragma unroll
    for (int h = 0; h < kHeld; ++h) row[h] = s + h * kLanes < n ? rows[s + h * kLanes] : -1;
  }
  __device__ __forceinline__ void LoadValues() {
#pragma unroll
    for (int h = 0; h < kHeld; ++h) val[h] = row[h] >= 0 ? vals[s + h * kLanes] : T(0);
  }
  template <class F>
  __device__ __forceinline__ void Rows(F f) const {
#pragma unroll
    for (int h = 0; h < kHeld; ++h) {
      if (row[h] >= 0) f(row[h]);
    }
#pragma unroll 1
    for (int e = s + kHeld * kLanes; e < n; e += kLanes) f(rows[e]);
  }
  template <class F>
  __device__ __forceinline__ void Entries(F f) const {
#pragma unroll
    for (int h = 0; h < kHeld; ++h) {
      if (row[h] >= 0) f(row[h], val[h]);
    }
#pragma unroll 1
    for (int e = s + kHeld * kLanes; e < n; e += kLanes) f(rows[e], vals[e]);
  }
};

// False when the group does not fit (nothing written): its columns go one by one.
template <class T, int kEll, int C>
__device__ __forceinline__ bool DropGroup(const FusedArgs<T>& a, unsigned char* base, int64_t j0, T step,
                                          int64_t parity, int lane, unsigned long long* written, int* overflow) {
  constexpr int kLanes = kWarp / C;  // lanes of one column
  RowWindow w = WindowAt(base, a.words, static_cast<int32_t>(j0) - a.words * 16);
  uint16_t* rows = reinterpret_cast<uint16_t*>(base);
  base += Round16(static_cast<size_t>(kGroupDropRows) * 2);
  using Values = GroupValues<T, C>;
  Values* own = reinterpret_cast<Values*>(base);
  Values* trans = own + kGroupDropRows;
  uint16_t* list = reinterpret_cast<uint16_t*>(own);  // free until the ranks are known
  const int c = lane / kLanes;
  const int s = lane % kLanes;
  const int home = lane - s;  // first lane of the column
  const int64_t j = j0 + c;
  const bool valid = j < a.n;
  const int nm = valid ? a.m_cnt[j] : 0;
  const int nz = valid ? a.z_cnt[j] : 0;
  const int nmt = valid ? a.mt_cnt[parity][j] : 0;
  const int32_t* m_rows = a.m_rows + j * a.topk;
  const int32_t* z_rows = a.z_rows + j * a.cap_z;
  const int32_t* mt_all = a.mt_cols[parity];
  const T* mt_vals = a.mt_vals[parity];
  bool lost = nmt > a.cap_mt;
  // lane s of the column holds entries s, s + kLanes, ... of row j of A and the lengths of those rows of M^T
  constexpr int kHeld = (kEll + kLanes - 1) / kLanes;
  int32_t k_held[kHeld];
  int n_held[kHeld];
  T a_held[kHeld];
#pragma unroll
  for (int h = 0; h < kHeld; ++h) {
    const int u = h * kLanes + s;
    k_held[h] = valid && u < kEll ? a.a_rows_ell[j * kEll + u] : -1;
    a_held[h] = k_held[h] >= 0 ? a.a_rows_ell_val[j * kEll + u] : T(0);
    n_held[h] = k_held[h] >= 0 ? a.mt_cnt[parity][k_held[h]] : 0;
    lost = lost || n_held[h] > a.cap_mt;
  }
  if (__any_sync(0xffffffffu, lost)) {
    *overflow |= kOverflowMt;
    return true;  // the whole solve is redone on the unfused kernels
  }
  HeldSlots<T, kLanes, kMaxTopK / kLanes> m_list(m_rows, a.m_vals + j * a.topk, nm, s);
  HeldSlots<T, kLanes, 64 / kLanes> z_list(z_rows, a.z_vals + j * a.cap_z, nz, s);
  HeldSlots<T, kLanes, 32 / kLanes> mt_list(mt_all + j * a.cap_mt, mt_vals + j * a.cap_mt, nmt, s);
  // the first entries of the rows k of M, k in row j of A (rows of M^T), for operators of up to eight
  // entries a row; the others are read where they are used
  constexpr bool kRowsHeld = kEll <= 8 && C == 4;  // in groups of two (small problems) fetching the code costs more
  constexpr int kPer = kRowsHeld ? 24 / kLanes + (24 % kLanes != 0 ? 1 : 0) : 1;  // at least 24 entries of each
  constexpr int kRows = kRowsHeld ? kEll : 1;
  int32_t r_row[kRows][kPer];
  T r_val[kRows][kPer];
  const auto row_of_mt = [&](int u, int32_t* k, int* nk, T* a_jk) {
    const int h = u / kLanes;
    int32_t kh = k_held[0];
    int nh = n_held[0];
    T ah = a_held[0];
#pragma unroll
    for (int q = 1; q < kHeld; ++q) {
      kh = h == q ? k_held[q] : kh;
      nh = h == q ? n_held[q] : nh;
      ah = h == q ? a_held[q] : ah;
    }
    *k = __shfl_sync(0xffffffffu, kh, home + u % kLanes);
    *nk = __shfl_sync(0xffffffffu, nh, home + u % kLanes);
    *a_jk = __shfl_sync(0xffffffffu, ah, home + u % kLanes);
  };
  if constexpr (kRowsHeld) {
#pragma unroll
    for (int u = 0; u < kEll; ++u) {
      int32_t k;
      int nk;
      T a_jk;
      row_of_mt(u, &k, &nk, &a_jk);
#pragma unroll
      for (int q = 0; q < kPer; ++q) {
        const int e = q * kLanes + s;
        r_row[u][q] = e < nk ? mt_all[static_cast<int64_t>(k) * a.cap_mt + e] : -1;
      }
    }
  }
  bool fits = true;
  const auto mark = [&](int32_t row) {
    if (w.Holds(row)) {
      w.Mark(row);
    } else {
      fits = false;
    }
  };
  if (valid && s == 0) mark(static_cast<int32_t>(j));
  m_list.Rows(mark);
  z_list.Rows(mark);
  mt_list.Rows(mark);
  constexpr int kSkip = kRowsHeld ? kPer * kLanes : 0;  // entries of a row of M^T that registers hold
  if constexpr (kRowsHeld) {
#pragma unroll
    for (int u = 0; u < kEll; ++u) {
#pragma unroll
      for (int q = 0; q < kPer; ++q) {
        if (r_row[u][q] >= 0) mark(r_row[u][q]);
      }
    }
  }
#pragma unroll 1
  for (int u = 0; u < kEll; ++u) {
    int32_t k;
    int nk;
    T a_jk;
    row_of_mt(u, &k, &nk, &a_jk);
    const int32_t* from = mt_all + static_cast<int64_t>(k) * a.cap_mt;
#pragma unroll 1
    for (int e = kSkip + s; e < nk; e += kLanes) mark(from[e]);
  }
  // the values travel while the rows are ranked
  m_list.LoadValues();
  z_list.LoadValues();
  mt_list.LoadValues();
  if constexpr (kRowsHeld) {
#pragma unroll
    for (int u = 0; u < kEll; ++u) {
      const int32_t k = __shfl_sync(0xffffffffu, k_held[0], home + u % kLanes);
      static_assert(kEll <= kLanes || !kRowsHeld, "one held entry per lane");
#pragma unroll
      for (int q = 0; q < kPer; ++q) {
        r_val[u][q] = r_row[u][q] >= 0 ? mt_vals[static_cast<int64_t>(k) * a.cap_mt + q * kLanes + s] : T(0);
      }
    }
  }
  int count = kGroupDropRows + 1;
  if (__all_sync(0xffffffffu, fits)) count = RankRows<true>(w, rows, list, kGroupDropRows, lane);
  if (count > kGroupDropRows) {
    ClearWindow(w, lane);
    return false;
  }
#pragma unroll 1
  for (int r = lane; r < count; r += kWarp) {
#pragma unroll
    for (int q = 0; q < C; ++q) own[r].v[q] = trans[r].v[q] = T(0);
  }
  __syncwarp();
  // U(:, j): M, then + alpha Z
  m_list.Entries([&](int32_t i, T v) { own[w.Rank(i)].v[c] = v; });
  __syncwarp();
  const T alpha = a.alpha != nullptr && valid ? static_cast<T>(a.alpha[j]) : step;
  z_list.Entries([&](int32_t i, T v) {
    T& u = own[w.Rank(i)].v[c];
    u = Add(u, Mul(alpha, v));
  });
  // row j of A M, terms in ascending k: one row of M^T after another
  const auto add = [&](int32_t i, T v, T a_jk) {
    T& t = trans[w.Rank(i)].v[c];
    t = Add(t, Mul(a_jk, v));
  };
  const auto add_rest = [&](int32_t k, int nk, T a_jk) {
    const int64_t at = static_cast<int64_t>(k) * a.cap_mt;
#pragma unroll 1
    for (int e = kSkip + s; e < nk; e += kLanes) add(mt_all[at + e], mt_vals[at + e], a_jk);
  };
  if constexpr (kRowsHeld) {
#pragma unroll
    for (int u = 0; u < kEll; ++u) {
      int32_t k;
      int nk;
      T a_jk;
      row_of_mt(u, &k, &nk, &a_jk);
#pragma unroll
      for (int q = 0; q < kPer; ++q) {
        if (r_row[u][q] >= 0) add(r_row[u][q], r_val[u][q], a_jk);
      }
      if (__any_sync(0xffffffffu, nk > kSkip)) add_rest(k, nk, a_jk);
      __syncwarp();
    }
  } else {
#pragma unroll 1
    for (int u = 0; u < kEll; ++u) {
      int32_t k;
      int nk;
      T a_jk;
      row_of_mt(u, &k, &nk, &a_jk);
      add_rest(k, nk, a_jk);
      __syncwarp();
    }
  }
  // alpha Z(j, :) = alpha pr_j (e_j - that), then + M(j, :)
  T pr[C];
  T steps[C];
#pragma unroll
  for (int q = 0; q < C; ++q) {
    pr[q] = j0 + q < a.n ? a.pr[j0 + q] : T(0);
    steps[q] = __shfl_sync(0xffffffffu, alpha, q * kLanes);
  }
#pragma unroll 1
  for (int r = lane; r < count; r += kWarp) {
    const int64_t i = static_cast<int64_t>(w.lo) + rows[r];
    Values t = trans[r];
#pragma unroll
    for (int q = 0; q < C; ++q) {
      T rv = -t.v[q];
      if (i == j0 + q) rv = Add(rv, T(1));
      t.v[q] = rv == T(0) ? T(0) : Mul(steps[q], Mul(pr[q], rv));
    }
    trans[r] = t;
  }
  __syncwarp();
  mt_list.Entries([&](int32_t i, T v) {
    T& t = trans[w.Rank(i)].v[c];
    t = Add(v, t);
  });
  __syncwarp();
#pragma unroll 1
  for (int r = lane; r < count; r += kWarp) {
    Values u = own[r];
    const Values t = trans[r];
#pragma unroll
    for (int q = 0; q < C; ++q) u.v[q] = Mul(T(0.5), Add(u.v[q], t.v[q]));
    own[r] = u;
  }
  __syncwarp();
  // each column's nonzero entries, compacted (over trans, which is done with), then decided
  T* column_vals = reinterpret_cast<T*>(trans);
  uint16_t* column_rows = reinterpret_cast<uint16_t*>(column_vals + kGroupDropRows);
  static_assert(kGroupDropRows * (sizeof(T) + sizeof(uint16_t)) <= kGroupDropRows * sizeof(Values), "the column fits");
#pragma unroll 1
  for (int q = 0; q < C; ++q) {
    if (j0 + q >= a.n) break;
    int entries = 0;
#pragma unroll 1
    for (int r0 = 0; r0 < count; r0 += kWarp) {
      const int r = r0 + lane;
      const T v = r < count ? reinterpret_cast<const T*>(own)[r * C + q] : T(0);
      const bool some = !(v == T(0));
      const unsigned mask = __ballot_sync(0xffffffffu, some);
      if (some) {
        const int o = entries + __popc(mask & LaneMaskBelow());
        column_vals[o] = v;
        column_rows[o] = rows[r];
      }
      entries += __popc(mask);
    }
    __syncwarp();
    const int kept = DropAndWrite<T>(a, [&](int r) { return w.lo + static_cast<int32_t>(column_rows[r]); },
                                     column_vals, entries, j0 + q, parity ^ 1, lane, overflow);
    *written += static_cast<unsigned long long>(kept);
    __syncwarp();
  }
  ClearRows(w, rows, count, lane);
  return true;
}

// A column of a group that does not fit (a call per column: over several
// columns the compiler keeps 157 registers in FP64, and groups of two then run
// in two waves).
template <class T>
__device__ __noinline__ int DropOneColumn(const FusedArgs<T>& a, unsigned char* base, bool clear, int64_t j,
                                          unsigned long long* written) {
  const DropSlab<T> slab(a, base, clear, threadIdx.x & 31);
  return DropColumn<T, 1>(a, slab, j, written);
}

// A warp's entries of M and its overflow bits into the loop's state.
template <class T>
__device__ __forceinline__ void FinishDrop(const FusedArgs<T>& a, unsigned long long written, int overflow, int lane) {
  overflow = __reduce_or_sync(0xffffffffu, overflow);
  if (lane == 0) {
    if (written != 0ull) atomicAdd(&a.state->nnz_m, written);
    if (overflow != 0) atomicOr(&a.state->overflow, overflow);
  }
}

template <class T, int kEll, int C>
__global__ void __launch_bounds__(kGroupWarps * kWarp) FusedDropKernel(const __grid_constant__ FusedArgs<T> a) {
  extern __shared__ __align__(16) unsigned char fused_drop_smem[];
  const int lane = threadIdx.x & 31;
  unsigned char* base = fused_drop_smem + (threadIdx.x >> 5) * a.drop_bytes;
  const int64_t parity = a.state->parity;
  const T alpha = static_cast<T>(a.state->alpha);
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  unsigned long long written = 0;
  int overflow = 0;
  unsigned int unfit = 0;
  bool clear = false;  // whether the window starts clear
#pragma unroll 1
  for (int64_t j0 = warp * C; j0 < a.n; j0 += warps * C) {
    if (!clear) {
      unsigned char* at = base;
      RowWindow w = WindowAt(at, a.words, 0);
      ClearWindow(w, lane);
      clear = true;
    }
    if (DropGroup<T, kEll, C>(a, base, j0, alpha, parity, lane, &written, &overflow)) continue;
    clear = false;
    ++unfit;
#pragma unroll 1
    for (int64_t j = j0; j < j0 + C && j < a.n; ++j) overflow |= DropOneColumn<T>(a, base, j == j0, j, &written);
  }
  if (lane == 0 && unfit != 0u) atomicAdd(&a.state->unfit, unfit);
  FinishDrop(a, written, overflow, lane);
}

// The drop step column by column, for operators whose groups have no window
// (GroupWords).  What bounds it: the latency of the hash updates and of the
// window's scans, so it is a kernel of its own with registers for 24 (FP32) or
// 20 warps an SM.  As the fallback inside the group kernel (168 registers, the
// window cleared for every column) it left 12, and six iterations on a randomly
// permuted 47^3 operator in FP32 storage, 16 entries a column, took 27.2 ms;
// now 19.2 (20.3 before there were groups).  At 90^3: 4.7 ms a launch in FP32
// storage, 6.5 in FP64.
template <class T>
__global__ void __launch_bounds__(kColumnWarps * kWarp, sizeof(T) == 4 ? 6 : 5)
    FusedDropColumnsKernel(const __grid_constant__ FusedArgs<T> a) {
  extern __shared__ __align__(16) unsigned char fused_drop_smem[];
  const int lane = threadIdx.x & 31;
  unsigned char* base = fused_drop_smem + (threadIdx.x >> 5) * a.drop_bytes;
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  unsigned long long written = 0;
  int overflow = 0;
  const DropSlab<T> slab(a, base, true, lane);
  for (int64_t j = warp; j < a.n; j += warps) overflow |= DropColumn<T, 4>(a, slab, j, &written);
  FinishDrop(a, written, overflow, lane);
}

// ---------------------------------------------------------------------------
// Residual kernel: R = I - A M(:, j), Z = Pr R, ||R(:, j)||^2, then the MR
// projection of A Z(:, j).  The arithmetic is ColumnProductKernel's
// (spgemm.cu): rows in ascending order from the window bitmap, each row of A
// (ELL copy) pulled in ascending k against a hash of the column, the
// accumulator started at -0.0, sums sequential in row order on one lane.

template <class T>
__host__ __device__ size_t ResidualSlabBytes(int m_slots, int z_slots) {
  return Round16(static_cast<size_t>(kWindowWords) * 4) + Round16(static_cast<size_t>(SummaryWords(kWindowWords)) * 4) +
         Round16(static_cast<size_t>(kRowsCap) * 2) + Round16(static_cast<size_t>(m_slots) * 4) +
         Round16(static_cast<size_t>(m_slots) * sizeof(T)) + Round16(static_cast<size_t>(z_slots) * 4) +
         Round16(static_cast<size_t>(z_slots) * sizeof(T)) + 2 * Round16(kWarp * sizeof(double));
}

// Sequential sum of `count` staged values onto s (one lane).
__device__ __forceinline__ double SumStaged(double s, const double* src, int count) {
  if (count == kWarp) {
    const double2* src2 = reinterpret_cast<const double2*>(src);
#pragma unroll
    for (int l = 0; l < kWarp / 2; ++l) {
      const double2 v = src2[l];
      s = Add(s, v.x);
      s = Add(s, v.y);
    }
  } else {
    for (int l = 0; l < count; ++l) s = Add(s, src[l]);
  }
  return s;
}

// A warp's shared memory while it goes column by column.
template <class T>
struct ResidualSlab {
  uint32_t* bm;
  uint32_t* summary;
  uint16_t* rows;
  int32_t* mkeys;
  T* mvals;
  int32_t* zkeys;
  T* zvals;
  double* stage;
  int mbits;  // buckets of two slots
  int zbits;

  // clear: whether the window has to be cleared.
  __device__ __forceinline__ ResidualSlab(const FusedArgs<T>& a, unsigned char* base, bool clear, int lane) {
    bm = reinterpret_cast<uint32_t*>(base);
    base += Round16(static_cast<size_t>(kWindowWords) * 4);
    summary = reinterpret_cast<uint32_t*>(base);
    base += Round16(static_cast<size_t>(kResidualSummary) * 4);
    rows = reinterpret_cast<uint16_t*>(base);
    base += Round16(static_cast<size_t>(kRowsCap) * 2);
    mkeys = reinterpret_cast<int32_t*>(base);
    base += Round16(static_cast<size_t>(a.m_hash_slots) * 4);
    mvals = reinterpret_cast<T*>(base);
    base += Round16(static_cast<size_t>(a.m_hash_slots) * sizeof(T));
    zkeys = reinterpret_cast<int32_t*>(base);
    base += Round16(static_cast<size_t>(a.z_hash_slots) * 4);
    zvals = reinterpret_cast<T*>(base);
    base += Round16(static_cast<size_t>(a.z_hash_slots) * sizeof(T));
    stage = reinterpret_cast<double*>(base);
    mbits = Log2(a.m_hash_slots) - 1;
    zbits = Log2(a.z_hash_slots) - 1;
    if (clear) {
      __syncwarp();
      ClearWords(bm, kWindowWords, lane);
      ClearWords(summary, kResidualSummary, lane);
      __syncwarp();
    }
  }
};

// One column on its own; its window is clear before and after.
template <class T, int kEll>
__device__ __forceinline__ void ResidualColumn(const FusedArgs<T>& a, const ResidualSlab<T>& slab, int64_t j,
                                               unsigned long long* written_out) {
  const int lane = threadIdx.x & 31;
  uint32_t* bm = slab.bm;
  uint32_t* summary = slab.summary;
  uint16_t* rows = slab.rows;
  int32_t* mkeys = slab.mkeys;
  T* mvals = slab.mvals;
  int32_t* zkeys = slab.zkeys;
  T* zvals = slab.zvals;
  double* stage0 = slab.stage;
  double* stage1 = stage0 + kWarp;
  const int mbits = slab.mbits;
  const int zbits = slab.zbits;
  {
    // ---- R(:, j) = e_j - A M(:, j) ----------------------------------------
    const int nm = a.m_cnt[j];
    ClearTable(mkeys, a.m_hash_slots, lane);
    __syncwarp();
    int32_t k_mine = -1;
    bool placed = true;
    if (lane < nm) {
      k_mine = a.m_rows[j * a.topk + lane];
      placed = BucketInsert(mkeys, mvals, mbits, k_mine, a.m_vals[j * a.topk + lane]);
    }
    const bool m_displaced = !__all_sync(0xffffffffu, placed);
    // the candidate rows: A(:, k) for k in M(:, j), and j itself
    int32_t cand[kEll];
    int32_t lo = static_cast<int32_t>(j);
    int32_t hi = static_cast<int32_t>(j);
#pragma unroll
    for (int u = 0; u < kEll / 4; ++u) {
      int4 r4 = make_int4(-1, -1, -1, -1);
      if (k_mine >= 0) r4 = reinterpret_cast<const int4*>(a.a_cols_ell + static_cast<int64_t>(k_mine) * kEll)[u];
      cand[4 * u] = r4.x;
      cand[4 * u + 1] = r4.y;
      cand[4 * u + 2] = r4.z;
      cand[4 * u + 3] = r4.w;
    }
#pragma unroll
    for (int u = 0; u < kEll; ++u) {
      if (cand[u] >= 0) {
        lo = min(lo, cand[u]);
        hi = max(hi, cand[u]);
      }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    int32_t* zr_out = a.z_rows + j * a.cap_z;
    T* zv_out = a.z_vals + j * a.cap_z;
    ClearTable(zkeys, a.z_hash_slots, lane);
    __syncwarp();
    int kept = 0;
    double sq = 0.0;
    bool z_placed = true;
    // the rows in ascending order, one window of kWindowRows rows at a time
    for (int32_t seg_lo = lo; seg_lo <= hi; seg_lo += kWindowRows) {
      const int32_t seg_hi = hi - seg_lo < kWindowRows ? hi : seg_lo + (kWindowRows - 1);
      const int words = (seg_hi - seg_lo) / 32 + 1;
      if (lane == 0 && j >= seg_lo && j <= seg_hi) MarkRow(bm, summary, static_cast<int>(j - seg_lo));
#pragma unroll
      for (int u = 0; u < kEll; ++u) {
        if (cand[u] >= seg_lo && cand[u] <= seg_hi) MarkRow(bm, summary, cand[u] - seg_lo);
      }
      __syncwarp();
      const int count = DrainRows(bm, summary, SummaryWords(words), rows, lane);
      for (int r0 = 0; r0 < count; r0 += kWarp) {
        const int r = r0 + lane;
        bool keep = false;
        int32_t i = 0;
        T v = T(0);
        if (r < count) {
          i = seg_lo + static_cast<int32_t>(rows[r]);
          T acc = T(-0.0);
          const int4* ks = reinterpret_cast<const int4*>(a.a_rows_ell + static_cast<int64_t>(i) * kEll);
          const T* vs = a.a_rows_ell_val + static_cast<int64_t>(i) * kEll;
#pragma unroll
          for (int u = 0; u < kEll / 4; ++u) {
            const int4 k4 = ks[u];
            T v4[4];
            LoadFour(vs + 4 * u, v4);
            const int32_t kk[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              T bv;
              if (kk[e] >= 0 && BucketFind(mkeys, mvals, mbits, m_displaced, kk[e], bv)) acc = Add(acc, Mul(v4[e], bv));
            }
          }
          v = -acc;
          if (static_cast<int64_t>(i) == j) v = Add(v, T(1));
          const double sd = static_cast<double>(v);
          stage0[lane] = Mul(sd, sd);
          keep = !(v == T(0));  // Eigen prune(0.0)
        }
        const unsigned mask = __ballot_sync(0xffffffffu, keep);
        if (keep) {
          const int o = kept + __popc(mask & LaneMaskBelow());
          const T z = Mul(a.pr[i], v);
          zr_out[o] = i;
          zv_out[o] = z;
          z_placed &= BucketInsert(zkeys, zvals, zbits, i, z);
        }
        kept += __popc(mask);
        __syncwarp();
        if (lane == 0) sq = SumStaged(sq, stage0, min(kWarp, count - r0));
        __syncwarp();
      }
    }
    if (lane == 0) {
      a.sq[j] = sq;
      a.z_cnt[j] = kept;
    }
    *written_out += static_cast<unsigned long long>(kept);
    const bool z_displaced = !__all_sync(0xffffffffu, z_placed);
    // ---- projection: tt = ||Pr A Z(:, j)||^2, bt = <Z(:, j), Pr A Z(:, j)> --
    lo = INT32_MAX;
    hi = -1;
    for (int e = lane; e < kept; e += kWarp) {
      const int4* src = reinterpret_cast<const int4*>(a.a_cols_ell + static_cast<int64_t>(zr_out[e]) * kEll);
#pragma unroll
      for (int u = 0; u < kEll / 4; ++u) {
        const int4 r4 = src[u];
        const int32_t rr[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          if (rr[t] >= 0) {
            lo = min(lo, rr[t]);
            hi = max(hi, rr[t]);
          }
        }
      }
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    double proj = 0.0;  // tt on lane 0, bt on lane 1
    for (int32_t seg_lo = lo; seg_lo <= hi; seg_lo += kWindowRows) {
      const int32_t seg_hi = hi - seg_lo < kWindowRows ? hi : seg_lo + (kWindowRows - 1);
      const int words2 = (seg_hi - seg_lo) / 32 + 1;
      for (int e = lane; e < kept; e += kWarp) {
        const int4* src = reinterpret_cast<const int4*>(a.a_cols_ell + static_cast<int64_t>(zr_out[e]) * kEll);
#pragma unroll
        for (int u = 0; u < kEll / 4; ++u) {
          const int4 r4 = src[u];
          const int32_t rr[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
          for (int t = 0; t < 4; ++t) {
            if (rr[t] >= seg_lo && rr[t] <= seg_hi) MarkRow(bm, summary, rr[t] - seg_lo);
          }
        }
      }
      __syncwarp();
      const int count2 = DrainRows(bm, summary, SummaryWords(words2), rows, lane);
      for (int r0 = 0; r0 < count2; r0 += kWarp) {
        const int r = r0 + lane;
        if (r < count2) {
          const int32_t i = seg_lo + static_cast<int32_t>(rows[r]);
          T acc = T(-0.0);
          const int4* ks = reinterpret_cast<const int4*>(a.a_rows_ell + static_cast<int64_t>(i) * kEll);
          const T* vs = a.a_rows_ell_val + static_cast<int64_t>(i) * kEll;
#pragma unroll
          for (int u = 0; u < kEll / 4; ++u) {
            const int4 k4 = ks[u];
            T v4[4];
            LoadFour(vs + 4 * u, v4);
            const int32_t kk[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              T bv;
              if (kk[e] >= 0 && BucketFind(zkeys, zvals, zbits, z_displaced, kk[e], bv)) acc = Add(acc, Mul(v4[e], bv));
            }
          }
          const double td = static_cast<double>(Mul(a.pr[i], acc));
          T zi;
          stage0[lane] = Mul(td, td);
          // rows of Z absent from the product add +0.0, which leaves a sum started at +0.0 unchanged
          stage1[lane] = BucketFind(zkeys, zvals, zbits, z_displaced, i, zi) ? Mul(static_cast<double>(zi), td) : 0.0;
        }
        __syncwarp();
        // lane 0 extends tt and lane 1 bt, side by side in one instruction stream
        const int span = min(kWarp, count2 - r0);
        if (lane < 2) proj = SumStaged(proj, lane == 0 ? stage0 : stage1, span);
        __syncwarp();
      }
    }
    if (lane == 0) a.tt[j] = proj;
    if (lane == 1) a.bt[j] = proj;
    __syncwarp();
  }
}

// ---------------------------------------------------------------------------
// The residual and projection of C adjacent columns (colgroup.cuh).  Two
// windows: one ranks the rows k of M and later the rows of A Z, the other the
// rows of R, whose ranks hold Z for the projection's lookups.  A product row i
// walks row i of A in ascending k, one lookup per k for all columns; a column
// that lacks k adds A(i, k) * 0, which changes at most the sign of a zero (the
// host takes this path only when A and Pr are finite).  The 3 C column sums
// run sequentially in row order, side by side on C or 2 C lanes.
//
// What bounds it: the sequential sums (a dependent FP64 addition a row) and
// the dependent reads window word -> rank -> value, over the warps its shared
// memory allows (12 an SM; 37 % of the issue slots).  Measured at 64^3, 16
// entries a column, FP32, four columns a warp: 1.08 ms and 1,680 warp
// instructions a column, against 1.85 ms and 4,300 with hashes and one column a
// warp; 47^3 FP64 0.47 against 0.83 ms.

constexpr int kGroupResidualRows = 192;  // rows of R of a group
constexpr int kGroupProductRows = 512;   // rows of A Z of a group taken at a time
constexpr int kStageStride = kWarp + 2;  // doubles between two columns' staged terms: lanes hit different banks

template <class T, int C>
__host__ __device__ size_t ResidualGroupBytes(int words, int topk) {
  return 2 * WindowBytes(words) + Round16(static_cast<size_t>(kGroupResidualRows) * 2) +
         Round16(static_cast<size_t>(kGroupProductRows) * 2) + Round16(2 * C * kStageStride * sizeof(double)) +
         Round16(static_cast<size_t>(C * topk + kGroupResidualRows + 2) * sizeof(GroupValues<T, C>));
}

// acc[q] += A(i, k) b_k[q] over row i of A, ascending k; an absent k reads the
// zeros at vals[zero], so that no lookup waits for another's outcome.  kUse:
// A's longest row (the slots past it are padding everywhere).
template <class T, int C, int kEll, int kUse, class Sum>
__device__ __forceinline__ void GroupRow(const FusedArgs<T>& a, const RowWindow& w, const GroupValues<T, C>* vals,
                                         int zero, int32_t i, Sum& acc) {
  const int4* ks = reinterpret_cast<const int4*>(a.a_rows_ell + static_cast<int64_t>(i) * kEll);
  const T* vs = a.a_rows_ell_val + static_cast<int64_t>(i) * kEll;
#pragma unroll
  for (int u = 0; u < kEll / 4; ++u) {
    const int4 k4 = ks[u];
    T v4[4];
    LoadFour(vs + 4 * u, v4);
    const int32_t kk[4] = {k4.x, k4.y, k4.z, k4.w};  // padding (-1) is never marked
    GroupValues<T, C> b[4];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (4 * u + e < kUse) b[e] = vals[w.FindOr(kk[e], zero)];
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      if (4 * u + e < kUse) {
#pragma unroll
        for (int q = 0; q < C; ++q) acc[q] = Add(acc[q], Mul(v4[e], b[e].v[q]));
      }
    }
  }
}

// False when the group does not fit (nothing written).
template <class T, int kEll, int kUse, int C>
__device__ __forceinline__ bool ResidualGroup(const FusedArgs<T>& a, unsigned char* base, int64_t j0, int lane,
                                              unsigned long long* written) {
  constexpr int kLanes = kWarp / C;
  using Values = GroupValues<T, C>;
  const int32_t lo = static_cast<int32_t>(j0) - a.words * 16;
  RowWindow wm = WindowAt(base, a.words, lo);  // rows of M, then of A Z
  RowWindow wr = WindowAt(base, a.words, lo);  // rows of R
  uint16_t* rows = reinterpret_cast<uint16_t*>(base);
  base += Round16(static_cast<size_t>(kGroupResidualRows) * 2);
  uint16_t* prod = reinterpret_cast<uint16_t*>(base);
  base += Round16(static_cast<size_t>(kGroupProductRows) * 2);
  double* stage = reinterpret_cast<double*>(base);
  base += Round16(2 * C * kStageStride * sizeof(double));
  Values* mv = reinterpret_cast<Values*>(base);  // M by rank
  Values* zv = mv + C * a.topk + 1;              // Z by rank
  uint16_t* list = prod;                         // scratch of the first two rankings
  const int c = lane / kLanes;
  const int s = lane % kLanes;
  const int64_t j = j0 + c;
  const bool valid = j < a.n;
  const int nm = valid ? a.m_cnt[j] : 0;
  bool fits = true;
  const auto mark = [&](RowWindow& w, int32_t row) {
    if (w.Holds(row)) {
      w.MarkNew(row);
    } else {
      fits = false;
    }
  };
  if (valid && s == 0) mark(wr, static_cast<int32_t>(j));
#pragma unroll 1
  for (int e = s; e < nm; e += kLanes) {
    const int32_t k = a.m_rows[j * a.topk + e];
    mark(wm, k);
    const int4* src = reinterpret_cast<const int4*>(a.a_cols_ell + static_cast<int64_t>(k) * kEll);
#pragma unroll
    for (int u = 0; u < kEll / 4; ++u) {
      const int4 r4 = src[u];
      if (r4.x >= 0) mark(wr, r4.x);
      if (r4.y >= 0) mark(wr, r4.y);
      if (r4.z >= 0) mark(wr, r4.z);
      if (r4.w >= 0) mark(wr, r4.w);
    }
  }
  int count = kGroupResidualRows + 1;
  if (__all_sync(0xffffffffu, fits)) count = RankRows<true>(wr, rows, list, kGroupResidualRows, lane);
  if (count > kGroupResidualRows) {
    ClearWindow(wm, lane);
    ClearWindow(wr, lane);
    return false;
  }
  const int distinct = RankRows<true>(wm, nullptr, list, min(C * a.topk, kGroupProductRows), lane);
#pragma unroll 1
  for (int r = lane; r <= distinct; r += kWarp) {  // the zeros of absent rows past the end
#pragma unroll
    for (int q = 0; q < C; ++q) mv[r].v[q] = T(0);
  }
  __syncwarp();
#pragma unroll 1
  for (int e = s; e < nm; e += kLanes) mv[wm.Rank(a.m_rows[j * a.topk + e])].v[c] = a.m_vals[j * a.topk + e];
  __syncwarp();
  // ---- R(:, j) = e_j - A M(:, j), Z = Pr R, ||R(:, j)||^2 on lane c ----------
  int kept[C];
#pragma unroll
  for (int q = 0; q < C; ++q) kept[q] = 0;
  double sq = 0.0;
#pragma unroll 1
  for (int r0 = 0; r0 <= count; r0 += kWarp) {
    const int r = r0 + lane;
    const int32_t i = r < count ? lo + static_cast<int32_t>(rows[r]) : -1;
    T acc[C];
#pragma unroll
    for (int q = 0; q < C; ++q) acc[q] = T(-0.0);
    T pri = T(0);
    if (i >= 0) {
      pri = a.pr[i];
      GroupRow<T, C, kEll, kUse>(a, wm, mv, distinct, i, acc);
    }
    Values z;
#pragma unroll
    for (int q = 0; q < C; ++q) {
      T v = -acc[q];
      if (static_cast<int64_t>(i) == j0 + q) v = Add(v, T(1));
      const bool keep = i >= 0 && j0 + q < a.n && !(v == T(0));  // Eigen prune(0.0)
      z.v[q] = keep ? Mul(pri, v) : T(0);
      const double sd = keep ? static_cast<double>(v) : 0.0;
      stage[q * kStageStride + lane] = Mul(sd, sd);
      const unsigned mask = __ballot_sync(0xffffffffu, keep);
      if (keep) {
        const int64_t o = (j0 + q) * a.cap_z + kept[q] + __popc(mask & LaneMaskBelow());
        a.z_rows[o] = i;
        a.z_vals[o] = z.v[q];
      }
      kept[q] += __popc(mask);
    }
    if (r <= count) zv[r] = z;  // zeros past the end
    __syncwarp();
    if (lane < C && r0 < count) sq = SumStaged(sq, stage + lane * kStageStride, min(kWarp, count - r0));
    __syncwarp();
  }
#pragma unroll
  for (int q = 0; q < C; ++q) {
    if (lane == q && j0 + q < a.n) {
      a.sq[j0 + q] = sq;
      a.z_cnt[j0 + q] = kept[q];
    }
    *written += static_cast<unsigned long long>(kept[q]);
  }
  // M's rows leave their window
#pragma unroll 1
  for (int e = s; e < nm; e += kLanes) wm.bits[(a.m_rows[j * a.topk + e] - lo) >> 5] = 0u;
#pragma unroll 1
  for (int t = lane; t < GroupSummaryWords(a.words); t += kWarp) wm.summary[t] = 0u;
  __syncwarp();
  // ---- projection: ||Pr A Z(:, j)||^2 on lane c, <Z(:, j), Pr A Z(:, j)> on lane C + c
  const int64_t first = max(static_cast<int64_t>(lo) + rows[0] - a.bandwidth, int64_t{0});
  const int64_t last = min(static_cast<int64_t>(lo) + rows[count - 1] + a.bandwidth, a.n - 1);
  double proj = 0.0;
  int span = a.words * 32;  // rows of the running piece
#pragma unroll 1
  for (int64_t piece = first; piece <= last;) {
    wm.lo = static_cast<int32_t>(piece);
    const int32_t end = static_cast<int32_t>(min(last, piece + span - 1));
#pragma unroll 1
    for (int r = lane; r < count; r += kWarp) {
      const int4* src = reinterpret_cast<const int4*>(a.a_cols_ell + (static_cast<int64_t>(lo) + rows[r]) * kEll);
#pragma unroll
      for (int u = 0; u < kEll / 4; ++u) {
        const int4 r4 = src[u];
        if (r4.x >= wm.lo && r4.x <= end) wm.MarkNew(r4.x);
        if (r4.y >= wm.lo && r4.y <= end) wm.MarkNew(r4.y);
        if (r4.z >= wm.lo && r4.z <= end) wm.MarkNew(r4.z);
        if (r4.w >= wm.lo && r4.w <= end) wm.MarkNew(r4.w);
      }
    }
    static_assert(2 * C * kStageStride * sizeof(double) >= kGroupProductRows * sizeof(uint16_t), "the list fits stage");
    const int np = RankRows<false>(wm, prod, reinterpret_cast<uint16_t*>(stage), kGroupProductRows, lane);
    if (np > kGroupProductRows) {
      ClearWindow(wm, lane);
      span >>= 1;  // fewer rows at a time; a piece of 256 rows always fits
      continue;
    }
#pragma unroll 1
    for (int r0 = 0; r0 < np; r0 += kWarp) {
      const int r = r0 + lane;
      if (r < np) {
        const int32_t i = static_cast<int32_t>(piece) + static_cast<int32_t>(prod[r]);
        T acc[C];
#pragma unroll
        for (int q = 0; q < C; ++q) acc[q] = T(-0.0);
        GroupRow<T, C, kEll, kUse>(a, wr, zv, count, i, acc);
        const T pri = a.pr[i];
        const Values z = zv[wr.FindOr(i, count)];
#pragma unroll
        for (int q = 0; q < C; ++q) {
          const double td = static_cast<double>(Mul(pri, acc[q]));
          stage[q * kStageStride + lane] = Mul(td, td);
          // rows that Z(:, j) lacks add 0, which leaves a sum started at +0.0 unchanged
          stage[(C + q) * kStageStride + lane] = z.v[q] == T(0) ? 0.0 : Mul(static_cast<double>(z.v[q]), td);
        }
      }
      __syncwarp();
      if (lane < 2 * C) proj = SumStaged(proj, stage + lane * kStageStride, min(kWarp, np - r0));
      __syncwarp();
    }
    ClearRows(wm, prod, np, lane);
    piece += span;
  }
  if (lane < C && j0 + lane < a.n) a.tt[j0 + lane] = proj;
  if (lane >= C && lane < 2 * C && j0 + lane - C < a.n) a.bt[j0 + lane - C] = proj;
  ClearRows(wr, rows, count, lane);
  return true;
}

// A column of a group that does not fit.
template <class T, int kEll>
__device__ __noinline__ void ResidualOneColumn(const FusedArgs<T>& a, unsigned char* base, bool clear, int64_t j,
                                               unsigned long long* written) {
  const ResidualSlab<T> slab(a, base, clear, threadIdx.x & 31);
  ResidualColumn<T, kEll>(a, slab, j, written);
}

template <class T, int kEll, int kUse, int C>
__global__ void __launch_bounds__(kGroupWarps * kWarp) FusedResidualKernel(const __grid_constant__ FusedArgs<T> a) {
  extern __shared__ __align__(16) unsigned char fused_res_smem[];
  const int lane = threadIdx.x & 31;
  unsigned char* base = fused_res_smem + (threadIdx.x >> 5) * a.residual_bytes;
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  if (a.state->overflow != 0) return;  // the step is void: M^T and Z stay what it started from
  const int64_t read_set = a.state->parity;  // the M^T set the drop kernel has just read
  unsigned long long written = 0;
  unsigned int unfit = 0;
  bool clear = false;  // whether the windows start clear
#pragma unroll 1
  for (int64_t j0 = warp * C; j0 < a.n; j0 += warps * C) {
    if (lane < C && j0 + lane < a.n) a.mt_cnt[read_set][j0 + lane] = 0;  // refilled from zero by the next drop kernel
    if (!clear) {
      unsigned char* at = base;
      RowWindow wm = WindowAt(at, a.words, 0);
      RowWindow wr = WindowAt(at, a.words, 0);
      ClearWindow(wm, lane);
      ClearWindow(wr, lane);
      clear = true;
    }
    if (ResidualGroup<T, kEll, kUse, C>(a, base, j0, lane, &written)) continue;
    clear = false;
    ++unfit;
#pragma unroll 1
    for (int64_t j = j0; j < j0 + C && j < a.n; ++j) ResidualOneColumn<T, kEll>(a, base, j == j0, j, &written);
  }
  if (lane == 0) {
    if (written != 0ull) atomicAdd(&a.state->nnz_z, written);
    if (unfit != 0u) atomicAdd(&a.state->unfit, unfit);
  }
}

// The residual and projection column by column, for operators whose groups
// have no window: 20 to 24 warps an SM, bound by the latency of hash lookups
// and sequential sums.  6.0 ms a launch at 90^3 in FP32 storage, 7.0 in FP64.
template <class T, int kEll>
__global__ void __launch_bounds__(kColumnWarps * kWarp)
    FusedResidualColumnsKernel(const __grid_constant__ FusedArgs<T> a) {
  extern __shared__ __align__(16) unsigned char fused_res_smem[];
  const int lane = threadIdx.x & 31;
  unsigned char* base = fused_res_smem + (threadIdx.x >> 5) * a.residual_bytes;
  const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
  if (a.state->overflow != 0) return;  // the step is void: M^T and Z stay what it started from
  const int64_t read_set = a.state->parity;  // the M^T set the drop kernel has just read
  unsigned long long written = 0;
  const ResidualSlab<T> slab(a, base, true, lane);
  for (int64_t j = warp; j < a.n; j += warps) {
    if (lane == 0) a.mt_cnt[read_set][j] = 0;  // refilled from zero by the next drop kernel
    ResidualColumn<T, kEll>(a, slab, j, &written);
  }
  if (lane == 0 && written != 0ull) atomicAdd(&a.state->nnz_z, written);
}

// ---------------------------------------------------------------------------
// Decide kernel: the three tree sums; the last block appends the history row,
// applies the stop rules (result_operations.cpp:53-67, minimal_residual.cpp:55-89),
// forms the next step length and, inside the graph, sets the loop condition.
template <class T>
__global__ void __launch_bounds__(kTreeLanes) FusedDecideKernel(FusedArgs<T> a, cudaGraphConditionalHandle loop,
                                                                bool in_graph) {
  __shared__ double shared[kTreeLanes];
  __shared__ int last;
  const int t = threadIdx.x;
  const int64_t base = static_cast<int64_t>(blockIdx.x) * kTreeChunk + t;
  double s_sq = 0.0;
  double s_bt = 0.0;
  double s_tt = 0.0;
#pragma unroll
  for (int m = 0; m < kTreeTerms; ++m) {
    const int64_t i = base + static_cast<int64_t>(kTreeLanes) * m;
    if (i < a.n) {
      s_sq = Add(s_sq, a.sq[i]);
      s_bt = Add(s_bt, a.bt[i]);
      s_tt = Add(s_tt, a.tt[i]);
    }
  }
  double total_sq = TreeButterfly(s_sq, shared);
  double total_bt = TreeButterfly(s_bt, shared);
  double total_tt = TreeButterfly(s_tt, shared);
  FusedState* state = a.state;
  if (gridDim.x > 1) {
    const int64_t chunks = gridDim.x;
    if (t == 0) {
      a.chunk[blockIdx.x] = total_sq;
      a.chunk[chunks + blockIdx.x] = total_bt;
      a.chunk[2 * chunks + blockIdx.x] = total_tt;
      __threadfence();
      last = atomicAdd(&state->arrive, 1u) == gridDim.x - 1 ? 1 : 0;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    total_sq = TreeLevel(a.chunk, chunks, shared);
    total_bt = TreeLevel(a.chunk + chunks, chunks, shared);
    total_tt = TreeLevel(a.chunk + 2 * chunks, chunks, shared);
  }
  if (t != 0) return;
  // the loads side by side, before the first store: 8.7 us at 64^2 against 11.9 with a load after each store
  const int64_t it = state->iteration + 1;
  const bool scattered = static_cast<int64_t>(state->unfit) > a.unfit_limit;
  const int32_t overflow = state->overflow;
  const unsigned long long nnz_m = state->nnz_m;
  const unsigned long long nnz_z = state->nnz_z;
  const unsigned long long nnz_dir = state->nnz_dir;
  const int64_t parity = state->parity;
  const int64_t bodies = state->bodies + 1;
  state->arrive = 0u;
  const double entries = Mul(static_cast<double>(a.n), static_cast<double>(a.n));
  FusedRow row;
  row.iteration = it;
  row.residual_norm = __dsqrt_rn(total_sq);
  row.density_m = __ddiv_rn(static_cast<double>(nnz_m), entries);
  // the row's direction is the Z the step M += alpha Z used, not the one just formed
  // (the history row is appended before Z is recomputed, minimal_residual.cpp:78-88)
  row.density_direction = __ddiv_rn(static_cast<double>(nnz_dir), entries);
  a.history[it] = row;
  state->iteration = it;
  state->last_nnz_m = nnz_m;
  state->last_nnz_z = nnz_z;
  state->nnz_dir = nnz_z;
  state->nnz_m = 0ull;
  state->nnz_z = 0ull;
  state->unfit = 0u;
  int stop = kRunning;
  if (overflow != 0) {
    stop = kOverflowStop;
  } else if (row.residual_norm < a.tolerance) {
    stop = kConverged;
  } else if (it >= a.max_iterations) {
    stop = kIterationLimit;
  } else {
    // the next iteration's step length (minimal_residual.cpp:55-60)
    const double num = total_bt;
    const double den = total_tt;
    if (!isfinite(den) || !(fabs(den) > 0.0)) {
      stop = kBreakdown;
    } else {
      const double alpha = __ddiv_rn(num, den);
      if (!isfinite(alpha)) {
        stop = kBreakdown;
      } else {
        state->alpha = alpha;
        if (scattered) stop = kScatteredStop;
      }
    }
  }
  state->stop = stop;
  state->parity = parity ^ 1;
  state->bodies = bodies;
  if (in_graph) {
    // the body count bounds the loop whatever the recurrence does
    const bool again = stop == kRunning && bodies < a.max_iterations + 1;
    cudaGraphSetConditional(loop, again ? 1u : 0u);
  }
}

// ---------------------------------------------------------------------------
// Conversions between compact CSC and the slots.

// Column j of a compact CSC into `cap` slots (count per column); when t_cnt is
// given, every entry (i, j) is also appended to row i of the transposed slots.
template <class T>
__global__ void ToSlotsKernel(CscView<T> x, int cap, int32_t* __restrict__ rows, T* __restrict__ vals,
                              int32_t* __restrict__ cnt, int t_cap, int32_t* __restrict__ t_cols, T* __restrict__ t_vals,
                              int32_t* __restrict__ t_cnt, FusedState* __restrict__ state) {
  int overflow = 0;
  for (int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < x.cols;
       j += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t b = x.ptr[j];
    const int64_t e = x.ptr[j + 1];
    const int len = static_cast<int>(e - b);
    if (len > cap) {
      overflow |= kOverflowSide;
      cnt[j] = 0;
      continue;
    }
    for (int q = 0; q < len; ++q) {
      const int32_t i = x.idx[b + q];
      const T v = x.val[b + q];
      rows[j * cap + q] = i;
      vals[j * cap + q] = v;
      if (t_cnt != nullptr) {
        const int slot = atomicAdd(&t_cnt[i], 1);
        if (slot < t_cap) {
          t_cols[static_cast<int64_t>(i) * t_cap + slot] = static_cast<int32_t>(j);
          t_vals[static_cast<int64_t>(i) * t_cap + slot] = v;
        } else {
          overflow |= kOverflowMt;
        }
      }
    }
    cnt[j] = len;
  }
  if (overflow != 0) atomicOr(&state->overflow, overflow);
}

// A batched step is over: the M^T sets change places (the decide kernel's part
// in single runs), unless the step is void.
__global__ void FlipKernel(FusedState* __restrict__ state) {
  if (state->overflow == 0) state->parity ^= 1;
  state->last_unfit = state->unfit;
  state->unfit = 0u;
}

// out[s] = the entries of M and out[count + s] those of Z in the columns [first[s], first[s + 1]); a block each.
__global__ void SegmentCountsKernel(const int32_t* __restrict__ m_cnt, const int32_t* __restrict__ z_cnt,
                                    const int64_t* __restrict__ first, int64_t count, int64_t* __restrict__ out) {
  __shared__ unsigned long long total[2];
  for (int64_t s = blockIdx.x; s < count; s += gridDim.x) {
    if (threadIdx.x < 2) total[threadIdx.x] = 0ull;
    __syncthreads();
    unsigned long long m = 0ull;
    unsigned long long z = 0ull;
    for (int64_t j = first[s] + threadIdx.x; j < first[s + 1]; j += blockDim.x) {
      m += static_cast<unsigned long long>(m_cnt[j]);
      z += static_cast<unsigned long long>(z_cnt[j]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      m += __shfl_xor_sync(0xffffffffu, m, o);
      z += __shfl_xor_sync(0xffffffffu, z, o);
    }
    if ((threadIdx.x & 31) == 0) {
      atomicAdd(&total[0], m);
      atomicAdd(&total[1], z);
    }
    __syncthreads();
    if (threadIdx.x < 2) out[threadIdx.x * count + s] = static_cast<int64_t>(total[threadIdx.x]);
    __syncthreads();
  }
}

__global__ void WidenCountsKernel(const int32_t* __restrict__ cnt, int64_t n, int64_t* __restrict__ out) {
  for (int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < n;
       j += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    out[j] = cnt[j];
  }
}

template <class T>
__global__ void FromSlotsKernel(int64_t n, int cap, const int32_t* __restrict__ rows, const T* __restrict__ vals,
                                const int64_t* __restrict__ ptr, int32_t* __restrict__ idx_out, T* __restrict__ val_out) {
  for (int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; j < n;
       j += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t o = ptr[j];
    const int len = static_cast<int>(ptr[j + 1] - o);
    for (int q = 0; q < len; ++q) {
      idx_out[o + q] = rows[j * cap + q];
      val_out[o + q] = vals[j * cap + q];
    }
  }
}

int CapZ(const FusedMrProblem& p) {
  const int64_t bound = 1 + static_cast<int64_t>(p.topk) * p.a_longest;
  return static_cast<int>(std::min<int64_t>(p.n, bound));
}

int NextPow2Int(int v) {
  int p = 1;
  while (p < v) p <<= 1;
  return p;
}

int CapMt(const FusedMrProblem& p) { return static_cast<int>(std::min<int64_t>(p.n, 4 * static_cast<int64_t>(p.topk))); }

// Slots of the drop kernel's hash of R(j, :): twice the row's bound (every entry of row j of A times a row of M)
// up to 256; a longer row flags an overflow.
int DropRowSlots(const FusedMrProblem& p) {
  const int64_t bound = static_cast<int64_t>(p.a_longest) * CapMt(p) + 1;
  return NextPow2Int(static_cast<int>(std::min<int64_t>(std::max<int64_t>(2 * bound, kWarp), 256)));
}

std::atomic<bool> g_fused_mr_enabled{true};

template <class T>
class FusedMr final : public FusedMrBase {
 public:
  ~FusedMr() override {
    if (exec_ != nullptr) cudaGraphExecDestroy(exec_);
  }

  FusedMrOutcome Run(Ctx& ctx, const FusedMrProblem& problem, void* m_csc, const void* z_csc, double alpha,
                     std::vector<SingleIterationData>& history) override {
    FusedMrOutcome outcome;
    if (!FusedMrApplicable(problem)) return outcome;
    auto& m = *static_cast<DevCsc<T>*>(m_csc);
    const auto& z = *static_cast<const DevCsc<T>*>(z_csc);
    const cudaStream_t st = ctx.stream;
    Start(ctx, problem, m, z, alpha, nullptr);
    FusedState out;
    if (prof::Enabled()) {
      out = RunStepwise(ctx, problem);
    } else {
      do {
        if (exec_ == nullptr) Capture();
        SPAI_CUDA(cudaGraphLaunch(exec_, st));
        SPAI_CUDA(cudaMemcpyAsync(host_state_, state_.data(), sizeof(FusedState), cudaMemcpyDeviceToHost, st));
        ctx.Sync();
        out = *host_state_;
        if (out.stop == kScatteredStop) LeaveGroups(problem);
      } while (out.stop == kScatteredStop);
      CountLaunches(3 * out.bodies);
    }
    outcome.ran = true;
    outcome.graph_bodies = out.bodies;
    if (out.stop == kOverflowStop || out.overflow != 0) {
      outcome.overflow = true;
      return outcome;
    }
    const int64_t rows = out.iteration;
    std::vector<FusedRow> host_rows(static_cast<size_t>(rows + 1));
    SPAI_CUDA(cudaMemcpyAsync(host_rows.data(), args_.history, sizeof(FusedRow) * (rows + 1), cudaMemcpyDeviceToHost,
                              st));
    CompactM(ctx, m);
    ctx.Sync();
    for (int64_t r = 1; r <= rows; ++r) {
      SingleIterationData row;
      row.iteration = host_rows[r].iteration;
      row.residual_norm = host_rows[r].residual_norm;
      row.density_m = host_rows[r].density_m;
      row.density_direction = host_rows[r].density_direction;
      history.push_back(row);
    }
    outcome.iterations = rows;
    outcome.converged = out.stop == kConverged;
    return outcome;
  }

  bool BeginBatch(Ctx& ctx, const FusedMrProblem& problem, const void* m_csc, const void* z_csc,
                  const double* alpha) override {
    if (!FusedMrApplicable(problem)) return false;
    Start(ctx, problem, *static_cast<const DevCsc<T>*>(m_csc), *static_cast<const DevCsc<T>*>(z_csc), 0.0, alpha);
    problem_ = problem;
    return true;
  }

  FusedBatchSums StepBatch(Ctx& ctx) override {
    const cudaStream_t st = ctx.stream;
    {
      prof::Scope scope(st, drop_class_, 0.0);
      drop_kernel_<<<drop_grid_, warps_ * kWarp, drop_smem_, st>>>(args_);
      SPAI_LAUNCH_CHECK();
    }
    {
      prof::Scope scope(st, res_class_, 0.0);
      res_kernel_<<<res_grid_, warps_ * kWarp, res_smem_, st>>>(args_);
      SPAI_LAUNCH_CHECK();
    }
    FlipKernel<<<1, 1, 0, st>>>(args_.state);
    SPAI_LAUNCH_CHECK();
    return FusedBatchSums{args_.sq, args_.bt, args_.tt};
  }

  bool BatchCounts(Ctx& ctx, const int64_t* first, int64_t segments, int64_t* out_dev, int64_t* out) override {
    const cudaStream_t st = ctx.stream;
    SegmentCountsKernel<<<static_cast<unsigned>(std::min<int64_t>(segments, 65535)), 256, 0, st>>>(
        args_.m_cnt, args_.z_cnt, first, segments, out_dev);
    SPAI_LAUNCH_CHECK();
    SPAI_CUDA(cudaMemcpyAsync(host_state_, state_.data(), sizeof(FusedState), cudaMemcpyDeviceToHost, st));
    SPAI_CUDA(cudaMemcpyAsync(out, out_dev, sizeof(int64_t) * 2 * segments, cudaMemcpyDeviceToHost, st));
    ctx.Sync();
    if (host_state_->overflow != 0) return false;
    if (prof::Enabled()) {
      int64_t m_entries = 0;
      int64_t z_entries = 0;
      for (int64_t s = 0; s < segments; ++s) {
        m_entries += out[s];
        z_entries += out[segments + s];
      }
      AddStepBytes(problem_, static_cast<double>(m_entries), static_cast<double>(z_entries));
    }
    if (host_state_->last_unfit > args_.unfit_limit) LeaveGroups(problem_);
    return true;
  }

  void CompactBatch(Ctx& ctx, void* m_csc) override { CompactM(ctx, *static_cast<DevCsc<T>*>(m_csc)); }

  void RecoverBatch(Ctx& ctx, void* m_csc, void* z_csc) override {
    // the drop kernel has overwritten M's columns, but not the M^T it read
    const int64_t set = host_state_->parity;
    DevCsc<T> mt;
    Compact(ctx, args_.cap_mt, args_.mt_cols[set], args_.mt_vals[set], args_.mt_cnt[set], mt);
    Transpose(ctx, mt, *static_cast<DevCsc<T>*>(m_csc));
    Compact(ctx, args_.cap_z, args_.z_rows, args_.z_vals, args_.z_cnt, *static_cast<DevCsc<T>*>(z_csc));
  }

 private:
  // The slots filled from M and Z, the state at iteration 0 (M^T set 0 current).
  void Start(Ctx& ctx, const FusedMrProblem& problem, const DevCsc<T>& m, const DevCsc<T>& z, double alpha,
             const double* alpha_columns) {
    const cudaStream_t st = ctx.stream;
    const int64_t n = problem.n;
    Reserve(ctx, problem);
    Configure(problem);
    args_.alpha = alpha_columns;
    m_entries_ = static_cast<double>(m.nnz);
    z_entries_ = static_cast<double>(z.nnz);
    FusedState init{};
    init.alpha = alpha;
    init.nnz_dir = static_cast<unsigned long long>(z.nnz);
    *host_state_ = init;
    SPAI_CUDA(cudaMemcpyAsync(state_.data(), host_state_, sizeof(FusedState), cudaMemcpyHostToDevice, st));
    for (int s = 0; s < 2; ++s) SPAI_CUDA(cudaMemsetAsync(mt_cnt_[s].data(), 0, sizeof(int32_t) * n, st));
    const int grid = GridFor(n, 128);
    ToSlotsKernel<T><<<grid, 128, 0, st>>>(View(m), args_.topk, args_.m_rows, args_.m_vals, args_.m_cnt, args_.cap_mt,
                                           args_.mt_cols[0], args_.mt_vals[0], args_.mt_cnt[0], args_.state);
    SPAI_LAUNCH_CHECK();
    ToSlotsKernel<T><<<grid, 128, 0, st>>>(View(z), args_.cap_z, args_.z_rows, args_.z_vals, args_.z_cnt, 0,
                                           nullptr, nullptr, nullptr, args_.state);
    SPAI_LAUNCH_CHECK();
  }

  // M back to compact CSC.
  void CompactM(Ctx& ctx, DevCsc<T>& m) { Compact(ctx, args_.topk, args_.m_rows, args_.m_vals, args_.m_cnt, m); }

  // Slots to compact columns, each column's entries in slot order.
  void Compact(Ctx& ctx, int cap, const int32_t* rows, const T* vals, const int32_t* cnt, DevCsc<T>& out) {
    const cudaStream_t st = ctx.stream;
    const int64_t n = args_.n;
    DevCsc<T> result;
    result.Shape(n, n, st);
    ctx.counts.Reserve(static_cast<size_t>(n + 1), st);
    WidenCountsKernel<<<GridFor(n, 256), 256, 0, st>>>(cnt, n, ctx.counts.data());
    SPAI_LAUNCH_CHECK();
    const int64_t nnz = ScanCounts(ctx, ctx.counts.data(), n, result.ptr.data());
    result.ReserveNnz(nnz, st);
    FromSlotsKernel<T><<<GridFor(n, 128), 128, 0, st>>>(n, cap, rows, vals, result.ptr.data(), result.idx.data(),
                                                        result.val.data());
    SPAI_LAUNCH_CHECK();
    out.Swap(result);
  }

  // Algorithmic bytes of a step that left m_new entries in M and z_new in Z: the
  // drop step reads M, Z and both transposes and writes M and M^T; the residual
  // step reads M, A and Pr, writes Z, Z^T and the three column sums.
  void AddStepBytes(const FusedMrProblem& p, double m_new, double z_new) {
    const double e = static_cast<double>(sizeof(T) + sizeof(int32_t));
    const double n = static_cast<double>(p.n);
    const double a_bytes = static_cast<double>(p.a_nnz) * e + 8.0 * (n + 1.0);
    prof::AddBytes(drop_class_, e * (2.0 * m_entries_ + 2.0 * z_entries_ + 2.0 * m_new) + 4.0 * 6.0 * n);
    prof::AddBytes(res_class_, e * m_new + a_bytes + sizeof(T) * n + 2.0 * e * z_new + 4.0 * 3.0 * n + 24.0 * n);
    m_entries_ = m_new;
    z_entries_ = z_new;
  }

  // The same three kernels launched one by one with the library's CUDA-event
  // accounting around each (spai_profile_enable): the decide kernel's result
  // is read back after every iteration, in place of the graph's condition.
  FusedState RunStepwise(Ctx& ctx, const FusedMrProblem& p) {
    const cudaStream_t st = ctx.stream;
    const double n = static_cast<double>(p.n);
    FusedState out{};
    for (int64_t body = 0; body <= p.max_iterations; ++body) {
      {
        prof::Scope scope(st, drop_class_, 0.0);
        drop_kernel_<<<drop_grid_, warps_ * kWarp, drop_smem_, st>>>(args_);
        SPAI_LAUNCH_CHECK();
      }
      {
        prof::Scope scope(st, res_class_, 0.0);
        res_kernel_<<<res_grid_, warps_ * kWarp, res_smem_, st>>>(args_);
        SPAI_LAUNCH_CHECK();
      }
      {
        prof::Scope scope(st, "fused_decide", 24.0 * n);
        FusedDecideKernel<T><<<decide_grid_, kTreeLanes, 0, st>>>(args_, 0, false);
        SPAI_LAUNCH_CHECK();
      }
      SPAI_CUDA(cudaMemcpyAsync(host_state_, state_.data(), sizeof(FusedState), cudaMemcpyDeviceToHost, st));
      ctx.Sync();
      out = *host_state_;
      AddStepBytes(p, static_cast<double>(out.last_nnz_m), static_cast<double>(out.last_nnz_z));
      if (out.stop == kScatteredStop) {
        LeaveGroups(p);
      } else if (out.stop != kRunning) {
        break;
      }
    }
    return out;
  }

  void Reserve(Ctx& ctx, const FusedMrProblem& p) {
    const cudaStream_t st = ctx.stream;
    const int64_t n = p.n;
    const int cap_z = CapZ(p);
    const int cap_mt = CapMt(p);
    const size_t un = static_cast<size_t>(n);
    m_rows_.Reserve(un * p.topk, st);
    m_vals_.Reserve(un * p.topk, st);
    m_cnt_.Reserve(un, st);
    for (int s = 0; s < 2; ++s) {
      mt_cols_[s].Reserve(un * cap_mt, st);
      mt_vals_[s].Reserve(un * cap_mt, st);
      mt_cnt_[s].Reserve(un, st);
    }
    z_rows_.Reserve(un * cap_z, st);
    z_vals_.Reserve(un * cap_z, st);
    z_cnt_.Reserve(un, st);
    sq_.Reserve(un, st);
    tt_.Reserve(un, st);
    bt_.Reserve(un, st);
    chunk_.Reserve(static_cast<size_t>(3 * CeilDiv(n, kTreeChunk)), st);
    history_.Reserve(static_cast<size_t>(p.max_iterations + 1), st);
    state_.Reserve(1, st);
    if (host_state_ == nullptr) {
      SPAI_CUDA(cudaMallocHost(reinterpret_cast<void**>(&host_state_), sizeof(FusedState)));
      host_state_holder_.reset(host_state_);
    }
    FusedArgs<T> a{};
    a.n = n;
    a.topk = p.topk;
    a.cap_z = cap_z;
    a.cap_mt = cap_mt;
    a.ell = p.ell_width;
    a.m_hash_slots = NextPow2Int(std::max(4 * p.topk, kWarp));
    a.z_hash_slots = NextPow2Int(std::max(2 * cap_z, kWarp));
    a.d_mt_slots = NextPow2Int(std::max(2 * cap_mt, kWarp));
    a.d_r_slots = DropRowSlots(p);
    a.words = scattered_ ? 0 : GroupWords(p);
    a.bandwidth = p.bandwidth;
    a.max_iterations = p.max_iterations;
    a.tolerance = p.tolerance;
    a.a_cols_ell = p.a_cols_ell;
    a.a_rows_ell = p.a_rows_ell;
    a.a_rows_ell_val = static_cast<const T*>(p.a_rows_ell_val);
    a.pr = static_cast<const T*>(p.pr);
    a.m_rows = m_rows_.data();
    a.m_vals = m_vals_.data();
    a.m_cnt = m_cnt_.data();
    for (int s = 0; s < 2; ++s) {
      a.mt_cols[s] = mt_cols_[s].data();
      a.mt_vals[s] = mt_vals_[s].data();
      a.mt_cnt[s] = mt_cnt_[s].data();
    }
    a.z_rows = z_rows_.data();
    a.z_vals = z_vals_.data();
    a.z_cnt = z_cnt_.data();
    a.sq = sq_.data();
    a.tt = tt_.data();
    a.bt = bt_.data();
    a.chunk = chunk_.data();
    a.history = history_.data();
    a.state = state_.data();
    // a captured graph holds the old pointers and sizes: capture again on any change
    if (exec_ != nullptr && !SameArgs(a, args_)) {
      cudaGraphExecDestroy(exec_);
      exec_ = nullptr;
    }
    args_ = a;
  }

  static bool SameArgs(const FusedArgs<T>& x, const FusedArgs<T>& y) {
    bool same = x.n == y.n && x.topk == y.topk && x.cap_z == y.cap_z && x.cap_mt == y.cap_mt &&
                x.ell == y.ell && x.words == y.words && x.bandwidth == y.bandwidth && x.m_hash_slots == y.m_hash_slots && x.d_r_slots == y.d_r_slots &&
                x.d_mt_slots == y.d_mt_slots &&
                x.z_hash_slots == y.z_hash_slots && x.max_iterations == y.max_iterations &&
                x.tolerance == y.tolerance && x.a_cols_ell == y.a_cols_ell && x.a_rows_ell == y.a_rows_ell &&
                x.a_rows_ell_val == y.a_rows_ell_val && x.pr == y.pr && x.m_rows == y.m_rows &&
                x.m_vals == y.m_vals && x.m_cnt == y.m_cnt && x.z_rows == y.z_rows && x.z_vals == y.z_vals &&
                x.z_cnt == y.z_cnt &&
                x.alpha == y.alpha && x.sq == y.sq && x.tt == y.tt && x.bt == y.bt && x.chunk == y.chunk && x.history == y.history &&
                x.state == y.state;
    for (int s = 0; s < 2; ++s) {
      same = same && x.mt_cols[s] == y.mt_cols[s] && x.mt_vals[s] == y.mt_vals[s] && x.mt_cnt[s] == y.mt_cnt[s];
    }
    return same;
  }

  // Words of a group's window: a little over four bandwidths of A on either
  // side of the group, which covers the drop step's and the residual's rows of
  // nearly every column (M reaches two to three bandwidths, R one more).  Wider
  // operators (a bandwidth above about 7,900: 3-D grids from 89^3 up, unordered
  // meshes), and operators with entries that are not finite (a column group
  // multiplies them by the 0 of an absent entry), go column by column.
  static int GroupWords(const FusedMrProblem& p) {
    if (!p.finite) return 0;
    const int64_t words = CeilDiv(8 * p.bandwidth + p.bandwidth / 4, 32) + 8;
    return words > kMaxGroupWords ? 0 : static_cast<int>(CeilDiv(words, 32) * 32);
  }

  // Columns per group: four, or two while four would leave the chip's warps
  // idle (below 16 groups of four per SM).  Drop and residual together, 5-point
  // FP64, 16 entries: 44 us in groups of two against 50 in groups of four at
  // n = 4,096, 69 against 71 at n = 8,100 (62 column by column at 4,096).
  // kUse: the longest row of A, compile time for the 5-point and 7-point
  // operators (2-D rows would else look up three slots of padding in eight).
  template <int kEll, int kUse, int C>
  void Choose() {
    res_kernel_ = FusedResidualKernel<T, kEll, kUse, C>;
    drop_kernel_ = FusedDropKernel<T, kEll, C>;
    columns_ = C;
    warps_ = kGroupWarps;
    drop_class_ = "fused_drop";
    res_class_ = "fused_residual";
    args_.drop_bytes = Round16(std::max(DropWarpBytes<T>(args_.topk + args_.cap_z, args_.d_mt_slots, args_.d_r_slots),
                                        DropGroupBytes<T, C>(args_.words)));
    args_.residual_bytes = Round16(std::max(ResidualSlabBytes<T>(args_.m_hash_slots, args_.z_hash_slots),
                                            ResidualGroupBytes<T, C>(args_.words, args_.topk)));
  }

  // Without a window (GroupWords): the kernels that take one column after another.
  void ChooseColumns(int ell) {
    switch (ell) {
      case 4: res_kernel_ = FusedResidualColumnsKernel<T, 4>; break;
      case 8: res_kernel_ = FusedResidualColumnsKernel<T, 8>; break;
      case 12: res_kernel_ = FusedResidualColumnsKernel<T, 12>; break;
      case 16: res_kernel_ = FusedResidualColumnsKernel<T, 16>; break;
      default: throw std::invalid_argument("fused MR: unsupported ELL width");
    }
    drop_kernel_ = FusedDropColumnsKernel<T>;
    columns_ = 1;
    warps_ = kColumnWarps;
    drop_class_ = "fused_drop_columns";
    res_class_ = "fused_residual_columns";
    args_.drop_bytes = Round16(DropWarpBytes<T>(args_.topk + args_.cap_z, args_.d_mt_slots, args_.d_r_slots));
    args_.residual_bytes = Round16(ResidualSlabBytes<T>(args_.m_hash_slots, args_.z_hash_slots));
  }

  template <int C>
  void ChooseEll(int ell, int64_t longest) {
    switch (ell) {
      case 4: Choose<4, 4, C>(); break;
      case 8:  // the 5-point and 7-point rows have kernels of their own length
        if (longest <= 5) {
          Choose<8, 5, C>();
        } else if (longest <= 7) {
          Choose<8, 7, C>();
        } else {
          Choose<8, 8, C>();
        }
        break;
      case 12: Choose<12, 12, C>(); break;
      case 16: Choose<16, 16, C>(); break;
      default: throw std::invalid_argument("fused MR: unsupported ELL width");
    }
  }

  // The following iterations, of this run and of later ones on this problem, go
  // column by column: more than a sixteenth of the two kernels' groups did not
  // fit.  Such a group costs its attempt and the slow way through its columns
  // (few warps, generic addresses).  47^3, 16 entries a column, FP32 storage, ten
  // iterations, rows shuffled within 10, 30, 100 and 2,000 so that 3, 16, 24 and
  // 45 % of the groups do not fit: 12.8, 21.5, 24.8 and 31.9 ms in groups against
  // 15.3, 14.6, 14.8 and 15.3 column by column (7.7 unshuffled); in FP64 16.3,
  // 26.5, 28.9 and 36.2 against 19.2, 18.3, 18.6 and 19.1.
  void LeaveGroups(const FusedMrProblem& p) {
    scattered_ = true;
    args_.words = 0;
    Configure(p);
    if (exec_ != nullptr) {
      cudaGraphExecDestroy(exec_);
      exec_ = nullptr;
    }
  }

  // Kernel choice, shared memory and grids (once per problem shape).
  void Configure(const FusedMrProblem& p) {
    int device = 0;
    SPAI_CUDA(cudaGetDevice(&device));
    int sms = 0;
    SPAI_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    if (args_.words == 0) {
      ChooseColumns(p.ell_width);
    } else if (args_.n >= int64_t{4} * 16 * sms) {
      ChooseEll<4>(p.ell_width, p.a_longest);
    } else {
      ChooseEll<2>(p.ell_width, p.a_longest);
    }
    drop_smem_ = static_cast<size_t>(warps_) * args_.drop_bytes;
    res_smem_ = static_cast<size_t>(warps_) * args_.residual_bytes;
    SPAI_CUDA(cudaFuncSetAttribute(drop_kernel_, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(drop_smem_)));
    SPAI_CUDA(cudaFuncSetAttribute(res_kernel_, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                   static_cast<int>(res_smem_)));
    int drop_blocks = 0;
    int res_blocks = 0;
    SPAI_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&drop_blocks, drop_kernel_, warps_ * kWarp, drop_smem_));
    SPAI_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&res_blocks, res_kernel_, warps_ * kWarp, res_smem_));
    if (drop_blocks < 1 || res_blocks < 1) throw std::runtime_error("fused MR: kernels do not fit on an SM");
    args_.unfit_limit = columns_ > 1 ? CeilDiv(args_.n, int64_t{columns_}) / 8 : INT64_MAX;
    const int64_t blocks = CeilDiv(args_.n, int64_t{warps_} * columns_);
    drop_grid_ = static_cast<unsigned>(std::min<int64_t>(blocks, int64_t{sms} * drop_blocks));
    res_grid_ = static_cast<unsigned>(std::min<int64_t>(blocks, int64_t{sms} * res_blocks));
    decide_grid_ = static_cast<unsigned>(CeilDiv(args_.n, kTreeChunk));
  }

  void Capture() {
    const FusedArgs<T> a = args_;
    cudaStream_t cs = nullptr;
    cudaStream_t bs = nullptr;
    cudaGraph_t graph = nullptr;
    SPAI_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
    try {
      SPAI_CUDA(cudaStreamCreateWithFlags(&bs, cudaStreamNonBlocking));
      SPAI_CUDA(cudaStreamBeginCapture(cs, cudaStreamCaptureModeThreadLocal));
      cudaStreamCaptureStatus status;
      cudaGraph_t capture_graph = nullptr;
      const cudaGraphNode_t* deps = nullptr;
      size_t num_deps = 0;
      SPAI_CUDA(cudaStreamGetCaptureInfo(cs, &status, nullptr, &capture_graph, &deps, &num_deps));
      cudaGraphConditionalHandle loop;
      SPAI_CUDA(cudaGraphConditionalHandleCreate(&loop, capture_graph, 1, cudaGraphCondAssignDefault));
      cudaGraphNodeParams params = {};
      params.type = cudaGraphNodeTypeConditional;
      params.conditional.handle = loop;
      params.conditional.type = cudaGraphCondTypeWhile;
      params.conditional.size = 1;
      cudaGraphNode_t loop_node;
      SPAI_CUDA(cudaGraphAddNode(&loop_node, capture_graph, deps, num_deps, &params));
      SPAI_CUDA(cudaStreamUpdateCaptureDependencies(cs, &loop_node, 1, cudaStreamSetCaptureDependencies));
      cudaGraph_t body = params.conditional.phGraph_out[0];
      SPAI_CUDA(cudaStreamBeginCaptureToGraph(bs, body, nullptr, nullptr, 0, cudaStreamCaptureModeThreadLocal));
      drop_kernel_<<<drop_grid_, warps_ * kWarp, drop_smem_, bs>>>(a);
      res_kernel_<<<res_grid_, warps_ * kWarp, res_smem_, bs>>>(a);
      FusedDecideKernel<T><<<decide_grid_, kTreeLanes, 0, bs>>>(a, loop, true);
      SPAI_CUDA(cudaGetLastError());
      cudaGraph_t body_out = nullptr;
      SPAI_CUDA(cudaStreamEndCapture(bs, &body_out));
      SPAI_CUDA(cudaStreamEndCapture(cs, &graph));
      SPAI_CUDA(cudaGraphInstantiate(&exec_, graph, 0));
    } catch (...) {
      cudaStreamCaptureStatus st;
      for (cudaStream_t stream : {bs, cs}) {
        if (stream != nullptr && cudaStreamIsCapturing(stream, &st) == cudaSuccess &&
            st != cudaStreamCaptureStatusNone) {
          cudaGraph_t dropped = nullptr;
          cudaStreamEndCapture(stream, &dropped);
          if (dropped != nullptr && stream == cs) cudaGraphDestroy(dropped);
        }
      }
      if (graph != nullptr) cudaGraphDestroy(graph);
      if (bs != nullptr) cudaStreamDestroy(bs);
      cudaStreamDestroy(cs);
      cudaGetLastError();
      exec_ = nullptr;
      throw;
    }
    cudaGraphDestroy(graph);
    cudaStreamDestroy(bs);
    cudaStreamDestroy(cs);
  }

  struct PinnedFree {
    void operator()(FusedState* p) const { cudaFreeHost(p); }
  };

  DevBuf<int32_t> m_rows_, m_cnt_, z_rows_, z_cnt_;
  DevBuf<T> m_vals_, z_vals_;
  DevBuf<int32_t> mt_cols_[2], mt_cnt_[2];
  DevBuf<T> mt_vals_[2];
  DevBuf<double> sq_, tt_, bt_, chunk_;
  DevBuf<FusedRow> history_;
  DevBuf<FusedState> state_;
  FusedState* host_state_ = nullptr;
  std::unique_ptr<FusedState, PinnedFree> host_state_holder_;
  FusedArgs<T> args_{};
  cudaGraphExec_t exec_ = nullptr;
  void (*res_kernel_)(const FusedArgs<T>) = nullptr;
  void (*drop_kernel_)(const FusedArgs<T>) = nullptr;
  FusedMrProblem problem_;   // of the running batch
  double m_entries_ = 0.0;   // entries of M and Z that the next step starts from
  double z_entries_ = 0.0;
  bool scattered_ = false;   // the problem's column groups do not fit
  int columns_ = 1;  // per warp
  int warps_ = 1;    // per block
  const char* drop_class_ = "";  // profile classes of the two kernels
  const char* res_class_ = "";
  size_t drop_smem_ = 0;
  size_t res_smem_ = 0;
  unsigned drop_grid_ = 1;
  unsigned res_grid_ = 1;
  unsigned decide_grid_ = 1;
};

}  // namespace

bool FusedMrEnabled() { return g_fused_mr_enabled.load(std::memory_order_relaxed); }
void SetFusedMrEnabled(bool enabled) { g_fused_mr_enabled.store(enabled, std::memory_order_relaxed); }

bool FusedMrApplicable(const FusedMrProblem& p) {
  if (p.n <= 0 || p.n > kTreeChunk * kTreeChunk) return false;
  if (p.topk <= 0 || p.topk > kMaxTopK) return false;
  if (p.ell_width != 4 && p.ell_width != 8 && p.ell_width != 12 && p.ell_width != 16) return false;
  if (p.a_longest <= 0 || p.a_longest > p.ell_width) return false;
  if (p.max_iterations < 1) return false;
  const int cap_z = CapZ(p);
  // a drop column's candidate rows and a product column's row lists must fit
  const int64_t drop_candidates = p.topk + cap_z + CapMt(p) + DropRowSlots(p) / 2 + 1;
  if (drop_candidates > kDropRowsCap) return false;
  if (static_cast<int64_t>(cap_z) * p.a_longest > kRowsCap) return false;
  return true;
}

template <class T>
std::unique_ptr<FusedMrBase> MakeFusedMr() {
  return std::unique_ptr<FusedMrBase>(new FusedMr<T>());
}

template std::unique_ptr<FusedMrBase> MakeFusedMr<double>();
template std::unique_ptr<FusedMrBase> MakeFusedMr<float>();

}  // namespace spai
