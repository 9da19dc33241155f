#pragma once
// A sequential floating-point sum s = fl(s + t) over t = t[0], t[1], ...,
// split into pieces that are summarised independently and still give the
// sequential sum's bits.
//
// While the running sum stays inside one binade [2^e, 2^(e+1)), it is m * u
// with u = 2^(e-52) and an integer m in [2^52, 2^53), and adding t rounds
// t / u to an integer: m -> m + round(t / u).  The rounded increment does not
// depend on m, except at an exact tie, where round-to-even looks at the parity
// of m.  A run of terms therefore maps m to m + inc[m & 1], and such maps
// compose (the second map's index is the parity after the first).  The map is
// the sequential sum as long as no intermediate m left the binade, which the
// smallest and largest intermediate offsets (lo, hi) decide once m is known.
// Where that check fails -- at a change of binade, a few dozen times in a long
// sum, or at zeros, subnormals and non-finite values -- the piece is added
// term by term.  Negative sums are the mirror image: round-to-even is
// symmetric.

#include <cstdint>
#include <cstring>
#include <cmath>

#ifdef __CUDACC__
#define SPAI_HD __host__ __device__ __forceinline__
#else
#define SPAI_HD inline
#endif

namespace spai {

constexpr int64_t kBinadeLow = int64_t{1} << 52;   // m of the binade's first value
constexpr int64_t kBinadeHigh = int64_t{1} << 53;  // first m past the binade
constexpr int64_t kNoOffset = int64_t{1} << 60;    // lo / -hi of an empty run

SPAI_HD uint64_t DoubleBits(double v) {
#ifdef __CUDA_ARCH__
  return static_cast<uint64_t>(__double_as_longlong(v));
#else
  uint64_t u;
  std::memcpy(&u, &v, sizeof(u));
  return u;
#endif
}

SPAI_HD double BitsDouble(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double(static_cast<long long>(u));
#else
  double v;
  std::memcpy(&v, &u, sizeof(v));
  return v;
#endif
}

// How a run acts on a running sum m * u of known binade, by the parity of m.
struct SumMap {
  int64_t inc[2];
  int64_t lo[2];  // smallest intermediate offset (one less where the step was downward)
  int64_t hi[2];  // largest
  int bad;        // 1: some term cannot stay in any binade of this u
};

SPAI_HD SumMap EmptyMap() { return SumMap{{0, 0}, {kNoOffset, kNoOffset}, {-kNoOffset, -kNoOffset}, 0}; }

// The running sum's binade: kNormal (scale = 1 / u, sign), kZero or kOther (added term by term).
enum SumState : int { kSumNormal = 0, kSumZero = 1, kSumOther = 2 };

SPAI_HD SumState Classify(double s, double* scale) {
  const uint64_t bits = DoubleBits(s);
  const int field = static_cast<int>((bits >> 52) & 0x7FF);
  *scale = 0.0;
  if ((bits << 1) == 0) return kSumZero;
  // 1 / u = 2^(52 - e), e = field - 1023, is a normal number for field >= 52
  if (field == 0x7FF || field < 52) return kSumOther;
  *scale = BitsDouble((static_cast<uint64_t>(2098 - field) << 52) | (bits & 0x8000000000000000ull));
  return kSumNormal;
}

// The map of one term; scale carries the running sum's sign, so q counts
// upward in magnitude.  The product is a power-of-two scaling: exact, or an
// underflow far below a tie, which rounds to no increment either way.
SPAI_HD SumMap TermMap(double t, double scale, SumState state) {
  if (state == kSumZero) return SumMap{{0, 0}, {0, 0}, {0, 0}, t == 0.0 ? 0 : 1};
  const double q = t * scale;
  if (!(fabs(q) < 4503599627370496.0)) return SumMap{{0, 0}, {0, 0}, {0, 0}, 1};
  const double k = floor(q);
  const double f = q - k;  // exact below 2^52
  const int64_t ki = static_cast<int64_t>(k);
  SumMap m;
  m.bad = 0;
  for (int p = 0; p < 2; ++p) {
    const int64_t up = f > 0.5 ? 1 : (f == 0.5 ? ((p + ki) & 1) : 0);
    m.inc[p] = ki + up;
    m.hi[p] = m.inc[p];
    // a step down from the binade's first value rounds on the finer grid below it
    m.lo[p] = m.inc[p] - (q < 0.0 || (t != 0.0 && (DoubleBits(q) >> 63)) ? 1 : 0);
  }
  return m;
}

// First a, then b.
SPAI_HD SumMap Then(const SumMap& a, const SumMap& b) {
  SumMap c;
  int bad = a.bad | b.bad;
  for (int p = 0; p < 2; ++p) {
    const int p2 = static_cast<int>((p + a.inc[p]) & 1);
    c.inc[p] = a.inc[p] + b.inc[p2];
    const int64_t lo = a.inc[p] + b.lo[p2];
    const int64_t hi = a.inc[p] + b.hi[p2];
    c.lo[p] = a.lo[p] < lo ? a.lo[p] : lo;
    c.hi[p] = a.hi[p] > hi ? a.hi[p] : hi;
    // an offset this far out has left every binade: no value below needs more than 54 bits
    if (c.hi[p] > kBinadeHigh || c.lo[p] < -kBinadeHigh) bad = 1;
  }
  c.bad = bad;
  if (bad) {
    c.inc[0] = c.inc[1] = 0;
    c.lo[0] = c.lo[1] = kNoOffset;
    c.hi[0] = c.hi[1] = -kNoOffset;
  }
  return c;
}

// True when the run keeps the sum s in its binade; *out is the sum after it.
SPAI_HD bool ApplyMap(const SumMap& map, double s, SumState state, double* out) {
  if (map.bad || state == kSumOther) return false;
  *out = s;
  if (state == kSumZero) return true;
  const uint64_t bits = DoubleBits(s);
  const int64_t m = static_cast<int64_t>((bits & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull);
  const int p = static_cast<int>(m & 1);
  if (m + map.lo[p] < kBinadeLow || m + map.hi[p] >= kBinadeHigh) return false;
  const uint64_t moved = static_cast<uint64_t>(m + map.inc[p]);
  *out = BitsDouble((bits & 0xFFF0000000000000ull) | (moved & 0x000FFFFFFFFFFFFFull));
  return true;
}

}  // namespace spai
