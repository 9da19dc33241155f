#pragma once
// A sequential floating-point sum s = fl(s + t) over t = t[0], t[1], ...,
// split into pieces that are summarised independently and still give the
// sequential sum's bits.
//
// While the running sum stays inside one binade [2^e, 2^(e+1)), it is m * u
// with u = 2^(e-52) and an integer m in [2^52, 2^53), and adding t rounds
// t / u to an integer: m -> m + round(t / u).  The rounded increment does not
// depend on m, except at an exact tie, where round-to-even looks at the parity
// of m.  A run of terms therefore moves m by inc[m & 1], and such maps compose
// (the second map's index is the parity after the first).  The map is the
// sequential sum as long as no intermediate m left the binade, which bounds on
// the intermediate offsets (lo, hi) decide once m is known.  Where that check
// fails -- at a change of binade, a few dozen times in a long sum, or at
// zeros, subnormals and non-finite values -- the piece is added term by term.
// Negative sums are the mirror image: round-to-even is symmetric.
//
// Increments and bounds are doubles: integers below 2^53 are exact, and a run
// that moves m by 2^51 or more counts as leaving the binade.

#include <cmath>
#include <cstdint>
#include <cstring>

#ifdef __CUDACC__
#define SPAI_HD __host__ __device__ __forceinline__
#else
#define SPAI_HD inline
#endif

namespace spai {

constexpr double kSumLimit = 2251799813685248.0;    // 2^51
constexpr double kSumMagic = 6755399441055744.0;    // 1.5 * 2^52: adding and taking it away rounds |q| < 2^51 to even
constexpr int64_t kBinadeLow = int64_t{1} << 52;    // m of the binade's first value
constexpr int64_t kBinadeHigh = int64_t{1} << 53;   // first m past the binade

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

// How a run of terms acts on a running sum m * u of known binade.
struct SumMap {
  double inc[2];  // by the parity of m
  double lo;      // at most every intermediate offset (one less where a step was downward)
  double hi;      // at least every intermediate offset
  int bad;        // 1: some term cannot stay in any binade of this u
};

SPAI_HD SumMap EmptyMap() { return SumMap{{0.0, 0.0}, 0.0, 0.0, 0}; }

// The running sum's binade: kSumNormal (scale = 1 / u with the sum's sign), kSumZero or kSumOther (term by term).
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

// Whether an integer of magnitude below 2^51 is odd.
SPAI_HD bool OddInteger(double v) { return (DoubleBits(v + kSumMagic) & 1u) != 0u; }

// The running map of a run of terms, extended by one term after another:
// inc, the sums of the upward and of the downward steps, and two flags.
struct TermRun {
  double inc[2] = {0.0, 0.0};
  double up = 0.0;
  double down = 0.0;
  bool far = false;       // a term cannot stay in the binade
  bool downward = false;  // a step below 0

  // scale carries the running sum's sign, so q counts upward in magnitude.
  // The product is a power-of-two scaling: exact, or an underflow far below a
  // tie, which rounds to no increment either way.
  SPAI_HD void Add(double t, double scale) {
    const double q = t * scale;
    const double r = (q + kSumMagic) - kSumMagic;  // ties to even
    far = far || !(fabs(q) < kSumLimit);
    // a step down from the binade's first value rounds on the finer grid below it
    downward = downward || q < 0.0 || (t != 0.0 && (DoubleBits(q) >> 63) != 0u);
    if (fabs(q - r) == 0.5) {
      const double k = floor(q);
      for (int p = 0; p < 2; ++p) {
        // m + k odd: up to the even neighbour
        const bool odd = (OddInteger(inc[p]) != (p == 1)) != OddInteger(k);
        inc[p] += odd ? k + 1.0 : k;
      }
      up += fmax(k + 1.0, 0.0);
      down += fmin(k, 0.0);
    } else {
      inc[0] += r;
      inc[1] += r;
      up += fmax(r, 0.0);
      down += fmin(r, 0.0);
    }
  }

  SPAI_HD SumMap Map() const { return SumMap{{inc[0], inc[1]}, down - (downward ? 1.0 : 0.0), up, far ? 1 : 0}; }
};

// First a, then b.
SPAI_HD SumMap Then(const SumMap& a, const SumMap& b) {
  SumMap c;
  c.inc[0] = a.inc[0] + (OddInteger(a.inc[0]) ? b.inc[1] : b.inc[0]);
  c.inc[1] = a.inc[1] + (OddInteger(a.inc[1]) ? b.inc[0] : b.inc[1]);
  c.lo = fmin(a.lo, fmin(a.inc[0], a.inc[1]) + b.lo);
  c.hi = fmax(a.hi, fmax(a.inc[0], a.inc[1]) + b.hi);
  // what lies further out than 2^51 counts as out of the binade, so every value kept is exact
  c.bad = a.bad | b.bad | (c.hi < kSumLimit && c.lo > -kSumLimit ? 0 : 1);
  return c;
}

// True when the run keeps the sum s in its binade; *out is the sum after it.
SPAI_HD bool ApplyMap(const SumMap& map, double s, SumState state, double* out) {
  *out = s;
  if (map.bad || state == kSumOther) return false;
  if (state == kSumZero) return true;
  if (!(map.hi < kSumLimit && map.lo > -kSumLimit)) return false;
  const uint64_t bits = DoubleBits(s);
  const int64_t m = static_cast<int64_t>((bits & 0x000FFFFFFFFFFFFFull) | 0x0010000000000000ull);
  if (m + static_cast<int64_t>(map.lo) < kBinadeLow || m + static_cast<int64_t>(map.hi) >= kBinadeHigh) return false;
  const uint64_t moved = static_cast<uint64_t>(m + static_cast<int64_t>((m & 1) != 0 ? map.inc[1] : map.inc[0]));
  *out = BitsDouble((bits & 0xFFF0000000000000ull) | (moved & 0x000FFFFFFFFFFFFFull));
  return true;
}

}  // namespace spai
