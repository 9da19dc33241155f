// The piecewise sequential sum (csrc/ordered_sum.cuh) against the plain loop:
// pieces of random length, summarised by a random two-way split, must leave
// the loop's bits whatever the terms are.  argv[1] selects the terms.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>

#include "ordered_sum.cuh"

using namespace spai;

namespace {

double Term(int kind, std::mt19937_64& gen) {
  std::normal_distribution<double> normal(0.0, 1.0);
  const double v = normal(gen);
  const auto die = [&](int n) { return static_cast<int>(gen() % static_cast<unsigned>(n)); };
  switch (kind) {
    case 0: return v * v;                                            // squares: steady growth
    case 1: return v;                                                // both signs: crossings of zero
    case 2: return (die(9) - 4) * 0.25;                              // dyadic: exact sums, powers of two
    case 3: return std::ldexp(v, die(120) - 60);                     // wide range
    case 4: return (die(5) - 2) * std::ldexp(1.0, -die(56));         // ties at every grid
    case 5: return die(3) != 0 ? 0.0 : v * v * 1e-300;               // long zero stretches, tiny sums
    case 6: return std::ldexp(v, -1060 + die(40));                   // subnormals
    default: return die(50) == 0 ? (die(2) != 0 ? INFINITY : NAN) : v;  // non-finite
  }
}

// The map of terms [first, last).
SumMap Summarise(const std::vector<double>& t, int first, int last, double scale, SumState state) {
  if (state == kSumZero) {
    SumMap m = EmptyMap();
    for (int i = first; i < last; ++i) m.bad |= t[i] == 0.0 ? 0 : 1;
    return m;
  }
  TermRun run;
  for (int i = first; i < last; ++i) run.Add(t[i], scale);
  return run.Map();
}

}  // namespace

int main(int argc, char** argv) {
  const int kind = argc > 1 ? std::atoi(argv[1]) : 0;
  std::mt19937_64 gen(static_cast<unsigned>(kind) + 1u);
  long summarised = 0;
  for (int trial = 0; trial < 4000; ++trial) {
    const int n = 1 + static_cast<int>(gen() % 300);
    const int piece = 1 + static_cast<int>(gen() % 64);
    std::vector<double> t(static_cast<size_t>(n));
    for (double& x : t) x = Term(kind, gen);
    double want = 0.0;
    for (const double x : t) want = want + x;
    double got = 0.0;
    for (int first = 0; first < n; first += piece) {
      const int last = first + piece < n ? first + piece : n;
      const int middle = first + static_cast<int>(gen() % static_cast<unsigned>(last - first + 1));
      double scale;
      const SumState state = Classify(got, &scale);
      SumMap left = EmptyMap();
      SumMap right = EmptyMap();
      if (state != kSumOther) {
        left = Summarise(t, first, middle, scale, state);
        right = Summarise(t, middle, last, scale, state);
      }
      double moved;
      if (ApplyMap(Then(left, right), got, state, &moved)) {
        got = moved;
        ++summarised;
      } else {
        for (int i = first; i < last; ++i) got = got + t[i];
      }
    }
    const bool same = DoubleBits(got) == DoubleBits(want) || (got != got && want != want);
    if (!same) {
      std::printf("kind %d, trial %d: %a != %a\n", kind, trial, got, want);
      return 1;
    }
  }
  std::printf("%ld\n", summarised);
  return 0;
}
