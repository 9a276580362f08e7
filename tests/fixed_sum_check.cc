// Sums of eight FP64 numbers in fixed point (fixed_sum.cuh) against sums in
// extended precision and against FP64 additions: one line per kind of numbers,
// "kind error_fixed error_fp64", the largest errors over the largest |x|.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <limits>
#include <random>
#include <string>

#include "../nimblesm_gb300/csrc/fixed_sum.cuh"

int main(int argc, char** argv)
{
  const int       n = argc > 1 ? std::atoi(argv[1]) : 1000;
  std::mt19937_64 rng(argc > 2 ? std::atoi(argv[2]) : 1);
  std::normal_distribution<double>      gauss;
  std::uniform_real_distribution<double> uni(-1.0, 1.0);
  const char* kinds[] = {"alike", "spread", "cancelling", "few", "tiny", "huge", "not_numbers", "zeros"};
  for (const char* kind : kinds) {
    const std::string k = kind;
    double            worst = 0.0, worst64 = 0.0;
    for (int t = 0; t < n; t++) {
      double x[8], most = 0.0, f64 = 0.0;
      for (int j = 0; j < 8; j++) {
        x[j] = gauss(rng);
        if (k == "spread") x[j] = std::ldexp(x[j], (int)(40 * uni(rng)));
        if (k == "cancelling" && j % 2) x[j] = -x[j - 1] * (1.0 + 1e-9 * uni(rng));
        if (k == "few" && j >= 1 + t % 3) x[j] = j % 2 ? 0.0 : -0.0;
        if (k == "tiny") x[j] = std::ldexp(x[j], -1022 + (int)(60 * uni(rng)));
        if (k == "huge") x[j] = std::ldexp(x[j] / 64, 1021);
        if (k == "not_numbers" && j == t % 8)
          x[j] = t % 3 == 0 ? std::numeric_limits<double>::infinity() : (t % 3 == 1 ? -std::numeric_limits<double>::infinity() : NAN);
        if (k == "zeros") x[j] = (t >> j) & 1 ? -0.0 : 0.0;
      }
      long double exact = 0.0L;
      for (int j = 0; j < 8; j++) {
        exact += x[j];
        f64 += x[j];
        most = std::max(most, std::fabs(x[j]));
      }
      const double s = nsm::fx::sum8(x);
      if (k == "not_numbers" || k == "tiny" || k == "huge" || k == "zeros") {
        // what FP64 additions give wherever the fixed point does not apply
        const bool same = std::memcmp(&s, &f64, 8) == 0 || (std::isnan(s) && std::isnan(f64));
        if (k != "huge" && k != "tiny" && !same) worst = INFINITY;
      }
      if (most > 0.0 && std::isfinite(most)) {
        worst   = std::max(worst, (double)(std::fabs((long double)s - exact) / most));
        worst64 = std::max(worst64, (double)(std::fabs((long double)f64 - exact) / most));
      }
    }
    std::printf("%s %.3e %.3e\n", kind, worst, worst64);
  }
  return 0;
}
