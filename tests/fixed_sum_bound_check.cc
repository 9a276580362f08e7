// The stated bound of sum8 (fixed_sum.cuh): eight terms cut below 2^-59 of the
// largest's power of two, and one rounding.  Numbers of which the large ones
// cancel, exactly or nearly, and smaller remainders.  Prints per kind the
// largest error over the bound (at most 1) and the error of FP64 additions in
// order over it.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <string>

#include "../nimblesm_gb300/csrc/fixed_sum.cuh"

int main(int argc, char** argv)
{
  const int       n = argc > 1 ? std::atoi(argv[1]) : 1000;
  std::mt19937_64 rng(3);
  std::normal_distribution<double>       gauss;
  std::uniform_real_distribution<double> uni(0.0, 1.0);
  for (std::string kind : {"pairs_and_remainder", "pairs_apart", "nearly", "spread", "alike"}) {
    double worst = 0.0, worst64 = 0.0;
    for (int t = 0; t < n; t++) {
      double       x[8] = {};
      const double scale = std::ldexp(1.0, (int)(200 * (uni(rng) - 0.5)));
      for (int j = 0; j < 8; j++) x[j] = gauss(rng);
      if (kind == "spread")
        for (double& v : x) v = std::ldexp(v, (int)(70 * (uni(rng) - 0.5)));
      if (kind == "pairs_and_remainder" || kind == "pairs_apart" || kind == "nearly") {
        for (int j = 0; j < 6; j += 2) x[j + 1] = -x[j] * (kind == "nearly" ? 1.0 + std::ldexp(gauss(rng), -30) : 1.0);
        const int down = (int)(75 * uni(rng));
        x[6] = std::ldexp(gauss(rng), -down), x[7] = std::ldexp(gauss(rng), -down);
        if (kind == "pairs_apart") std::shuffle(x, x + 8, rng);
      }
      long double exact = 0.0L, most = 0.0L;
      double      f64 = 0.0;
      for (double& v : x) {
        v *= scale;
        exact += v;  // (64 bits: off by less than 2^-62 of the largest)
        f64 += v;
        most = std::max(most, std::fabs((long double)v));
      }
      const long double bound = 8 * std::ldexp(1.0L, std::ilogb(most) - 59) + std::ldexp(std::fabs(exact), -53) +
                                std::ldexp(most, -61);
      worst   = std::max(worst, (double)(std::fabs((long double)nsm::fx::sum8(x) - exact) / bound));
      worst64 = std::max(worst64, (double)(std::fabs((long double)f64 - exact) / bound));
    }
    std::printf("%s %.3e %.3e\n", kind.c_str(), worst, worst64);
  }
}
