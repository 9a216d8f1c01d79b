// Sums of 32 float pairs as integers (float_fixed), against long double and against
// FP64 adds of the pairs in a tree: never further off than the tree's own bound, and
// exact where the terms are within 2^-32 of the largest.
#include <cmath>
#include <cstdio>
#include <random>

#include "../../manybody_gb300/csrc/mb_internal.h"

int main() {
  std::mt19937_64 rng(5);
  std::uniform_real_distribution<double> u(-1.0, 1.0);
  int bad = 0;
  double worst = 0.0, worst_tree = 0.0;
  // binades that the terms spread over, and where the largest lies (subnormals and the
  // largest floats among them)
  for (int spread : {0, 3, 20, 31, 60, 250})
    for (int top : {-126, -100, 0, 20, 127})
      for (int rep = 0; rep < 400; ++rep) {
        float hi[32], lo[32];
        int t = 0;
        for (int l = 0; l < 32; ++l) {
          const int e = top - (spread ? (int)(rng() % (unsigned)(spread + 1)) : 0);
          hi[l] = (float)std::ldexp(rep % 2 ? u(rng) : std::fabs(u(rng)), e);
          // a pair's second part is below 2^-20 of the first after some terms
          lo[l] = (float)std::ldexp(u(rng), e - 20 - (int)(rng() % 8));
          t = std::max({t, mb::float_top(hi[l]), mb::float_top(lo[l])});
        }
        long long a = 0;
        long double want = 0.0, size = 0.0;
        double tree[32];
        bool near = true;
        for (int l = 0; l < 32; ++l) {
          a += mb::float_fixed(hi[l], t) + mb::float_fixed(lo[l], t);
          want += (long double)hi[l] + (long double)lo[l];
          size += std::fabs((long double)hi[l]) + std::fabs((long double)lo[l]);
          tree[l] = (double)hi[l] + (double)lo[l];
          for (float v : {hi[l], lo[l]})
            near = near && (v == 0.0f || std::max(mb::float_top(v), 1) >= t - 32);
        }
        for (int o = 16; o > 0; o >>= 1)
          for (int l = 0; l < o; ++l) tree[l] += tree[l + o];
        const long double got = std::ldexp((long double)a, t - 183);
        const long double off = std::fabs(got - want), off_tree = std::fabs((long double)tree[0] - want);
        // 64 cuts of a unit; six roundings of the partial sums by the tree
        const long double unit = std::ldexp(1.0L, t - 183);
        if (off > 64 * unit || (near && off != 0)) ++bad;
        if (off > 6 * std::ldexp(size, -53)) ++bad;
        worst = std::fmax(worst, (double)(off / size));
        worst_tree = std::fmax(worst_tree, (double)(off_tree / size));
      }
  std::printf("worst error of sum |term|: integers %.3g, FP64 tree %.3g; %d bad\n", worst, worst_tree, bad);
  return bad ? 1 : 0;
}
