// The integer hop sums' headroom (mb_isum.h, isum_base), restated for the host:
// four decoded terms' high parts meet in 32 bits and all terms in 64, also where
// every term is just below a power of two and floored away from zero.  The sums
// run over the sliced down tables that the apply reads, against long double.
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <map>
#include <vector>

#include "../../manybody_gb300/csrc/mb_internal.h"

namespace {

// isum_pack and ISum2::add_packed of one component; *fits: no 32- or 64-bit wrap
struct Packed {
  int base, e = 512;
  __int128 a = 0;
  bool fits = true;

  static long long pack(double v) {
    unsigned long long h;
    std::memcpy(&h, &v, 8);
    const int ex = (int)(h >> 52 & 0x7FF);
    if (ex <= 512) return 0;
    const unsigned long long m = ((h & ((1ull << 52) - 1)) | 1ull << 52) << 10;
    return (long long)((h >> 63 ? 0ull - m : m) | (unsigned long long)(ex - 512));
  }
  void add(const long long (&v)[4], const bool (&neg)[4]) {
    int s[4], least = 0;
    for (int k = 0; k < 4; ++k) {
      s[k] = e - ((int)(v[k] & 1023) + 512);
      least = std::min(least, s[k]);
    }
    if (least < 0) {
      a >>= std::min(1 - least, 63);
      e += 1 - least;
      for (int& x : s) x += 1 - least;
    }
    long long hi = 0, lo = 0;
    for (int k = 0; k < 4; ++k) {
      const long long r = (v[k] & ~1023ll) >> std::min(s[k] + base - 4, 63);
      const int sign = neg[k] ? -1 : 1;
      hi += sign * (r >> 32);
      lo += sign * (long long)((uint32_t)r >> 3);
    }
    fits = fits && hi >= INT_MIN && hi <= INT_MAX && lo >= INT_MIN && lo <= INT_MAX;
    a += (__int128)hi * (1 << 29) + lo;
    fits = fits && a >= LLONG_MIN && a <= LLONG_MAX;
  }
  long double value() const { return std::ldexp((long double)a, e + base - 1023 - 63); }
};

mb::HopTable hops(int L, int n, const std::vector<std::pair<int, int>>& bonds) {
  const std::vector<uint32_t> m = mb::make_spin_sector(L, n).masks;
  std::map<uint32_t, int32_t> rank;
  for (size_t i = 0; i < m.size(); ++i) rank[m[i]] = (int32_t)i;
  mb::HopTable t;
  t.off.push_back(0);
  for (uint32_t s : m) {
    for (const auto& b : bonds)
      for (int dir = 0; dir < 2; ++dir) {
        const int a = dir ? b.second : b.first, c = dir ? b.first : b.second;
        if (!(s >> a & 1u) || (s >> c & 1u)) continue;
        const uint32_t between = s & ((1u << std::max(a, c)) - 1u) & ~((1u << (std::min(a, c) + 1)) - 1u);
        t.ent.push_back((uint32_t)rank[s ^ (1u << a) ^ (1u << c)] << 8 |
                        ((uint32_t)__builtin_popcount(between) & 1u));
      }
    t.off.push_back((int32_t)t.ent.size());
  }
  return t;
}

int check(const char* name, int L, int n, const std::vector<std::pair<int, int>>& bonds, int lanes) {
  const mb::HopTable t = hops(L, n, bonds);
  const int64_t D = (int64_t)t.off.size() - 1;
  const mb::SlicedTable s = mb::sliced_table(t, D, lanes);
  int words = 0;
  for (size_t g = 1; g < s.grp.size(); g += 2) words = std::max(words, (s.grp[g] + 3) / 4);
  // both spins have this table
  const int64_t terms = 8 * words;
  int bad = 0;
  // values of the neighbours with a negative and a positive hop
  const double top = 1.0 - std::ldexp(1.0, -53), near_top = 1.0 - std::ldexp(1.0, -40);
  const double kinds[][2] = {{-top, 0.4}, {-near_top, 0.4}, {-top, top}, {0.4, -top}, {top, -top}};
  for (int64_t c = 0; c < D; ++c)
    for (const auto& kind : kinds) {
      Packed sum{mb::isum_base(terms, mb::kISumDecoded)};
      long double want = 0.0, size = 0.0;
      const int32_t base = s.grp[(size_t)(2 * (c / 32))], k = s.grp[(size_t)(2 * (c / 32) + 1)];
      for (int j = 0; j < k; j += 4) {
        long long v[4];
        bool neg[4];
        for (int q = 0; q < 4; ++q) {
          const uint32_t e = s.ent[(size_t)base + 32 * (size_t)j + 4 * (size_t)(c % 32) + (size_t)q];
          neg[q] = e >> 31;
          const double x = (e & 0x7FFFFFFFu) < (uint32_t)D ? kind[neg[q] ? 0 : 1] : 0.0;
          v[q] = Packed::pack(x);
          want += neg[q] ? -(long double)x : (long double)x;
          size += std::fabs((long double)x);
        }
        sum.add(v, neg);
      }
      if (size > 0 && (!sum.fits || std::fabs(sum.value() - want) > terms * std::ldexp(1.0L, -53) * size)) {
        if (!bad) std::printf("%s: column %lld gives %.17Lg, not %.17Lg\n", name, (long long)c, sum.value(), want);
        ++bad;
      }
    }
  std::printf("%s: D=%lld base %d, %d bad\n", name, (long long)D, mb::isum_base(terms, mb::kISumDecoded), bad);
  return bad;
}

std::vector<std::pair<int, int>> square(int lx, int ly) {
  std::vector<std::pair<int, int>> b;
  for (int y = 0; y < ly; ++y)
    for (int x = 0; x < lx; ++x) {
      b.push_back({x + lx * y, (x + 1) % lx + lx * y});
      b.push_back({x + lx * y, x + lx * ((y + 1) % ly)});
    }
  return b;
}

// As many floored terms of one kind and sign as a base is chosen for, the first
// word a binade lower: the worst case of both widths.
int worst() {
  int bad = 0;
  const double top = 1.0 - std::ldexp(1.0, -53);
  for (int64_t terms = 4; terms <= 512; ++terms)
    for (int sign = 0; sign < 4; ++sign) {
      Packed sum{mb::isum_base(terms, mb::kISumDecoded)};
      const double x = sign & 1 ? -top : top;
      const bool neg = sign & 2;
      for (int64_t j = 0; j < terms; j += 4) {
        long long v[4];
        const bool n[4] = {neg, neg, neg, neg};
        for (int64_t q = 0; q < 4; ++q) v[q] = j + q < terms ? Packed::pack(j ? x : x / 2) : 0;
        sum.add(v, n);
      }
      bad += !sum.fits;
    }
  std::printf("worst cases: %d bad\n", bad);
  return bad;
}

}  // namespace

int main() {
  std::vector<std::pair<int, int>> ring;
  for (int i = 0; i < 12; ++i) ring.push_back({i, (i + 1) % 12});
  int bad = worst();
  for (int lanes : {8, 16}) {
    bad += check("4x4 n=3", 16, 3, square(4, 4), lanes);
    bad += check("4x4 n=4", 16, 4, square(4, 4), lanes);
    bad += check("4x4 n=6", 16, 6, square(4, 4), lanes);
    bad += check("3x3 n=4", 9, 4, square(3, 3), lanes);
    bad += check("ring 12 n=6", 12, 6, ring, lanes);
  }
  return bad ? 1 : 0;
}
