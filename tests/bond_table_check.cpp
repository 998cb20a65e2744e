// Accuracy harness for gpuga_b200/csrc/bond_table.cuh on the host (built and run by tests/test_bond_table_cpu.py): every
// entry that is accepted, evaluated in FP32 as the items do, against b and b' in long double.
// Arguments: n, first and last beta s.  Prints: entries, accepted; for the plain and the fine evaluation the largest error of b
// (of its size) and of b' (of the entry's largest, or of 1e-3 / s); and the largest mean error of the fine b' over an
// entry (1024 points, every 20th beta).
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "../gpuga_b200/csrc/bond_table.cuh"

static float from_bits(int i) {
  float f;
  memcpy(&f, &i, 4);
  return f;
}
static int bits(float f) {
  int i;
  memcpy(&i, &f, 4);
  return i;
}

static void closed(long double n, long double beta, long double s, long double& b, long double& db) {
  const long double z = n * std::log(beta * s), l = z > 0 ? z + std::log1p(std::exp(-z)) : std::log1p(std::exp(z));
  b = std::exp(-l / (2 * n));
  db = -0.5L * b / s * std::exp(z - l);
}

int main(int argc, char** argv) {
  const double n = atof(argv[1]), z0 = atof(argv[2]), z1 = atof(argv[3]);
  long total = 0, accepted = 0;
  double eb[2] = {0, 0}, ed[2] = {0, 0}, bias = 0;
  for (int k = 0; k <= 400; ++k) {
    const double beta = k == 400 ? 0.33675f : (double)(float)(0.02 * std::pow(300.0, k / 399.0));
    const double lbeta = std::log(beta), mh = -0.5 / n;
    for (int i = bits((float)(z0 / beta)) >> 20; i <= bits((float)(z1 / beta)) >> 20; ++i) {
      const float c = from_bits((i << 20) | 0x00080000), lo = from_bits(i << 20);
      const double h = (double)c - lo;
      double f[gpuga::kBondPoints], at, bc = 0;
      for (int k = 0; k < gpuga::kBondPoints; ++k) {
        const double x = c + h * gpuga::kBondPoint[k];
        gpuga::bond_order(n, mh, beta, lbeta, x, std::log(x), at, f[k]);
        f[k] *= h;
        if (k == gpuga::kBondCenter) bc = at;
      }
      const gpuga::BondEntry e = gpuga::bond_fit(f, bc, c, h);
      ++total;
      if (!e.ok) continue;
      ++accepted;
      long double top = 1e-3L / c, worst[2] = {0, 0};
      auto eval = [&](bool fine, float s, float& b, float& d) {
        auto f = fine ? gpuga::bond_eval<true> : gpuga::bond_eval<false>;
        f(e.b0, e.lo, e.k[0], e.k[1], e.k[2], e.k[3], e.k[4], e.k[5], s - c, b, d);
      };
      for (int x = 0; x <= 64; ++x) {
        const float s = x < 64 ? from_bits((i << 20) + x * 0x4000) : std::nextafter(from_bits((i + 1) << 20), 0.0f);
        long double b, db;
        closed(n, beta, s, b, db);
        top = std::fmax(top, std::fabs(db));
        for (int fine = 0; fine < 2; ++fine) {
          float bo, d;
          eval(fine, s, bo, d);
          eb[fine] = std::fmax(eb[fine], (double)(std::fabs(bo - b) / b));
          worst[fine] = std::fmax(worst[fine], std::fabs(d - db));
        }
      }
      for (int fine = 0; fine < 2; ++fine) ed[fine] = std::fmax(ed[fine], (double)(worst[fine] / top));
      if (k % 20 > 0) continue;
      long double sum = 0;
      for (int x = 0; x < 1024; ++x) {
        const float s = from_bits((i << 20) + x * 0x400 + 0x200);
        float bo, d;
        eval(true, s, bo, d);
        long double b, db;
        closed(n, beta, s, b, db);
        sum += d - db;
      }
      bias = std::fmax(bias, (double)(std::fabs(sum / 1024) / top));
    }
  }
  printf("%ld %ld %.4e %.4e %.4e %.4e %.4e\n", total, accepted, eb[0], ed[0], eb[1], ed[1], bias);
  return 0;
}
