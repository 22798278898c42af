// Host build of the device edge builder (edge_build.cuh): curves split in the steps a warp's lanes share
// (curve_poly, cubic_candidates, sorted cuts, poly_piece) against split_cubic and split_quad, bit for
// bit: random curves, control points on each other, on a line, on whole pixels, loops and cusps.
// Usage: split_steps_check <seed> <curves>; exit status 0 when all match.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#define __device__
#define __forceinline__ inline
using std::max;
using std::min;
static inline long long __double_as_longlong(double x) { long long v; memcpy(&v, &x, 8); return v; }
static inline int __double2hiint(double x) { return int(uint64_t(__double_as_longlong(x)) >> 32); }
static inline int __double2loint(double x) { return int(uint32_t(uint64_t(__double_as_longlong(x)))); }
static inline double __hiloint2double(int hi, int lo) {
  const uint64_t b = (uint64_t(uint32_t(hi)) << 32) | uint32_t(lo);
  double v; memcpy(&v, &b, 8); return v;
}
static inline uint32_t atomicAdd(uint32_t* p, uint32_t v) { uint32_t o = *p; *p += v; return o; }
#include "edge_build.cuh"

using namespace blgpu::eb;

static bool same_points(const Pt* a, const Pt* b, int n) { return memcmp(a, b, sizeof(Pt) * size_t(n)) == 0; }

int main(int argc, char** argv) {
  std::mt19937_64 rng(argc > 1 ? strtoull(argv[1], nullptr, 10) : 1);
  const long n = argc > 2 ? atol(argv[2]) : 10000;
  std::uniform_real_distribution<double> u(0.0, 1.0);
  long bad = 0, pieces[9] = {};
  for (long it = 0; it < n; it++) {
    const double span = std::pow(65535.0, u(rng)) * 256.0;
    const int grid = int(rng() % 3);
    Pt c[4];
    for (Pt& p : c) {
      p = Pt{(u(rng) - 0.3) * span, (u(rng) - 0.3) * span};
      if (grid == 1) p = Pt{std::floor(p.x / 256.0) * 256.0, std::floor(p.y / 256.0) * 256.0};
    }
    switch (rng() % 10) {
      case 0: c[1] = c[0]; break;
      case 1: c[2] = c[3]; break;
      case 2: c[3] = c[0]; break;
      case 3: c[1].y = c[0].y; c[2].x = c[3].x; break;
      case 4: for (int i = 1; i < 4; i++) c[i] = Pt{c[0].x + i * 7.0, c[0].y + i * 3.0}; break;
      case 5: std::swap(c[1], c[2]); c[1].x = c[3].x + span * 0.1; c[2].x = c[0].x - span * 0.1; break;
      default: break;
    }
    {
      Pt want[25];
      for (int i = 0; i < 4; i++) want[i] = c[i];
      int nout = split_cubic(want);
      if (nout == 0) nout = 3;
      const Poly<3> p = curve_poly(c[0], c[1], c[2], c[3]);
      std::vector<double> t;
      for (int set = 0; set < kCubicSets; set++) {
        double o[2];
        cubic_candidates(p, set, o);
        for (double v : o) if (v != kNoCut) t.push_back(v);
      }
      std::sort(t.begin(), t.end());
      t.erase(std::unique(t.begin(), t.end()), t.end());
      Pt got[25];
      if (t.empty()) for (int i = 0; i < 4; i++) got[i] = c[i];
      else
        for (size_t k = 0; k <= t.size(); k++)
          poly_piece(p, k ? t[k - 1] : 0.0, k < t.size() ? t[k] : 1.0, k ? poly_point(p, t[k - 1]) : c[0], k < t.size() ? poly_point(p, t[k]) : c[3], got + 3 * k);
      pieces[min<size_t>(t.size(), 8)]++;
      if (nout != int(3 * (t.size() + 1)) || !same_points(want, got, nout + 1))
        if (++bad <= 5) printf("cubic %ld: %d points against %zu cuts\n", it, nout, t.size());
    }
    {
      Pt want[7];
      for (int i = 0; i < 3; i++) want[i] = c[i];
      int nout = split_quad(want);
      if (nout == 0) nout = 2;
      const Poly<2> p = curve_poly(c[0], c[1], c[2]);
      const double ex = (c[0].x - c[1].x) / (c[0].x - c[1].x * 2.0 + c[2].x);
      const double ey = (c[0].y - c[1].y) / (c[0].y - c[1].y * 2.0 + c[2].y);
      const double t0 = dmin(ex, ey), t1 = dmax(ex, ey);
      std::vector<double> t;
      if ((t0 > 0.0) & (t0 < 1.0)) t.push_back(t0);
      if ((t1 > dmax(t0, 0.0)) & (t1 < 1.0)) t.push_back(t1);
      Pt got[7];
      if (t.empty()) for (int i = 0; i < 3; i++) got[i] = c[i];
      else
        for (size_t k = 0; k <= t.size(); k++)
          poly_piece(p, k ? t[k - 1] : 0.0, k < t.size() ? t[k] : 1.0, k ? poly_point(p, t[k - 1]) : c[0], k < t.size() ? poly_point(p, t[k]) : c[2], got + 2 * k);
      if (nout != int(2 * (t.size() + 1)) || !same_points(want, got, nout + 1))
        if (++bad <= 5) printf("quad %ld: %d points against %zu cuts\n", it, nout, t.size());
    }
  }
  printf("cuts:");
  for (long v : pieces) printf(" %ld", v);
  printf(", mismatches %ld\n", bad);
  return bad ? 1 : 0;
}
