// Host build of the device edge builder (edge_build.cuh): the 32-bit flatness test (flat_guess) against
// the FP64 one (Mono::is_flat) on every node of random curve pieces inside the clip box: where it
// decides, it must decide alike. Sizes from a pixel to 65,535 px, whole and half pixels among them.
// Usage: flat_guess_check <seed> <pieces>; exit status 0 when no decision differs.
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

using namespace blgpu;
using namespace blgpu::eb;

static long g_nodes = 0, g_unsure = 0, g_bad = 0;

template<int DEG>
static void walk(const Pt* pts, std::mt19937_64& rng) {
  const double tol = 0.20 * 256.0;
  uint32_t sign;
  std::vector<TreeNode<DEG>> pending{tree_root<DEG>(pts, sign)};
  for (long guard = 0; !pending.empty() && guard < 4000; guard++) {
    const size_t pick = size_t(rng() % pending.size());
    const TreeNode<DEG> n = pending[pick];
    pending[pick] = pending.back();
    pending.pop_back();
    Mono<DEG, NoStack> mc;
    mc.tol_sq = tol * tol;
    for (int i = 0; i <= DEG; i++) mc.p[i] = n.p[i];
    Step st;
    const bool flat = mc.is_flat(st);
    const int guess = flat_guess<DEG>(n.p);
    g_nodes++;
    if (guess < 0) g_unsure++;
    else if ((guess > 0) != flat && ++g_bad <= 5) printf("differs: degree %d, value / limit = %.9g, guess %d\n", DEG, st.value / st.limit, guess);
    TreeNode<DEG> l, r;
    if (!tree_step<DEG>(n, tol * tol, l, r)) { pending.push_back(l); pending.push_back(r); }
  }
}

int main(int argc, char** argv) {
  std::mt19937_64 rng(argc > 1 ? strtoull(argv[1], nullptr, 10) : 1);
  const long n = argc > 2 ? atol(argv[2]) : 10000;
  std::uniform_real_distribution<double> u(0.0, 1.0);
  for (long it = 0; it < n; it++) {
    const double w = std::pow(65535.0, u(rng)), h = std::pow(65535.0, u(rng));
    // a fifth of the curves lie along the box's left or top side, where split points may fall outside
    const double ox = rng() % 5 ? u(rng) * (65535.0 - w) : 0.0, oy = rng() % 5 ? u(rng) * (65535.0 - h) : 0.0;
    const int grid = int(rng() % 4);             // 0: any; whole, half, 1/256 pixels
    auto coord = [&](double o, double s) {
      double v = o + (u(rng) < 0.1 ? (rng() & 1u ? s : 0.0) : u(rng) * s);
      if (grid == 1) v = std::floor(v);
      if (grid == 2) v = std::floor(v * 2.0) * 0.5;
      if (grid == 3) v = std::floor(v * 256.0) / 256.0;
      return v * 256.0;
    };
    Pt p[25];
    for (int i = 0; i < 4; i++) p[i] = Pt{coord(ox, w), coord(oy, h)};
    if (rng() % 8 == 0) p[1] = p[0];
    if (rng() % 8 == 0) p[2].y = p[1].y;
    // starting or ending along the box's side: an extremum there, split off with a rounding error
    if (rng() % 4 == 0) p[0].y = p[1].y = oy * 256.0;
    if (rng() % 4 == 0) p[2].x = p[3].x = ox * 256.0;
    if (it & 1) {
      int nout = split_cubic(p);
      for (int k = 0; k < (nout ? nout : 3); k += 3) walk<3>(p + k, rng);
    }
    else {
      int nout = split_quad(p);
      for (int k = 0; k < (nout ? nout : 2); k += 2) walk<2>(p + k, rng);
    }
  }
  printf("nodes %ld unsure %ld differ %ld\n", g_nodes, g_unsure, g_bad);
  return g_bad || g_unsure * 20 > g_nodes ? 1 : 0;
}
