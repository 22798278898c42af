// Host build of the device edge builder (edge_build.cuh): clipped monotonic pieces flattened by the
// lane flattener with subtrees handed over (LaneCurve::step<true>, skip_node; some of them refused,
// split_node) and walked as trees in a random order, against the lane flattener on its own: the same
// multiset of segments; and pieces outside the box (piece_outside) against it. Cubic and quadratic
// curves around and across the clip box.
// Usage: subtree_check <seed> <curves>; exit status 0 when all match.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <tuple>
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

using Seg = std::tuple<int, int, int, int, uint32_t>;
static std::vector<DevSeg> g_segs(1 << 16);
static std::vector<uint32_t> g_meta(1 << 16);
static uint32_t g_counter;

static void init_builder(Builder& b, double w, double h) {
  b.cx0 = 0.0; b.cy0 = 0.0; b.cx1 = w * 256.0; b.cy1 = h * 256.0;
  b.icx0 = trunc_i(b.cx0); b.icx1 = trunc_i(b.cx1);
  const double tol = 0.20 * 256.0;
  b.tol_sq = tol * tol;
  b.acc_x0_y0 = b.acc_x0_y1 = b.acc_x1_y0 = b.acc_x1_y1 = b.cy0;
  b.px = b.py = 0; b.psign = 0; b.pasc = false;
  g_counter = 0;
  b.sink.init(g_segs.data(), g_meta.data(), &g_counter, uint32_t(g_segs.size()), 7u);
}

static std::vector<Seg> taken(Builder& b) {
  b.done(); b.sink.flush();
  std::vector<Seg> v;
  for (uint32_t i = 0; i < g_counter; i++) v.push_back(Seg{g_segs[i].x0, g_segs[i].y0, g_segs[i].x1, g_segs[i].y1, g_meta[i]});
  return v;
}

static long g_handed = 0, g_refused = 0, g_outside[4] = {};

template<int DEG>
static bool same(const Pt* pts, uint32_t any, double w, double h, std::mt19937_64& rng) {
  Builder b;
  init_builder(b, w, h);
  LaneCurve<DEG, CachedStack<DEG>> lc;
  bool busy = lc.begin_piece(b, pts, any);
  while (busy) {
    lc.step(b);
    if (lc.state == kLsDone && !lc.next_piece(b, true)) busy = false;
  }
  std::vector<Seg> want = taken(b), got;
  // a piece outside the box: nothing, or a run at its side
  double y0, y1;
  uint32_t sign;
  const PieceOutside where = piece_outside(pts, DEG, b, y0, y1, sign);
  g_outside[where]++;
  if (where != kCrosses) {
    Builder o;
    init_builder(o, w, h);
    if (where == kLeftRun) o.acc_left_s(y0, y1, sign);
    if (where == kRightRun) o.acc_right_s(y0, y1, sign);
    std::vector<Seg> run = taken(o);
    std::sort(run.begin(), run.end());
    std::sort(want.begin(), want.end());
    return run == want;
  }
  Builder c;
  init_builder(c, w, h);
  LaneCurve<DEG, CachedStack<DEG>> lh;
  busy = lh.begin_piece(c, pts, any);
  while (busy) {
    const int r = lh.template step<true>(c);
    if (r == LaneCurve<DEG, CachedStack<DEG>>::kStepLeaf) lh.leaf(c);
    if (r == LaneCurve<DEG, CachedStack<DEG>>::kStepHand) {
      if (rng() % 8 == 0) { g_refused++; lh.split_node(c); }
      else {
        g_handed++;
        TreeNode<DEG> root;
        for (int i = 0; i <= DEG; i++) root.p[i] = lh.mc.p[i];
        root.level = lh.mc.sp;
        std::vector<TreeNode<DEG>> pending{root};
        while (!pending.empty()) {
          const size_t pick = size_t(rng() % pending.size());
          const TreeNode<DEG> n = pending[pick];
          pending[pick] = pending.back();
          pending.pop_back();
          TreeNode<DEG> l, r;
          if (tree_step<DEG>(n, c.tol_sq, l, r)) {
            const int x0 = trunc_i(n.p[0].x), y0 = trunc_i(n.p[0].y), x1 = trunc_i(n.p[DEG].x), y1 = trunc_i(n.p[DEG].y);
            if (y0 != y1) got.push_back(Seg{x0, y0, x1, y1, (7u << 1) | lh.sign});
          }
          else { pending.push_back(l); pending.push_back(r); }
        }
        lh.skip_node(c);
      }
    }
    if (lh.state == kLsDone && !lh.next_piece(c, true)) busy = false;
  }
  const std::vector<Seg> rest = taken(c);
  got.insert(got.end(), rest.begin(), rest.end());
  std::sort(want.begin(), want.end());
  std::sort(got.begin(), got.end());
  return want == got;
}

template<int DEG>
static long check(std::mt19937_64& rng, long n) {
  std::uniform_real_distribution<double> u(0.0, 1.0);
  long bad = 0;
  for (long it = 0; it < n; it++) {
    const double span = it % 4 ? 200.0 : 3000.0;
    const double w = 16 + std::floor(u(rng) * span), h = 16 + std::floor(u(rng) * span);
    auto coord = [&](double lim) {
      const double r = u(rng);
      if (r < 0.06) return 0.0;
      if (r < 0.12) return lim * 256.0;
      if (r < 0.16) return 256.0 * (-1e5 + 2e5 * u(rng));
      if (r < 0.5) return 256.0 * (std::floor(-0.25 * lim + 1.5 * lim * u(rng)) + (u(rng) < 0.5 ? 0.5 : 0.0));
      return 256.0 * (-0.5 * lim + 2.0 * lim * u(rng));
    };
    Pt spline[DEG == 3 ? 25 : 7];
    Builder b;
    init_builder(b, w, h);
    uint32_t any = 0, common = 15;
    for (int i = 0; i <= DEG; i++) {
      spline[i] = Pt{coord(w), coord(h)};
      const uint32_t fl = b.fxy(spline[i]);
      any |= fl; common &= fl;
    }
    if (common || !any) continue;
    int nout = DEG == 3 ? split_cubic(spline) : split_quad(spline);
    if (nout == 0) nout = DEG;
    for (int k = 0; k < nout; k += DEG)
      if (!same<DEG>(spline + k, any, w, h, rng) && ++bad <= 5) printf("mismatch: degree %d curve %ld piece %d\n", DEG, it, k / DEG);
  }
  return bad;
}

int main(int argc, char** argv) {
  std::mt19937_64 rng(argc > 1 ? strtoull(argv[1], nullptr, 10) : 1);
  const long n = argc > 2 ? atol(argv[2]) : 10000;
  const long bad = check<3>(rng, n) + check<2>(rng, n);
  printf("handed %ld refused %ld, outside: none %ld left %ld right %ld, mismatches %ld\n", g_handed, g_refused,
         g_outside[kNothing], g_outside[kLeftRun], g_outside[kRightRun], bad);
  return bad || !g_handed || !g_outside[kNothing] || !g_outside[kLeftRun] || !g_outside[kRightRun] ? 1 : 0;
}
