// The margins of the Delaunay finder's local search, compiled for the host:
// what it calls certain has to be so in 64 bits.
//
//   delaunay_margins_host normals
//     open faces of cells with two others nearly on one line, on a grid of the
//     size of 40,000 cells: prints "<angle> <faces> <refused> <points> <missed>",
//     missed being points on the open side that the rows looked up leave out.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "tecs/device/delaunay_star.cuh"

using namespace tecs::dl;

static int normals() {
  const unsigned n = 40000;
  std::mt19937 rng(5);
  std::uniform_real_distribution<double> u01(0.0, 1.0), u11(-1.0, 1.0);
  std::vector<Pt> P(n);
  double mn[3] = {1e300, 1e300, 1e300}, mx[3] = {-1e300, -1e300, -1e300};
  for (auto& p : P) {
    double q[3];
    for (int d = 0; d < 3; ++d) q[d] = 34.0 * u01(rng) - 17.0;
    p = Pt{(float)q[0], (float)q[1], (float)q[2], 0.f};
    const double f[3] = {p.x, p.y, p.z};
    for (int d = 0; d < 3; ++d) {
      mn[d] = f[d] < mn[d] ? f[d] : mn[d];
      mx[d] = f[d] > mx[d] ? f[d] : mx[d];
    }
  }
  Grid g{};
  plan_grid<3>(g, mn, mx, n, n + 64u);
  std::vector<unsigned> off(g.nbins + 1, 0u), key(n), idx(n);
  std::vector<Pt> sp(n);
  for (unsigned i = 0; i < n; ++i) {
    const double q[3] = {P[i].x, P[i].y, P[i].z};
    int b[3];
    bin_of<3>(g, q, b);
    key[i] = flat(g, b[0], b[1], b[2]);
    ++off[key[i] + 1];
  }
  for (unsigned b = 0; b < g.nbins; ++b) off[b + 1] += off[b];
  std::vector<unsigned> cur(off.begin(), off.end() - 1);
  for (unsigned i = 0; i < n; ++i) {
    const unsigned at = cur[key[i]]++;
    idx[at] = i;
    sp[at] = P[i];
  }
  g.off = off.data();
  g.idx = idx.data();
  g.sp = sp.data();
  g.P = P.data();
  g.n = n;
  std::vector<char> seen(n);
  for (const double angle : {1e-1, 1e-3, 1e-4, 3e-5, 1.5e-5, 1e-5, 3e-6, 1e-6}) {
    unsigned faces = 0, refused = 0;
    unsigned long long points = 0, missed = 0;
    for (; faces < 60; ++faces) {
      // a cell and two others, at an angle of about `angle` between them
      const Pt pi = P[rng() % n];
      double e[3], t[3], len = 0.0;
      for (int d = 0; d < 3; ++d) { e[d] = u11(rng); t[d] = u11(rng) * angle; len += e[d] * e[d]; }
      len = std::sqrt(len);
      const Pt pa{(float)(pi.x + e[0] / len), (float)(pi.y + e[1] / len), (float)(pi.z + e[2] / len), 0.f};
      const Pt pb{(float)(pi.x + 1.3 * e[0] / len + t[0]), (float)(pi.y + 1.3 * e[1] / len + t[1]),
                  (float)(pi.z + 1.3 * e[2] / len + t[2]), 0.f};
      const double o[3] = {pi.x, pi.y, pi.z};
      const double a[3] = {pa.x - o[0], pa.y - o[1], pa.z - o[2]}, b[3] = {pb.x - o[0], pb.y - o[1], pb.z - o[2]};
      double nn[3], slack;
      if (!plane_normal(a, b, nn, slack)) { ++refused; continue; }
      std::memset(seen.data(), 0, n);
      visit_half<3>(Solo{}, g, o, nn, [&](unsigned id, const Pt&) { seen[id] = 1; return true; });
      double x[3];
      cross3(a, b, x);
      const double xl = std::sqrt(x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
      for (unsigned i = 0; i < n; ++i) {
        const double v[3] = {P[i].x - o[0], P[i].y - o[1], P[i].z - o[2]};
        if (!(x[0] * v[0] + x[1] * v[1] + x[2] * v[2] > 1.0e-9 * xl)) continue;
        ++points;
        if (!seen[i]) ++missed;
      }
    }
    std::printf("%g %u %u %llu %llu\n", angle, faces, refused, points, missed);
  }
  return 0;
}

int main(int argc, char** argv) {
  if (argc == 2 && !std::strcmp(argv[1], "normals")) return normals();
  return 2;
}
