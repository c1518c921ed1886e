// The margins of the Delaunay finder's local search, compiled for the host:
// what it calls certain has to be so in 64 bits.
//
//   delaunay_margins_host normals
//     open faces of cells with two others nearly on one line, on a grid of the
//     size of 40,000 cells: prints "<angle> <faces> <refused> <points> <missed>",
//     missed being points on the open side that the rows looked up leave out.
//   delaunay_margins_host lines
//     the lines that may bound the Voronoi faces of a cell among its neighbours,
//     cut in float as the search does and in double: prints
//     "<set> <unit of length> <lines without a rest in float> <looked at in double>
//     <doubtful> <wrong>",
//     wrong being those called certain of which more bits leave something.
//   delaunay_margins_host spheres
//     tetrahedra from thin to regular, most of them with five or more points on
//     their sphere but for rounding: prints "<refused> <outside>" and the five
//     positions (the cell, three others, a fifth), in which outside says that
//     the fifth is certainly outside of the first four's sphere.
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

// Neighbourhoods: random cells, lattices with jitter (near-ties), a cell that
// is nearly on one line with many pairs of others.
static std::vector<Pt> cloud(int set, double unit, unsigned seed) {
  std::mt19937 rng(seed);
  std::normal_distribution<double> nd(0.0, 1.0);
  std::uniform_real_distribution<double> u11(-1.0, 1.0);
  std::vector<Pt> p{Pt{0.f, 0.f, 0.f, 0.f}};
  auto put = [&](double x, double y, double z) {
    p.push_back(Pt{(float)(unit * x), (float)(unit * y), (float)(unit * z), 0.f});
  };
  if (set == 0) {
    while (p.size() < 90) put(2.8 * u11(rng), 2.8 * u11(rng), 2.8 * u11(rng));
  } else if (set <= 3) {
    const double jitter = set == 1 ? 1e-2 : set == 2 ? 1e-4 : 1e-6;
    for (int x = -2; x <= 2; ++x)
      for (int y = -2; y <= 2; ++y)
        for (int z = -1; z <= 1; ++z)
          if (x || y || z) put(x + jitter * nd(rng), y + jitter * nd(rng), z + jitter * nd(rng));
  } else {
    while (p.size() < 90) {
      const double t = 2.5 * u11(rng);
      put(t + 1e-3 * nd(rng), 0.3 * t + 1e-3 * nd(rng), 0.5 + (p.size() % 2) * 1e-4 * nd(rng));
    }
  }
  return p;
}

// What the other points leave of the line of j and k, in long double
// (80 or 128 bits: below the rounding of cuts_cross).
static bool rest(const std::vector<Pt>& p, int j, int k) {
  using L = long double;
  const L a[3] = {p[j].x, p[j].y, p[j].z}, b[3] = {p[k].x, p[k].y, p[k].z};
  L ha = 0, hb = 0, w[3], x[3], w2 = 0, hi = 1e300L, lo = -1e300L;
  for (int d = 0; d < 3; ++d) {
    const int e = (d + 1) % 3, f = (d + 2) % 3;
    w[d] = a[e] * b[f] - a[f] * b[e];
    ha += a[d] * a[d] / 2;
    hb += b[d] * b[d] / 2;
    w2 += w[d] * w[d];
  }
  for (int d = 0; d < 3; ++d) {
    const int e = (d + 1) % 3, f = (d + 2) % 3;
    x[d] = (ha * (b[e] * w[f] - b[f] * w[e]) + hb * (w[e] * a[f] - w[f] * a[e])) / w2;
  }
  for (int l = 1; l < (int)p.size(); ++l) {
    if (l == j || l == k) continue;
    const L v[3] = {p[l].x, p[l].y, p[l].z};
    L h = 0, wl = 0, xl = 0;
    for (int d = 0; d < 3; ++d) {
      h += v[d] * v[d] / 2;
      wl += w[d] * v[d];
      xl += x[d] * v[d];
    }
    const L t = (h - xl) / wl;
    if (wl > 0 && t < hi) hi = t;
    if (wl < 0 && t > lo) lo = t;
  }
  return lo < hi;
}

static int lines() {
  for (int set = 0; set < 5; ++set)
    for (const double unit : {1.0, 37.0, 1000.0, 1024.0, 1.0 / 8192.0, 1e-4}) {
      unsigned long long none = 0, again = 0, doubtful = 0, wrong = 0;
      for (unsigned seed = 1; seed <= 6; ++seed) {
        const std::vector<Pt> p = cloud(set, unit, seed);
        const int n = (int)p.size();
        std::vector<float> h(n);
        for (int a = 0; a < n; ++a) h[a] = 0.5f * (p[a].x * p[a].x + p[a].y * p[a].y + p[a].z * p[a].z);
        for (int j = 1; j < n; ++j)
          for (int k = 1; k < n; ++k) {
            if (k == j) continue;
            const FaceLine<float> f = face_line(p[j].x, p[j].y, p[j].z, h[j], p[k].x, p[k].y, p[k].z, h[k]);
            if (!(f.w2 > kLineMin)) continue;
            float hi = 1e15f, lo = -1e15f;
            int hl = -1, ll = -1;
            for (int l = 1; l < n; ++l) {
              if (l == j || l == k) continue;
              const float wl = std::fmaf(f.wz, p[l].z, std::fmaf(f.wy, p[l].y, f.wx * p[l].x));
              const float t = (h[l] - std::fmaf(f.z, p[l].z, std::fmaf(f.y, p[l].y, f.x * p[l].x))) / wl;
              if (wl > 0.f && t < hi) { hi = t; hl = l; }
              if (wl < 0.f && t > lo) { lo = t; ll = l; }
            }
            if (lo < hi) continue;
            ++none;
            const CutError<float> err(f, h[j], h[k]);
            const bool close = !(hl >= 0 && ll >= 0 &&
                                 (lo - hi) * err.len > err.of(f, p[hl].x, p[hl].y, p[hl].z, h[hl], hi) +
                                                           err.of(f, p[ll].x, p[ll].y, p[ll].z, h[ll], lo));
            const bool apart = !close || (hl >= 0 && ll >= 0 && cuts_cross(p[0], p[j], p[k], p[hl], p[ll]));
            again += close ? 1u : 0u;
            if (!apart) ++doubtful;
            else if (rest(p, j, k)) ++wrong;
          }
      }
      std::printf("%d %.9g %llu %llu %llu %llu\n", set, unit, none, again, doubtful, wrong);
    }
  return 0;
}

static int spheres() {
  std::mt19937 rng(11);
  std::normal_distribution<double> nd(0.0, 1.0);
  std::uniform_real_distribution<double> u11(-1.0, 1.0);
  for (int t = 0; t < 6000; ++t) {
    // corners of a turned and shifted unit cube, off by the jitter
    const double jitter = t % 3 == 0 ? 0.0 : t % 3 == 1 ? 1e-6 : 1e-3;
    double q[4], len = 0.0, shift[3];
    for (double& v : q) { v = nd(rng); len += v * v; }
    for (double& v : q) v /= std::sqrt(len);
    for (double& v : shift) v = 3.0 * u11(rng);
    const double r[3][3] = {
        {1 - 2 * (q[2] * q[2] + q[3] * q[3]), 2 * (q[1] * q[2] - q[0] * q[3]), 2 * (q[1] * q[3] + q[0] * q[2])},
        {2 * (q[1] * q[2] + q[0] * q[3]), 1 - 2 * (q[1] * q[1] + q[3] * q[3]), 2 * (q[2] * q[3] - q[0] * q[1])},
        {2 * (q[1] * q[3] - q[0] * q[2]), 2 * (q[2] * q[3] + q[0] * q[1]), 1 - 2 * (q[1] * q[1] + q[2] * q[2])}};
    unsigned pick[5] = {0, 1, 2, 3, 4 + (unsigned)(rng() % 4)};  // the face z = 0, and a corner above it
    if (t % 2) pick[3] = 4 + (unsigned)(rng() % 4), pick[4] = 3;  // or a fat one, and the face's last corner
    Pt p[5];
    for (int k = 0; k < 5; ++k) {
      double c[3], w[3];
      for (int d = 0; d < 3; ++d) c[d] = ((pick[k] >> d) & 1u) + jitter * nd(rng);
      for (int d = 0; d < 3; ++d) w[d] = r[d][0] * c[0] + r[d][1] * c[1] + r[d][2] * c[2] + shift[d];
      p[k] = Pt{(float)w[0], (float)w[1], (float)w[2], 0.f};
    }
    const double pi[3] = {p[0].x, p[0].y, p[0].z};
    double x[3], thin2;
    tet_centre(pi, p[1], p[2], p[3], x, thin2);
    const bool refused = !(thin2 < kThin * kThin);
    std::printf("%d %d", refused ? 1 : 0, !refused && sphere_leaves_out(pi, x, thin2, p[4]) ? 1 : 0);
    for (const Pt& v : p) std::printf(" %.9g %.9g %.9g", v.x, v.y, v.z);
    std::printf("\n");
  }
  return 0;
}

int main(int argc, char** argv) {
  if (argc == 2 && !std::strcmp(argv[1], "normals")) return normals();
  if (argc == 2 && !std::strcmp(argv[1], "lines")) return lines();
  if (argc == 2 && !std::strcmp(argv[1], "spheres")) return spheres();
  return 2;
}
