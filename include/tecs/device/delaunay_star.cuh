// delaunay_star.cuh -- the Delaunay finder for any number of cells.
//
// The reference's NaiveDelaunay (include/pair_finders/naive_delaunay.hpp:31-294)
// applies an in-cutoff pair (i, j)
//   2-D (:45-99):   once per third point k whose float circumcircle through
//                   i, j, k is non-degenerate (|den| > FLT_EPSILON) and holds
//                   no other point (distance^2 <= r^2 rejects);
//   3-D (:158-292): once per third point k for which some l > k spans a
//                   non-degenerate tetrahedron whose sphere holds no other
//                   point.
// It tries every k (and l) over all cells: O(N^3) work per cell.  This file
// finds the multiplicities from each cell's Delaunay star:
//
//  1. A counting-sorted copy of the positions on a uniform grid (about two
//     cells per bin) answers every geometric search below exactly: a search
//     visits every row of bins that its region (the shells around a point, a
//     ball, an open half-space, a band along a line) can touch, each row cut
//     to the region.
//  2. Star of cell i, in double.  From i's nearest neighbour a, the walk
//     moves through i's Voronoi cell: from a point x on it along a direction
//     w, the first point p that becomes as close to x + s w as i is the one
//     with the least s = (|x - p|^2 - |x - i|^2) / (2 w.(p - i)) over the
//     points with w.(p - i) > 0 (ties by index).  The midpoint of (i, a)
//     leads to a Voronoi edge (2-D: a vertex), each Voronoi edge to its
//     vertices, each vertex's faces to the next vertices; every vertex is the
//     centre of one empty circle/sphere through i ("star sphere"), and the
//     points on it with i form a simplex of i's star.
//  3. 2-D: the reference's float predicate decides, not the double geometry.
//     A triangle the float test can accept has an almost empty circumcircle,
//     so its points lie on, or within rounding of, one of i's star circles.
//     Every star circle collects the points within a tolerance of it (the
//     rounding of the float circumcentre, from the coordinates' size and the
//     triangle's shape, times a safety factor), and the reference's own float
//     test (with its emptiness check over every point the test can reach,
//     found through the grid) runs on every (j, k) drawn from that set.  On
//     the hull, the points near the line of each hull edge at i form one more
//     set (three collinear points can pass the float test there).  mult(i, j)
//     is the number of distinct k accepted: the reference's multiplicities,
//     bit for bit.
//  4. 3-D: the reference's quotients solve 2 (x_m - x_i).c = |x_m|^2 -
//     |x_i|^2, so they are the circumcentre itself; it adds x_i once more, and
//     its sphere (centre x_i + c, radius |c|) passes through i but not through
//     j, k or l.  Its test accepts simplices whose number grows with the cell
//     count, which no local search can enumerate.  The 3-D form here applies
//     the reference's counting rule to the Delaunay tetrahedra: mult(i, j) is
//     the number of distinct k = min(k, l) over the star tetrahedra
//     (i, j, k, l).
//
// The same code runs on the device (one warp per cell, k_dl_mult; Warp
// below) and on the host (the tests' driver; Solo), so the walk can be
// checked on the CPU against the naive restatement (2-D) and an independent
// Delaunay triangulation (3-D).
#pragma once

#include <float.h>
#include <math.h>
#include <stdint.h>
#include <string.h>

#if defined(__CUDACC__)
#define TECS_DL_HD __host__ __device__ __forceinline__
#define TECS_DL_CALL __host__ __device__ __noinline__
#else
#define TECS_DL_HD inline
#define TECS_DL_CALL inline
#endif

namespace tecs {
namespace dl {

struct alignas(16) Pt {
  float x, y, z, w;  // a position (w unused)
};

// The grid in float, for the row ranges (grid_f).
struct GridF {
  float lo[3], h, inv, m;
  int dims[3];
};

// Bin grid of the active cells.  Bin b along dimension d covers
// [lo + b h, lo + (b + 1) h); bin1() is the one binning function, used for
// the points and for every search range, so a point inside a range's bounds
// is always inside the range's bins (floor and the affine map are monotone).
struct Grid {
  double lo[3];
  double h, inv;
  int dims[3];
  unsigned nbins;
  const unsigned* off;  // bin offsets, nbins + 1
  const unsigned* idx;  // slot of each sorted entry
  const Pt* sp;         // positions in sorted order
  const Pt* P;          // positions by slot
  unsigned n;           // active cells
  float rc2;            // cutoff^2 of the in-cutoff test
  GridF f;              // set by plan_grid
};

// error bits of one cell's search
enum : unsigned {
  kErrStar = 1u,   // more star simplices or spheres than the local arrays hold
  kErrNear = 2u,   // more points near one circle than the local array holds
  kErrPairs = 4u,  // more accepted (j, k) than the local array holds
  kErrList = 8u    // more partners than the output row holds
};

constexpr int kMaxTet = 192;     // star simplices (3-D tetrahedra, 2-D triangles)
constexpr int kMaxSph = 192;     // distinct star spheres (3-D: one per tetrahedron)
constexpr int kMaxNear = 48;     // points near one circle (2-D)
constexpr int kMaxPairs = 320;   // accepted (j, k)
constexpr int kMaxKill = 64;     // points tested first (2-D)
// Sets up to this size are walked without them: a triangle's test over the grid is
// short there (64 cells, cutoff past all: 0.23 ms a pass without, 0.28 with; 1,000
// cells 0.37 and 0.42, 2,000 cells 4.0 and 0.66).
constexpr unsigned kKillFrom = 512;
constexpr double kInf = 1.0e300;
constexpr double kEps = (double)FLT_EPSILON;

// Lane policies.  Every search visits entries; Solo visits them in one
// thread (the host), Warp in the 32 lanes of a warp, each lane taking every
// 32nd entry.  Every result of a visit is combined across the warp (a vote,
// a minimum, candidates merged in lane order) before anything depends on it.
// The star and the candidate lists (Scratch) are one copy per warp, in
// shared memory on the device: every lane reads them, the leader lane writes
// them between two sync() calls.
struct Solo {
  static constexpr unsigned width = 1;
  TECS_DL_HD unsigned lane() const { return 0u; }
  TECS_DL_HD bool leader() const { return true; }
  TECS_DL_HD void sync() const {}
  TECS_DL_HD bool any(bool b) const { return b; }
  TECS_DL_HD unsigned ballot(bool b) const { return b ? 1u : 0u; }
  TECS_DL_HD unsigned bcast(unsigned v, int) const { return v; }
  TECS_DL_HD double bcast(double v, int) const { return v; }
  TECS_DL_HD unsigned most(unsigned v) const { return v; }
  TECS_DL_HD unsigned least(unsigned v) const { return v; }
};

#if defined(__CUDACC__)
struct Warp {
  static constexpr unsigned width = 32;
  __device__ __forceinline__ unsigned lane() const { return threadIdx.x & 31u; }
  __device__ __forceinline__ bool leader() const { return (threadIdx.x & 31u) == 0u; }
  __device__ __forceinline__ void sync() const { __syncwarp(); }
  __device__ __forceinline__ bool any(bool b) const { return __any_sync(0xffffffffu, b); }
  __device__ __forceinline__ unsigned ballot(bool b) const { return __ballot_sync(0xffffffffu, b); }
  __device__ __forceinline__ unsigned bcast(unsigned v, int src) const { return __shfl_sync(0xffffffffu, v, src); }
  __device__ __forceinline__ double bcast(double v, int src) const { return __shfl_sync(0xffffffffu, v, src); }
  __device__ __forceinline__ unsigned most(unsigned v) const { return __reduce_max_sync(0xffffffffu, v); }
  __device__ __forceinline__ unsigned least(unsigned v) const { return __reduce_min_sync(0xffffffffu, v); }
};
#endif

// the lowest set bit's index
TECS_DL_HD int low_bit(unsigned m) {
#if defined(__CUDA_ARCH__)
  return __ffs((int)m) - 1;
#endif
  int b = 0;
  while (!(m & 1u)) { m >>= 1; ++b; }
  return b;
}

// the least (key, id) over the lanes, in every lane
template <class W>
TECS_DL_HD void lane_min(const W& w, double& key, unsigned& id) {
  for (unsigned sh = W::width / 2; sh > 0; sh >>= 1) {
    const int src = (int)(w.lane() ^ sh);
    const double k2 = w.bcast(key, src);
    const unsigned i2 = w.bcast(id, src);
    if (k2 < key || (k2 == key && i2 < id)) { key = k2; id = i2; }
  }
}

// the first index below n for which pred holds, or -1; the lanes take the
// indices in turn
template <class W, class F>
TECS_DL_HD int find_first(const W& w, int n, F&& pred) {
  for (int q0 = 0; q0 < n; q0 += (int)W::width) {
    const int q = q0 + (int)w.lane();
    const unsigned m = w.ballot(q < n && pred(q));
    if (m) return q0 + low_bit(m);
  }
  return -1;
}

struct NoRound {
  TECS_DL_HD void operator()() const {}
};

// the bits of a float that is not negative, which order as the floats do
TECS_DL_HD unsigned float_order(float f) {
#if defined(__CUDA_ARCH__)
  return __float_as_uint(f);
#else
  unsigned u;
  memcpy(&u, &f, sizeof u);
  return u;
#endif
}

TECS_DL_HD double dmax(double a, double b) { return a > b ? a : b; }
TECS_DL_HD int imax(int a, int b) { return a > b ? a : b; }
TECS_DL_HD int imin(int a, int b) { return a < b ? a : b; }

TECS_DL_HD int bin1(const Grid& g, int d, double x) {
  const double t = floor((x - g.lo[d]) * g.inv);
  if (!(t >= 0.0)) return 0;  // also NaN
  if (t >= (double)(g.dims[d] - 1)) return g.dims[d] - 1;
  return (int)t;
}

// Row ranges in float.  A search region's rows are the same in every lane
// of a warp, and FP64 is scarce on this part, so the bounds are formed in
// float with a margin m far above float rounding (1e-3 of a bin plus the
// rounding of bin numbers and coordinates of the grid's size): a range can
// only grow, so no point is lost, and the tests on the points stay exact.
TECS_DL_HD GridF grid_f(const Grid& g) {
  GridF f;
  double span = 0.0;
  int dm = 1;
  for (int d = 0; d < 3; ++d) {
    f.lo[d] = (float)g.lo[d];
    f.dims[d] = g.dims[d];
    span = dmax(span, fabs(g.lo[d]) + (double)g.dims[d] * g.h);
    dm = imax(dm, g.dims[d]);
  }
  f.h = (float)g.h;
  f.inv = (float)g.inv;
  f.m = (float)(g.h * (1.0e-3 + 1.0e-6 * (double)dm) + 2.0e-6 * span);
  return f;
}

// Bin edge and extents from the cells' bounding box [mn, mx]: about two cells
// per bin over the dimensions the cells spread along (a flat dimension gets
// one bin), at most max_bins bins.
template <int D>
TECS_DL_HD void plan_grid(Grid& g, const double* mn, const double* mx, unsigned n, unsigned max_bins) {
  double ext[3] = {0.0, 0.0, 0.0};
  // a span that is not finite (a cell at infinity) gets one bin
  for (int d = 0; d < D; ++d) ext[d] = (mx[d] - mn[d] > 0.0 && mx[d] - mn[d] < 1.0e30) ? mx[d] - mn[d] : 0.0;
  double target = n > 2u ? 0.5 * (double)n : 1.0;
  if (target > (double)max_bins) target = (double)max_bins;
  bool thin[3] = {false, false, false};
  double h = 1.0;
  for (int it = 0; it < 3; ++it) {
    double vol = 1.0;
    int k = 0;
    for (int d = 0; d < D; ++d)
      if (!thin[d]) { vol *= ext[d]; ++k; }
    if (k == 0 || !(vol > 0.0)) {
      // every spread dimension is flat: one bin per dimension of zero extent
      double m = 0.0;
      for (int d = 0; d < D; ++d) m = dmax(m, ext[d]);
      h = m > 0.0 ? m : 1.0;
      break;
    }
    h = pow(vol / target, 1.0 / (double)k);
    bool changed = false;
    for (int d = 0; d < D; ++d)
      if (!thin[d] && ext[d] < h) { thin[d] = true; changed = true; }
    if (!changed) break;
  }
  if (!(h > 0.0) || !(h < 1.0e300)) h = 1.0;
  for (;;) {
    double prod = 1.0;
    for (int d = 0; d < 3; ++d) {
      const double q = d < D ? floor(ext[d] / h) + 1.0 : 1.0;
      g.dims[d] = q < 1.0 ? 1 : (q > 2.0e9 ? 2000000000 : (int)q);
      prod *= (double)g.dims[d];
    }
    if (prod <= (double)max_bins) break;
    h *= 1.25;
  }
  for (int d = 0; d < 3; ++d) g.lo[d] = d < D ? mn[d] : 0.0;
  g.h = h;
  g.inv = 1.0 / h;
  g.nbins = (unsigned)g.dims[0] * (unsigned)g.dims[1] * (unsigned)g.dims[2];
  g.f = grid_f(g);
}

TECS_DL_HD unsigned flat(const Grid& g, int x, int y, int z) {
  return ((unsigned)z * (unsigned)g.dims[1] + (unsigned)y) * (unsigned)g.dims[0] + (unsigned)x;
}

// Every entry of nrows rows; range(r, lo, hi) gives row r's entries [lo, hi)
// and may differ from lane to lane in what it computes, not in what it gives.
// f(slot, pos) returns false to stop (the warp stops when any lane does).
// round() runs in every lane after each round of entries (one entry per lane),
// where the caller merges what the lanes found.  One thread loads four
// entries at a time, to keep several loads in flight.  A warp's lanes form the
// ranges of 32 rows side by side and take the rows' entries as one list, 32 at
// a time: most rows hold fewer than ten entries, and the ranges cost more than
// the entries (one row after the other, every lane forming every range: 54 ms
// where this takes 32 for all of 40k cells in 3-D).
template <class W, class RF, class F, class R = NoRound>
TECS_DL_HD bool visit_rows(const W& w, const Grid& g, int nrows, RF&& range, F&& f, R&& round = R{}) {
  if (W::width == 1) {
    for (int r = 0; r < nrows; ++r) {
      unsigned e = 0, hi = 0;
      range(r, e, hi);
      for (; e + 4 <= hi; e += 4) {
        const unsigned i0 = g.idx[e], i1 = g.idx[e + 1], i2 = g.idx[e + 2], i3 = g.idx[e + 3];
        const Pt p0 = g.sp[e], p1 = g.sp[e + 1], p2 = g.sp[e + 2], p3 = g.sp[e + 3];
        if (!f(i0, p0)) return false;
        round();
        if (!f(i1, p1)) return false;
        round();
        if (!f(i2, p2)) return false;
        round();
        if (!f(i3, p3)) return false;
        round();
      }
      for (; e < hi; ++e) {
        if (!f(g.idx[e], g.sp[e])) return false;
        round();
      }
    }
    return true;
  }
  for (int r0 = 0; r0 < nrows; r0 += (int)W::width) {
    const int r = r0 + (int)w.lane();
    unsigned lo = 0, hi = 0;
    if (r < nrows) range(r, lo, hi);
    const unsigned len = hi > lo ? hi - lo : 0u;
    unsigned end = len;  // of this row in the list
    for (unsigned sh = 1; sh < W::width; sh <<= 1) {
      const unsigned y = w.bcast(end, (int)(w.lane() - sh) & (int)(W::width - 1));
      if (w.lane() >= sh) end += y;
    }
    const unsigned total = w.bcast(end, (int)W::width - 1);
    const unsigned base = lo - (end - len);
    for (unsigned t0 = 0; t0 < total; t0 += W::width) {
      const unsigned t = t0 + w.lane();
      // the row of place t: the first whose end is past it
      int q = 0;
      for (unsigned sh = W::width / 2; sh > 0; sh >>= 1)
        if (w.bcast(end, q + (int)sh - 1) <= t) q += (int)sh;
      const unsigned e = t + w.bcast(base, q & (int)(W::width - 1));
      bool stop = false;
      if (t < total) stop = !f(g.idx[e], g.sp[e]);
      if (w.any(stop)) return false;
      round();
    }
  }
  return true;
}

// The entries of bins [a, b] of row (y, z).
TECS_DL_HD void row_entries(const Grid& g, int a, int b, int y, int z, unsigned& lo, unsigned& hi) {
  const unsigned k = flat(g, 0, y, z);
  lo = g.off[k + (unsigned)a];
  hi = g.off[k + (unsigned)b + 1u];
}

// The bins at Chebyshev distance k from bc.
template <int D, class W, class F, class R = NoRound>
TECS_DL_HD bool visit_shell(const W& w, const Grid& g, const int* bc, int k, F&& f, R&& round = R{}) {
  const int side = 2 * k + 1;
  // two parts a row: the whole row on a face of the shell, else its two ends
  return visit_rows(w, g, 2 * side * (D >= 3 ? side : 1), [&](int r, unsigned& lo, unsigned& hi) {
    const int part = r & 1, q = r >> 1;
    const int y = bc[1] - k + q % side, z = D >= 3 ? bc[2] - k + q / side : 0;
    if (y < 0 || y >= g.dims[1] || z < 0 || z >= g.dims[2]) return;
    const bool full = y == bc[1] - k || y == bc[1] + k || (D >= 3 && (z == bc[2] - k || z == bc[2] + k));
    int a, b;
    if (full) {
      if (part) return;
      a = imax(bc[0] - k, 0);
      b = imin(bc[0] + k, g.dims[0] - 1);
      if (a > b) return;
    } else {
      a = b = part ? bc[0] + k : bc[0] - k;
      if (a < 0 || a >= g.dims[0]) return;
    }
    row_entries(g, a, b, y, z, lo, hi);
  }, f, round);
}

TECS_DL_HD int bin1f(const GridF& f, int d, float x) {
  const float t = floorf((x - f.lo[d]) * f.inv);
  if (!(t >= 0.0f)) return 0;  // also NaN
  if (t >= (float)(f.dims[d] - 1)) return f.dims[d] - 1;
  return (int)t;
}

// Distance from v to the interval that bin b of dimension d covers (0
// inside), the interval widened by the margin.
TECS_DL_HD float gap_to_bin(const GridF& f, int d, int b, float v) {
  const float lo = f.lo[d] + (float)b * f.h - f.m, hi = f.lo[d] + (float)(b + 1) * f.h + f.m;
  return v < lo ? lo - v : (v > hi ? v - hi : 0.0f);
}

// The bins [a, b] of row (y, z) that can hold a point p with w.(p - o) > 0.
template <int D>
TECS_DL_HD void half_range(const GridF& f, int y, int z, const float* o, const float* w, int& a, int& b) {
  // the largest w1 (y - o1) + w2 (z - o2) over the row's box, then its margin
  float off = 0.0f, aw = 0.0f;
  for (int d = 1; d < D; ++d) {
    const int bb = d == 1 ? y : z;
    const float lo = f.lo[d] + (float)bb * f.h - f.m, hi = f.lo[d] + (float)(bb + 1) * f.h + f.m;
    off += w[d] > 0.0f ? w[d] * (hi - o[d]) : w[d] * (lo - o[d]);
    aw += fabsf(w[d]);
  }
  off += aw * f.m;
  // need w0 (x - o0) + off > 0
  a = 0;
  b = f.dims[0] - 1;
  if (w[0] > 0.0f) a = bin1f(f, 0, o[0] - off / w[0] - f.m);
  else if (w[0] < 0.0f) b = bin1f(f, 0, o[0] - off / w[0] + f.m);
  else if (!(off >= 0.0f)) { a = 1; b = 0; }
}

// Every entry within distance rad of c (and a few just outside): the rows
// of bins (along x) that the ball touches, each cut to the ball's chord --
// and, given a plane (o, w), to the bins that reach its open side.
template <int D, class W, class F, class R = NoRound>
TECS_DL_HD bool visit_ball(const W& ln, const Grid& g, const double* c, double rad, F&& f, const double* o = nullptr,
                           const double* w = nullptr, R&& round = R{}) {
  if (!(rad < 1.0e18)) {
    return visit_rows(ln, g, g.dims[1] * g.dims[2], [&](int r, unsigned& lo, unsigned& hi) {
      row_entries(g, 0, g.dims[0] - 1, r % g.dims[1], r / g.dims[1], lo, hi);
    }, f, round);
  }
  const GridF& gf = g.f;
  const float cf[3] = {(float)c[0], (float)c[1], (float)c[2]};
  const float rf = (float)rad * 1.00001f + gf.m;
  float of[3] = {0.f, 0.f, 0.f}, wf[3] = {0.f, 0.f, 0.f};
  if (w)
    for (int d = 0; d < 3; ++d) { of[d] = (float)o[d]; wf[d] = (float)w[d]; }
  const int z0 = D >= 3 ? bin1f(gf, 2, cf[2] - rf) : 0, z1 = D >= 3 ? bin1f(gf, 2, cf[2] + rf) : 0;
  const int y0 = bin1f(gf, 1, cf[1] - rf), y1 = bin1f(gf, 1, cf[1] + rf);
  const int ny = y1 - y0 + 1;
  const float r2 = rf * rf;
  return visit_rows(ln, g, ny * (z1 - z0 + 1), [&](int r, unsigned& lo, unsigned& hi) {
    const int z = z0 + r / ny, y = y0 + r % ny;
    const float gz = D >= 3 ? gap_to_bin(gf, 2, z, cf[2]) : 0.0f;
    const float gy = gap_to_bin(gf, 1, y, cf[1]);
    const float rem2 = r2 - gy * gy - gz * gz + 1.0e-5f * r2;
    if (rem2 < 0.0f) return;
    const float rem = sqrtf(rem2) + gf.m;
    int a = bin1f(gf, 0, cf[0] - rem), b = bin1f(gf, 0, cf[0] + rem);
    if (w) {
      int ha, hb;
      half_range<D>(gf, y, z, of, wf, ha, hb);
      a = imax(a, ha);
      b = imin(b, hb);
      if (a > b) return;
    }
    row_entries(g, a, b, y, z, lo, hi);
  }, f, round);
}

// Every entry p with w.(p - o) > 0 (and a few on the boundary): each row of
// bins cut to the part that can reach the open side.
template <int D, class W, class F>
TECS_DL_HD bool visit_half(const W& ln, const Grid& g, const double* o, const double* w, F&& f) {
  const GridF& gf = g.f;
  const float of[3] = {(float)o[0], (float)o[1], (float)o[2]}, wf[3] = {(float)w[0], (float)w[1], (float)w[2]};
  return visit_rows(ln, g, g.dims[1] * (D >= 3 ? g.dims[2] : 1), [&](int r, unsigned& lo, unsigned& hi) {
    int a, b;
    half_range<D>(gf, r % g.dims[1], r / g.dims[1], of, wf, a, b);
    if (a <= b) row_entries(g, a, b, r % g.dims[1], r / g.dims[1], lo, hi);
  }, f);
}

// The unit normal of the plane through a cell and two others, at a and b from
// it; slack: |a| |b| over the length of a x b, by which the rounding of a x b
// (a few 2^-53 |a| |b|) turns the normal.  False where a and b are so nearly on
// one line that a x b in float (off by up to 7 2^-24 |a| |b|) may point
// elsewhere, and with it the side of the plane that a float search took.
TECS_DL_HD bool plane_normal(const double* a, const double* b, double* n, double& slack) {
  const double c[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
  const double len = sqrt(c[0] * c[0] + c[1] * c[1] + c[2] * c[2]);
  const double ab = sqrt((a[0] * a[0] + a[1] * a[1] + a[2] * a[2]) * (b[0] * b[0] + b[1] * b[1] + b[2] * b[2]));
  if (!(len > 1.0e-5 * ab)) return false;
  for (int d = 0; d < 3; ++d) n[d] = c[d] / len;
  slack = ab / len;
  return true;
}

// The local search in space (delaunay_local.cuh): the line in which the planes
// halfway to two others, at vj and vk from the cell, meet -- x + t w with x its
// point nearest to the cell.  h: half a squared length.
template <class T>
struct FaceLine {
  T wx, wy, wz, w2, inv, x, y, z;
};

// Lines with a lesser w^2 are not formed in float: their products may underflow.
constexpr float kLineMin = 1.0e-28f;

template <class T>
TECS_DL_HD FaceLine<T> face_line(T jx, T jy, T jz, T jh, T kx, T ky, T kz, T kh) {
  FaceLine<T> l;
  l.wx = jy * kz - jz * ky;
  l.wy = jz * kx - jx * kz;
  l.wz = jx * ky - jy * kx;
  l.w2 = l.wx * l.wx + l.wy * l.wy + l.wz * l.wz;
  l.inv = (T)1 / l.w2;
  l.x = (jh * (ky * l.wz - kz * l.wy) + kh * (l.wy * jz - l.wz * jy)) * l.inv;
  l.y = (jh * (kz * l.wx - kx * l.wz) + kh * (l.wz * jx - l.wx * jz)) * l.inv;
  l.z = (jh * (kx * l.wy - ky * l.wx) + kh * (l.wx * jy - l.wy * jx)) * l.inv;
  return l;
}

// How far rounding may move the cut that a point makes on a line, as a length.
// With u the unit roundoff, S the sine of the angle between vj and vk and Q
// that of a point's v with the plane across the line, rounding moves
//   w   by 7 u |vj| |vk|                     (a turn of 7 u / S),
//   x   by 18 u (|vj| + |vk|) / S^2          (|x| <= (|vj| + |vk|) / 2 S),
//   T   by u (2.5 |v| + 18 (|vj| + |vk|) / S^2 + 4 |x| + |T| (7 / S + 4)) / Q + 3 u |T|
// of a cut at T = t |w| from x.  Twice that is allowed for, which covers the
// second order and the rounding here; it holds in any unit of length.
TECS_DL_HD float root(float v) { return sqrtf(v); }
TECS_DL_HD double root(double v) { return sqrt(v); }
TECS_DL_HD float size(float v) { return fabsf(v); }
TECS_DL_HD double size(double v) { return fabs(v); }

template <class T>
struct CutError {
  T len, turn, near;  // |w|, 1 / S, 20 (|vj| + |vk|) / S^2
  TECS_DL_HD CutError(const FaceLine<T>& l, T jh, T kh) {
    len = root(l.w2);
    turn = (T)2 * root(jh) * root(kh) / len;
    near = (T)28.3 * (root(jh) + root(kh)) * turn * turn;
  }
  TECS_DL_HD T of(const FaceLine<T>& l, T vx, T vy, T vz, T vh, T t) const {
    constexpr T u2 = sizeof(T) == 4 ? (T)1.3e-7 : (T)2.4e-16;
    const T v = (T)1.4143 * root(vh);
    const T q = size(l.wx * vx + l.wy * vy + l.wz * vz);
    return u2 * ((T)3 * v + near + (T)14 * size(t) * len * turn) * (len * v / q);
  }
};

// In double: whether the line of the planes halfway to pj and pk is cut off at
// t < hi by ph and at t > lo by pl with hi < lo, with certainty.
template <class P>
TECS_DL_CALL bool cuts_cross(const P& pi, const P& pj, const P& pk, const P& ph, const P& pl) {
  double v[4][3], h[4];
  const P* p[4] = {&pj, &pk, &ph, &pl};
  for (int q = 0; q < 4; ++q) {
    v[q][0] = (double)p[q]->x - (double)pi.x;
    v[q][1] = (double)p[q]->y - (double)pi.y;
    v[q][2] = (double)p[q]->z - (double)pi.z;
    h[q] = 0.5 * (v[q][0] * v[q][0] + v[q][1] * v[q][1] + v[q][2] * v[q][2]);
  }
  const FaceLine<double> l = face_line(v[0][0], v[0][1], v[0][2], h[0], v[1][0], v[1][1], v[1][2], h[1]);
  const CutError<double> err(l, h[0], h[1]);
  double t[2], e[2];
  for (int q = 0; q < 2; ++q) {
    const double* c = v[2 + q];
    const double wl = l.wx * c[0] + l.wy * c[1] + l.wz * c[2];
    if (!(q ? wl < 0.0 : wl > 0.0)) return false;
    t[q] = (h[2 + q] - (l.x * c[0] + l.y * c[1] + l.z * c[2])) / wl;
    e[q] = err.of(l, c[0], c[1], c[2], h[2 + q], t[q]);
  }
  return (t[1] - t[0]) * err.len > e[0] + e[1];
}

// The circumcentre x of the cell at pi and three others, relative to the cell;
// thin2: (|a| |b| |c| / det)^2 of the three relative positions, by which rounding
// is enlarged: x is off by at most 2^-53 thin (15 max |a| + 8 |x|).
template <class P>
TECS_DL_HD void tet_centre(const double* pi, const P& pa, const P& pb, const P& pc, double* x, double& thin2) {
  const double a[3] = {pa.x - pi[0], pa.y - pi[1], pa.z - pi[2]}, b[3] = {pb.x - pi[0], pb.y - pi[1], pb.z - pi[2]},
               c[3] = {pc.x - pi[0], pc.y - pi[1], pc.z - pi[2]};
  double ha = 0.0, hb = 0.0, hc = 0.0;
  for (int d = 0; d < 3; ++d) {
    ha += a[d] * a[d];
    hb += b[d] * b[d];
    hc += c[d] * c[d];
  }
  const double bc[3] = {b[1] * c[2] - b[2] * c[1], b[2] * c[0] - b[0] * c[2], b[0] * c[1] - b[1] * c[0]};
  const double ca[3] = {c[1] * a[2] - c[2] * a[1], c[2] * a[0] - c[0] * a[2], c[0] * a[1] - c[1] * a[0]};
  const double ab[3] = {a[1] * b[2] - a[2] * b[1], a[2] * b[0] - a[0] * b[2], a[0] * b[1] - a[1] * b[0]};
  const double det = a[0] * bc[0] + a[1] * bc[1] + a[2] * bc[2];
  const double inv = 0.5 / det;
  for (int d = 0; d < 3; ++d) x[d] = (ha * bc[d] + hb * ca[d] + hc * ab[d]) * inv;
  thin2 = 4.0 * ha * inv * hb * inv * hc;
}

// Tetrahedra thinner than this are not decided by their centre: at 2^-53 thin its
// error stays far below that of a float test of a point against the sphere.
constexpr double kThin = 1.0e6;

// The share of |v|^2 + |x|^2 that a point's power |v|^2 / 2 - x.v in a sphere has
// to exceed to be certain: the centre's error (with max |a| <= 2 |x|) moves it by
// up to 19 2^-53 thin of that, the point's own products by less than 1e-15.
TECS_DL_HD double sphere_margin(double thin2) { return 1.0e-11 + 4.0e-15 * sqrt(thin2); }

template <class P>
TECS_DL_HD bool sphere_leaves_out(const double* pi, const double* x, double thin2, const P& p) {
  const double v[3] = {p.x - pi[0], p.y - pi[1], p.z - pi[2]};
  const double vv = v[0] * v[0] + v[1] * v[1] + v[2] * v[2], xx = x[0] * x[0] + x[1] * x[1] + x[2] * x[2];
  return 0.5 * vv - (v[0] * x[0] + v[1] * x[1] + v[2] * x[2]) > sphere_margin(thin2) * (vv + xx);
}

// 2-D: every entry within distance del of the line through o with unit
// normal nrm (and a few just outside): each row of bins cut to the band.
template <class W, class F, class R>
TECS_DL_HD bool visit_band(const W& w, const Grid& g, const double* o, const double* nrm, double del, F&& f,
                           R&& round) {
  const double m = 1.0e-9 * g.h;
  return visit_rows(w, g, g.dims[1], [&](int y, unsigned& lo, unsigned& hi) {
    const double ylo = g.lo[1] + (double)y * g.h - m, yhi = g.lo[1] + (double)(y + 1) * g.h + m;
    int a = 0, b = g.dims[0] - 1;
    if (fabs(nrm[0]) > 1.0e-12) {
      // n0 (x - o0) + n1 (y - o1) in [-del, del] over the row's y interval
      double xmn = kInf, xmx = -kInf;
      for (int e = 0; e < 4; ++e) {
        const double yy = (e & 1) ? yhi : ylo, sg = (e & 2) ? del : -del;
        const double x = o[0] + (sg - nrm[1] * (yy - o[1])) / nrm[0];
        xmn = x < xmn ? x : xmn;
        xmx = x > xmx ? x : xmx;
      }
      a = bin1(g, 0, xmn - m);
      b = bin1(g, 0, xmx + m);
    } else {
      const double half = del / fabs(nrm[1]);
      if (yhi < o[1] - half || ylo > o[1] + half) return;
    }
    row_entries(g, a, b, y, 0, lo, hi);
  }, f, round);
}

template <int D>
TECS_DL_HD int shells_to_cover(const Grid& g, const int* bc) {
  int k = 0;
  for (int d = 0; d < D; ++d) k = imax(k, imax(bc[d], g.dims[d] - 1 - bc[d]));
  return k;
}

template <int D>
TECS_DL_HD void bin_of(const Grid& g, const double* x, int* b) {
  for (int d = 0; d < 3; ++d) b[d] = d < D ? bin1(g, d, x[d]) : 0;
}

TECS_DL_HD void load(const Pt& p, double* q) { q[0] = p.x; q[1] = p.y; q[2] = p.z; }

// ---------------------------------------------------------------------------
// The reference's float predicates, operation for operation.

TECS_DL_HD float sqlen2(const Pt& p) { return p.x * p.x + p.y * p.y; }
TECS_DL_HD float sqlen3(const Pt& p) { return (p.x * p.x + p.y * p.y) + p.z * p.z; }

// in-cutoff test: displacement = x_i - x_j, length_squared() < cutoff^2
template <int D>
TECS_DL_HD bool in_cutoff(const Grid& g, const Pt& pi, const Pt& pj) {
  const float e0 = pi.x - pj.x, e1 = pi.y - pj.y;
  float d2 = e0 * e0 + e1 * e1;
  if (D >= 3) { const float e2 = pi.z - pj.z; d2 = d2 + e2 * e2; }
  return d2 < g.rc2;
}

// Whether the triangle (i, j, k) is not degenerate and none of the points
// around i (Scratch::kill) rejects it: the start of tri_pass, for one lane.
template <class S>
TECS_DL_HD bool tri_near(const Grid& g, unsigned i, unsigned j, unsigned k, const S& sc) {
  const Pt pi = g.P[i], pj = g.P[j], pk = g.P[k];
  const float den = 2.0f * (pi.x * (pj.y - pk.y) + pj.x * (pk.y - pi.y) + pk.x * (pi.y - pj.y));
  if (fabsf(den) <= FLT_EPSILON) return false;
  const float li = sqlen2(pi), lj = sqlen2(pj), lk = sqlen2(pk);
  float c[2];
  c[0] = (li * (pj.y - pk.y) + lj * (pk.y - pi.y) + lk * (pi.y - pj.y)) / den;
  c[1] = (li * (pk.x - pj.x) + lj * (pi.x - pk.x) + lk * (pj.x - pi.x)) / den;
  const float e0 = pi.x - c[0], e1 = pi.y - c[1];
  const float r2 = e0 * e0 + e1 * e1;
  for (int q = 0; q < sc.n_kill; ++q) {
    const float f0 = sc.kill[q].x - c[0], f1 = sc.kill[q].y - c[1];
    if (f0 * f0 + f1 * f1 <= r2 && sc.kill_id[q] != j && sc.kill_id[q] != k) return false;
  }
  return true;
}

// naive_delaunay.hpp:62-99: triangle (i, j, k) accepted
template <class W, class S>
TECS_DL_CALL bool tri_pass(const W& w, const Grid& g, unsigned i, unsigned j, unsigned k, const S& sc) {
  const Pt pi = g.P[i], pj = g.P[j], pk = g.P[k];
  const float den = 2.0f * (pi.x * (pj.y - pk.y) + pj.x * (pk.y - pi.y) + pk.x * (pi.y - pj.y));
  if (fabsf(den) <= FLT_EPSILON) return false;
  const float li = sqlen2(pi), lj = sqlen2(pj), lk = sqlen2(pk);
  float c[2];
  c[0] = (li * (pj.y - pk.y) + lj * (pk.y - pi.y) + lk * (pi.y - pj.y)) / den;
  c[1] = (li * (pk.x - pj.x) + lj * (pi.x - pk.x) + lk * (pj.x - pi.x)) / den;
  const float e0 = pi.x - c[0], e1 = pi.y - c[1];
  const float r2 = e0 * e0 + e1 * e1;
  if (find_first(w, sc.n_kill, [&](int q) {
        const float f0 = sc.kill[q].x - c[0], f1 = sc.kill[q].y - c[1];
        return f0 * f0 + f1 * f1 <= r2 && sc.kill_id[q] != j && sc.kill_id[q] != k;
      }) >= 0)
    return false;
  // every point the test can reach: float distance^2 <= r2 means a true
  // distance within sqrt(r2) (1 + a few eps)
  const double cc[3] = {c[0], c[1], 0.0};
  const double reach = (double)sqrtf(r2) * (1.0 + 8.0 * kEps) + 1.0e-30;
  const bool finite = cc[0] > -1.0e30 && cc[0] < 1.0e30 && cc[1] > -1.0e30 && cc[1] < 1.0e30;
  return visit_ball<2>(w, g, cc, finite ? reach : kInf, [&](unsigned m, const Pt& pm) {
    if (m == i || m == j || m == k) return true;
    const float f0 = pm.x - c[0], f1 = pm.y - c[1];
    return !(f0 * f0 + f1 * f1 <= r2);
  });
}

// ---------------------------------------------------------------------------
// Geometry of the star, in double.

struct Hit {
  unsigned id;
  double s;
};

// The first point p (not in ex) that becomes as close to x0 + s w as i is:
// the least s = (|x0 - p|^2 - |x0 - i|^2) / (2 w.(p - i)) over w.(p - i) > 0.
// Every point with parameter <= s lies in the ball B(s) about x0 + s w
// through i (on the open side of the plane through i), and B(s) grows with
// s.  So: a bound from the points near i (2-D), else balls of doubling s until
// one holds a point; its least parameter is then the answer (after one more
// ball at that parameter, for points just outside the last ball's bins); each
// ball cut to the open side; past the grid's size, every bin on the open side
// of the plane.
template <int D, class W>
TECS_DL_CALL Hit shoot(const W& ln, const Grid& g, const double* x0, const double* w, const double* pi,
                     const unsigned* ex, int nex) {
  double pow0 = 0.0;
  for (int d = 0; d < D; ++d) { const double v = x0[d] - pi[d]; pow0 += v * v; }
  Hit best{~0u, kInf};  // this lane's, then the warp's after each visit
  auto take = [&](unsigned id, const Pt& p) {
    for (int e = 0; e < nex; ++e)
      if (id == ex[e]) return true;
    double q[3];
    load(p, q);
    double wp = 0.0, nn = 0.0, num = 0.0;
    for (int d = 0; d < D; ++d) {
      const double v = q[d] - pi[d], u = q[d] - x0[d];
      wp += w[d] * v;
      nn += v * v;
      num += u * u;
    }
    if (!(wp > 0.0) || wp * wp <= 1.0e-18 * nn) return true;  // on or behind the plane through i
    const double s = (num - pow0) / (2.0 * wp);
    if (s < best.s || (s == best.s && id < best.id)) best = Hit{id, s};
    return true;
  };
  auto reduce = [&]() { lane_min(ln, best.s, best.id); };
  // visits B(s) (with a margin)
  auto ball_at = [&](double s) {
    double c[3] = {0.0, 0.0, 0.0}, r2 = 0.0;
    for (int d = 0; d < D; ++d) {
      c[d] = x0[d] + s * w[d];
      const double v = c[d] - pi[d];
      r2 += v * v;
    }
    visit_ball<D>(ln, g, c, sqrt(r2) * (1.0 + 1.0e-9) + 1.0e-9 * g.h, take, pi, w);
    reduce();
  };
  // 2-D: the points near i bound the parameter, and B(best.s) holds few
  // points.  (3-D: the first ball below finds as much by itself; with the
  // bound in front the walk's 9 cells of 40k take 2.1 ms instead of 0.8.)
  if (D == 2) {
    visit_ball<D>(ln, g, pi, 2.0 * g.h, take, pi, w);
    reduce();
    if (best.id != ~0u) {
      ball_at(best.s);
      return best;
    }
    // a hull edge has no point at all on its open side
    bool some = false;
    visit_half<D>(ln, g, pi, w, [&](unsigned id, const Pt& p) {
      for (int e = 0; e < nex; ++e)
        if (id == ex[e]) return true;
      double q[3], wp = 0.0, nn = 0.0;
      load(p, q);
      for (int d = 0; d < D; ++d) {
        const double v = q[d] - pi[d];
        wp += w[d] * v;
        nn += v * v;
      }
      some = wp > 0.0 && !(wp * wp <= 1.0e-18 * nn);
      return !some;
    });
    if (!ln.any(some)) return best;
  }
  // balls of growing s (doubling in 3-D): in 3-D from the distance from x0 to i (the radius of
  // the empty ball that the search starts from), at least a twentieth of a
  // bin, in 2-D, with no point near i on the open side, from half a bin
  double span2 = 0.0;
  for (int d = 0; d < D; ++d) { const double e = (double)g.dims[d] * g.h; span2 += e * e; }
  const double span = sqrt(span2);
  for (double s = D == 2 ? 0.5 * g.h : dmax(sqrt(pow0), 0.05 * g.h); s < 4.0 * span;
       s *= D == 2 ? 4.0 : 2.0) {
    ball_at(s);
    if (best.id != ~0u) {
      if (best.s > s) ball_at(best.s);
      return best;
    }
  }
  visit_half<D>(ln, g, pi, w, take);
  reduce();
  return best;
}

// i's nearest other cell at a non-zero distance (ties by index).
template <int D, class W>
TECS_DL_HD unsigned nearest(const W& ln, const Grid& g, const double* pi, unsigned self) {
  double bd = kInf;
  unsigned bid = ~0u;
  int bc[3];
  bin_of<D>(g, pi, bc);
  const int kmax = shells_to_cover<D>(g, bc);
  for (int k = 0; k <= kmax; ++k) {
    visit_shell<D>(ln, g, bc, k, [&](unsigned id, const Pt& p) {
      if (id == self) return true;
      double q[3];
      load(p, q);
      double d2 = 0.0;
      for (int d = 0; d < D; ++d) { const double v = q[d] - pi[d]; d2 += v * v; }
      if (d2 > 0.0 && (d2 < bd || (d2 == bd && id < bid))) { bd = d2; bid = id; }
      return true;
    });
    lane_min(ln, bd, bid);
    if (bid != ~0u && ((double)k - 1.0e-3) * g.h >= sqrt(bd)) break;
  }
  return bid;
}

struct Tet {
  unsigned v[3];  // the simplex's other points, ascending (2-D: v[2] unused)
  int sph;
  unsigned done;  // bit f: the face opposite v[f] has been crossed
};

struct Sph {
  double c[3];
  double R;    // squared radius
  double tol;  // half-width of the near shell, in units of |p - c|^2 - R
};

struct Star {
  Tet t[kMaxTet];
  Sph s[kMaxSph];
  int nt, ns;
  unsigned err;
  unsigned open_end[2];  // 2-D: the neighbours at which the walk left the grid (i on the hull)
  int n_open;
};

struct JK {
  unsigned j, k;
};

// One cell's working state: the star, the accepted (j, k), one circle's
// candidate points.
struct Scratch {
  Star st;
  JK pairs[kMaxPairs];
  unsigned near[kMaxNear];
  double dev[kMaxNear];
  // 2-D: points around the cell, tested first against every triangle's circle
  Pt kill[kMaxKill];
  unsigned kill_id[kMaxKill];
  int n_kill;
};

// Rounding of the reference's float circumcentre for a simplex of this shape
// and coordinate size, as a tolerance on |p - c|^2 - R, with a safety factor.
template <int D>
TECS_DL_HD double shell_tol(const double* pi, const double (*e)[3], double R) {
  double L = 0.0, hm = 0.0;
  for (int d = 0; d < D; ++d) L = dmax(L, fabs(pi[d]));
  for (int q = 0; q < D; ++q) {
    double n2 = 0.0;
    for (int d = 0; d < D; ++d) { n2 += e[q][d] * e[q][d]; L = dmax(L, fabs(pi[d] + e[q][d])); }
    hm = dmax(hm, sqrt(n2));
  }
  double det;
  if (D == 2) det = e[0][0] * e[1][1] - e[0][1] * e[1][0];
  else det = e[0][0] * (e[1][1] * e[2][2] - e[1][2] * e[2][1]) - e[0][1] * (e[1][0] * e[2][2] - e[1][2] * e[2][0]) +
             e[0][2] * (e[1][0] * e[2][1] - e[1][1] * e[2][0]);
  const double den = dmax(2.0 * fabs(det), 1.0e-300);
  double hp = 1.0;
  for (int q = 0; q < D - 1; ++q) hp *= hm;
  // Centre error (u = eps/2, the unit roundoff): the |x|^2 terms carry about
  // 3 u L^2 each, times cofactors of size h^(D-1), summed over D + 1 terms
  // with as many roundings of partial sums of size L^2 h^(D-1); the
  // determinant's own relative error (about 6 u L h^(D-1) / den) moves a
  // centre of size L by as much again: about 21 u L^2 h^(D-1) / den in all,
  // taken here with a factor 2 to spare.
  const double u = 0.5 * kEps;
  const double dc = 48.0 * u * (L * L + hm * hm) * hp / den + 8.0 * u * L;
  // |p - c|^2 - R moves by 2 r dc + dc^2 with the centre; the distance
  // test's own roundings add a few u (R + L r); a factor 4 over both
  const double r = sqrt(R);
  return 4.0 * (2.0 * r * dc + dc * dc) + 32.0 * u * (R + L * r);
}

template <int D, class W>
TECS_DL_HD int find_sphere(const W& w, Star& st, const double* c, double R) {
  const double rr = sqrt(R);
  return find_first(w, st.ns, [&](int q) {
    double d2 = 0.0;
    for (int d = 0; d < D; ++d) { const double v = st.s[q].c[d] - c[d]; d2 += v * v; }
    const double lim = 1.0e-9 * (rr + sqrt(st.s[q].R)) + 1.0e-200;
    return d2 <= lim * lim;
  });
}

// Adds the simplex (i, a, b[, d]) with circumcentre c; returns its index.
// Every lane computes the same values from the same snapshot; the leader
// writes them.
template <int D, class W>
TECS_DL_HD int add_simplex(const W& ln, const Grid& g, Star& st, const double* pi, unsigned a, unsigned b,
                           unsigned d3, const double* c) {
  unsigned v[3] = {a, b, D == 3 ? d3 : ~0u};
  // ascending (three elements)
  for (int x = 0; x < 2; ++x)
    for (int y = 0; y < 2 - x; ++y)
      if (v[y] > v[y + 1]) { const unsigned t = v[y]; v[y] = v[y + 1]; v[y + 1] = t; }
  const int nt = st.nt, ns = st.ns;
  const int known = find_first(ln, nt, [&](int q) {
    return st.t[q].v[0] == v[0] && st.t[q].v[1] == v[1] && st.t[q].v[2] == v[2];
  });
  if (known >= 0) return known;
  double R = 0.0;
  for (int d = 0; d < D; ++d) { const double u = c[d] - pi[d]; R += u * u; }
  // 3-D counts come from the tetrahedra; their centres only start the next
  // searches, so each keeps its own (no merging, no tolerance)
  double tol = 0.0;
  int sp = -1;
  if (D == 2) {
    double e[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}};
    for (int q = 0; q < D; ++q) {
      double p[3];
      load(g.P[v[q]], p);
      for (int d = 0; d < D; ++d) e[q][d] = p[d] - pi[d];
    }
    tol = shell_tol<D>(pi, e, R);
    sp = find_sphere<D>(ln, st, c, R);
  }
  const bool fresh = sp < 0;
  const bool full = nt >= kMaxTet || (fresh && ns >= kMaxSph);
  const double old_tol = fresh ? 0.0 : st.s[sp].tol;
  ln.sync();  // every lane has read what the leader writes next
  if (ln.leader()) {
    if (full) {
      st.err |= kErrStar;
    } else {
      const int spw = fresh ? ns : sp;
      if (fresh) {
        for (int d = 0; d < 3; ++d) st.s[spw].c[d] = d < D ? c[d] : 0.0;
        st.s[spw].R = R;
        st.s[spw].tol = tol;
        st.ns = ns + 1;
      } else if (tol > old_tol) {
        st.s[spw].tol = tol;
      }
      st.t[nt].v[0] = v[0];
      st.t[nt].v[1] = v[1];
      st.t[nt].v[2] = v[2];
      st.t[nt].sph = spw;
      st.t[nt].done = 0u;
      st.nt = nt + 1;
    }
  }
  ln.sync();
  return full ? -1 : nt;
}

template <class W>
TECS_DL_HD void mark_face(const W& ln, Star& st, int q, unsigned opposite) {
  if (q < 0) return;
  unsigned bits = st.t[q].done;
  for (int f = 0; f < 3; ++f)
    if (st.t[q].v[f] == opposite) bits |= 1u << f;
  ln.sync();
  if (ln.leader()) st.t[q].done = bits;
  ln.sync();
}

template <class W>
TECS_DL_HD void add_open_end(const W& ln, Star& st, unsigned e) {
  const int k = st.n_open;
  ln.sync();
  if (ln.leader() && k < 2) {
    st.open_end[k] = e;
    st.n_open = k + 1;
  }
  ln.sync();
}

TECS_DL_HD void normalize3(double* v, int D) {
  double n = 0.0;
  for (int d = 0; d < D; ++d) n += v[d] * v[d];
  n = sqrt(n);
  if (n > 0.0)
    for (int d = 0; d < D; ++d) v[d] /= n;
}

TECS_DL_HD void cross3(const double* a, const double* b, double* c) {
  c[0] = a[1] * b[2] - a[2] * b[1];
  c[1] = a[2] * b[0] - a[0] * b[2];
  c[2] = a[0] * b[1] - a[1] * b[0];
}

// 2-D: walk around i's Voronoi polygon from the edge of its nearest
// neighbour a: from the midpoint of (i, a) to the vertex on one side, then
// from vertex to vertex, each time across the edge of the newest neighbour,
// until the walk is back at a (closed) or leaves the grid (i on the hull);
// then the same from the other side.
template <class W>
TECS_DL_HD void star2(const W& ln, const Grid& g, unsigned i, Star& st) {
  double pi[3];
  load(g.P[i], pi);
  const unsigned a = nearest<2>(ln, g, pi, i);
  if (a == ~0u) return;
  double pa[3];
  load(g.P[a], pa);
  const double x0[3] = {(pi[0] + pa[0]) * 0.5, (pi[1] + pa[1]) * 0.5, 0.0};
  double u[3] = {-(pa[1] - pi[1]), pa[0] - pi[0], 0.0};
  normalize3(u, 2);
  for (int side = 0; side < 2; ++side) {
    const double w[3] = {side ? -u[0] : u[0], side ? -u[1] : u[1], 0.0};
    const unsigned ex[2] = {i, a};
    const Hit h = shoot<2>(ln, g, x0, w, pi, ex, 2);
    if (h.id == ~0u) {
      add_open_end(ln, st, a);  // (i, a) is a hull edge
      continue;
    }
    const double c[3] = {x0[0] + h.s * w[0], x0[1] + h.s * w[1], 0.0};
    const int nt0 = st.nt;
    int q = add_simplex<2>(ln, g, st, pi, a, h.id, ~0u, c);
    if (q < 0 || (side == 1 && st.nt == nt0)) return;
    unsigned prev = a, cur = h.id;
    double v[3] = {c[0], c[1], 0.0};
    bool closed = false;
    for (int guard = 0; guard < kMaxTet && !closed; ++guard) {
      double pc[3], pp[3];
      load(g.P[cur], pc);
      load(g.P[prev], pp);
      double n[3] = {-(pc[1] - pi[1]), pc[0] - pi[0], 0.0};
      if (n[0] * (pp[0] - pi[0]) + n[1] * (pp[1] - pi[1]) > 0.0) { n[0] = -n[0]; n[1] = -n[1]; }
      normalize3(n, 2);
      const unsigned ex2[3] = {i, cur, prev};
      const Hit h2 = shoot<2>(ln, g, v, n, pi, ex2, 3);
      if (h2.id == ~0u) {  // open: (i, cur) is a hull edge
        add_open_end(ln, st, cur);
        break;
      }
      const double c2[3] = {v[0] + h2.s * n[0], v[1] + h2.s * n[1], 0.0};
      const int cur_sph = st.t[q].sph, ns0 = st.ns, nt1 = st.nt;
      const int q2 = add_simplex<2>(ln, g, st, pi, cur, h2.id, ~0u, c2);
      if (q2 < 0) return;
      // back at a, at a triangle met before, or at an earlier vertex: closed
      closed = h2.id == a || st.nt == nt1 || (st.ns == ns0 && st.t[q2].sph != cur_sph);
      prev = cur;
      cur = h2.id;
      v[0] = c2[0];
      v[1] = c2[1];
      q = q2;
    }
    if (closed) return;
  }
}

// 3-D: breadth-first over i's Voronoi vertices, crossing each face of each
// star tetrahedron that contains i once.
template <class W>
TECS_DL_HD void star3(const W& ln, const Grid& g, unsigned i, Star& st) {
  double pi[3];
  load(g.P[i], pi);
  const unsigned a = nearest<3>(ln, g, pi, i);
  if (a == ~0u) return;
  double pa[3];
  load(g.P[a], pa);
  const double ea[3] = {pa[0] - pi[0], pa[1] - pi[1], pa[2] - pi[2]};
  double x0[3] = {(pi[0] + pa[0]) * 0.5, (pi[1] + pa[1]) * 0.5, (pi[2] + pa[2]) * 0.5};
  // a direction across the bisector plane of (i, a)
  int ax = 0;
  if (fabs(ea[1]) < fabs(ea[ax])) ax = 1;
  if (fabs(ea[2]) < fabs(ea[ax])) ax = 2;
  double unit[3] = {0, 0, 0};
  unit[ax] = 1.0;
  double u[3];
  cross3(ea, unit, u);
  normalize3(u, 3);
  const unsigned ex[2] = {i, a};
  Hit h = shoot<3>(ln, g, x0, u, pi, ex, 2);
  if (h.id == ~0u) {
    for (int d = 0; d < 3; ++d) u[d] = -u[d];
    h = shoot<3>(ln, g, x0, u, pi, ex, 2);
  }
  if (h.id == ~0u) return;  // every other point on the line through i and a
  const unsigned b = h.id;
  const double x1[3] = {x0[0] + h.s * u[0], x0[1] + h.s * u[1], x0[2] + h.s * u[2]};
  double pb[3];
  load(g.P[b], pb);
  const double eb[3] = {pb[0] - pi[0], pb[1] - pi[1], pb[2] - pi[2]};
  double n[3];
  cross3(ea, eb, n);
  normalize3(n, 3);
  const unsigned ex3[3] = {i, a, b};
  int q0[2] = {-1, -1};
  unsigned apex[2] = {~0u, ~0u};
  for (int side = 0; side < 2; ++side) {
    double w[3] = {side ? -n[0] : n[0], side ? -n[1] : n[1], side ? -n[2] : n[2]};
    const Hit hd = shoot<3>(ln, g, x1, w, pi, ex3, 3);
    if (hd.id == ~0u) continue;
    const double c[3] = {x1[0] + hd.s * w[0], x1[1] + hd.s * w[1], x1[2] + hd.s * w[2]};
    q0[side] = add_simplex<3>(ln, g, st, pi, a, b, hd.id, c);
    apex[side] = hd.id;
  }
  // the face (i, a, b) between the two first tetrahedra is crossed
  mark_face(ln, st, q0[0], apex[0]);
  mark_face(ln, st, q0[1], apex[1]);
  for (int q = 0; q < st.nt; ++q) {
    for (int f = 0; f < 3; ++f) {
      const unsigned done = st.t[q].done;
      if (done & (1u << f)) continue;
      ln.sync();
      if (ln.leader()) st.t[q].done = done | (1u << f);
      ln.sync();
      const unsigned O = st.t[q].v[f], A = st.t[q].v[(f + 1) % 3], B = st.t[q].v[(f + 2) % 3];
      double pA[3], pB[3], pO[3];
      load(g.P[A], pA);
      load(g.P[B], pB);
      load(g.P[O], pO);
      const double eA[3] = {pA[0] - pi[0], pA[1] - pi[1], pA[2] - pi[2]};
      const double eB[3] = {pB[0] - pi[0], pB[1] - pi[1], pB[2] - pi[2]};
      double w[3];
      cross3(eA, eB, w);
      if (w[0] * (pO[0] - pi[0]) + w[1] * (pO[1] - pi[1]) + w[2] * (pO[2] - pi[2]) > 0.0)
        for (int d = 0; d < 3; ++d) w[d] = -w[d];
      normalize3(w, 3);
      const Sph& S = st.s[st.t[q].sph];
      const unsigned exf[4] = {i, A, B, O};
      const Hit hf = shoot<3>(ln, g, S.c, w, pi, exf, 4);
      if (hf.id == ~0u) continue;  // open face: i is on the hull
      const double c[3] = {S.c[0] + hf.s * w[0], S.c[1] + hf.s * w[1], S.c[2] + hf.s * w[2]};
      const int q2 = add_simplex<3>(ln, g, st, pi, A, B, hf.id, c);
      if (q2 < 0) return;
      mark_face(ln, st, q2, hf.id);
    }
  }
}

// ---------------------------------------------------------------------------
// One cell: its partners and how often the reference applies each pair.
// out[0..return) = (j, reps), ascending j (written by the lanes together: one
// copy per warp); *err gets the error bits.

template <int D, class W>
TECS_DL_HD unsigned cell_mult(const W& ln, const Grid& g, unsigned i, unsigned* out_j, unsigned* out_r, unsigned cap,
                              unsigned* err, Scratch& sc) {
  Star& st = sc.st;
  JK* pairs = sc.pairs;
  unsigned* near = sc.near;
  double* dev = sc.dev;
  ln.sync();
  if (ln.leader()) {
    st.nt = 0;
    st.ns = 0;
    st.err = 0u;
    st.n_open = 0;
    sc.n_kill = 0;
  }
  ln.sync();
  if (D == 2 && g.n > kKillFrom) {
    // the points around i, as many as fit
    double pi[3];
    load(g.P[i], pi);
    int nk = 0;
    bool has = false;
    Pt pt{0.0f, 0.0f, 0.0f, 0.0f};
    unsigned id = 0u;
    visit_ball<2>(ln, g, pi, 2.0 * g.h, [&](unsigned q, const Pt& p) {
      has = q != i;
      pt = p;
      id = q;
      return true;
    }, nullptr, nullptr, [&]() {
      const unsigned m = ln.ballot(has);
      unsigned before = 0;
      for (unsigned b = m & ((1u << ln.lane()) - 1u); b; b &= b - 1u) ++before;
      const int at = nk + (int)before;
      if (has && at < kMaxKill) {
        sc.kill[at] = pt;
        sc.kill_id[at] = id;
      }
      for (unsigned b = m; b; b &= b - 1u) ++nk;
      has = false;
    });
    ln.sync();
    if (ln.leader()) sc.n_kill = imin(nk, kMaxKill);
    ln.sync();
  }
  if (D == 2) star2(ln, g, i, st);
  else star3(ln, g, i, st);
  unsigned e = st.err;
  int np = 0;
  const Pt Pi = g.P[i];
  auto record = [&](unsigned j, unsigned k) {
    if (find_first(ln, np, [&](int p) { return pairs[p].j == j && pairs[p].k == k; }) >= 0) return;
    if (np >= kMaxPairs) { e |= kErrPairs; return; }
    ln.sync();
    if (ln.leader()) pairs[np] = JK{j, k};
    ln.sync();
    ++np;
  };
  if (D == 3) {
    // every star tetrahedron (i, a, b, c): j one of them, k the lesser other
    for (int q = 0; q < st.nt; ++q) {
      const unsigned* v = st.t[q].v;
      for (int f = 0; f < 3; ++f) {
        const unsigned j = v[f], k = v[f == 0 ? 1 : 0];
        if (in_cutoff<3>(g, Pi, g.P[j])) record(j, k);
      }
    }
  } else {
    // the star circles, then one group per hull edge at i
    for (int q = 0; q < st.ns + st.n_open; ++q) {
      // the circle's own triangle points first (deviation -1: never dropped),
      // then every point on or near it, or inside; when the array is full
      // the point farthest from the circle gives way
      int nn = 0;
      double far = kInf;  // of a full array: the largest deviation, and its place
      int far_at = 0;
      auto put = [&](unsigned id, double f) {
        // (a warp's lanes leave out what a full array would refuse: a wide
        // tolerance takes in hundreds of points)
        if (W::width > 1 && nn >= kMaxNear && !(f < far)) return;
        if (find_first(ln, nn, [&](int x) { return near[x] == id; }) >= 0) return;
        int at = nn;
        if (nn >= kMaxNear) {
          e |= kErrNear;
          at = far_at;
          if (!(f < far)) return;
        }
        ln.sync();
        if (ln.leader()) { near[at] = id; dev[at] = f; }
        ln.sync();
        if (at == nn) ++nn;
        if (nn >= kMaxNear) {
          // the farthest, the first of equals
          if (W::width > 1 && q < st.ns) {
            // A circle's deviations are floats, or -1: as whole numbers in
            // their order, so two warp reductions take the place of five
            // rounds of exchanged doubles.  The hull cells' sets, a few
            // hundred points put one by one, are the walk's longest: 0.90 to
            // 0.78 ms a pass over a disk of 30 000, mean of twelve passes.
            unsigned key = 0u, who = ~0u;
            for (int x = (int)ln.lane(); x < nn; x += (int)W::width) {
              const unsigned k = dev[x] < 0.0 ? 0u : float_order((float)dev[x]) + 1u;
              if (who == ~0u || k > key) { key = k; who = (unsigned)x; }
            }
            const unsigned top = ln.most(key);
            far_at = (int)ln.least(key == top ? who : ~0u);
            far = dev[far_at];
          } else {
            double key = kInf;
            unsigned who = ~0u;
            for (int x = (int)ln.lane(); x < nn; x += (int)W::width)
              if (-dev[x] < key) { key = -dev[x]; who = (unsigned)x; }
            lane_min(ln, key, who);
            far = -key;
            far_at = (int)who;
          }
        }
      };
      // a lane's candidate of the current round, put by every lane in lane order
      bool has = false;
      unsigned cid = 0u;
      double cdev = 0.0;
      auto merge = [&]() {
        if (W::width > 1 && nn >= kMaxNear && !(cdev < far)) has = false;
        unsigned m = ln.ballot(has);
        while (m) {
          const int src = low_bit(m);
          m &= m - 1u;
          put(ln.bcast(cid, src), ln.bcast(cdev, src));
        }
        has = false;
      };
      if (q < st.ns) {
        const Sph S = st.s[q];
        double pi2[3], hm = 0.0;
        load(Pi, pi2);
        for (int t = 0; t < st.nt; ++t)
          if (st.t[t].sph == q)
            for (int v = 0; v < 2; ++v) {
              put(st.t[t].v[v], -1.0);
              double pv[3];
              load(g.P[st.t[t].v[v]], pv);
              hm = dmax(hm, sqrt((pv[0] - pi2[0]) * (pv[0] - pi2[0]) + (pv[1] - pi2[1]) * (pv[1] - pi2[1])));
            }
        // |p - c|^2 - R <= tol, in float with a margin above its rounding:
        // the set may only grow (every member's triangles are tested by the
        // reference's float test), so no double work is needed per point
        const float cx = (float)S.c[0], cy = (float)S.c[1], Rf = (float)S.R, tf = (float)S.tol;
        const float reach = sqrtf(fmaxf(Rf + tf, 0.0f));
        const float slack = 1.0e-5f * (Rf + tf + 2.0f * reach * (fabsf(cx) + fabsf(cy) + reach)) + 1.0e-30f;
        auto near_test = [&](unsigned id, const Pt& p) {
          if (id == i) return true;
          const float u0 = p.x - cx, u1 = p.y - cy;
          const float f = u0 * u0 + u1 * u1 - Rf;
          if (f <= tf + slack) { has = true; cid = id; cdev = fabs((double)f); }
          return true;
        };
        // An alternative triangle to the circle's own is local: its points
        // lie within a few of the triangle's edges of i.  A circle much
        // larger than its triangle (a hull triangle, bulging out of the
        // hull) meets the other cells only along the hull, where a wide
        // float tolerance would take in cells far from i whose triangles
        // with i enclose the hull's interior; those are searched near i.
        const double rad = sqrt(S.R + S.tol) * (1.0 + 1.0e-9) + 1.0e-9 * g.h;
        const double local = 4.0 * hm + 4.0 * g.h;
        if (local < rad) visit_ball<2>(ln, g, pi2, local, near_test, nullptr, nullptr, merge);
        else visit_ball<2>(ln, g, S.c, rad, near_test, nullptr, nullptr, merge);
      } else {
        // A hull edge (i, e): three points that are collinear in exact
        // arithmetic can still give the reference a determinant above
        // FLT_EPSILON (it rounds products of size L h, L the coordinates'
        // size), and the huge circle of such a triangle holds no point when
        // it bulges out of the hull, along a supporting line of i.  So the
        // points near the line of each hull edge form one more group.
        const unsigned e_id = st.open_end[q - st.ns];
        double pi2[3], pe[3];
        load(Pi, pi2);
        load(g.P[e_id], pe);
        double nrm[3] = {-(pe[1] - pi2[1]), pe[0] - pi2[0], 0.0};
        normalize3(nrm, 2);
        const double L = dmax(dmax(fabs(g.lo[0]), fabs(g.lo[0] + g.dims[0] * g.h)),
                              dmax(fabs(g.lo[1]), fabs(g.lo[1] + g.dims[1] * g.h)));
        const double span = (double)(g.dims[0] + g.dims[1]) * g.h;
        const double del = 64.0 * 0.5 * kEps * L * (1.0 + span) + (double)FLT_EPSILON;
        put(e_id, -1.0);
        visit_band(ln, g, pi2, nrm, del, [&](unsigned id, const Pt& p) {
          if (id == i) return true;
          const double f = fabs(((double)p.x - pi2[0]) * nrm[0] + ((double)p.y - pi2[1]) * nrm[1]);
          if (f <= del) { has = true; cid = id; cdev = f; }
          return true;
        }, merge);
      }
      // the reference's test on every choice of j (in cutoff) and k among them
      for (int a = 0; a < nn; ++a) {
        const unsigned j = near[a];
        if (!in_cutoff<2>(g, Pi, g.P[j])) continue;
        // a warp's lanes first put the k to the points around the cell, 32 at a
        // time: few triangles are left for the test over the grid
        unsigned left = 0u;
        for (int b = 0; b < nn; ++b) {
          if (W::width > 1) {
            const int b0 = b & ~(int)(W::width - 1);
            if (b == b0) {
              const int mine = b0 + (int)ln.lane();
              left = ln.ballot(mine < nn && near[mine] != j && tri_near(g, i, j, near[mine], sc));
            }
            if (!(left >> (b - b0) & 1u)) continue;
          }
          const unsigned k = near[b];
          if (k == j) continue;
          const bool have = find_first(ln, np, [&](int p) { return pairs[p].j == j && pairs[p].k == k; }) >= 0;
          if (!have && tri_pass(ln, g, i, j, k, sc)) record(j, k);
        }
      }
    }
  }
  // (j, number of distinct k), ascending j: the pairs are distinct; the first
  // of each j is marked, and its place is the number of marked lesser j
  constexpr unsigned kFirst = 0x80000000u;  // slots are below 2^30
  ln.sync();
  unsigned len = 0;
  for (int x0 = 0; x0 < np; x0 += (int)W::width) {
    const int x = x0 + (int)ln.lane();
    bool first = x < np;
    for (int y = 0; y < x && first; ++y) first = pairs[y].j != pairs[x].j;
    for (unsigned m = ln.ballot(first); m; m &= m - 1u) ++len;
    ln.sync();
    if (first) pairs[x].k |= kFirst;
  }
  ln.sync();
  for (int x = (int)ln.lane(); x < np; x += (int)W::width) {
    if (!(pairs[x].k & kFirst)) continue;
    const unsigned j = pairs[x].j;
    unsigned at = 0, reps = 0;
    for (int y = 0; y < np; ++y) {
      reps += pairs[y].j == j ? 1u : 0u;
      at += ((pairs[y].k & kFirst) && pairs[y].j < j) ? 1u : 0u;
    }
    if (at < cap) {
      out_j[at] = j;
      out_r[at] = reps;
    }
  }
  if (len > cap) {
    e |= kErrList;
    len = cap;
  }
  ln.sync();
  *err = e;
  return len;
}

}  // namespace dl
}  // namespace tecs
