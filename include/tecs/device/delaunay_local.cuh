// delaunay_local.cuh -- the Delaunay finder's fast path: cells whose star lies
// within a gathered neighbourhood, one warp per cell, without FP64 searches.
//
// delaunay_star.cuh walks a cell's Voronoi cell in double, one search of the
// grid after the other; FP64 is scarce on this part (about two lanes an SM and
// clock) and the searches depend on each other.  Here a warp gathers the
// points of a box of bins around the cell once (relative to it, in shared
// memory), finds the cell's partners from them in float with all lanes, and
// keeps the result only where it is certain; any doubt -- a point nearer to a
// circle or sphere than the rounding, a sphere that reaches out of the gathered
// ball, a hull face, a duplicate -- hands the cell on: to a second search (2-D:
// over a larger box; 3-D: that looks up what lies beyond the ball), then to the
// walk in double.
//
// 3-D.  For an in-cutoff j the Voronoi face of (i, j) is a polygon in their
// bisector plane.  Each third point k bounds it by a line; a lane takes a k
// and cuts its line by every other point, which leaves an interval if (i, j,
// k) is a triangle of the triangulation, with the fourth points of its two
// tetrahedra at the ends.  Each tetrahedron is met from both of its third
// points (checked), so the tetrahedra around (i, j) form a closed ring, and
// each one's circumcentre is solved in double and every gathered point tested
// against its sphere with a margin above the float rounding: empty spheres are
// the Delaunay tetrahedra, whichever way they were found.
//
// 2-D.  The reference's float test decides (delaunay_star.cuh, 3): every
// triangle (i, j, k) of an in-cutoff j and a gathered k is put to it, the lanes
// taking the k.  The cell's own triangles are found in float as well (each
// lane takes a neighbour and the nearest parameter on either side), to make
// sure that the circles, with the tolerance inside which delaunay_star.cuh looks for
// further third points, lie within the gathered disk.
//
// The margins hold in any unit of length: they are shares of the cells' own
// distances, each at least twice its rounding bound (tests/cpp/
// delaunay_margins_host.cpp compares them with more bits).  A missed face cannot
// pass: where some lines bound it, its tetrahedra are met from one third point
// only, and where none does, every line has to be certain.
//
// What bounds it: instruction issue, then the latency of the few cells left to
// the walk.  40k cells in space, one pass: 54 ms (the walk for every cell) ->
// 1.7-2.1 (1.0 the first search, 0.6 the second over 7 % of the cells, 0-0.4 the
// walk of a few cells); 30k in the plane, two passes: 27-42 -> 2.7-3.0 ms.
#pragma once

#include "delaunay_star.cuh"

namespace tecs {
namespace dl {

constexpr int kLocalThreads = 128;
constexpr unsigned kNoEnd = 0xffffu;
// A point's power (|v|^2 - 2 x.v) / 2 in a sphere about x through the cell has
// to exceed kPowerV |v|^2 / 2 + kPowerX |x|^2.  Its float error (u = 6e-8 for
// each product and sum, for v and for x) is at most 6 u (|x| |v| + |v|^2 / 2)
// <= 1.8e-7 |x|^2 + 3.6e-7 |v|^2: the margin is five times that.
constexpr float kPowerV = 4.0e-6f, kPowerX = 1.0e-6f;

// The points within rho of cell i -- REACH / 100 bins, less where the box of BOX
// bins to every side ends before that or they are too many: position relative to i and half the squared distance
// (3-D), or absolute and relative position (2-D).  Returns the number of
// points, LOC + 1 or more if they do not fit.
template <int D, int BOX, int REACH, int LOC>
__device__ __forceinline__ unsigned gather_local(const Warp& w, const Grid& g, unsigned i, const Pt& pi, float4* p,
                                                 unsigned* id, float& rho) {
  const GridF& gf = g.f;
  const float c[3] = {pi.x, pi.y, pi.z};
  int b0[3] = {0, 0, 0}, b1[3] = {0, 0, 0};
  rho = 1.0e9f;  // the box holds the whole grid
#pragma unroll
  for (int d = 0; d < D; ++d) {
    const int b = bin1f(gf, d, c[d]);
    b0[d] = imax(b - BOX, 0);
    b1[d] = imin(b + BOX, gf.dims[d] - 1);
    if (b0[d] > 0) rho = fminf(rho, c[d] - (gf.lo[d] + (float)b0[d] * gf.h) - 2.0f * gf.m);
    if (b1[d] < gf.dims[d] - 1) rho = fminf(rho, gf.lo[d] + (float)(b1[d] + 1) * gf.h - c[d] - 2.0f * gf.m);
  }
  rho = fminf(rho, REACH * 0.01f * gf.h);
  if (!(rho > 0.0f)) return (unsigned)LOC + 1u;
  const int ny = b1[1] - b0[1] + 1, nz = b1[2] - b0[2] + 1;
  unsigned n = 0u;
  // a ball that holds too many points shrinks (twice at most)
  for (int turn = 0; turn < 3; ++turn) {
    const float rho2 = rho * rho;
    n = 0u;
    bool has = false;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    unsigned vid = 0u;
    visit_rows(w, g, ny * nz, [&](int r, unsigned& lo, unsigned& hi) {
      row_entries(g, b0[0], b1[0], b0[1] + r % ny, b0[2] + r / ny, lo, hi);
    }, [&](unsigned e, const Pt& q) {
      const float x = q.x - pi.x, y = q.y - pi.y, z = D >= 3 ? q.z - pi.z : 0.0f;
      float d2 = x * x + y * y;
      if (D >= 3) d2 = d2 + z * z;
      has = e != i && d2 <= rho2;
      v = D >= 3 ? make_float4(x, y, z, 0.5f * d2) : make_float4(q.x, q.y, x, y);
      vid = e;
      return true;
    }, [&]() {
      const unsigned m = w.ballot(has);
      const unsigned at = n + (unsigned)__popc(m & ((1u << w.lane()) - 1u));
      if (has && at < (unsigned)LOC) {
        p[at] = v;
        id[at] = vid;
      }
      n += (unsigned)__popc(m);
      has = false;
    });
    if (n <= (unsigned)LOC) break;
    const float f = 0.85f * (float)LOC / (float)n;
    rho *= D >= 3 ? cbrtf(f) : sqrtf(f);
  }
  __syncwarp();
  return n;
}

// One warp's working memory.
template <int LOC>
struct LocalScratch {
  float4 p[LOC];
  unsigned id[LOC];
  unsigned short list[LOC];     // third points whose line may bound the face
  unsigned long long done[64];  // 3-D: spheres and open faces that verify_far found certain
  ushort4 tet[160];             // 3-D: tetrahedra to verify (indices into p); z = kNoEnd: an open face, w its side
  float4 cen[160];              // their centres (relative) and squared radii
  unsigned rj[64], rr[64];      // partners and their counts
};

// Partners in ascending j to the cell's row.
template <int LOC>
__device__ __forceinline__ void write_row(const Warp& w, const LocalScratch<LOC>& sc, unsigned m, uint2* row, unsigned* len) {
  __syncwarp();
  for (unsigned e = w.lane(); e < m; e += 32u) {
    const unsigned j = sc.rj[e];
    unsigned rank = 0u;
    for (unsigned k = 0; k < m; ++k) rank += sc.rj[k] < j ? 1u : 0u;
    row[rank] = make_uint2(j, sc.rr[e]);
  }
  if (w.leader()) *len = m;
}

// The gathered points put in order of their distance, by eighths of rho^2: a
// search may stop where every later point is too far (the first search of 40k
// cells 1.4 -> 0.9 ms).
constexpr int kShells = 8;
template <int LOC>
__device__ __forceinline__ void order_points(const Warp& w, LocalScratch<LOC>& sc, unsigned n, float rho) {
  constexpr int C = (LOC + 31) / 32;
  float4 v[C];
  unsigned id[C], to[C];
  const float inv = (float)kShells / (rho * rho);
  unsigned base = 0u;
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const unsigned k = 32u * c + w.lane();
    v[c] = sc.p[k < n ? k : 0u];
    id[c] = sc.id[k < n ? k : 0u];
    to[c] = 0u;
  }
  for (int s = 0; s < kShells; ++s) {
#pragma unroll
    for (int c = 0; c < C; ++c) {
      const unsigned k = 32u * c + w.lane();
      const bool here = k < n && min((int)(2.0f * v[c].w * inv), kShells - 1) == s;
      const unsigned b = __ballot_sync(0xffffffffu, here);
      if (here) to[c] = base + (unsigned)__popc(b & ((1u << w.lane()) - 1u));
      base += (unsigned)__popc(b);
    }
  }
  __syncwarp();
#pragma unroll
  for (int c = 0; c < C; ++c)
    if (32u * c + w.lane() < n) {
      sc.p[to[c]] = v[c];
      sc.id[to[c]] = id[c];
    }
  __syncwarp();
}

// The circumcentres of the listed tetrahedra, and whether every gathered point
// lies outside their spheres with certainty.
template <int LOC>
__device__ __forceinline__ bool verify_tets(const Warp& w, const Grid& g, unsigned i, LocalScratch<LOC>& sc, unsigned n,
                                            unsigned m, float rho) {
  double pi[3];
  load(g.P[i], pi);
  bool bad = false;
  for (unsigned t0 = 0; t0 < m; t0 += 32u) {
    const unsigned t = t0 + w.lane();
    const ushort4 q = sc.tet[t < m ? t : t0];
    const bool closed = q.z != kNoEnd;
    double xd[3], thin2;
    tet_centre(pi, g.P[sc.id[q.x]], g.P[sc.id[q.y]], g.P[sc.id[closed ? q.z : q.x]], xd, thin2);
    const float x = (float)xd[0], y = (float)xd[1], z = (float)xd[2];
    const float r2 = x * x + y * y + z * z;
    if (t < m) sc.cen[t] = make_float4(x, y, z, r2);
    if (closed && !(r2 < 2.5e11f * rho * rho && thin2 < kThin * kThin)) bad = true;
    const float m0 = kPowerX * r2;
    for (unsigned k = 0; k < n; ++k) {
      const float4 v = sc.p[k];
      const float pw = v.w - (x * v.x + y * v.y + z * v.z);
      if (closed && !(pw > kPowerV * v.w + m0) && k != q.x && k != q.y && k != q.z) {
        // too near for float: once more in double
        if (!sphere_leaves_out(pi, xd, thin2, g.P[sc.id[k]])) bad = true;
      }
    }
    if (__any_sync(0xffffffffu, bad)) return false;
  }
  return true;
}

// Beyond the gathered ball: every cell outside the spheres that reach out of
// it, and none on the open side of the open faces.  0: certain; 1: a cell
// breaks one -- it joins the gathered points; 2: a cell is too near to tell,
// or there is no room.  What was certain in an earlier turn (done, ndone of
// them: the points keep their places) is not looked up again: an empty sphere
// of a surface cell is the costliest look-up, all its cells are read (the second
// search of a 40k ball 1.03 -> 0.82 ms, mean of six sets).
template <int LOC>
__device__ __forceinline__ int verify_far(const Warp& w, const Grid& g, unsigned i, LocalScratch<LOC>& sc, unsigned& n,
                                          unsigned m, float rho, unsigned& ndone) {
  const Pt Pi = g.P[i];
  const double pi[3] = {Pi.x, Pi.y, Pi.z};
  int state = 0;
  for (unsigned t = 0; t < m; ++t) {
    const ushort4 q = sc.tet[t];
    const float4 c = sc.cen[t];
    const bool closed = q.z != kNoEnd;
    if (closed && 4.0f * c.w <= rho * rho * 0.9999f) continue;
    // the same from each of its partners: in one order
    const unsigned q0 = min(q.x, q.y), q1 = max(q.x, q.y);
    const unsigned long long key =
        closed ? (unsigned long long)min(q0, (unsigned)q.z) << 32 | max(q0, min(q1, (unsigned)q.z)) << 16 | max(q1, (unsigned)q.z)
               : (unsigned long long)(q.x < q.y ? q.w : 3 - q.w) << 48 | (unsigned long long)q0 << 16 | q1;
    bool seen = false;
    for (unsigned k = w.lane(); k < ndone; k += 32u) seen = seen || sc.done[k] == key;
    if (__any_sync(0xffffffffu, seen)) continue;
    const unsigned ia = sc.id[q.x], ib = sc.id[q.y], ic = closed ? sc.id[q.z] : i;
    // An open face's normal is formed in double: a float one of a thin face may
    // lean so far that the rows of bins it leaves out hold cells on the open side.
    double nn[3] = {0.0, 0.0, 0.0}, slack = 0.0;
    if (!closed) {
      double a[3], b[3];
      load(g.P[ia], a);
      load(g.P[ib], b);
      for (int d = 0; d < 3; ++d) {
        const double va = a[d] - pi[d], vb = b[d] - pi[d];
        a[d] = q.w == 2 ? vb : va;
        b[d] = q.w == 2 ? va : vb;
      }
      if (!plane_normal(a, b, nn, slack)) return 2;
    }
    const float nx = (float)nn[0], ny = (float)nn[1], nz = (float)nn[2];
    bool hit = false;
    unsigned hid = 0u;
    float deep = 0.0f;
    float4 hv = make_float4(0.f, 0.f, 0.f, 0.f);
    // in float, and where a cell is too near to tell, once more in double
    for (int dbl = 0; dbl < 2; ++dbl) {
      bool doubt = false;
      double xd[3] = {0.0, 0.0, 0.0}, thin2 = 0.0, margin = 0.0;
      if (dbl && closed) {
        tet_centre(pi, g.P[ia], g.P[ib], g.P[ic], xd, thin2);
        margin = sphere_margin(thin2);
      }
      auto test = [&](unsigned e, const Pt& p) {
        if (e == i || e == ia || e == ib || e == ic) return true;
        const float x = p.x - Pi.x, y = p.y - Pi.y, z = p.z - Pi.z;
        const float h = 0.5f * (x * x + y * y + z * z);
        bool out, in;
        float depth;
        if (!dbl) {
          // (of the plane: the rounding of n and of the products, 16 u |v|)
          const float lim = closed ? kPowerV * h + kPowerX * c.w : 1.0e-6f * sqrtf(2.0f * h);
          const float pw = closed ? h - (c.x * x + c.y * y + c.z * z) : -(nx * x + ny * y + nz * z);
          out = pw > lim;
          in = pw < -lim;
          depth = -pw;
        } else {
          const double v[3] = {p.x - pi[0], p.y - pi[1], p.z - pi[2]};
          const double vv = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
          const double* to = closed ? xd : nn;
          const double dt = v[0] * to[0] + v[1] * to[1] + v[2] * to[2];
          const double pw = closed ? 0.5 * vv - dt : -dt;
          const double xx = xd[0] * xd[0] + xd[1] * xd[1] + xd[2] * xd[2];
          const double lim = closed ? margin * (vv + xx) : 1.0e-13 * slack * sqrt(vv);
          out = pw > lim;
          in = pw < -lim;
          depth = (float)-pw;
        }
        if (out) return true;
        deep = depth;
        hit = in;
        doubt = !in;
        hid = e;
        hv = make_float4(x, y, z, h);
        return false;
      };
      if (closed) {
        const double cc[3] = {pi[0] + c.x, pi[1] + c.y, pi[2] + c.z};
        visit_ball<3>(w, g, cc, (double)(sqrtf(c.w) * 1.0001f), test);
      } else {
        visit_half<3>(w, g, pi, nn, test);
      }
      if (!__any_sync(0xffffffffu, doubt)) break;
      if (dbl) return 2;
      hit = false;
    }
    const unsigned b = __ballot_sync(0xffffffffu, hit);
    if (b) {
      // of the cells that break it, the deepest one of the round that found
      // them: fewer turns than with the first lane's (0.82 -> 0.65 ms)
      const unsigned order = hit ? float_order(deep) : 0u;
      const unsigned top = __reduce_max_sync(0xffffffffu, order);
      const bool first = hit && order == top;
      const int src = __ffs(__ballot_sync(0xffffffffu, first)) - 1;
      hid = __shfl_sync(0xffffffffu, hid, src);
      bool known = false;
      for (unsigned k = w.lane(); k < n; k += 32u) known = known || sc.id[k] == hid;
      state = 1;
      if (!__any_sync(0xffffffffu, known)) {
        if (n >= (unsigned)LOC) return 2;
        if ((int)w.lane() == src) {
          sc.p[n] = hv;
          sc.id[n] = hid;
        }
        ++n;
        __syncwarp();
      }
    } else if (ndone < 64u) {
      if (w.leader()) sc.done[ndone] = key;
      ++ndone;
      __syncwarp();
    }
  }
  return state;
}

// Whether two cuts of a line, t < hi by vh and t > lo by vl, cross by more than
// their rounding in float.  Out of line: it is asked of few lines, and its
// registers in the search cost the first level of 40k cells 1.12 ms where this
// takes 1.00.
static __device__ __noinline__ bool cuts_apart(const FaceLine<float> l, float jh, float kh, const float4 vh, float hi,
                                               const float4 vl, float lo) {
  const CutError<float> err(l, jh, kh);
  return (lo - hi) * err.len > err.of(l, vh.x, vh.y, vh.z, vh.w, hi) + err.of(l, vl.x, vl.y, vl.z, vl.w, lo);
}

// FAR: the spheres may reach out of the gathered ball and the cell may lie on
// the hull; what lies beyond is looked up (verify_far), and cells that break a
// sphere join the gathered points, until none does.
template <int BOX, int REACH, int LOC, bool FAR>
__device__ __forceinline__ bool cell_local3(const Warp& w, const Grid& g, unsigned i, LocalScratch<LOC>& sc, uint2* row,
                                            unsigned* len) {
  const unsigned lane = w.lane();
  float rho;
  unsigned n = gather_local<3, BOX, REACH, LOC>(w, g, i, g.P[i], sc.p, sc.id, rho);
  if (n > (unsigned)LOC || n < 4u) return false;
  if (!(rho * rho > g.rc2 * 1.0001f)) return false;
  order_points(w, sc, n, rho);
  const float shell = rho * rho / (float)kShells;
  const float r2max = 0.25f * rho * rho;
  unsigned ndone = 0u;
  const unsigned near_n = n;  // the in-cutoff cells are among the gathered ball's
  for (int turn = 0; turn < 32; ++turn) {
  unsigned rows = 0u, tets = 0u;
  bool big = false;  // a sphere reaches out of the ball
  for (unsigned t0 = 0; t0 < near_n; t0 += 32u) {
    bool in = false;
    if (t0 + lane < near_n) {
      const float4 v = sc.p[t0 + lane];
      float d2 = v.x * v.x + v.y * v.y;
      d2 = d2 + v.z * v.z;
      in = d2 < g.rc2;
    }
    for (unsigned bits = __ballot_sync(0xffffffffu, in); bits; bits &= bits - 1u) {
      const unsigned J = t0 + (unsigned)__ffs(bits) - 1u;
      const float4 vj = sc.p[J];
      unsigned reps = 0u, members = 0u, mix = 0u;
      // First the k whose triangle (i, j, k) has a circumradius below the
      // largest sphere's, their lines cut off there.  Where these give no
      // face, it is empty or lies farther out: then every gathered k, with its
      // whole line; no interval means that the gathered points alone leave
      // no face.
      for (int wide = FAR ? 1 : 0; wide < 2 && members == 0u; ++wide) {
        unsigned nk = 0u;
        __syncwarp();
        for (unsigned k0 = 0; k0 < n; k0 += 32u) {
          const unsigned k = k0 + lane;
          bool keep = false;
          if (k < n && k != J) {
            const float4 v = sc.p[k];
            const float dt = vj.x * v.x + vj.y * v.y + vj.z * v.z;
            const float jj = 2.0f * vj.w, kk = 2.0f * v.w;
            const float w2 = jj * kk - dt * dt;
            keep = wide || jj * kk * (jj + kk - 2.0f * dt) < 4.04f * r2max * w2 + 1.0e-5f * jj * kk * (jj + kk);
          }
          const unsigned b = __ballot_sync(0xffffffffu, keep);
          if (keep) sc.list[nk + (unsigned)__popc(b & ((1u << lane) - 1u))] = (unsigned short)k;
          nk += (unsigned)__popc(b);
        }
        __syncwarp();
        bool doubt = false;  // a line that may bound the face
        for (unsigned k0 = 0; k0 < nk; k0 += 32u) {
          const bool act = k0 + lane < nk;
          const unsigned k = act ? sc.list[k0 + lane] : J;
          const float4 vk = sc.p[k];
          const FaceLine<float> ln = face_line(vj.x, vj.y, vj.z, vj.w, vk.x, vk.y, vk.z, vk.w);
          const float wx = ln.wx, wy = ln.wy, wz = ln.wz, w2 = ln.w2, inv = ln.inv, x0 = ln.x, y0 = ln.y, z0 = ln.z;
          const float room = 1.02f * r2max - (x0 * x0 + y0 * y0 + z0 * z0);
          const bool line = act && w2 > kLineMin;
          const bool alive = line && (wide || room > 0.0f);
          float hi = !alive ? -1.0f : wide ? 1.0e15f : sqrtf(room * inv), lo = -hi;
          unsigned hl = kNoEnd, ll = kNoEnd;
          for (unsigned l0 = 0; l0 < n;) {
            // a point cuts an interval only from within twice its ends' distance
            // to the cell; the points come in shells of growing distance
            const float end = fmaxf(hi, -lo);
            const float r2 = lo < hi ? x0 * x0 + y0 * y0 + z0 * z0 + end * end * w2 : 0.0f;
            const float far2 = 4.001f * __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(r2)));
            if (far2 == 0.0f) break;
            if (l0 < near_n && floorf(2.0f * sc.p[l0].w / shell * 0.99999f) * shell > far2) {
              l0 = near_n;  // only points looked up from beyond the ball are left
              if (l0 >= n) break;
            }
            const unsigned l1 = min(l0 + 8u, l0 < near_n ? near_n : n);
#pragma unroll 4
            for (unsigned l = l0; l < l1; ++l) {
              if (l == J) continue;
              const float4 v = sc.p[l];
              const float wl = fmaf(wz, v.z, fmaf(wy, v.y, wx * v.x));
              const float nm = v.w - fmaf(z0, v.z, fmaf(y0, v.y, x0 * v.x));
              const float t = __fdividef(nm, wl);
              if (l != k) {
                if (wl > 0.0f && t < hi) { hi = t; hl = l; }
                if (wl < 0.0f && t > lo) { lo = t; ll = l; }
              }
            }
            l0 = l1;
          }
          const bool member = alive && lo < hi;
          if (wide && act && !member) {
            // certain only where the two cuts cross by more than their rounding,
            // in float or else in double
            bool apart = false;
            if (line && hl != kNoEnd && ll != kNoEnd) {
              const float4 vh = sc.p[hl], vl = sc.p[ll];
              apart = cuts_apart(ln, vj.w, vk.w, vh, hi, vl, lo) ||
                      cuts_cross(g.P[i], g.P[sc.id[J]], g.P[sc.id[k]], g.P[sc.id[hl]], g.P[sc.id[ll]]);
            }
            doubt = doubt || !apart;
          }
          // an end at the largest sphere: its tetrahedron reaches out of the ball
          if (!FAR && __any_sync(0xffffffffu, member && (wide || hl == kNoEnd || ll == kNoEnd))) return false;
          members += (unsigned)__popc(__ballot_sync(0xffffffffu, member));
          bool counted = false;
          unsigned code = 0u;
          if (member) {
            if (hl != kNoEnd) {
              counted = sc.id[hl] > sc.id[k];
              code = (min(k, hl) << 16 | max(k, hl)) * 2654435761u;
            }
            if (ll != kNoEnd) {
              counted = counted || sc.id[ll] > sc.id[k];
              code ^= (min(k, ll) << 16 | max(k, ll)) * 2654435761u;
            }
          }
          reps += (unsigned)__popc(__ballot_sync(0xffffffffu, counted));
          mix ^= __reduce_xor_sync(0xffffffffu, code);
          // each tetrahedron once, from its lesser third point
#pragma unroll
          for (int end = 0; end < 2; ++end) {
            const unsigned l = end ? ll : hl;
            const bool put = member && k < l;
            const unsigned b = __ballot_sync(0xffffffffu, put);
            const unsigned at = tets + (unsigned)__popc(b & ((1u << lane) - 1u));
            if (put && at < 160u) 
              sc.tet[at] = make_ushort4((unsigned short)J, (unsigned short)k, (unsigned short)l, (unsigned short)(end + 1));
            tets += (unsigned)__popc(b);
          }
          if (tets > 160u) return false;
        }
        // No face: certain where every line is.  (Where some lines bound the face
        // and one was missed, its tetrahedra are met from the other third point
        // alone, and mix is not zero.)
        if (wide && members == 0u && __any_sync(0xffffffffu, doubt)) return false;
      }
      if (mix != 0u) return false;
      if (reps) {
        if (rows >= 64u) return false;
        if (w.leader()) {
          sc.rj[rows] = sc.id[J];
          sc.rr[rows] = reps;
        }
        ++rows;
      }
      if (!FAR && tets > 96u) {
        __syncwarp();
        if (!verify_tets(w, g, i, sc, n, tets, rho)) return false;
        for (unsigned t = lane; t < tets; t += 32u)
          if (!(4.0f * sc.cen[t].w <= rho * rho * 0.9999f)) big = true;
        __syncwarp();
        tets = 0u;
      }
    }
  }
  __syncwarp();
  if (!verify_tets(w, g, i, sc, n, tets, rho)) return false;
  if (FAR) {
    __syncwarp();
    const int far = verify_far(w, g, i, sc, n, tets, rho, ndone);
    if (far == 2) return false;
    if (far == 1) continue;
  } else {
    for (unsigned t = lane; t < tets; t += 32u)
      if (!(4.0f * sc.cen[t].w <= rho * rho * 0.9999f)) big = true;
    if (__any_sync(0xffffffffu, big)) return false;
  }
  write_row(w, sc, rows, row, len);
  return true;
  }
  return false;
}


template <int BOX, int REACH, int LOC>
__device__ __forceinline__ bool cell_local2(const Warp& w, const Grid& g, unsigned i, LocalScratch<LOC>& sc, uint2* row,
                                            unsigned* len) {
  const unsigned lane = w.lane();
  float rho;
  const Pt Pi = g.P[i];
  const unsigned n = gather_local<2, BOX, REACH, LOC>(w, g, i, Pi, sc.p, sc.id, rho);
  if (n > (unsigned)LOC || n < 3u) return false;
  if (!(rho * rho > g.rc2 * 1.0001f)) return false;
  // the star: the circles through i and a with the least parameter on either
  // side; those of an edge (or of one that the rounding may make an edge)
  // have to lie within the disk with their tolerance
  const float L0 = fmaxf(fabsf(Pi.x), fabsf(Pi.y));
  bool bad = false;
  unsigned edges = 0u;
  for (unsigned a0 = 0; a0 < n; a0 += 32u) {
    const bool act = a0 + lane < n;
    const unsigned a = act ? a0 + lane : 0u;
    const float4 va = sc.p[a];
    const float a2 = va.z * va.z + va.w * va.w;
    float left = 1.0e30f, right = -1.0e30f;
    unsigned kl = kNoEnd, kr = kNoEnd;
    for (unsigned q = 0; q < n; ++q) {
      const float4 v = sc.p[q];
      const float cr = va.z * v.w - va.w * v.z;
      const float nm = (v.z * v.z + v.w * v.w) - (va.z * v.z + va.w * v.w);
      const float s = __fdividef(nm, 2.0f * cr);
      if (q != a) {
        if (cr > 0.0f && s < left) { left = s; kl = q; }
        if (cr < 0.0f && s > right) { right = s; kr = q; }
      }
    }
    const bool edge = act && a2 > 0.0f && right <= left + 1.0e-3f * (1.0f + fabsf(left) + fabsf(right));
    edges += (unsigned)__popc(__ballot_sync(0xffffffffu, edge));
    if (edge) {
      if (kl == kNoEnd || kr == kNoEnd) {
        bad = true;
      } else {
#pragma unroll
        for (int side = 0; side < 2; ++side) {
          const float s = side ? right : left;
          const float4 vk = sc.p[side ? kr : kl];
          const float R = a2 * (0.25f + s * s), r = sqrtf(R);
          // shell_tol of the triangle (i, a, k), and the near test's slack
          const float h2 = fmaxf(a2, vk.z * vk.z + vk.w * vk.w), hm = sqrtf(h2);
          const float L = fmaxf(L0, fmaxf(fmaxf(fabsf(va.x), fabsf(va.y)), fmaxf(fabsf(vk.x), fabsf(vk.y))));
          const float den = 2.0f * fabsf(va.z * vk.w - va.w * vk.z);
          const float u = 0.5f * FLT_EPSILON;
          const float dc = 48.0f * u * (L * L + h2) * hm / den + 8.0f * u * L;
          const float tol = 1.01f * (4.0f * (2.0f * r * dc + dc * dc) + 32.0f * u * (R + L * r));
          const float reach = sqrtf(R + tol);
          const float slack = 1.0e-5f * (R + tol + 2.0f * reach * (2.0f * (L + r) + reach)) + 1.0e-30f;
          if (!(1.01f * r + sqrtf(R + tol + slack) * 1.01f <= rho)) bad = true;
          // the walk keeps at most kMaxNear points near a circle: a cell where
          // it may drop some is the walk's
          if (n >= (unsigned)kMaxNear) {
            // centre relative to i: a / 2 + s (-a.y, a.x)
            const float cx = 0.5f * va.z - s * va.w, cy = 0.5f * va.w + s * va.z;
            const float lim = (R + tol + slack) * 1.01f;
            unsigned near = 0u;
            for (unsigned q = 0; q < n; ++q) {
              const float e0 = sc.p[q].z - cx, e1 = sc.p[q].w - cy;
              near += e0 * e0 + e1 * e1 <= lim ? 1u : 0u;
            }
            if (near >= (unsigned)kMaxNear) bad = true;
          }
        }
      }
    }
  }
  if (edges < 3u || __any_sync(0xffffffffu, bad)) return false;
  const float li = sqlen2(Pi);
  unsigned rows = 0u;
  for (unsigned t0 = 0; t0 < n; t0 += 32u) {
    bool in = false;
    if (t0 + lane < n) {
      const float4 v = sc.p[t0 + lane];
      in = in_cutoff<2>(g, Pi, Pt{v.x, v.y, 0.0f, 0.0f});
    }
    for (unsigned bits = __ballot_sync(0xffffffffu, in); bits; bits &= bits - 1u) {
      const unsigned J = t0 + (unsigned)__ffs(bits) - 1u;
      const Pt pj{sc.p[J].x, sc.p[J].y, 0.0f, 0.0f};
      const float lj = sqlen2(pj);
      unsigned reps = 0u;
      for (unsigned k0 = 0; k0 < n; k0 += 32u) {
        const unsigned k = k0 + lane;
        bool open = k < n && k != J;
        float c[2] = {0.f, 0.f}, r2 = 0.f;
        if (open) {
          // naive_delaunay.hpp:62-99, as tri_pass
          const Pt pk{sc.p[k].x, sc.p[k].y, 0.0f, 0.0f};
          const float den = 2.0f * (Pi.x * (pj.y - pk.y) + pj.x * (pk.y - Pi.y) + pk.x * (Pi.y - pj.y));
          open = !(fabsf(den) <= FLT_EPSILON);
          const float lk = sqlen2(pk);
          c[0] = (li * (pj.y - pk.y) + lj * (pk.y - Pi.y) + lk * (Pi.y - pj.y)) / den;
          c[1] = (li * (pk.x - pj.x) + lj * (Pi.x - pk.x) + lk * (pj.x - Pi.x)) / den;
          const float e0 = Pi.x - c[0], e1 = Pi.y - c[1];
          r2 = e0 * e0 + e1 * e1;
        }
        for (unsigned m0 = 0; m0 < n; m0 += 8u) {
          if (!__any_sync(0xffffffffu, open)) break;
          const unsigned m1 = min(m0 + 8u, n);
          for (unsigned m = m0; m < m1; ++m) {
            const float4 v = sc.p[m];
            const float f0 = v.x - c[0], f1 = v.y - c[1];
            if (f0 * f0 + f1 * f1 <= r2 && m != J && m != k) open = false;
          }
        }
        // a circle without a gathered point has to lie within the disk
        const float r = sqrtf(r2);
        if (__any_sync(0xffffffffu, open && !(2.0f * r * 1.00001f <= rho))) return false;
        reps += (unsigned)__popc(__ballot_sync(0xffffffffu, open));
      }
      if (reps) {
        if (rows >= 64u) return false;
        if (w.leader()) {
          sc.rj[rows] = sc.id[J];
          sc.rr[rows] = reps;
        }
        ++rows;
      }
    }
  }
  write_row(w, sc, rows, row, len);
  return true;
}

template <int D, int BOX, int REACH, int LOC, bool FAR>
__device__ __forceinline__ bool cell_local(const Warp& w, const Grid& g, unsigned i, LocalScratch<LOC>& sc, uint2* row,
                                           unsigned* len) {
  if (D == 3) return cell_local3<BOX, REACH, LOC, FAR>(w, g, i, sc, row, len);
  return cell_local2<BOX, REACH, LOC>(w, g, i, sc, row, len);
}

}  // namespace dl
}  // namespace tecs
