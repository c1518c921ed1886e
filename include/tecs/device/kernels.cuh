// kernels.cuh -- device kernels of one cell step on sm_103a.
//
// State layout in HBM (per simulation, capacity-sized):
//   A      float4[cap]  x, y, z, cell id (uint bits)   state between steps
//   B      float4[cap]  A reordered by (bin, cell id)   working copy of a step
//   Xt     float4[cap]  Heun predictor x~ (sorted order)
//   d1,d2  float4[cap]  pass-1 / pass-2 position deltas (sorted order)
//   PA,PB,Pt,dp1,dp2    float2 polarity counterparts
//   key,rank,src        uint[cap] bin key, tentative rank, sorted -> unsorted slot
//   cnt,off             uint[nbins+1] bin counts (zero between steps), offsets
#pragma once

#include <cfloat>

#include "common.cuh"
#include "forces.cuh"
#include "delaunay_star.cuh"
#include "delaunay_local.cuh"

namespace tecs {

enum PassMode : int {
  kStore = 0,       // d_out[i] = sum of pair deltas
  kEulerFused = 1,  // A[i] = B[i] + sum * dt                               (euler.hpp:52-68, no COM)
  kHeun1Fused = 2,  // d_out[i] = sum; Xt[i] = B[i] + sum * dt             (heun.hpp:54-68, no COM)
  kHeun2Fused = 3   // A[i] = B[i] + ((d1[i] + sum) * 0.5) * dt            (heun.hpp:78-98, no COM)
};

struct Counters {
  unsigned n;           // active cells
  unsigned div_count;   // daughters requested this step
  unsigned done[2];     // last-block counters of the two COM reductions
  unsigned error;       // bit 0: capacity overflow on division; bit 1: a user law set drag, no old velocities kept;
                        // bit 2: a Delaunay cell search overflowed its arrays (more than kDlRow partners)
  unsigned done_div;    // last-block counter of the division fixup
  unsigned long long step;        // integrator steps taken (keys the division RNG)
  unsigned long long pair_count;  // pairs recorded by the capture hook
};

struct PassArgs {
  const float4* X;      // positions read by the pass (B or Xt)
  const float2* P;      // polarities read by the pass (PB or Pt) or null
  const unsigned* off;  // bin offsets
  Counters* ctr;
  // outputs
  float4* d_out;
  float2* dp_out;
  // fused epilogues
  const float4* Bx;     // x_n (sorted) for the fused updates
  const float2* Bp;
  const float4* d1;     // pass-1 deltas (Heun pass 2)
  const float2* dp1;
  float4* A;            // state written by the fused Euler / Heun-2 epilogue
  float2* PA;
  float4* Xt;           // predictor written by the fused Heun-1 epilogue
  float2* Pt;
  float dt;
  int mode;
  // centre-of-mass reduction (GlobalComFixer) fused into kStore
  double* com_part;     // fixed-point (2^-32) int64 sums, 3 per slot, reused as such
  float* com_out;       // 3 floats
  int com_slot;         // 0 or 1 (which done counter)
  unsigned capacity;
  // division (fused into kEulerFused / kHeun2Fused): a cell divides when
  // (hash >> 11) <= div_thresh = floor(p * 2^53), i.e. u01(hash) <= p exactly
  int div_enabled;
  unsigned long long div_thresh;
  float div_offset;
  unsigned long long seed;
  unsigned* div_parent;
  unsigned* div_slot;
  // pair capture hook
  uint2* pairs;
  unsigned long long pair_cap;
  // cell ids of the sorted slots (binned finders keep the bin key in X.w);
  // null when X.w holds the id (naive finders)
  const unsigned* Bid;
  // bin count of the next step's rebuild, fused into the state write
  int count_next;
  unsigned* key;
  unsigned* rank;
  unsigned* cnt;
  unsigned* part;       // scan chunk totals formed while counting (count_bin), or null
  // naive Delaunay: how many times each directed pair is applied, row i at i * capacity
  const unsigned short* dmult;
  // Delaunay (any capacity): cell i's partners and their applications,
  // dl_row[i * kDlRow + t] = (j, reps) for t < dl_len[i], ascending j
  const uint2* dl_row;
  const unsigned* dl_len;
  // links of each cell id, in link order: link_ent[link_off[id] .. link_off[id + 1])
  // = (other cell id, (link index << 1) | 1 when this cell is the link's b
  // end); slot_of maps an id to its slot in X (null when X is in id order)
  const unsigned* link_off;
  const uint2* link_ent;
  const unsigned* slot_of;
  float link_k;
  // the integrator's is_full_step of this evaluation (Euler, Heun pass 1: 1; Heun pass 2: 0), for user laws
  int full_step;
  // the integrator's old velocities by cell id (integrators/base.hpp:74), or
  // null when the simulation does not keep them: user laws that set drag
  // read them (binned_gabriel.hpp:225-226, 356-357), and k_finish writes the
  // step's velocity there (euler.hpp:59, heun.hpp:87)
  float4* old_vel;
  // extra fields: E float components per cell beyond position and polarity
  // (the config's other fields), stored component-major (component k of
  // slot s at k * capacity + s).  Bit k of ex_dbl: component k belongs to a
  // Scalar field, which the reference's integrators update in double
  // (float += delta * double dt); Vector and Polarity components update in
  // float (VectorN * Scalar).
  unsigned E;
  unsigned ex_dbl;
  const float* EX;   // extras read by the pass (EB or Et)
  const float* EBx;  // x_n extras (sorted) for the fused updates
  float* ed_out;     // extra deltas written (kStore, kHeun1Fused)
  const float* ed1;  // pass-1 extra deltas (Heun pass 2, k_finish)
  const float* ed2;  // pass-2 extra deltas (k_finish)
  float* EA;         // extras of the next state
  float* Et;         // extras of the predictor
  double dt64;       // the step's dt as the caller gave it
};

// at most this many extra components per cell
constexpr unsigned kMaxExtra = 8;

// What the user-law pass keeps per cell besides the position and polarity
// sums: the drag sums (the pairs' drag and drag * the other cell's old
// velocity, in pair order, binned_gabriel.hpp:105-106, 225-226) and the NE
// extra components' values and delta sums.
template <unsigned NE>
struct LawCell {
  float drag;
  float v[3];
  float ex_self[NE > 0 ? NE : 1];
  float ex_delta[NE > 0 ? NE : 1];
};

// ---------------------------------------------------------------------------
// binning: key + count, exclusive scan, scatter, per-bin id sort + gather

constexpr int kScanThreads = 256;
constexpr int kScanPer = 16;
constexpr int kScanChunk = kScanThreads * kScanPer;
// The bin scan keeps one partial sum per chunk of kScanChunk bins and, after
// those, one sum per kScanSuper chunks, so a chunk's prefix adds up at most
// len / (kScanChunk * kScanSuper) super sums and kScanSuper - 1 chunk sums:
// linear in the bin count (a server's bin space reaches billions of bins).
constexpr unsigned kScanSuper = 4096;
constexpr size_t scan_part_words(size_t len) {
  const size_t chunks = (len + kScanChunk - 1) / kScanChunk;
  return chunks + (chunks + kScanSuper - 1) / kScanSuper;
}

// Count a cell into bin b and return its tentative rank.  With part set, the
// cell is also added to its scan chunk's total -- what k_scan_reduce would
// form from the finished counts -- with one atomic per group of lanes that
// share the chunk (consecutive cells mostly do: they are in bin order).  The
// super-chunk totals, needed past kScanSuper chunks only, come from
// k_scan_super.
static __device__ __noinline__ void add_chunk_total(unsigned* part, unsigned b) {
  const unsigned c = b / (unsigned)kScanChunk;
  const unsigned grp = __match_any_sync(__activemask(), c);
  if ((threadIdx.x & 31u) == (unsigned)(__ffs(grp) - 1)) atomicAdd(&part[c], (unsigned)__popc(grp));
}
__device__ __forceinline__ unsigned count_bin(unsigned* cnt, unsigned* part, unsigned b) {
  const unsigned r = atomicAdd(&cnt[b], 1u);
  if (part) add_chunk_total(part, b);
  return r;
}

// Super-chunk totals part[chunks + j] = sum of chunk totals j*kScanSuper ..,
// one block per super-chunk.
static __global__ void k_scan_super(unsigned* __restrict__ part, unsigned chunks) {
  __shared__ unsigned sh[32];
  const unsigned lo = blockIdx.x * kScanSuper, hi = min(chunks, lo + kScanSuper);
  unsigned v = 0u;
  for (unsigned c = lo + threadIdx.x; c < hi; c += blockDim.x) v += part[c];
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31u) == 0u) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned t = 0u;
    for (unsigned w = 0; w < blockDim.x / 32u; ++w) t += sh[w];
    part[chunks + blockIdx.x] = t;
  }
}

static __global__ void k_count(const float4* __restrict__ A, const Counters* __restrict__ ctr, GridP g, int dims,
                               unsigned* __restrict__ key, unsigned* __restrict__ rank, unsigned* __restrict__ cnt,
                               unsigned* __restrict__ part) {
  const unsigned n = ctr->n;
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
    float4 v = A[s];
    float p[3] = {v.x, v.y, v.z};
    int c[3] = {0, 0, 0};
    unsigned b;
    if (dims == 3) { bin_coords_div<3>(g, p, c); b = flatten<3>(g, c); }
    else { bin_coords_div<2>(g, p, c); b = flatten<2>(g, c); }
    key[s] = b;
    rank[s] = count_bin(cnt, part, b);
  }
}

__device__ __forceinline__ unsigned block_sum(unsigned v, unsigned* sh) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
  __syncthreads();
  unsigned t = 0;
  if (threadIdx.x < 32) {
    t = threadIdx.x < (blockDim.x >> 5) ? sh[threadIdx.x] : 0u;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  }
  __syncthreads();
  if (threadIdx.x == 0) sh[0] = t;
  __syncthreads();
  t = sh[0];
  __syncthreads();
  return t;
}

// Per-chunk totals of cnt[0..len).
static __global__ void k_scan_reduce(const unsigned* __restrict__ cnt, unsigned len, unsigned* __restrict__ part) {
  __shared__ unsigned sh[32];
  const unsigned base = blockIdx.x * kScanChunk;
  unsigned v = 0;
  for (int k = 0; k < kScanPer; ++k) {
    unsigned idx = base + k * kScanThreads + threadIdx.x;
    if (idx < len) v += cnt[idx];
  }
  unsigned t = block_sum(v, sh);
  if (threadIdx.x == 0) {
    part[blockIdx.x] = t;
    // the super sums follow the chunk partials; k_scan_apply reads them past the
    // first kScanSuper chunks only, and only then they are zeroed before this kernel
    if (gridDim.x > kScanSuper) atomicAdd(&part[gridDim.x + blockIdx.x / kScanSuper], t);
  }
}

// Exclusive scan of cnt into off, zeroing cnt for the next step.  Each warp
// owns 512 consecutive counts, read 32 at a time (coalesced): a first sweep
// forms the warp totals, the block combines them with the earlier chunks'
// totals, a second sweep (L1 hits) scans and writes.
static __global__ void k_scan_apply(unsigned* __restrict__ cnt, unsigned len, const unsigned* __restrict__ part,
                             unsigned* __restrict__ off) {
  __shared__ unsigned sh[32];
  __shared__ unsigned wtot[kScanThreads / 32];
  unsigned pre = 0;
  const unsigned s0 = blockIdx.x / kScanSuper;
  for (unsigned j = threadIdx.x; j < s0; j += blockDim.x) pre += part[gridDim.x + j];
  for (unsigned b = s0 * kScanSuper + threadIdx.x; b < blockIdx.x; b += blockDim.x) pre += part[b];
  pre = block_sum(pre, sh);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int kPerWarp = kScanChunk / (kScanThreads / 32);
  const unsigned base = blockIdx.x * kScanChunk + warp * kPerWarp;
  unsigned tot = 0;
  for (int it = 0; it < kPerWarp / 32; ++it) {
    const unsigned idx = base + it * 32 + lane;
    tot += idx < len ? cnt[idx] : 0u;
  }
  for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
  if (lane == 0) wtot[warp] = tot;
  __syncthreads();
  unsigned carry = pre;
  for (int w = 0; w < warp; ++w) carry += wtot[w];
  for (int it = 0; it < kPerWarp / 32; ++it) {
    const unsigned idx = base + it * 32 + lane;
    const unsigned v = idx < len ? cnt[idx] : 0u;
    unsigned incl = v;
    for (int o = 1; o < 32; o <<= 1) {
      const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (idx < len) {
      off[idx] = carry + incl - v;
      cnt[idx] = 0u;
    }
    carry += __shfl_sync(0xffffffffu, incl, 31);
  }
}

// (part_words > 0: the scan has read the chunk totals that the counting
// formed; they start again from zero for the next step's count)
static __global__ void k_scatter(const Counters* __restrict__ ctr, const unsigned* __restrict__ key,
                          const unsigned* __restrict__ rank, const unsigned* __restrict__ off,
                          unsigned* __restrict__ src, unsigned* __restrict__ part, unsigned part_words) {
  const unsigned n = ctr->n;
  if (blockIdx.x == 0)
    for (unsigned w = threadIdx.x; w < part_words; w += blockDim.x) part[w] = 0u;
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x)
    src[off[key[s]] + rank[s]] = s;
}

// id of sorted slot j
__device__ __forceinline__ unsigned id_at(const float4* X, const unsigned* Bid, unsigned j) {
  return Bid ? __ldg(&Bid[j]) : id_of(__ldg(&X[j]));
}

// One thread per sorted slot: the cell that the scatter put at slot t moves to
// lo + (number of cells of its bin with a smaller id), so every bin lists its
// cells in ascending id -- the order of Kokkos BinSort's binning loop on the
// Serial backend.  Single-cell bins (most of them) copy straight through.
// the extra fields moved along with a state copy
struct ExtraMove {
  unsigned E;
  size_t C;  // capacity (component stride)
  const float* EA;
  float* EB;
};

static __global__ void k_order_gather(const Counters* __restrict__ ctr, const unsigned* __restrict__ key,
                                      const unsigned* __restrict__ off, const unsigned* __restrict__ src,
                                      const float4* __restrict__ A, const float2* __restrict__ PA,
                                      float4* __restrict__ B, float2* __restrict__ PB, unsigned* __restrict__ Bid,
                                      unsigned* __restrict__ slot_of, ExtraMove ex) {
  const unsigned n = ctr->n;
  for (unsigned t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
    const unsigned s = src[t];
    const unsigned b = key[s];
    const unsigned lo = off[b], hi = off[b + 1];
    const float4 v = A[s];
    unsigned dst = t;
    if (hi - lo > 1u) {
      const unsigned me = id_of(v);
      unsigned r = 0;
      for (unsigned k = lo; k < hi; ++k) r += id_of(A[src[k]]) < me ? 1u : 0u;
      dst = lo + r;
    }
    // the sorted copy carries the bin key in w (read by the passes with the
    // position); the id moves to Bid
    B[dst] = make_float4(v.x, v.y, v.z, __uint_as_float(b));
    Bid[dst] = id_of(v);
    if (slot_of) slot_of[id_of(v)] = dst;  // links find their other end by id
    if (PB) PB[dst] = PA[s];
    for (unsigned k = 0; k < ex.E; ++k) ex.EB[k * ex.C + dst] = ex.EA[k * ex.C + s];
  }
}

// A step without a rebuild (rebuild_every_n > 1): the working copy takes the
// new positions in the same slot order and keeps each slot's bin key in w.
static __global__ void k_refresh(const Counters* __restrict__ ctr, const float4* __restrict__ A,
                                 const float2* __restrict__ PA, float4* __restrict__ B, float2* __restrict__ PB,
                                 ExtraMove ex) {
  const unsigned n = ctr->n;
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
    const float4 v = A[s];
    B[s] = make_float4(v.x, v.y, v.z, B[s].w);
    if (PB) PB[s] = PA[s];
    for (unsigned k = 0; k < ex.E; ++k) ex.EB[k * ex.C + s] = ex.EA[k * ex.C + s];
  }
}

// Naive finders keep the working copy in cell-id order.
static __global__ void k_id_scatter(const Counters* __restrict__ ctr, const float4* __restrict__ A,
                             const float2* __restrict__ PA, float4* __restrict__ B, float2* __restrict__ PB,
                             ExtraMove ex) {
  const unsigned n = ctr->n;
  for (unsigned s = blockIdx.x * blockDim.x + threadIdx.x; s < n; s += gridDim.x * blockDim.x) {
    float4 v = A[s];
    unsigned id = id_of(v);
    B[id] = v;
    if (PB) PB[id] = PA[s];
    for (unsigned k = 0; k < ex.E; ++k) ex.EB[k * ex.C + id] = ex.EA[k * ex.C + s];
  }
}

// ---------------------------------------------------------------------------
// block reduction of the COM partials + last-block finalisation

// Centre-of-mass partial sums in 64-bit fixed point (2^-32 units): integer
// addition is associative, so the sum -- and the mean -- is the same whatever
// order the blocks finish in, and no FP64 (slow on this part) is needed.  Each
// block adds its totals to three global accumulators; the last block forms
// mean = sum / capacity (com_fixers.hpp:43 divides by the stage view's extent,
// i.e. the capacity) and clears the accumulators for the next use.
__device__ __forceinline__ long long com_fixed(float v) { return __float2ll_rn(v * 4294967296.0f); }

static __device__ void com_reduce_block(const PassArgs& a, long long x, long long y, long long z) {
  __shared__ long long sh[3][32];
  __shared__ bool last;
  for (int o = 16; o > 0; o >>= 1) {
    x += __shfl_xor_sync(0xffffffffu, x, o);
    y += __shfl_xor_sync(0xffffffffu, y, o);
    z += __shfl_xor_sync(0xffffffffu, z, o);
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  if (lane == 0) { sh[0][warp] = x; sh[1][warp] = y; sh[2][warp] = z; }
  __syncthreads();
  unsigned long long* acc = reinterpret_cast<unsigned long long*>(a.com_part) + 3 * a.com_slot;
  if (threadIdx.x == 0) {
    long long sx = 0, sy = 0, sz = 0;
    for (int w = 0; w < nw; ++w) { sx += sh[0][w]; sy += sh[1][w]; sz += sh[2][w]; }
    atomicAdd(&acc[0], (unsigned long long)sx);
    atomicAdd(&acc[1], (unsigned long long)sy);
    atomicAdd(&acc[2], (unsigned long long)sz);
    __threadfence();
    last = atomicAdd(&a.ctr->done[a.com_slot], 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (last && threadIdx.x == 0) {
    __threadfence();
    const double scale = 1.0 / (4294967296.0 * (double)a.capacity);
    for (int d = 0; d < 3; ++d) {
      const long long v = (long long)atomicExch(&acc[d], 0ull);
      a.com_out[d] = (float)((double)v * scale);
    }
    a.ctr->done[a.com_slot] = 0u;
  }
}

// Bin key and tentative rank of a freshly written cell for the next rebuild
// (what k_count does, fused into the state write).
template <int D>
__device__ __forceinline__ void count_cell(const GridP& g, const PassArgs& a, unsigned slot, const float* x) {
  int c[3] = {0, 0, 0};
  bin_coords_div<D>(g, x, c);
  const unsigned b = flatten<D>(g, c);
  a.key[slot] = b;
  a.rank[slot] = count_bin(a.cnt, a.part, b);
}

// ---------------------------------------------------------------------------
// division: decide (RNG keyed by cell id and step), append daughter at A[n + k]

template <int D>
__device__ __forceinline__ void maybe_divide(const GridP& g, const PassArgs& a, unsigned n, unsigned id,
                                             const float* xnew, float2 pnew, unsigned long long step,
                                             unsigned parent_slot) {
  if (!a.div_enabled) return;
  if ((hash64(a.seed, step, id, 0) >> 11) > a.div_thresh) return;
  unsigned k = atomicAdd(&a.ctr->div_count, 1u);
  unsigned slot = n + k;
  if (slot >= a.capacity) { atomicOr(&a.ctr->error, 1u); return; }
  double th = acos(2.0 * u01(hash64(a.seed, step, id, 1)) - 1.0);
  double ph = u01(hash64(a.seed, step, id, 2)) * 2.0 * 3.14159265358979323846;
  float v[3];
  pol_to_vec3((float)th, (float)ph, v);
  float4 o = make_float4(0.f, 0.f, 0.f, __uint_as_float(0xffffffffu));
  o.x = xnew[0] + a.div_offset * v[0];
  if (D >= 2) o.y = xnew[1] + a.div_offset * v[1];
  if (D >= 3) o.z = xnew[2] + a.div_offset * v[2];
  a.A[slot] = o;
  if (a.PA) a.PA[slot] = pnew;
  // the daughter takes the parent's new extra fields (written before this)
  for (unsigned c = 0; c < a.E; ++c) a.EA[c * (size_t)a.capacity + slot] = a.EA[c * (size_t)a.capacity + parent_slot];
  a.div_parent[k] = id;
  a.div_slot[k] = slot;
  if (a.count_next) {
    const float xd[3] = {o.x, o.y, o.z};
    count_cell<D>(g, a, slot, xd);
  }
}

// Daughter ids: n + rank of the parent id among this step's parents, then
// (last block) n += daughters.  Deterministic: ids depend only on parent ids.
static __global__ void k_divide_commit(Counters* __restrict__ ctr, unsigned capacity, const unsigned* __restrict__ parent,
                                const unsigned* __restrict__ slot, float4* __restrict__ A) {
  __shared__ bool last;
  const unsigned n = ctr->n;
  unsigned k = ctr->div_count;
  if (k > capacity - n) k = capacity - n;
  for (unsigned d = blockIdx.x * blockDim.x + threadIdx.x; d < k; d += gridDim.x * blockDim.x) {
    const unsigned p = parent[d];
    unsigned r = 0;
    for (unsigned e = 0; e < k; ++e) r += parent[e] < p ? 1u : 0u;
    A[slot[d]].w = __uint_as_float(n + r);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&ctr->done_div, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (last && threadIdx.x == 0) {
    ctr->n = n + k;
    ctr->div_count = 0u;
    ctr->step += 1ull;
    ctr->done_div = 0u;
  }
}
static __global__ void k_step_commit(Counters* __restrict__ ctr) { ctr->step += 1ull; }

// ---------------------------------------------------------------------------
// the force pass

// Gabriel witness test over the bins that overlap the ball around the
// midpoint (binned_gabriel.hpp:133-209).  true = some k blocks the pair.
template <int D>
__device__ __forceinline__ bool gabriel_blocked(const GridP& g, const ForceP& fp, const float4* __restrict__ X,
                                                const unsigned* __restrict__ off, unsigned i, unsigned j,
                                                const float* xi, const float* disp, float d2) {
  float m[3];
#pragma unroll
  for (int d = 0; d < D; ++d) m[d] = xi[d] - disp[d] * 0.5f;
  const float rsq = d2 * fp.gab_factor;
  const float r = sqrtf(rsq);
  int mn[3] = {0, 0, 0}, mx[3] = {0, 0, 0};
#pragma unroll
  for (int d = 0; d < D; ++d) {
    mn[d] = clampi((int)floorf((m[d] - r - g.mn[d]) * g.inv_bin), g.ext[d] - 1);
    mx[d] = clampi((int)floorf((m[d] + r - g.mn[d]) * g.inv_bin), g.ext[d] - 1);
  }
  const int z0 = D >= 3 ? mn[2] : 0, z1 = D >= 3 ? mx[2] : 0;
  for (int z = z0; z <= z1; ++z) {
    for (int y = mn[1]; y <= mx[1]; ++y) {
      // a row of bins along x is one contiguous segment in sorted order
      int c0[3] = {mn[0], y, z}, c1[3] = {mx[0], y, z};
      const unsigned lo = off[flatten<D>(g, c0)], hi = off[flatten<D>(g, c1) + 1];
      for (unsigned k = lo; k < hi; ++k) {
        if (k == i || k == j) continue;
        const float4 v = X[k];
        const float e0 = v.x - m[0], e1 = v.y - m[1];
        float s = e0 * e0 + e1 * e1;
        if (D >= 3) { const float e2 = v.z - m[2]; s = s + e2 * e2; }
        if (s < rsq) return true;
      }
    }
  }
  return false;
}

// naive_gabriel.hpp:71-80: every k, radius (d2 * 0.25) * c^2
template <int D>
__device__ __forceinline__ bool gabriel_blocked_naive(const ForceP& fp, const float4* __restrict__ X, unsigned n,
                                                      unsigned i, unsigned j, const float* xi, const float* disp,
                                                      float d2) {
  float m[3];
#pragma unroll
  for (int d = 0; d < D; ++d) m[d] = xi[d] - disp[d] * 0.5f;
  const float rsq = d2 * 0.25f * fp.gab_csq;
  for (unsigned k = 0; k < n; ++k) {
    if (k == i || k == j) continue;
    const float4 v = X[k];
    const float e0 = v.x - m[0], e1 = v.y - m[1];
    float s = e0 * e0 + e1 * e1;
    if (D >= 3) { const float e2 = v.z - m[2]; s = s + e2 * e2; }
    if (s < rsq) return true;
  }
  return false;
}

// ---------------------------------------------------------------------------
// Naive Delaunay (naive_delaunay.hpp).  The reference applies the pair (i, j)
// once per accepted simplex: in 2-D per third point k whose circumcircle
// through i, j, k is non-degenerate (|den| > FLT_EPSILON) and holds no other
// point (distance^2 <= r^2 rejects); in 3-D per third point k for which some
// l > k spans a non-degenerate tetrahedron with an empty circumsphere (a point
// outside the axis-aligned box |p - c| <= r is skipped before its distance
// test).  k_delaunay_mult counts the applications of every in-cutoff pair,
// one block per cell i with the threads spread over k; the force pass then
// adds the pair's force that many times, in j order -- the Serial order.
template <int D>
__device__ __forceinline__ float sq_len(const float4& v) {
  float s = v.x * v.x + v.y * v.y;
  if (D >= 3) s = s + v.z * v.z;
  return s;
}

template <int D>
__device__ __forceinline__ float sq_dist(const float4& v, const float* c) {
  const float e0 = v.x - c[0], e1 = v.y - c[1];
  float s = e0 * e0 + e1 * e1;
  if (D >= 3) { const float e2 = v.z - c[2]; s = s + e2 * e2; }
  return s;
}

// The circumcircle (2-D) or the reference's sphere (3-D) of i, j and the third
// (and fourth) point: false when degenerate.  r2 is the squared distance from
// the centre to i.
__device__ __forceinline__ bool delaunay_circle(const float4& pi, const float4& pj, const float4& pk, float li,
                                                float lj, float* c, float& r2) {
  const float den = 2.0f * (pi.x * (pj.y - pk.y) + pj.x * (pk.y - pi.y) + pk.x * (pi.y - pj.y));
  if (fabsf(den) <= FLT_EPSILON) return false;
  const float lk = sq_len<2>(pk);
  c[0] = (li * (pj.y - pk.y) + lj * (pk.y - pi.y) + lk * (pi.y - pj.y)) / den;
  c[1] = (li * (pk.x - pj.x) + lj * (pi.x - pk.x) + lk * (pj.x - pi.x)) / den;
  r2 = sq_dist<2>(pi, c);
  return true;
}

__device__ __forceinline__ bool delaunay_sphere(const float4& pi, const float4& pj, const float4& pk, const float4& pl,
                                                float li, float lj, float lk, float* c, float& r2) {
  const float e1[3] = {pj.x - pi.x, pj.y - pi.y, pj.z - pi.z};
  const float e2[3] = {pk.x - pi.x, pk.y - pi.y, pk.z - pi.z};
  const float e3[3] = {pl.x - pi.x, pl.y - pi.y, pl.z - pi.z};
  const float den = 2.0f * (e1[0] * (e2[1] * e3[2] - e2[2] * e3[1]) - e1[1] * (e2[0] * e3[2] - e2[2] * e3[0]) +
                            e1[2] * (e2[0] * e3[1] - e2[1] * e3[0]));
  if (fabsf(den) <= FLT_EPSILON) return false;
  const float b1 = lj - li, b2 = lk - li, b3 = sq_len<3>(pl) - li;
  c[0] = pi.x + (b1 * (e2[1] * e3[2] - e2[2] * e3[1]) - e1[1] * (b2 * e3[2] - e2[2] * b3) +
                 e1[2] * (b2 * e3[1] - e2[1] * b3)) / den;
  c[1] = pi.y + (e1[0] * (b2 * e3[2] - e2[2] * b3) - b1 * (e2[0] * e3[2] - e2[2] * e3[0]) +
                 e1[2] * (e2[0] * b3 - b2 * e3[0])) / den;
  c[2] = pi.z + (e1[0] * (e2[1] * b3 - b2 * e3[1]) - e1[1] * (e2[0] * b3 - b2 * e3[0]) +
                 b1 * (e2[0] * e3[1] - e2[1] * e3[0])) / den;
  r2 = sq_dist<3>(pi, c);
  return true;
}

// m rejects the simplex: 2-D distance^2 <= r^2; 3-D first inside the box of half edge r
template <int D>
__device__ __forceinline__ bool delaunay_inside(const float4& pm, const float* c, float r, float r2) {
  if (D == 3 && (fabsf(pm.x - c[0]) > r || fabsf(pm.y - c[1]) > r || fabsf(pm.z - c[2]) > r)) return false;
  return sq_dist<D>(pm, c) <= r2;
}

constexpr int kDelaunayThreads = 256;
constexpr unsigned kDelaunayMaxCells = 4096;  // the pair-count table is capacity^2 x 2 bytes
// Blocks per cell: the third points are dealt to their warps in turn, so that
// a cell with many pairs takes no longer than its share of the GPU (with the
// pairs dealt to four blocks the SMs waited 36 % of 2.0 ms for the last ones,
// 400 cells in 3-D).
constexpr unsigned kDelaunaySplit = 16;
// Up to so many cells a block takes a cell by itself and writes its row, without
// the clearing of the table before: launches are what such a call costs (2 cells
// 8.9 us a step against 13.0; past 10 cells in space the one block takes longer).
constexpr unsigned kDelaunayOne = 8;
constexpr unsigned kDelaunayNear = 64;  // points near i that each simplex is tested against first

// Every simplex is an existence test over all points: one point inside rejects
// it, so the order of the tests does not change a count.  A sphere through i is
// mostly rejected by a point near i, so each lane tests its simplex against
// the points near i first, and the few that are left are tested against all
// points by the whole warp, 32 at a time.  3-D: a warp takes one third point k
// and its lanes the fourth points l > k; the first accepted l ends k.  2-D:
// the lanes take the third points.
// What bounds it: instruction issue (the spheres' arithmetic).  One thread per
// third point that walks every l and every m in index order takes 400-660 ms
// on 400 cells in 3-D, this form 1.7 ms.
template <int D>
static __global__ void __launch_bounds__(kDelaunayThreads)
k_delaunay_mult(const float4* __restrict__ X, const Counters* __restrict__ ctr, float rc2, unsigned stride,
                unsigned short* __restrict__ mult) {  // (cleared before, unless a block takes a cell by itself)
  __shared__ float4 near[kDelaunayNear];  // w: the point's index
  __shared__ unsigned nnear, row[kDelaunayOne];
  const unsigned n = ctr->n;
  const unsigned i = blockIdx.x, split = gridDim.y;
  if (i >= n) return;
  const unsigned t = threadIdx.x, lane = t & 31u, warp = t >> 5;
  if (t < kDelaunayOne) row[t] = 0u;
  const float4 pi = __ldg(&X[i]);
  const float li = sq_len<D>(pi);
  const float ci[3] = {pi.x, pi.y, pi.z};
  // a ball around i that holds between 16 and kDelaunayNear points (or the
  // last one tried: any subset of the points is a valid first test)
  for (float rr = rc2 * 2.0f, it = 0.0f; it < 24.0f; it += 1.0f) {
    if (t == 0) nnear = 0u;
    __syncthreads();
    for (unsigned m = t; m < n; m += kDelaunayThreads) {
      const float4 v = __ldg(&X[m]);
      if (m != i && sq_dist<D>(v, ci) < rr) {
        const unsigned at = atomicAdd(&nnear, 1u);
        if (at < kDelaunayNear) near[at] = make_float4(v.x, v.y, v.z, __uint_as_float(m));
      }
    }
    __syncthreads();
    const unsigned got = nnear;
    if ((got >= 16u && got <= kDelaunayNear) || got + 1u >= n) break;
    rr = got < 16u ? rr * 2.0f : rr * 0.7f;
    __syncthreads();
  }
  const unsigned nn = min(nnear, kDelaunayNear);
  // nearest first: most spheres fall to the first few
  {
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    unsigned rank = 0u;
    if (t < nn) {
      v = near[t];
      const float d = sq_dist<D>(v, ci);
      for (unsigned m = 0; m < nn; ++m) {
        const float e = sq_dist<D>(near[m], ci);
        rank += (e < d || (e == d && m < t)) ? 1u : 0u;
      }
    }
    __syncthreads();
    if (t < nn) near[rank] = v;
    __syncthreads();
  }
  for (unsigned j0 = 0; j0 < n; j0 += 32u) {
    const unsigned jl = j0 + lane;
    bool in = false;
    if (jl < n && jl != i) {
      const float4 v = __ldg(&X[jl]);
      const float e0 = pi.x - v.x, e1 = pi.y - v.y;
      float d2 = e0 * e0 + e1 * e1;
      if (D >= 3) { const float e2 = pi.z - v.z; d2 = d2 + e2 * e2; }
      in = !(d2 >= rc2);
    }
    for (unsigned bits = __ballot_sync(0xffffffffu, in); bits; bits &= bits - 1u) {
      const unsigned j = j0 + (unsigned)__ffs(bits) - 1u;
      const float4 pj = __ldg(&X[j]);
      const float lj = sq_len<D>(pj);
      unsigned local = 0;
      const unsigned items = D == 3 ? n : (n + 31u) / 32u;
      for (unsigned q = blockIdx.y + warp * split; q < items; q += kDelaunayThreads / 32 * split) {
        if (D == 3 && (q == i || q == j)) continue;
        const float4 pq = D == 3 ? __ldg(&X[q]) : pj;
        const float lq = sq_len<3>(pq);
        for (unsigned b0 = D == 3 ? q + 1u : q * 32u, b1 = D == 3 ? n : min(n, q * 32u + 32u); b0 < b1; b0 += 32u) {
          const unsigned l = b0 + lane;
          bool open = l < b1 && l != i && l != j;
          float c[3] = {0.f, 0.f, 0.f}, r2 = 0.f;
          if (open) {
            const float4 pl = __ldg(&X[l]);
            open = D == 3 ? delaunay_sphere(pi, pj, pq, pl, li, lj, lq, c, r2)
                          : delaunay_circle(pi, pj, pl, li, lj, c, r2);
          }
          const float r = D == 3 ? sqrtf(r2) : 0.f;
          for (unsigned m = 0; m < nn; ++m) {
            if (!__any_sync(0xffffffffu, open)) break;
            const float4 v = near[m];
            const unsigned id = __float_as_uint(v.w);
            if (open && id != j && id != l && (D == 2 || id != q) && delaunay_inside<D>(v, c, r, r2)) open = false;
          }
          unsigned left = __ballot_sync(0xffffffffu, open), accepted = 0u;
          for (; left; left &= left - 1u) {
            const int src = __ffs(left) - 1;
            const float cc[3] = {__shfl_sync(0xffffffffu, c[0], src), __shfl_sync(0xffffffffu, c[1], src),
                                 __shfl_sync(0xffffffffu, c[2], src)};
            const float rr = __shfl_sync(0xffffffffu, r, src), rr2 = __shfl_sync(0xffffffffu, r2, src);
            const unsigned ll = b0 + (unsigned)src;
            bool hit = false;
            for (unsigned m = lane; m < n; m += 32u) {
              if (m != i && m != j && m != ll && (D == 2 || m != q))
                hit = delaunay_inside<D>(__ldg(&X[m]), cc, rr, rr2);
              if (hit) break;
            }
            if (!__any_sync(0xffffffffu, hit)) {
              ++accepted;
              if (D == 3) break;
            }
          }
          local += accepted;
          if (D == 3 && accepted) break;
        }
      }
      if (lane == 0u && local && split == 1u) {
        atomicAdd(&row[j], local);
      } else if (lane == 0u && local) {
        // a count is below 2^16, so adding it to its half of a word carries nothing over
        const size_t at = (size_t)i * stride + j;
        atomicAdd(reinterpret_cast<unsigned*>(mult) + at / 2, local << (at & 1 ? 16 : 0));
      }
    }
  }
  if (split == 1u) {
    __syncthreads();
    if (t < n) mult[(size_t)i * stride + t] = (unsigned short)row[t];
  }
}

// ---------------------------------------------------------------------------
// Delaunay finder for any capacity (tecs/device/delaunay_star.cuh).  Before
// each pass: the bounding box of the pass's positions, a bin grid of about
// two cells per bin, a counting sort into it, then each cell's partners and
// multiplicities (k_dl_local and k_dl_mult, one warp per cell).  The pass applies each
// listed pair reps times in ascending j, as FINDER 4 does.
constexpr unsigned kDlRow = 64;  // partners per cell
constexpr int kDlThreads = 64;

struct DlState {
  unsigned mm[6];  // ordered-integer min (0..2) and max (3..5) of the coordinates
  double lo[3];
  double h, inv;
  int dims[3];
  unsigned nbins;
  dl::GridF f;
  // cells handed on by the local search's levels, and the cells taken from
  // each list so far
  unsigned left[2], taken[3];
};

__device__ __forceinline__ unsigned f2ord(float f) {
  const unsigned u = __float_as_uint(f);
  return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float ord2f(unsigned u) {
  return __uint_as_float((u & 0x80000000u) ? (u & 0x7fffffffu) : ~u);
}

static __global__ void k_dl_reset(DlState* st) {
  if (threadIdx.x < 3) {
    st->mm[threadIdx.x] = 0xffffffffu;
    st->mm[3 + threadIdx.x] = 0u;
    st->taken[threadIdx.x] = 0u;
    if (threadIdx.x < 2) st->left[threadIdx.x] = 0u;
  }
}

template <int D>
static __global__ void k_dl_bounds(const float4* __restrict__ X, const Counters* __restrict__ ctr, DlState* st) {
  const unsigned n = ctr->n;
  unsigned lo[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu}, hi[3] = {0u, 0u, 0u};
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 v = X[i];
    const float c[3] = {v.x, v.y, v.z};
#pragma unroll
    for (int d = 0; d < D; ++d) {
      const unsigned o = f2ord(c[d]);
      lo[d] = min(lo[d], o);
      hi[d] = max(hi[d], o);
    }
  }
#pragma unroll
  for (int d = 0; d < D; ++d) {
    for (int sh = 16; sh > 0; sh >>= 1) {
      lo[d] = min(lo[d], __shfl_xor_sync(0xffffffffu, lo[d], sh));
      hi[d] = max(hi[d], __shfl_xor_sync(0xffffffffu, hi[d], sh));
    }
    if ((threadIdx.x & 31) == 0) { atomicMin(&st->mm[d], lo[d]); atomicMax(&st->mm[3 + d], hi[d]); }
  }
}

template <int D>
static __global__ void k_dl_plan(const Counters* __restrict__ ctr, unsigned max_bins, DlState* st) {
  if (threadIdx.x != 0 || blockIdx.x != 0) return;
  const unsigned n = ctr->n;
  double mn[3] = {0.0, 0.0, 0.0}, mx[3] = {0.0, 0.0, 0.0};
  if (n > 0)
    for (int d = 0; d < D; ++d) { mn[d] = ord2f(st->mm[d]); mx[d] = ord2f(st->mm[3 + d]); }
  dl::Grid g{};
  dl::plan_grid<D>(g, mn, mx, n, max_bins);
  for (int d = 0; d < 3; ++d) { st->lo[d] = g.lo[d]; st->dims[d] = g.dims[d]; }
  st->h = g.h;
  st->inv = g.inv;
  st->nbins = g.nbins;
  st->f = g.f;
}

__device__ __forceinline__ dl::Grid dl_view(const DlState* st) {
  dl::Grid g{};
  for (int d = 0; d < 3; ++d) { g.lo[d] = st->lo[d]; g.dims[d] = st->dims[d]; }
  g.h = st->h;
  g.inv = st->inv;
  g.nbins = st->nbins;
  g.f = st->f;
  return g;
}

template <int D>
__device__ __forceinline__ unsigned dl_bin(const dl::Grid& g, const float4& v) {
  const double q[3] = {v.x, v.y, v.z};
  int b[3];
  dl::bin_of<D>(g, q, b);
  return dl::flat(g, b[0], b[1], b[2]);
}

template <int D>
static __global__ void k_dl_count(const float4* __restrict__ X, const Counters* __restrict__ ctr,
                                  const DlState* __restrict__ st, unsigned* __restrict__ cnt) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ctr->n) return;
  const dl::Grid g = dl_view(st);
  atomicAdd(&cnt[dl_bin<D>(g, X[i])], 1u);
}

// exclusive scan of the bin counts into off (off[nbins] = cells), one block;
// the counts are cleared for the scatter's cursors
static __global__ void __launch_bounds__(1024) k_dl_scan(const DlState* __restrict__ st, unsigned* __restrict__ cnt,
                                                         unsigned* __restrict__ off) {
  __shared__ unsigned part[1024];
  const unsigned nb = st->nbins, t = threadIdx.x;
  const unsigned per = (nb + 1023u) / 1024u, b0 = min(nb, t * per), b1 = min(nb, b0 + per);
  unsigned sum = 0;
  for (unsigned b = b0; b < b1; ++b) sum += cnt[b];
  part[t] = sum;
  __syncthreads();
  for (unsigned sh = 1; sh < 1024u; sh <<= 1) {
    const unsigned v = t >= sh ? part[t - sh] : 0u;
    __syncthreads();
    part[t] += v;
    __syncthreads();
  }
  unsigned run = part[t] - sum;
  for (unsigned b = b0; b < b1; ++b) {
    const unsigned c = cnt[b];
    off[b] = run;
    run += c;
    cnt[b] = 0u;
  }
  if (t == 1023u) off[nb] = part[1023];
}

template <int D>
static __global__ void k_dl_scatter(const float4* __restrict__ X, const Counters* __restrict__ ctr,
                                    const DlState* __restrict__ st, unsigned* __restrict__ cnt,
                                    const unsigned* __restrict__ off, unsigned* __restrict__ idx,
                                    float4* __restrict__ sp) {
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= ctr->n) return;
  const dl::Grid g = dl_view(st);
  const float4 v = X[i];
  const unsigned b = dl_bin<D>(g, v);
  const unsigned at = off[b] + atomicAdd(&cnt[b], 1u);
  idx[at] = i;
  sp[at] = v;
}

__device__ __forceinline__ dl::Grid dl_grid(const float4* X, const Counters* ctr, const DlState* st, const unsigned* off,
                                            const unsigned* idx, const float4* sp, float rc2) {
  dl::Grid g = dl_view(st);
  g.off = off;
  g.idx = idx;
  g.sp = reinterpret_cast<const dl::Pt*>(sp);
  g.P = reinterpret_cast<const dl::Pt*>(X);
  g.n = ctr->n;
  g.rc2 = rc2;
  return g;
}

// The local search (delaunay_local.cuh), one warp per cell.  LEVEL 0: every
// cell, in bin order; LEVEL 1: the cells that level 0 handed on, in 2-D over a
// larger box, in 3-D looking up what lies beyond the gathered ball.  The cells
// that a level is not certain of go to its list.
// Radii: 1.75 bins hold about 85 points in a ball of cells (two cells a bin of
// its bounding box), enough for 97 % of the interior cells (spheres of 1.4 cell
// spacings); in 2-D 2.25 bins hold about 40, enough for all but the hull.
template <int D, int LEVEL>
static __global__ void __launch_bounds__(dl::kLocalThreads, LEVEL == 0 ? 6 : 5)
    k_dl_local(const float4* __restrict__ X, const Counters* __restrict__ ctr, DlState* __restrict__ st,
               const unsigned* __restrict__ off, const unsigned* __restrict__ idx, const float4* __restrict__ sp,
               float rc2, uint2* __restrict__ row, unsigned* __restrict__ len, const unsigned* __restrict__ in,
               unsigned* __restrict__ out) {
  constexpr int BOX = LEVEL == 1 && D == 2 ? 4 : 2;
  constexpr int REACH = D == 3 ? 175 : (LEVEL == 0 ? 225 : 450);
  constexpr int LOC = LEVEL == 0 ? 112 : (D == 3 ? 192 : 320);
  __shared__ dl::LocalScratch<LOC> scratch[dl::kLocalThreads / 32];
  dl::LocalScratch<LOC>& sc = scratch[threadIdx.x >> 5];
  const dl::Grid g = dl_grid(X, ctr, st, off, idx, sp, rc2);
  const dl::Warp lanes;
  const unsigned count = LEVEL == 0 ? g.n : st->left[0];
  for (;;) {
    unsigned at = 0u;
    if (lanes.leader()) at = atomicAdd(&st->taken[LEVEL], 1u);
    at = lanes.bcast(at, 0);
    if (at >= count) return;
    const unsigned i = in[at];
    __syncwarp();
    if (!dl::cell_local<D, BOX, REACH, LOC, LEVEL == 1>(lanes, g, i, sc, row + (size_t)i * kDlRow, len + i) && lanes.leader())
      out[atomicAdd(&st->left[LEVEL], 1u)] = i;
    __syncwarp();
  }
}

// The cells that the local search was not certain of (all: every cell, in bin
// order): the walk in double, one warp per cell, the lanes sharing each search's
// entries (dl::Warp).
template <int D>
static __global__ void __launch_bounds__(kDlThreads) k_dl_mult(const float4* __restrict__ X, Counters* __restrict__ ctr,
                                                               DlState* __restrict__ st,
                                                               const unsigned* __restrict__ off,
                                                               const unsigned* __restrict__ idx,
                                                               const float4* __restrict__ sp, float rc2,
                                                               uint2* __restrict__ row, unsigned* __restrict__ len,
                                                               const unsigned* __restrict__ in, bool all) {
  // the warp's star and candidate lists: one copy, in shared memory
  __shared__ __align__(16) unsigned char scratch[(kDlThreads / 32) * sizeof(dl::Scratch)];
  dl::Scratch& sc = reinterpret_cast<dl::Scratch*>(scratch)[threadIdx.x >> 5];
  __shared__ unsigned out_j[kDlThreads / 32][kDlRow], out_r[kDlThreads / 32][kDlRow];
  unsigned *oj = out_j[threadIdx.x >> 5], *orp = out_r[threadIdx.x >> 5];
  const dl::Grid g = dl_grid(X, ctr, st, off, idx, sp, rc2);
  const dl::Warp lanes;
  const unsigned count = all ? g.n : st->left[1];
  for (;;) {
    unsigned at = 0u;
    if (lanes.leader()) at = atomicAdd(&st->taken[2], 1u);
    at = lanes.bcast(at, 0);
    if (at >= count) return;
    const unsigned i = in[at];
    unsigned err = 0;
    const unsigned m = dl::cell_mult<D>(lanes, g, i, oj, orp, kDlRow, &err, sc);
    for (unsigned t = lanes.lane(); t < m; t += 32u) row[(size_t)i * kDlRow + t] = make_uint2(oj[t], orp[t]);
    __syncwarp();
    if (lanes.leader()) {
      len[i] = m;
      // a full near-circle list keeps the points nearest the circle (no error);
      // any other overflow leaves the row incomplete
      if (err & (dl::kErrStar | dl::kErrPairs | dl::kErrList)) atomicOr(&ctr->error, 4u);
    }
  }
}

template <int D, int FINDER, int FORCE>
__device__ __forceinline__ void visit(const GridP& g, const ForceP& fp, const PassArgs& a, unsigned n, unsigned i,
                                      unsigned j, const float* xi, float2 pi, Acc& acc, unsigned idi,
                                      unsigned reps5 = 1u) {
  const float4 vj = a.X[j];
  float disp[3];
  disp[0] = xi[0] - vj.x;
  if (D >= 2) disp[1] = xi[1] - vj.y;
  if (D >= 3) disp[2] = xi[2] - vj.z;
  float d2 = disp[0] * disp[0] + disp[1] * disp[1];
  if (D >= 3) d2 = d2 + disp[2] * disp[2];
  if (d2 >= fp.rc2) return;
  if (FINDER == 3 && gabriel_blocked<D>(g, fp, a.X, a.off, i, j, xi, disp, d2)) return;
  const unsigned reps = FINDER == 5 ? reps5 : 1u;
  if (a.pairs) {
    unsigned long long s = atomicAdd(&a.ctr->pair_count, (unsigned long long)reps);
    for (unsigned r = 0; r < reps; ++r)
      if (s + r < a.pair_cap) a.pairs[s + r] = make_uint2(idi, id_at(a.X, a.Bid, j));
  }
  const float dist = sqrtf(d2);
  const float2 pj = (FORCE == 2 && a.P) ? a.P[j] : make_float2(0.f, 0.f);
  for (unsigned r = 0; r < reps; ++r) pair_force<D, FORCE>(fp, disp, dist, pi, pj, acc);
}

// Commit of one cell: out(i) = 0 + sum (views(i) += values on cleared stage
// buffers); the drag term adds exactly zero for the built-in laws
// (pairwise_drag = 0).  Then the fused integrator epilogue of the mode.
// One link's force on this cell, added after the pairwise sum: the
// constant-pull law of examples/intercalation.cpp:65-71 -- cell a gets
// k*(x_b - x_a)/|x_b - x_a|, cell b its negative -- in the Serial order of
// integrators/base.hpp:205-233 (link order, each term from a zero accumulator).
// A link to an id beyond the active cells sees the zero position of an unused
// view slot.
template <int D>
__device__ __forceinline__ void add_link(const PassArgs& a, unsigned n, const float* xs, unsigned e, float* s) {
  const uint2 le = a.link_ent[e];
  const bool b_end = (le.y & 1u) != 0u;
  float xo[3] = {0.f, 0.f, 0.f};
  if (le.x < n) {
    const float4 v = a.X[a.slot_of ? a.slot_of[le.x] : le.x];
    xo[0] = v.x; xo[1] = v.y; xo[2] = v.z;
  }
  float disp[3] = {0.f, 0.f, 0.f};
#pragma unroll
  for (int d = 0; d < D; ++d) disp[d] = b_end ? xs[d] - xo[d] : xo[d] - xs[d];
  float d2 = disp[0] * disp[0] + disp[1] * disp[1];
  if (D >= 3) d2 = d2 + disp[2] * disp[2];
  const float dist = sqrtf(d2);
  const float k = b_end ? -a.link_k : a.link_k;
#pragma unroll
  for (int d = 0; d < D; ++d) s[d] = s[d] + (0.0f + (k * disp[d]) / dist);
}

// One extra component's update, in double for Scalar fields (the reference's
// float += float * double) and in float otherwise.
__device__ __forceinline__ float ex_update(float x, float d, float dt, double dt64, bool dbl) {
  return dbl ? (float)((double)x + (double)d * dt64) : x + d * dt;
}

// The extra fields of one active cell (slot i): the mode's delta store and
// state update, as cell_commit does for the position.  exd: the cell's extra
// deltas, 0 + its sums (null: zero).
__device__ __forceinline__ void commit_extras(const PassArgs& a, unsigned i, const float* exd) {
  const size_t C = a.capacity;
  for (unsigned k = 0; k < a.E; ++k) {
    const float d = exd ? exd[k] : 0.0f;
    const bool dbl = (a.ex_dbl >> k) & 1u;
    const size_t at = k * C + i;
    if (a.mode == kStore) {
      a.ed_out[at] = d;
    } else if (a.mode == kHeun1Fused) {
      a.ed_out[at] = d;
      a.Et[at] = ex_update(a.EX[at], d, a.dt, a.dt64, dbl);
    } else if (a.mode == kEulerFused) {
      a.EA[at] = ex_update(a.EBx[at], d, a.dt, a.dt64, dbl);
    } else {
      // Heun: x += (d1 + d2) * 0.5 * dt (heun.hpp:89-90)
      const float h = a.ed1[at] + d;
      const float xb = a.EBx[at];
      a.EA[at] = dbl ? (float)((double)xb + ((double)h * 0.5) * a.dt64) : xb + (h * 0.5f) * a.dt;
    }
  }
}

// The library's link law: the constant pull (add_link).  A user LINK_FORCE
// law takes its place in the user-law pass (tecs/pairwise.cuh).
struct BuiltinLinks {
  template <int D>
  __device__ __forceinline__ void add(const PassArgs& a, unsigned n, unsigned id, const float* xs, float2 ps,
                                      unsigned e, float* s, float* sp, float* se) const {
    add_link<D>(a, n, xs, e, s);
  }
};

// The write of one active cell: links, then the mode's store or fused
// integrator update, the next rebuild's bin count and division.  s receives
// the cell's position delta (for the COM partials).
// NE: the extra components the pass carries (the user-law pass of a config
// with extra fields; the built-in passes carry none and leave the extra
// fields to k_predict / k_finish, see enqueue_step).
template <int D, class Links = BuiltinLinks, unsigned NE = 0>
__device__ __forceinline__ void cell_commit(const GridP& g, const PassArgs& a, unsigned n, unsigned i,
                                            const float* xi, const float4& vi, const float2& pi, const Acc& acc,
                                            float* s, const Links& links = Links{}, const float* exd = nullptr) {
#pragma unroll
  for (int d = 0; d < 3; ++d) s[d] = 0.0f + acc.x[d];
  float sp[2] = {0.0f + acc.p[0], 0.0f + acc.p[1]};
  float se[NE > 0 ? NE : 1];
  if constexpr (NE > 0) {
#pragma unroll
    for (unsigned k = 0; k < NE; ++k) se[k] = 0.0f + exd[k];
  }
  if (a.link_off) {
    const unsigned id = a.Bid ? a.Bid[i] : id_of(vi);
    const unsigned e1 = a.link_off[id + 1];
    for (unsigned e = a.link_off[id]; e < e1; ++e) links.template add<D>(a, n, id, xi, pi, e, s, sp, se);
  }
  if constexpr (NE > 0) commit_extras(a, i, se);
  const float sp0 = sp[0], sp1 = sp[1];
  if (a.mode == kStore) {
    a.d_out[i] = make_float4(s[0], s[1], s[2], 0.f);
    if (a.dp_out) a.dp_out[i] = make_float2(sp0, sp1);
    return;
  }
  const float dt = a.dt;
  if (a.mode == kHeun1Fused) {
    a.d_out[i] = make_float4(s[0], s[1], s[2], 0.f);
    a.Xt[i] = make_float4(xi[0] + s[0] * dt, xi[1] + s[1] * dt, xi[2] + s[2] * dt, vi.w);
    if (a.P) {
      a.dp_out[i] = make_float2(sp0, sp1);
      a.Pt[i] = make_float2(pi.x + sp0 * dt, pi.y + sp1 * dt);
    }
    return;
  }
  // kEulerFused / kHeun2Fused: write the next state into A (w = cell id)
  const float4 xb = a.Bx[i];
  const unsigned idb = a.Bid ? a.Bid[i] : id_of(xb);
  float xn[3];
  float2 pn = make_float2(0.f, 0.f);
  if (a.mode == kEulerFused) {
    xn[0] = xb.x + s[0] * dt; xn[1] = xb.y + s[1] * dt; xn[2] = xb.z + s[2] * dt;
    if (a.P) { const float2 pb = a.Bp[i]; pn = make_float2(pb.x + sp0 * dt, pb.y + sp1 * dt); }
  } else {
    const float4 d1 = a.d1[i];
    const float h0 = d1.x + s[0], h1 = d1.y + s[1], h2 = d1.z + s[2];
    xn[0] = xb.x + (h0 * 0.5f) * dt; xn[1] = xb.y + (h1 * 0.5f) * dt; xn[2] = xb.z + (h2 * 0.5f) * dt;
    if (a.P) {
      const float2 pb = a.Bp[i], q1 = a.dp1[i];
      const float g0 = q1.x + sp0, g1 = q1.y + sp1;
      pn = make_float2(pb.x + (g0 * 0.5f) * dt, pb.y + (g1 * 0.5f) * dt);
    }
  }
  if (D < 3) xn[2] = 0.f;
  a.A[i] = make_float4(xn[0], xn[1], xn[2], __uint_as_float(idb));
  if (a.PA) a.PA[i] = pn;
  if (a.count_next) count_cell<D>(g, a, i, xn);
  maybe_divide<D>(g, a, n, idb, xn, pn, a.ctr->step, i);
}

// cell_commit for an active cell, then (every thread of the block) the COM
// partials of kStore.
template <int D, class Links = BuiltinLinks, unsigned NE = 0>
__device__ __forceinline__ void pass_epilogue(const GridP& g, const PassArgs& a, bool active, unsigned n, unsigned i,
                                              const float* xi, const float4& vi, const float2& pi, const Acc& acc,
                                              const Links& links = Links{}, const float* exd = nullptr) {
  float s[3] = {0.f, 0.f, 0.f};
  if (active) cell_commit<D, Links, NE>(g, a, n, i, xi, vi, pi, acc, s, links, exd);
  if (a.mode == kStore && a.com_part)
    com_reduce_block(a, active ? com_fixed(s[0]) : 0ll, active ? com_fixed(s[1]) : 0ll,
                     active ? com_fixed(s[2]) : 0ll);
}


// ---------------------------------------------------------------------------
// Gabriel fast path.
//
// A witness k that blocks the pair (i, j) lies inside the ball of radius
// r = c*d/2 around the midpoint m, and |x_i - m| = d/2, so |x_k - x_i| < d(1+c)/2.
// For c <= 0.9 and d < cutoff that is < 0.95 * cutoff: every witness is itself
// one of i's in-cutoff neighbours, found in i's 27 candidate bins.  The
// cooperative pass (k_pass_gabriel) therefore lists i's in-cutoff neighbours
// (candidate order = the reference's summation order) in shared memory and
// tests each pair against the others, keeping the reference's bin-range
// restriction on k exactly (binned_gabriel.hpp:142-207).  A cell with more
// than kMaxNb neighbours takes the general path.
constexpr int kMaxNb = 24;     // (4 on average at one cell per bin, 12 in packed tissue; a count is a class: at most 31)
// Candidates in a z-plane of the bins around a cell past which it takes the
// general path unwalked: about 33 of 3 x 72 are in cutoff in space (0.155 of
// them) and 25 of 72 in the plane (0.35).  200,000 cells at nine a bin,
// all-pairs, a Heun step: 766 us with every cell walked to the end first, 688 with
// this, 718 with a thread a cell throughout.
constexpr int kCrowd = 72;
constexpr int kPool = 224;     // neighbours of a warp's cells at a time (about 130 at one cell per bin)
// Threads (cells) per block of the passes; of the cooperative pass over the
// grid by the law: the spring laws four warps at 72 registers, so that seven
// blocks (28 warps) share an SM (at 96 threads and nine blocks 136 us a pass of
// 1M cells, here 126; at 64 and 32 threads 138 and 150); the polarity law three
// warps, seven blocks (21 warps at 96 registers): a 100k-cell pass runs in a
// single wave on 152 SMs (six blocks: 53 us, seven 44, four warps 47 to 49).
constexpr int kPassThreads = 96;
template <int FORCE>
constexpr int kCoopThreads = FORCE == 2 ? 96 : 128;
constexpr int kCoopBlocks = 7;  // an SM
// Position arrays that the cooperative pass scans hold this many float4 past
// their capacity: the candidate scan reads rounds of four places past a
// list's end and leaves their bits out.
constexpr unsigned kRowPad = 64;

template <int D, int FINDER, int FORCE>
__device__ __forceinline__ void cell_general(const GridP& g, const ForceP& fp, const PassArgs& a, unsigned n, unsigned i,
                                          const float* xi, float2 pi, unsigned idi, Acc& acc);

template <int D, int FINDER, int FORCE>
static __global__ void __launch_bounds__(kPassThreads) k_pass(GridP g, ForceP fp, PassArgs a) {
  const unsigned n = a.ctr->n;
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < n;
  Acc acc = {{0.f, 0.f, 0.f}, {0.f, 0.f}};
  float xi[3] = {0.f, 0.f, 0.f};
  float4 vi = make_float4(0.f, 0.f, 0.f, 0.f);
  float2 pi = make_float2(0.f, 0.f);
  if (active) {
    vi = a.X[i];
    xi[0] = vi.x; xi[1] = vi.y; xi[2] = vi.z;
    if (a.P) pi = a.P[i];
    const unsigned idi = id_at(a.X, a.Bid, i);
    cell_general<D, FINDER, FORCE>(g, fp, a, n, i, xi, pi, idi, acc);
  }
  pass_epilogue<D>(g, a, active, n, i, xi, vi, pi, acc);
}

// The general path: the reference's loops (27 bins, then the ball's bins per pair).
template <int D, int FINDER, int FORCE>
__device__ __forceinline__ void cell_general(const GridP& g, const ForceP& fp, const PassArgs& a, unsigned n, unsigned i,
                                          const float* xi, float2 pi, unsigned idi, Acc& acc) {
    static_assert(FINDER == 1 || FINDER == 3 || FINDER == 5, "the naive finders run in k_pass_naive");
    if (FINDER == 1 || FINDER == 3) {
      int bc[3] = {0, 0, 0};
      if (FINDER == 1) bin_coords_mul<D>(g, xi, bc);
      else bin_coords_div<D>(g, xi, bc);
      // neighbour bins in the reference's task order (x fastest); each row of
      // bins along x is one contiguous range of the sorted arrays
      const int R = g.R;
      const int z0 = D >= 3 ? -R : 0, z1 = D >= 3 ? R : 0;
      for (int dz = z0; dz <= z1; ++dz) {
        const int cz = D >= 3 ? bc[2] + dz : 0;
        if (D >= 3 && (cz < 0 || cz >= g.ext[2])) continue;
        for (int dy = -R; dy <= R; ++dy) {
          const int cy = bc[1] + dy;
          if (cy < 0 || cy >= g.ext[1]) continue;
          const int x0 = max(bc[0] - R, 0), x1 = min(bc[0] + R, g.ext[0] - 1);
          int c0[3] = {x0, cy, cz}, c1[3] = {x1, cy, cz};
          const unsigned lo = a.off[flatten<D>(g, c0)], hi = a.off[flatten<D>(g, c1) + 1];
          for (unsigned j = lo; j < hi; ++j) {
            if (j == i) continue;
            visit<D, FINDER, FORCE>(g, fp, a, n, i, j, xi, pi, acc, idi);
          }
        }
      }
    } else {
      // FINDER 5: the cell's Delaunay partners, ascending j, each applied reps times
      const unsigned m = a.dl_len[i];
      for (unsigned t = 0; t < m; ++t) {
        const uint2 e = a.dl_row[(size_t)i * kDlRow + t];
        visit<D, FINDER, FORCE>(g, fp, a, n, i, e.x, xi, pi, acc, idi, e.y);
      }
    }
}

// The naive finders' pass (FINDER 0, 2, 4: every j is a candidate), one warp
// per CELLS cells: the lanes test 32 candidates at a time and the in-cutoff
// lanes form their pairs' terms side by side and hand them over in shared
// memory.  Lane 8 c + d adds component d of cell c, in j order -- the
// reference's order, so the sums are those of cell_general bit for bit.  A
// Gabriel pair's witnesses are tested by all lanes.
// What bounds it: instruction issue and L1/L2 reads of the positions.  One
// thread per cell walks the n candidates in one dependent chain and fills 21 of
// 152 SMs at 2,003 cells: 280 us a pass there.  Terms passed on by shuffles,
// every lane adding every term, cost as many instructions a pair as forming it
// takes a warp: with all of 60,013 cells in cutoff 74.8 ms a pass, where one
// thread per cell takes 18.1 and this 12.2.
constexpr int kNaiveThreads = 256;

template <int D, int FINDER, int FORCE, int CELLS>
static __global__ void __launch_bounds__(kNaiveThreads, FINDER == 0 && CELLS == 1 ? 5 : 4) k_pass_naive(GridP g, ForceP fp, PassArgs a) {
  static_assert(FINDER == 0 || FINDER == 2 || FINDER == 4, "the naive finders");
  static_assert(CELLS == 1 || (FINDER == 0 && FORCE != 2), "several cells a warp: all pairs, spring laws");
  const unsigned n = a.ctr->n;
  const unsigned lane = threadIdx.x & 31u;
  const unsigned i0 = (blockIdx.x * (kNaiveThreads / 32) + (threadIdx.x >> 5)) * CELLS;
  float xs[CELLS][3];
  float2 ps[CELLS];
  unsigned ids[CELLS];
#pragma unroll
  for (int c = 0; c < CELLS; ++c) {
    const unsigned i = i0 + c;
    // (a place past the last cell is infinitely far from every cell)
    const float4 v = i < n ? __ldg(&a.X[i]) : make_float4(INFINITY, INFINITY, INFINITY, 0.f);
    xs[c][0] = v.x; xs[c][1] = v.y; xs[c][2] = v.z;
    ids[c] = id_of(v);
    ps[c] = (FORCE == 2 && a.P && i < n) ? a.P[i] : make_float2(0.f, 0.f);
  }
  PolTrig ti[FORCE == 2 ? CELLS : 1];
  if (FORCE == 2)
#pragma unroll
    for (int c = 0; c < CELLS; ++c) ti[c] = pol_trig(ps[c]);
  // A round's terms: for each cell its kTerms components of 32 pairs (the
  // spring's three, with the polarity law also the bending vector and two pairs
  // of angles).  kLine: a component's 32 places, padded so that the lanes that
  // add different components read different banks.
  constexpr int kTerms = FORCE == 2 ? 10 : D, kLine = 36;
  __shared__ __align__(16) float terms_s[FORCE == 0 ? 1 : kNaiveThreads / 32 * CELLS * kTerms * kLine];
  float* const terms = terms_s + (FORCE == 0 ? 0 : (threadIdx.x >> 5) * CELLS * kTerms * kLine);
  const unsigned comp = lane & 7u, of = lane >> 3 < (unsigned)CELLS ? lane >> 3 : 0u;
  // (the components in order: s, bv; bp, al: a polar lane adds two of each pair)
  const float* const first =
      terms + (of * kTerms + (comp < (unsigned)D ? comp : comp < 5u && FORCE == 2 ? comp + 3u : 0u)) * kLine;
  const float* const second = first + (comp < 3u ? 3 : 2) * kLine;  // FORCE 2: added right after
  float own = 0.f;
  constexpr int U = CELLS == 1 && FORCE != 2 ? 4 : 2;  // rounds of 32 candidates in flight
  for (unsigned j0 = 0; j0 < (i0 < n ? n : 0u); j0 += 32u * U) {
    float4 v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned j = j0 + 32u * u + lane;
      v[u] = j < n ? __ldg(&a.X[j]) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const unsigned j = j0 + 32u * u + lane;
      unsigned any = 0u, reps = 1u;  // any: lanes with a pair of one of the cells
      unsigned accepted[CELLS];
      float2 pj = make_float2(0.f, 0.f);
      PolTrig tj{0.f, 0.f, 0.f, 0.f};
      bool have = false;
#pragma unroll
      for (int c = 0; c < CELLS; ++c) {
        const unsigned i = i0 + c;
        accepted[c] = 0u;
        float disp[3] = {xs[c][0] - v[u].x, xs[c][1] - v[u].y, 0.f};
        float d2 = disp[0] * disp[0] + disp[1] * disp[1];
        if (D >= 3) { disp[2] = xs[c][2] - v[u].z; d2 = d2 + disp[2] * disp[2]; }
        bool in = j < n && j != i && !(d2 >= fp.rc2);
        unsigned bits = __ballot_sync(0xffffffffu, in);
        if (!bits) continue;
        if (FINDER == 2) {
          // one in-cutoff pair at a time: a witness in the ball around its midpoint
          unsigned keep = 0u;
          for (unsigned b = bits; b; b &= b - 1u) {
            const int src = __ffs(b) - 1;
            const unsigned jj = j0 + 32u * u + (unsigned)src;
            float m[3] = {0.f, 0.f, 0.f};
#pragma unroll
            for (int d = 0; d < D; ++d) m[d] = xs[c][d] - __shfl_sync(0xffffffffu, disp[d], src) * 0.5f;
            const float rsq = __shfl_sync(0xffffffffu, d2, src) * 0.25f * fp.gab_csq;
            bool blocked = false;
            for (unsigned k0 = 0; k0 < n && !blocked; k0 += 64u) {
              bool hit = false;
#pragma unroll
              for (int w = 0; w < 2; ++w) {
                const unsigned k = k0 + 32u * w + lane;
                if (k < n && k != i && k != jj) {
                  const float4 q = __ldg(&a.X[k]);
                  const float e0 = q.x - m[0], e1 = q.y - m[1];
                  float s = e0 * e0 + e1 * e1;
                  if (D >= 3) { const float e2 = q.z - m[2]; s = s + e2 * e2; }
                  hit = hit || s < rsq;
                }
              }
              blocked = __any_sync(0xffffffffu, hit);
            }
            if (!blocked) keep |= 1u << src;
          }
          bits = keep;
          in = (keep >> lane) & 1u;
        }
        if (FINDER == 4) {
          reps = in ? a.dmult[(size_t)i * a.capacity + j] : 0u;
          in = reps != 0u;
          bits = __ballot_sync(0xffffffffu, in);
        }
        if (!bits) continue;
        accepted[c] = bits;
        any |= bits;
        float s[3] = {0.f, 0.f, 0.f}, bv[3] = {0.f, 0.f, 0.f}, bp[2] = {0.f, 0.f}, al[2] = {0.f, 0.f};
        if (in) {
          if (a.pairs && (CELLS == 1 || i < n)) {
            const unsigned long long at = atomicAdd(&a.ctr->pair_count, (unsigned long long)reps);
            for (unsigned r = 0; r < reps; ++r)
              if (at + r < a.pair_cap) a.pairs[at + r] = make_uint2(ids[c], id_of(v[u]));
          }
          const float dist = sqrtf(d2);
          if (FORCE != 0) spring_term<D>(fp, disp, dist, s);
          if (FORCE == 2) {
            if (!have) {
              if (a.P) pj = a.P[j];
              tj = pol_trig(pj);
              have = true;
            }
            polarity_terms(fp, disp, dist, ps[c], ti[c], pj, tj, bv, bp, al);
          }
        }
        // (the +0 of a lane without a pair, or of a pair at distance zero,
        // leaves a sum unchanged that is never -0)
        float* const t = terms + c * kTerms * kLine + lane;
        if (FORCE != 0)
#pragma unroll
          for (int d = 0; d < D; ++d) t[d * kLine] = s[d];
        if (FORCE == 2) {
#pragma unroll
          for (int d = 0; d < 3; ++d) t[(3 + d) * kLine] = bv[d];
#pragma unroll
          for (int d = 0; d < 2; ++d) {
            t[(6 + d) * kLine] = bp[d];
            t[(8 + d) * kLine] = al[d];
          }
        }
      }
      if constexpr (FORCE != 0) {
        if (!any) continue;
        if (FINDER != 4 && __popc(any) > 8) {
#pragma unroll
          for (int c = 0; c < CELLS; ++c)
            if (CELLS > 1 && !accepted[c])
#pragma unroll
              for (int k = 0; k < kTerms; ++k) terms[(c * kTerms + k) * kLine + lane] = 0.f;
          __syncwarp();
#pragma unroll 2
          for (int src = 0; src < 32; src += 4) {
            const float4 t0 = *reinterpret_cast<const float4*>(first + src);
            const float4 t1 = FORCE == 2 ? *reinterpret_cast<const float4*>(second + src) : t0;
            own = own + t0.x;
            if (FORCE == 2) own = own + t1.x;
            own = own + t0.y;
            if (FORCE == 2) own = own + t1.y;
            own = own + t0.z;
            if (FORCE == 2) own = own + t1.z;
            own = own + t0.w;
            if (FORCE == 2) own = own + t1.w;
          }
        } else {
          // few pairs: the places that one of the cells has, each lane those of its own
          __syncwarp();
          unsigned here = accepted[0];
#pragma unroll
          for (int c = 1; c < CELLS; ++c)
            if (of == (unsigned)c) here = accepted[c];
          for (; any; any &= any - 1u) {
            const int src = __ffs(any) - 1;
            const float t0 = first[src], t1 = FORCE == 2 ? second[src] : 0.f;
            const unsigned rr = FINDER == 4 ? __shfl_sync(0xffffffffu, reps, src) : here >> src & 1u;
            for (unsigned r = 0; r < rr; ++r) {
              own = own + t0;
              if (FORCE == 2) own = own + t1;
            }
          }
        }
        __syncwarp();
      }
    }
  }
  // lane c commits cell c
  Acc mine = {{0.f, 0.f, 0.f}, {0.f, 0.f}};
  if (FORCE != 0) {
#pragma unroll
    for (int d = 0; d < D; ++d) mine.x[d] = __shfl_sync(0xffffffffu, own, (int)(lane & 3u) * 8 + d);
    if (FORCE == 2)
#pragma unroll
      for (int d = 0; d < 2; ++d) mine.p[d] = __shfl_sync(0xffffffffu, own, (int)(lane & 3u) * 8 + 3 + d);
  }
  float2 pi = ps[0];
#pragma unroll
  for (int c = 1; c < CELLS; ++c)
    if (lane == (unsigned)c) pi = ps[c];
  const unsigned i = i0 + lane;
  const bool active = lane < (unsigned)CELLS && i < n;
  const float4 vi = active ? a.X[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  const float xi[3] = {vi.x, vi.y, vi.z};
  if (active && FORCE != 2 && a.P) pi = a.P[i];
  pass_epilogue<D>(g, a, active, n, i, xi, vi, pi, mine);
}

// ---------------------------------------------------------------------------
// User pairwise laws: a PAIRWISE_FORCE lambda or functor compiled into the
// calling program (include/tecs/pairwise.cuh) takes pair_force's place in the
// general pass.  Candidate order, pair predicates, per-cell sums and the
// epilogues (COM, links, fused integrator modes, division) are those of
// k_pass, so a law written like a built-in one gives the built-in's bits.
// Law is a device callable adding the pair (self = i, other = j) to acc:
//   law(a, id_i, id_j, x_i, x_j (w = key or id), displacement x_i - x_j, distance, p_i, p_j, acc)
// with displacement[2] = 0 in 2-D and p = 0 without polarity.  With
// Law::kGeneric it also carries a per-cell (GENERIC_FORCE) law,
//   law.generic(a, id_i, x_i, p_i, g)
// adding to a zero g; the reference evaluates it before the pairwise forces
// (integrators/base.hpp:116-142, kernel_fuser.hpp:148-156), into the cleared
// stage buffer that the pair sums are then added to, so the cell's delta is
// 0 + (g + pair sum) -- the reference's ((0 + g) + pair sum) + 0 bit for bit.

template <int D, int FINDER, class Law>
__device__ __forceinline__ void visit_law(const GridP& g, const ForceP& fp, const PassArgs& a, unsigned n, unsigned i,
                                          unsigned j, const float* xi, float2 pi, Acc& acc,
                                          typename Law::Cell& dacc, unsigned idi, const Law& law,
                                          unsigned reps5 = 1u) {
  const float4 vj = a.X[j];
  float disp[3] = {xi[0] - vj.x, xi[1] - vj.y, D >= 3 ? xi[2] - vj.z : 0.f};
  float d2 = disp[0] * disp[0] + disp[1] * disp[1];
  if (D >= 3) d2 = d2 + disp[2] * disp[2];
  if (d2 >= fp.rc2) return;
  if (FINDER == 3 && gabriel_blocked<D>(g, fp, a.X, a.off, i, j, xi, disp, d2)) return;
  if (FINDER == 2 && gabriel_blocked_naive<D>(fp, a.X, n, i, j, xi, disp, d2)) return;
  // Delaunay: the law is called once per accepted simplex, in j order
  unsigned reps = FINDER == 5 ? reps5 : 1u;
  if (FINDER == 4 && (reps = a.dmult[(size_t)i * a.capacity + j]) == 0u) return;
  const unsigned idj = id_at(a.X, a.Bid, j);
  if (a.pairs) {
    const unsigned long long s = atomicAdd(&a.ctr->pair_count, (unsigned long long)reps);
    for (unsigned r = 0; r < reps; ++r)
      if (s + r < a.pair_cap) a.pairs[s + r] = make_uint2(idi, idj);
  }
  const float dist = sqrtf(d2);
  const float2 pj = a.P ? a.P[j] : make_float2(0.f, 0.f);
  for (unsigned r = 0; r < reps; ++r) law(a, idi, idj, j, xi, vj, disp, dist, pi, pj, acc, dacc);
}

// cell_general's loops with a user law
template <int D, int FINDER, class Law>
__device__ __forceinline__ void cell_law(const GridP& g, const ForceP& fp, const PassArgs& a, unsigned n, unsigned i,
                                         const float* xi, float2 pi, unsigned idi, Acc& acc,
                                         typename Law::Cell& dacc, const Law& law) {
  if (FINDER == 1 || FINDER == 3) {
    int bc[3] = {0, 0, 0};
    if (FINDER == 1) bin_coords_mul<D>(g, xi, bc);
    else bin_coords_div<D>(g, xi, bc);
    const int R = g.R;
    const int z0 = D >= 3 ? -R : 0, z1 = D >= 3 ? R : 0;
    for (int dz = z0; dz <= z1; ++dz) {
      const int cz = D >= 3 ? bc[2] + dz : 0;
      if (D >= 3 && (cz < 0 || cz >= g.ext[2])) continue;
      for (int dy = -R; dy <= R; ++dy) {
        const int cy = bc[1] + dy;
        if (cy < 0 || cy >= g.ext[1]) continue;
        const int x0 = max(bc[0] - R, 0), x1 = min(bc[0] + R, g.ext[0] - 1);
        int c0[3] = {x0, cy, cz}, c1[3] = {x1, cy, cz};
        const unsigned lo = a.off[flatten<D>(g, c0)], hi = a.off[flatten<D>(g, c1) + 1];
        for (unsigned j = lo; j < hi; ++j) {
          if (j == i) continue;
          visit_law<D, FINDER>(g, fp, a, n, i, j, xi, pi, acc, dacc, idi, law);
        }
      }
    }
  } else if (FINDER == 5) {
    const unsigned m = a.dl_len[i];
    for (unsigned t = 0; t < m; ++t) {
      const uint2 e = a.dl_row[(size_t)i * kDlRow + t];
      visit_law<D, FINDER>(g, fp, a, n, i, e.x, xi, pi, acc, dacc, idi, law, e.y);
    }
  } else {
    for (unsigned j = 0; j < n; ++j) {
      if (j == i) continue;
      visit_law<D, FINDER>(g, fp, a, n, i, j, xi, pi, acc, dacc, idi, law);
    }
  }
}

template <int D, int FINDER, class Law>
static __global__ void __launch_bounds__(kPassThreads) k_pass_law(GridP g, ForceP fp, PassArgs a,
                                                                  const Law* __restrict__ lawp) {
  const Law& law = *lawp;
  constexpr unsigned NE = Law::kExtra;
  const unsigned n = a.ctr->n;
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool active = i < n;
  Acc acc = {{0.f, 0.f, 0.f}, {0.f, 0.f}};
  typename Law::Cell cell;
  float xi[3] = {0.f, 0.f, 0.f};
  float4 vi = make_float4(0.f, 0.f, 0.f, 0.f);
  float2 pi = make_float2(0.f, 0.f);
  if (active) {
    vi = a.X[i];
    xi[0] = vi.x; xi[1] = vi.y; xi[2] = vi.z;
    if (a.P) pi = a.P[i];
    const unsigned idi = id_at(a.X, a.Bid, i);
    cell.drag = 0.f;
#pragma unroll
    for (int d = 0; d < 3; ++d) cell.v[d] = 0.f;
    if constexpr (NE > 0) {
#pragma unroll
      for (unsigned k = 0; k < NE; ++k) {
        cell.ex_self[k] = a.EX[k * (size_t)a.capacity + i];
        cell.ex_delta[k] = 0.f;
      }
    }
    cell_law<D, FINDER>(g, fp, a, n, i, xi, pi, idi, acc, cell, law);
    if constexpr (Law::kGeneric) {
      Acc gen = {{0.f, 0.f, 0.f}, {0.f, 0.f}};
      float gex[NE > 0 ? NE : 1] = {};
      law.generic(a, idi, xi, pi, gen, cell.ex_self, gex);
#pragma unroll
      for (int d = 0; d < 3; ++d) acc.x[d] = gen.x[d] + acc.x[d];
      acc.p[0] = gen.p[0] + acc.p[0];
      acc.p[1] = gen.p[1] + acc.p[1];
      if constexpr (NE > 0) {
#pragma unroll
        for (unsigned k = 0; k < NE; ++k) cell.ex_delta[k] = gex[k] + cell.ex_delta[k];
      }
    }
    // out(i) += total_velocity / fmax(total_drag, epsilon), after the pair
    // sums (binned_gabriel.hpp:356-357); with no drag this adds +0
    if constexpr (Law::kPairwise) {
      const float den = fmaxf(cell.drag, FLT_EPSILON);
#pragma unroll
      for (int d = 0; d < D; ++d) acc.x[d] = acc.x[d] + cell.v[d] / den;
    }
  }
  // a LINK_FORCE law evaluates the cell's links in place of the built-in pull
  if constexpr (NE > 0) {
    if constexpr (Law::kLink) pass_epilogue<D, Law, NE>(g, a, active, n, i, xi, vi, pi, acc, law, cell.ex_delta);
    else pass_epilogue<D, BuiltinLinks, NE>(g, a, active, n, i, xi, vi, pi, acc, BuiltinLinks{}, cell.ex_delta);
  } else {
    if constexpr (Law::kLink) pass_epilogue<D>(g, a, active, n, i, xi, vi, pi, acc, law);
    else pass_epilogue<D>(g, a, active, n, i, xi, vi, pi, acc);
  }
}

// One force evaluation handed to a user law's launcher (tecs_sim_set_pair_law).
// size is sizeof(UserPassCall) of the library that filled it: a program built
// against other headers is refused.
struct UserPassCall {
  unsigned size;
  int device;           // the simulation's GPU
  int dims;
  int finder;           // TECS_FINDER_NAIVE_ALL_PAIRS .. TECS_FINDER_DELAUNAY
  unsigned blocks;      // of kPassThreads threads
  GridP g;
  ForceP fp;
  PassArgs a;
};

// Launches the pass of one evaluation with the law, on the library's stream,
// for the finder and dimension count the program was compiled for.  0 on
// success; 1 the call's layout differs; 2 a launch error; 3 the simulation's
// finder or dimension count is not the program's.
// A program compiled for the naive Delaunay finder runs with the Delaunay
// finder of any capacity (FINDER 5) too: the library takes that one past the
// naive finder's capacity.
template <int D, int FINDER, class Law>
int launch_user_pass(const UserPassCall* c, cudaStream_t stream, const Law* law) {
  static_assert(FINDER >= 0 && FINDER <= 5, "user laws run with the all-pairs, Gabriel and Delaunay finders");
  if (!c || c->size != sizeof(UserPassCall)) return 1;
  const bool dl5 = FINDER == 4 && c->finder == 5;
  if (c->dims != D || (c->finder != FINDER && !dl5) || c->a.E != Law::kExtra) return 3;
  int cur = -1;
  if (cudaGetDevice(&cur) != cudaSuccess || (cur != c->device && cudaSetDevice(c->device) != cudaSuccess)) return 2;
  if (dl5) k_pass_law<D, 5, Law><<<c->blocks, kPassThreads, 0, stream>>>(c->g, c->fp, c->a, law);
  else k_pass_law<D, FINDER, Law><<<c->blocks, kPassThreads, 0, stream>>>(c->g, c->fp, c->a, law);
  return cudaGetLastError() == cudaSuccess ? 0 : 2;
}

// Loads the law's pass on the device before the library first launches it,
// which may be while it captures a step graph: 0 on success.
template <int D, int FINDER, class Law>
int prepare_user_pass(int device) {
  cudaFuncAttributes fa;
  if (cudaSetDevice(device) != cudaSuccess) return 2;
  if (FINDER == 4 && cudaFuncGetAttributes(&fa, k_pass_law<D, 5, Law>) != cudaSuccess) return 2;
  return cudaFuncGetAttributes(&fa, k_pass_law<D, FINDER, Law>) == cudaSuccess ? 0 : 2;
}

// ---------------------------------------------------------------------------
// Warp-cooperative pass of the binned finders (spring laws and the 3-D
// polarity law): same pair semantics as cell_general on the fast path's
// geometry, reorganised so that the lanes stay busy.  Its phases and the
// reasons for them stand in pass_gabriel_body.inc.
// FINDER 3: binned Gabriel; FINDER 1: binned all-pairs (i's bin by
// multiplication, binned_all_pairs.hpp:103-109, and every in-cutoff pair
// accepted: no witness test).

// binned_gabriel.hpp:142-153: a witness in the ball (m, r) blocks only from a
// bin of the ball's bin range.
template <int D>
struct BallBins {
  int lo[3], hi[3];
  __device__ __forceinline__ BallBins(const GridP& g, const float* m, float r) {
#pragma unroll
    for (int d = 0; d < D; ++d) {
      lo[d] = clampi((int)floorf((m[d] - r - g.mn[d]) * g.inv_bin), g.ext[d] - 1);
      hi[d] = clampi((int)floorf((m[d] + r - g.mn[d]) * g.inv_bin), g.ext[d] - 1);
    }
  }
  __device__ __forceinline__ bool holds(const GridP& g, unsigned key) const {
    const unsigned row = grid_div(key, g.div_x);
    const int kx = (int)(key - row * (unsigned)g.ext[0]);
    const int kz = D >= 3 ? (int)grid_div(row, g.div_y) : 0;
    const int ky = (int)row - kz * g.ext[1];
    return kx >= lo[0] && kx <= hi[0] && ky >= lo[1] && ky <= hi[1] && (D < 3 || (kz >= lo[2] && kz <= hi[2]));
  }
};

constexpr unsigned kNoRow = 0xffffffffu;

// The slots of n rows of bins [lo, hi), from the bin offsets.
template <int N>
__device__ __forceinline__ void row_slots(const unsigned* __restrict__ off, unsigned* lo, unsigned* hi) {
#pragma unroll
  for (int r = 0; r < N; ++r) {
    const bool ok = lo[r] != kNoRow;
    const unsigned b = lo[r], e = hi[r];
    lo[r] = ok ? __ldg(&off[b]) : 0u;
    hi[r] = ok ? __ldg(&off[e]) : 0u;
  }
}

#define TECS_NO_ROW kNoRow
#define TECS_LOAD(p) __ldg(p)
#define TECS_ROW_SLOTS(N, lo, hi) row_slots<N>(off, lo, hi)
#define TECS_WITNESS (FINDER == 3)
#define TECS_ANY_WITNESS (FINDER == 3)
#define TECS_PAIR_G(c) g
#define TECS_PAIR_FP(c) fp
#define TECS_PAIR_KEY0(c) 0u
#define TECS_SPRING(fpc) (FORCE != 0)
#define TECS_POLAR(fpc) true
#define TECS_CAPTURING (a.pairs != nullptr)
#define TECS_CAPTURE(c, jj)                                                                   \
  if (a.pairs) {                                                                              \
    const unsigned long long s_ = atomicAdd(&a.ctr->pair_count, 1ull);                        \
    if (s_ < a.pair_cap)                                                                      \
      a.pairs[s_] = make_uint2(id_at(a.X, a.Bid, i - (unsigned)lane + (c)), id_at(a.X, a.Bid, (jj))); \
  }
#define TECS_PASS_BODY                                                                        \
  static_assert(FORCE <= 1 || (FORCE == 2 && D == 3), "spring laws, or the 3-D polarity law"); \
  static_assert(FINDER == 1 || FINDER == 3, "the binned finders");                            \
  constexpr bool POL = FORCE == 2;                                                            \
  constexpr int TB = kCoopThreads<FORCE>;                                                     \
  const unsigned n = a.ctr->n;                                                                \
  const unsigned i = blockIdx.x * TB + threadIdx.x;                                           \
  const bool run = i < n;                                                                     \
  const float4* const X = a.X;                                                                \
  const float2* const P = a.P;                                                                \
  const unsigned* const off = a.off;                                                          \
  const float rc2 = fp.rc2;                                                                   \
  float xi[3] = {0.f, 0.f, 0.f};                                                              \
  float4 vi = make_float4(0.f, 0.f, 0.f, 0.f);                                                \
  float2 pi = make_float2(0.f, 0.f);                                                          \
  int bc[3] = {0, 0, 0};                                                                      \
  bool fb = false;                                                                            \
  Acc acc = {{0.f, 0.f, 0.f}, {0.f, 0.f}};                                                    \
  if (run) {                                                                                  \
    vi = __ldg(&X[i]);                                                                        \
    xi[0] = vi.x; xi[1] = vi.y; xi[2] = vi.z;                                                 \
    if (P) pi = P[i];                                                                         \
    if (FINDER == 1) bin_coords_mul<D>(g, xi, bc);                                            \
    else bin_coords_div<D>(g, xi, bc);                                                        \
  }
#define TECS_PASS_END                                                                         \
  if (fb) cell_general<D, FINDER, FORCE>(g, fp, a, n, i, xi, pi, id_at(a.X, a.Bid, i), acc);  \
  pass_epilogue<D>(g, a, run, n, i, xi, vi, pi, acc);

// The grid pass: block blockIdx.x's cells.
template <int D, int FORCE, int FINDER = 3>
static __global__ void __launch_bounds__(kCoopThreads<FORCE>, kCoopBlocks)
    k_pass_gabriel(GridP g, ForceP fp, PassArgs a) {
  TECS_PASS_BODY
#include "pass_gabriel_body.inc"
  TECS_PASS_END
}

// ---------------------------------------------------------------------------
// Euler steps of a small simulation in one launch of one cluster of
// kSmallCtas blocks (up to kSmallCells = 1536 cells and kSmallBins bins; the
// binned finders on the geometry of the cooperative pass, no COM fix, no
// division, no links, no extra fields, built-in laws).
//
// What bounds such a step is the chain of dependent memory round trips and
// barriers, so there are few of either.  Every block reads all cells and
// sorts them by (bin, id) for itself, in shared memory: a coarse histogram of
// the bin numbers, its scan, the cells grouped by it, and each cell's place
// among the few of its group.  The rows' slots come from the
// sorted keys, so no bin counts, offsets or sorted arrays pass between blocks.
// Each block then takes its own share of the cells, a warp a cell (with a lane
// a cell, as in the pass over the grid, the two warps of a share take 24,000
// cycles a step: nothing else runs beside them).  A block writes its cells' new state once
// all blocks have read the old one: they arrive at the cluster's barrier after
// their reads and wait before their writes, a whole pass later.  A second
// barrier ends a step, and the next one follows in the same launch.
// The arithmetic is that of the passes over the grid: bit-identical runs.
// 1000 cells, all-pairs: 25 -> 8.1 us a step (counts, scan, scatter and gather
// through global memory between four cluster barriers, one launch a step: 21;
// over the grid: 23).
// The cluster size is set at launch (16 blocks: past the portable 8, opted
// into per kernel).
constexpr int kSmallCtas = 16;
constexpr int kSmallShare = 96;  // cells of a block, at most
constexpr unsigned kSmallCells = kSmallCtas * kSmallShare;
constexpr unsigned kSmallBins = 16384;
constexpr int kSmallThreads = 1024;
constexpr unsigned kSmallGroups = 2048;                         // of the coarse histogram, four a thread of the scan
constexpr unsigned kSmallNear = 64;                             // neighbours of a cell
constexpr int kSmallPer = (int)((kSmallCells + kSmallThreads - 1) / kSmallThreads);  // cells per thread of the sort
static_assert(kSmallCells <= 2048 && kSmallGroups / 4 <= kSmallThreads, "cells and slots in 11 bits");

// A block's shared memory beside the pass's own.
struct SmallScratch {
  float4 x[kSmallCells];                      // sorted positions, w = bin key
  float2 p[kSmallCells];
  unsigned long long group[kSmallCells];      // (bin << 22 | id << 11 | slot) grouped by the histogram
  unsigned key[kSmallCells], id[kSmallCells]; // sorted
  __align__(16) unsigned coarse[kSmallGroups + 4];  // start of each group
  unsigned wsum[kSmallThreads / 32];
  uint2 rows[kSmallShare * 9];                // the share's rows of bins: their slots
  float4 near[kSmallThreads / 32][kSmallNear];
  Acc acc[kSmallShare];                       // the share's sums
  unsigned crowded, list[kSmallShare];        // cells of more neighbours than a list holds
};

// The arrive half of the cluster's barrier and the wait half.
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

// The first of the sorted keys not below b: in b's group.
__device__ __forceinline__ unsigned first_key(const SmallScratch& sm, unsigned shift, unsigned b) {
  unsigned e = sm.coarse[b >> shift];
  const unsigned end = sm.coarse[(b >> shift) + 1u];
  while (e < end && sm.key[e] < b) ++e;
  return e;
}

// A cell's rows as one list of candidates: lane r's row is the places up to
// end, at slots base further on.
__device__ __forceinline__ void small_rows(const uint2* rows, int n, unsigned& end, unsigned& base) {
  const unsigned lane = threadIdx.x & 31u;
  const uint2 row = lane < (unsigned)n ? rows[lane] : make_uint2(0u, 0u);
  end = row.y - row.x;
#pragma unroll
  for (int o = 1; o < 16; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, end, o);
    if (lane >= (unsigned)o) end += y;
  }
  base = row.y - end;
}

// A cell of more neighbours than the list holds, by one warp: a lane a
// candidate, 32 at a time; a pair's witnesses are looked for among all the
// candidates (row by row, each read by all lanes at once), and the terms added in
// candidate order.
// What bounds it: instruction issue, (candidates / 32) x candidates x about 14.
// A thread a cell over the general path (each pair's witnesses one after
// another, three warps a block) takes 20.5 ms a step for 1,500 cells in a ball
// of radius 1.5, where this takes 1.
template <int D, int FINDER, int FORCE>
__device__ __forceinline__ void small_cell_crowded(const GridP& g, const ForceP& fp, const SmallScratch& sm, unsigned i,
                                                   const uint2* rows, float4* near, Acc& acc) {
  constexpr int kRows = D >= 3 ? 9 : 3;
  const unsigned lane = threadIdx.x & 31u;
  acc = Acc{{0.f, 0.f, 0.f}, {0.f, 0.f}};
  unsigned end, base;
  small_rows(rows, kRows, end, base);
  const unsigned total = __shfl_sync(0xffffffffu, end, kRows - 1);
  const float4 h = sm.x[i];
  PolTrig ti{0.f, 0.f, 0.f, 0.f};
  float2 pi = make_float2(0.f, 0.f);
  if (FORCE == 2) {
    pi = sm.p[i];
    ti = pol_trig(pi);
  }
  float sum = 0.f;  // of component `lane`
  for (unsigned t0 = 0u; t0 < total; t0 += 32u) {
    const unsigned t = t0 + lane;
    unsigned r = 0u;
#pragma unroll
    for (int k = 0; k < kRows - 1; ++k) r += t >= __shfl_sync(0xffffffffu, end, k) ? 1u : 0u;
    const unsigned j = t + __shfl_sync(0xffffffffu, base, (int)r);
    const float4 v = t < total ? sm.x[j] : h;
    float disp[3] = {h.x - v.x, h.y - v.y, D >= 3 ? h.z - v.z : 0.f};
    float d2 = disp[0] * disp[0] + disp[1] * disp[1];
    if (D >= 3) d2 = d2 + disp[2] * disp[2];
    bool open = t < total && j != i && d2 < fp.rc2;
    if (!__any_sync(0xffffffffu, open)) continue;
    if (FINDER == 3) {
      const float m[3] = {h.x - disp[0] * 0.5f, h.y - disp[1] * 0.5f, D >= 3 ? h.z - disp[2] * 0.5f : 0.f};
      const float rsq = d2 * fp.gab_factor;
      const BallBins<D> range(g, m, sqrtf(rsq));
      for (int k = 0; k < kRows && __any_sync(0xffffffffu, open); ++k) {
        const unsigned b = __shfl_sync(0xffffffffu, base, k), e1 = __shfl_sync(0xffffffffu, end, k) + b;
        for (unsigned w0 = (k ? __shfl_sync(0xffffffffu, end, k - 1) : 0u) + b; w0 < e1; w0 += 8u) {
          if (!__any_sync(0xffffffffu, open)) break;
          unsigned in = 0u;  // (a row's last witness is tested again in place of those past its end)
#pragma unroll
          for (unsigned u = 0u; u < 8u; ++u) {
            const unsigned w = min(w0 + u, e1 - 1u);
            const float4 vk = sm.x[w];
            const float e0 = vk.x - m[0], f0 = vk.y - m[1];
            float q = e0 * e0 + f0 * f0;
            if (D >= 3) { const float e2 = vk.z - m[2]; q = q + e2 * e2; }
            if (q < rsq && w != i && w != j) in |= 1u << u;
          }
          for (; in && open; in &= in - 1u)
            open = !range.holds(g, sm.key[min(w0 + (unsigned)__ffs(in) - 1u, e1 - 1u)]);
        }
      }
    }
    const float dist = sqrtf(d2);
    float s[3] = {0.f, 0.f, 0.f}, bv[3] = {0.f, 0.f, 0.f}, bp[2] = {0.f, 0.f}, al[2] = {0.f, 0.f};
    if (open) {
      if (FORCE != 0) spring_term<D>(fp, disp, dist, s);
      if (FORCE == 2) {
        const float2 pj = sm.p[j];
        polarity_terms(fp, disp, dist, pi, ti, pj, pol_trig(pj), bv, bp, al);
      }
    }
    if (FORCE == 1) {
      // (lane d adds component d; the other lanes' +0 leave a sum unchanged)
      near[lane] = make_float4(s[0], s[1], s[2], 0.f);
      __syncwarp();
      const float* term = reinterpret_cast<const float*>(near) + (lane < 3u ? lane : 0u);
#pragma unroll 8
      for (int k = 0; k < 32; ++k) sum = sum + term[4 * k];
      __syncwarp();
    }
    for (unsigned m = FORCE == 2 ? __ballot_sync(0xffffffffu, open) : 0u; m; m &= m - 1u) {
      const int k = __ffs(m) - 1;
#pragma unroll
      for (int d = 0; d < D; ++d) acc.x[d] = acc.x[d] + __shfl_sync(0xffffffffu, s[d], k);
#pragma unroll
      for (int d = 0; d < 3; ++d) acc.x[d] = acc.x[d] + __shfl_sync(0xffffffffu, bv[d], k);
#pragma unroll
      for (int d = 0; d < 2; ++d) acc.p[d] = acc.p[d] + __shfl_sync(0xffffffffu, bp[d], k);
#pragma unroll
      for (int d = 0; d < 2; ++d) acc.p[d] = acc.p[d] + __shfl_sync(0xffffffffu, al[d], k);
    }
  }
  if (FORCE == 1)
#pragma unroll
    for (int d = 0; d < 3; ++d) acc.x[d] = __shfl_sync(0xffffffffu, sum, d);
}

// One cell's sums by one warp: its candidates 32 at a time, a lane each; the
// in-cutoff ones listed in candidate order; a lane a pair for the witness test
// and the terms, which every lane then adds in that order.  False: more
// neighbours than the list holds.
template <int D, int FINDER, int FORCE>
__device__ __forceinline__ bool small_cell(const GridP& g, const ForceP& fp, const SmallScratch& sm, unsigned i,
                                           const uint2* rows, float4* near, Acc& acc) {
  constexpr int kRows = D >= 3 ? 9 : 3;
  const unsigned lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  acc = Acc{{0.f, 0.f, 0.f}, {0.f, 0.f}};
  const float4 h = sm.x[i];
  unsigned end, base;
  small_rows(rows, kRows, end, base);
  const unsigned total = __shfl_sync(0xffffffffu, end, kRows - 1);
  unsigned cnt = 0u;
  for (unsigned t0 = 0u; t0 < total; t0 += 32u) {
    const unsigned t = t0 + lane;
    unsigned r = 0u;
#pragma unroll
    for (int k = 0; k < kRows - 1; ++k) r += t >= __shfl_sync(0xffffffffu, end, k) ? 1u : 0u;
    const unsigned j = t + __shfl_sync(0xffffffffu, base, (int)r);
    bool in = false;
    float4 v = h;
    if (t < total) {
      v = sm.x[j];
      const float e0 = h.x - v.x, e1 = h.y - v.y;
      float d2 = e0 * e0 + e1 * e1;
      if (D >= 3) { const float e2 = h.z - v.z; d2 = d2 + e2 * e2; }
      in = d2 < fp.rc2 && j != i;
    }
    const unsigned m = __ballot_sync(0xffffffffu, in);
    const unsigned at = cnt + (unsigned)__popc(m & below);
    if (in && at < kSmallNear) near[at] = make_float4(v.x, v.y, v.z, __uint_as_float(j));
    cnt += (unsigned)__popc(m);
  }
  if (cnt > kSmallNear) return false;
  __syncwarp();
  PolTrig ti{0.f, 0.f, 0.f, 0.f};
  float2 pi = make_float2(0.f, 0.f);
  if (FORCE == 2) {
    pi = sm.p[i];
    ti = pol_trig(pi);
  }
  for (unsigned q0 = 0u; q0 < cnt; q0 += 32u) {
    const unsigned q = q0 + lane;
    const bool act = q < cnt;
    const float4 vj = near[act ? q : 0u];
    float disp[3] = {h.x - vj.x, h.y - vj.y, D >= 3 ? h.z - vj.z : 0.f};
    float d2 = disp[0] * disp[0] + disp[1] * disp[1];
    if (D >= 3) d2 = d2 + disp[2] * disp[2];
    bool blocked = !act;
    if (FINDER == 3 && cnt > 1u) {
      const float m[3] = {h.x - disp[0] * 0.5f, h.y - disp[1] * 0.5f, D >= 3 ? h.z - disp[2] * 0.5f : 0.f};
      const float rsq = d2 * fp.gab_factor;
      unsigned long long in = 0ull;
      for (unsigned w = 0u; w < cnt; ++w) {
        const float4 vk = near[w];
        const float e0 = vk.x - m[0], e1 = vk.y - m[1];
        float s = e0 * e0 + e1 * e1;
        if (D >= 3) { const float e2 = vk.z - m[2]; s = s + e2 * e2; }
        if (s < rsq && w != q) in |= 1ull << w;
      }
      if (act && in) {
        const BallBins<D> range(g, m, sqrtf(rsq));
        for (; in && !blocked; in &= in - 1ull)
          blocked = range.holds(g, sm.key[__float_as_uint(near[__ffsll((long long)in) - 1].w)]);
      }
    }
    const float dist = sqrtf(d2);
    float s[3] = {0.f, 0.f, 0.f}, bv[3] = {0.f, 0.f, 0.f}, bp[2] = {0.f, 0.f}, al[2] = {0.f, 0.f};
    if (!blocked) {
      if (FORCE != 0) spring_term<D>(fp, disp, dist, s);
      if (FORCE == 2) {
        const float2 pj = sm.p[__float_as_uint(vj.w)];
        polarity_terms(fp, disp, dist, pi, ti, pj, pol_trig(pj), bv, bp, al);
      }
    }
    if (FORCE == 1 && cnt <= 32u) {
      // (all witnesses have been read: the terms take the list's places, a
      // blocked pair's +0 leaving the sum, which is never -0, unchanged; lane d
      // adds component d)
      __syncwarp();
      if (act) near[q] = make_float4(s[0], s[1], s[2], 0.f);
      __syncwarp();
      float sum = 0.f;
      const float* term = reinterpret_cast<const float*>(near) + (lane < 3u ? lane : 0u);
      for (unsigned k = 0u; k < cnt; ++k) sum = sum + term[4u * k];
#pragma unroll
      for (int d = 0; d < 3; ++d) acc.x[d] = __shfl_sync(0xffffffffu, sum, d);
      __syncwarp();
      return true;
    }
    for (unsigned m = __ballot_sync(0xffffffffu, !blocked); m && FORCE != 0; m &= m - 1u) {
      const int k = __ffs(m) - 1;
#pragma unroll
      for (int d = 0; d < D; ++d) acc.x[d] = acc.x[d] + __shfl_sync(0xffffffffu, s[d], k);
      if (FORCE == 2) {
#pragma unroll
        for (int d = 0; d < 3; ++d) acc.x[d] = acc.x[d] + __shfl_sync(0xffffffffu, bv[d], k);
#pragma unroll
        for (int d = 0; d < 2; ++d) acc.p[d] = acc.p[d] + __shfl_sync(0xffffffffu, bp[d], k);
#pragma unroll
        for (int d = 0; d < 2; ++d) acc.p[d] = acc.p[d] + __shfl_sync(0xffffffffu, al[d], k);
      }
    }
  }
  return true;
}

template <int D, int FINDER, int FORCE>
static __global__ void __launch_bounds__(kSmallThreads)
    k_step_small(GridP g, ForceP fp, PassArgs p1, int steps, const float4* A, const float2* PA, float4* B, float2* PB,
                 unsigned* Bid, unsigned* off_out) {
  static_assert(FORCE <= 1 || (FORCE == 2 && D == 3), "spring laws, or the 3-D polarity law");
  extern __shared__ __align__(16) unsigned char small_smem[];
  SmallScratch& sm = *reinterpret_cast<SmallScratch*>(small_smem);
  const unsigned n = p1.ctr->n, tid = threadIdx.x;
  // the block's share: whole warps of cells, spread over the blocks
  const unsigned share = ((n + kSmallCtas - 1) / kSmallCtas + 31u) & ~31u;
  const unsigned i0 = min(n, blockIdx.x * share), i1 = min(n, i0 + share);
  unsigned shift = 0u;
  while ((g.nbins >> shift) >= kSmallGroups) ++shift;
  for (int step = 0; step < steps; ++step) {
    // 1. every block: all cells, counted into groups of bins
    for (unsigned k = tid; k <= kSmallGroups; k += kSmallThreads) sm.coarse[k] = 0u;
    float4 v[kSmallPer];
    unsigned bin[kSmallPer], at[kSmallPer];
#pragma unroll
    for (int k = 0; k < kSmallPer; ++k) {
      const unsigned c = tid + k * kSmallThreads;
      if (c < n) v[k] = __ldcg(&A[c]);
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSmallPer; ++k) {
      const unsigned c = tid + k * kSmallThreads;
      if (c < n) {
        const float q[3] = {v[k].x, v[k].y, v[k].z};
        int b3[3] = {0, 0, 0};
        bin_coords_div<D>(g, q, b3);
        bin[k] = flatten<D>(g, b3);
        at[k] = atomicAdd(&sm.coarse[bin[k] >> shift], 1u);
      }
    }
    __syncthreads();
    // 2. exclusive scan of the groups' counts, four a thread
    {
      const int lane = tid & 31, warp = tid >> 5;
      const bool part = 4u * tid < kSmallGroups;
      uint4 c = make_uint4(0u, 0u, 0u, 0u);
      if (part) c = *reinterpret_cast<const uint4*>(&sm.coarse[4u * tid]);
      const unsigned own = (c.x + c.y) + (c.z + c.w);
      unsigned incl = own;
      if (part) {  // whole warps
        for (int o = 1; o < 32; o <<= 1) {
          const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        if (lane == 31) sm.wsum[warp] = incl;
      }
      __syncthreads();
      if (part) {
        const unsigned before = __reduce_add_sync(0xffffffffu, lane < warp ? sm.wsum[lane] : 0u) + incl - own;
        const uint4 e = make_uint4(before, before + c.x, before + c.x + c.y, before + c.x + c.y + c.z);
        *reinterpret_cast<uint4*>(&sm.coarse[4u * tid]) = e;
        if (4u * tid + 4u == kSmallGroups) sm.coarse[kSmallGroups] = e.w + c.w;
      }
    }
    __syncthreads();
    // 3. the cells grouped, 4. each one's place by (bin, id)
#pragma unroll
    for (int k = 0; k < kSmallPer; ++k) {
      const unsigned c = tid + k * kSmallThreads;
      if (c < n)
        sm.group[sm.coarse[bin[k] >> shift] + at[k]] =
            (unsigned long long)bin[k] << 22 | (unsigned long long)id_of(v[k]) << 11 | c;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kSmallPer; ++k) {
      const unsigned c = tid + k * kSmallThreads;
      if (c < n) {
        const unsigned q = bin[k] >> shift, lo = sm.coarse[q], hi = sm.coarse[q + 1u];
        const unsigned long long me = (unsigned long long)bin[k] << 22 | (unsigned long long)id_of(v[k]) << 11 | c;
        unsigned dst = lo;
        for (unsigned e = lo; e < hi; ++e) dst += sm.group[e] < me ? 1u : 0u;
        sm.x[dst] = make_float4(v[k].x, v[k].y, v[k].z, __uint_as_float(bin[k]));
        sm.key[dst] = bin[k];
        sm.id[dst] = id_of(v[k]);
        if (PA) sm.p[dst] = __ldcg(&PA[c]);
      }
    }
    __syncthreads();
    cluster_arrive();  // this block has read the state
    // the sorted copy, by shares
    for (unsigned s = i0 + tid; s < i1; s += kSmallThreads) {
      B[s] = sm.x[s];
      Bid[s] = sm.id[s];
      if (PB) PB[s] = sm.p[s];
    }
    // 5. the slots of the rows of bins around the share's cells
    constexpr int kRows = D >= 3 ? 9 : 3;
    const unsigned cells = i1 - i0;
    if (tid == 0) sm.crowded = 0u;
    for (unsigned q = tid; q < cells * kRows; q += kSmallThreads) {
      const unsigned r = q % kRows;
      const float4 v4 = sm.x[i0 + q / kRows];
      const float q3[3] = {v4.x, v4.y, v4.z};
      int bc[3] = {0, 0, 0};
      if (FINDER == 1) bin_coords_mul<D>(g, q3, bc);
      else bin_coords_div<D>(g, q3, bc);
      const int cy = bc[1] + (int)(r % 3u) - 1, cz = D >= 3 ? bc[2] + (int)(r / 3u) - 1 : 0;
      unsigned lo = 0u, hi = 0u;
      if (cy >= 0 && cy < g.ext[1] && (D < 3 || (cz >= 0 && cz < g.ext[2]))) {
        int c0[3] = {max(bc[0] - 1, 0), cy, cz}, c1[3] = {min(bc[0] + 1, g.ext[0] - 1), cy, cz};
        lo = first_key(sm, shift, flatten<D>(g, c0));
        hi = first_key(sm, shift, flatten<D>(g, c1) + 1u);
      }
      sm.rows[q] = make_uint2(lo, hi);
    }
    __syncthreads();
    // 6. the cells' forces, one warp a cell
    for (unsigned c = tid >> 5; c < cells; c += kSmallThreads / 32) {
      Acc acc;
      const bool ok = small_cell<D, FINDER, FORCE>(g, fp, sm, i0 + c, sm.rows + c * kRows, sm.near[tid >> 5], acc);
      if ((tid & 31u) == 0u) {
        if (!ok) sm.list[atomicAdd(&sm.crowded, 1u)] = c;
        sm.acc[c] = acc;
      }
    }
    __syncthreads();
    if (sm.crowded) {
      for (unsigned q = tid >> 5; q < sm.crowded; q += kSmallThreads / 32) {
        const unsigned c = sm.list[q];
        Acc acc;
        small_cell_crowded<D, FINDER, FORCE>(g, fp, sm, i0 + c, sm.rows + c * kRows, sm.near[tid >> 5], acc);
        if ((tid & 31u) == 0u) sm.acc[c] = acc;
      }
      __syncthreads();
    }
    // the bin offsets, for later steps that keep this sort
    if (off_out && blockIdx.x == 0)
      for (unsigned b = tid; b <= g.nbins; b += kSmallThreads) off_out[b] = first_key(sm, shift, b);
    PassArgs a = p1;
    a.X = sm.x;
    a.Bx = sm.x;
    a.P = PA ? sm.p : nullptr;
    a.Bp = a.P;
    a.Bid = sm.id;
    cluster_wait();  // every block has read the state
    if (tid < cells) {
      const unsigned i = i0 + tid;
      const float4 vi = sm.x[i];
      const float xi[3] = {vi.x, vi.y, vi.z};
      float s3[3];
      cell_commit<D>(g, a, n, i, xi, vi, PA ? sm.p[i] : make_float2(0.f, 0.f), sm.acc[tid], s3);
    }
    if (step + 1 < steps) {
      __syncwarp();
      cluster_arrive();
      cluster_wait();
    }
  }
}
#undef TECS_NO_ROW
#undef TECS_LOAD
#undef TECS_ROW_SLOTS
#undef TECS_WITNESS
#undef TECS_ANY_WITNESS
#undef TECS_PAIR_G
#undef TECS_PAIR_FP
#undef TECS_PAIR_KEY0
#undef TECS_SPRING
#undef TECS_POLAR
#undef TECS_CAPTURING
#undef TECS_CAPTURE
#undef TECS_PASS_BODY
#undef TECS_PASS_END

// Symmetric finders (…_symmetric.hpp): only j with a smaller id, +delta to the
// evaluating cell and -delta to j for every field.  Float atomics: the
// accumulation order is not fixed, results agree to rounding.
template <int D, int FINDER, int FORCE>
static __global__ void __launch_bounds__(128) k_pass_sym(GridP g, ForceP fp, PassArgs a) {
  const unsigned n = a.ctr->n;
  const unsigned i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float4 vi = a.X[i];
  const float xi[3] = {vi.x, vi.y, vi.z};
  const float2 pi = a.P ? a.P[i] : make_float2(0.f, 0.f);
  const unsigned idi = id_at(a.X, a.Bid, i);
  auto one = [&](unsigned j) {
    if (id_at(a.X, a.Bid, j) >= idi) return;
    Acc acc = {{0.f, 0.f, 0.f}, {0.f, 0.f}};
    const unsigned long long before = a.pairs ? 1ull : 0ull;
    (void)before;
    // pair (self = i, other = j)
    const float4 vj = a.X[j];
    float disp[3];
    disp[0] = xi[0] - vj.x;
    disp[1] = xi[1] - vj.y;
    disp[2] = D >= 3 ? xi[2] - vj.z : 0.f;
    float d2 = disp[0] * disp[0] + disp[1] * disp[1];
    if (D >= 3) d2 = d2 + disp[2] * disp[2];
    if (d2 >= fp.rc2) return;
    if (FINDER == 3 && gabriel_blocked<D>(g, fp, a.X, a.off, i, j, xi, disp, d2)) return;
    if (FINDER == 2 && gabriel_blocked_naive<D>(fp, a.X, n, i, j, xi, disp, d2)) return;
    if (a.pairs) {
      unsigned long long s = atomicAdd(&a.ctr->pair_count, 1ull);
      if (s < a.pair_cap) a.pairs[s] = make_uint2(idi, id_at(a.X, a.Bid, j));
    }
    const float dist = sqrtf(d2);
    const float2 pj = (FORCE == 2 && a.P) ? a.P[j] : make_float2(0.f, 0.f);
    pair_force<D, FORCE>(fp, disp, dist, pi, pj, acc);
    for (int d = 0; d < D; ++d) {
      atomicAdd(&((float*)&a.d_out[i])[d], acc.x[d]);
      atomicAdd(&((float*)&a.d_out[j])[d], -acc.x[d]);
    }
    if (a.dp_out) {
      atomicAdd(&a.dp_out[i].x, acc.p[0]); atomicAdd(&a.dp_out[i].y, acc.p[1]);
      atomicAdd(&a.dp_out[j].x, -acc.p[0]); atomicAdd(&a.dp_out[j].y, -acc.p[1]);
    }
  };
  if (FINDER == 1 || FINDER == 3) {
    int bc[3] = {0, 0, 0};
    bin_coords_div<D>(g, xi, bc);
    const int R = g.R;
    const int z0 = D >= 3 ? -R : 0, z1 = D >= 3 ? R : 0;
    for (int dz = z0; dz <= z1; ++dz) {
      const int cz = D >= 3 ? bc[2] + dz : 0;
      if (D >= 3 && (cz < 0 || cz >= g.ext[2])) continue;
      for (int dy = -R; dy <= R; ++dy) {
        const int cy = bc[1] + dy;
        if (cy < 0 || cy >= g.ext[1]) continue;
        const int x0 = max(bc[0] - R, 0), x1 = min(bc[0] + R, g.ext[0] - 1);
        int c0[3] = {x0, cy, cz}, c1[3] = {x1, cy, cz};
        const unsigned lo = a.off[flatten<D>(g, c0)], hi = a.off[flatten<D>(g, c1) + 1];
        for (unsigned j = lo; j < hi; ++j) one(j);
      }
    }
  } else {
    for (unsigned j = 0; j < n; ++j) one(j);
  }
}

// Plain COM reduction over a delta buffer (used after the symmetric pass).
static __global__ void k_com(const float4* __restrict__ d, PassArgs a) {
  const unsigned n = a.ctr->n;
  long long x = 0, y = 0, z = 0;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 v = d[i];
    x += com_fixed(v.x); y += com_fixed(v.y); z += com_fixed(v.z);
  }
  com_reduce_block(a, x, y, z);
}

// ---------------------------------------------------------------------------
// integrator epilogues when the COM fix (or the symmetric finder) forbids
// fusing them into the pass

// heun.hpp:54-68: d1' = d1 - c1; x~ = x + d1' * dt (every field).  d1' is not
// stored: the corrector forms it again with the same operations.
static __global__ void k_predict(const Counters* __restrict__ ctr, const float* __restrict__ com, float dt,
                          const float4* __restrict__ B, const float2* __restrict__ PB, const float4* __restrict__ d1,
                          const float2* __restrict__ dp1, float4* __restrict__ Xt, float2* __restrict__ Pt,
                          PassArgs ex) {
  const unsigned n = ctr->n;
  const float c0 = com[0], c1 = com[1], c2 = com[2];
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    // the extra fields' predictor: x~ = x + d1 * dt (no COM fix: it acts on
    // the first field only)
    for (unsigned k = 0; k < ex.E; ++k) {
      const size_t at = k * (size_t)ex.capacity + i;
      ex.Et[at] = ex_update(ex.EBx[at], ex.ed1[at], dt, ex.dt64, (ex.ex_dbl >> k) & 1u);
    }
    float4 v = d1[i];
    v.x = v.x - c0; v.y = v.y - c1; v.z = v.z - c2;  // d1 - c1 (re-formed by k_finish)
    const float4 x = B[i];
    Xt[i] = make_float4(x.x + v.x * dt, x.y + v.y * dt, x.z + v.z * dt, x.w);
    if (Pt) {
      const float2 p = PB[i], q = dp1[i];
      Pt[i] = make_float2(p.x + q.x * dt, p.y + q.y * dt);
    }
  }
}

// heun.hpp:78-98 (corrector) and euler.hpp:49-69 with the COM subtraction,
// the old velocities when the simulation keeps them, plus division.  Heun: s = d1 + (d2 - c); x += (s * 0.5) * dt.
// Euler:  s = d1 - c; x += s * dt.
template <int D>
static __global__ void k_finish(int heun, GridP g, PassArgs a, const float* __restrict__ com, const float4* __restrict__ d2,
                         const float2* __restrict__ dp2) {
  const unsigned n = a.ctr->n;
  // Euler: com = c (slot 0).  Heun: com = c1 (slot 0), com + 4 = c2 (slot 1)
  const float c0 = com[heun ? 4 : 0], c1 = com[heun ? 5 : 1], c2 = com[heun ? 6 : 2];
  const float p0 = com[0], p1 = com[1], p2 = com[2];
  const float dt = a.dt;
  const unsigned long long step = a.ctr->step;
  for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float4 xb = a.Bx[i];
    const float4 v1 = a.d1[i];
    float xn[3];
    float2 pn = make_float2(0.f, 0.f);
    if (heun) {
      const float4 v2 = d2[i];
      const float f0 = v1.x - p0, f1 = v1.y - p1, f2 = v1.z - p2;  // d1 - c1 (predictor)
      const float e0 = v2.x - c0, e1 = v2.y - c1, e2 = v2.z - c2;  // d2 - c2 (corrector)
      const float h0 = f0 + e0, h1 = f1 + e1, h2 = f2 + e2;
      xn[0] = xb.x + (h0 * 0.5f) * dt; xn[1] = xb.y + (h1 * 0.5f) * dt; xn[2] = xb.z + (h2 * 0.5f) * dt;
      // old_velocities(i) = (d1' + d2') * 0.5 (heun.hpp:87)
      if (a.old_vel) a.old_vel[a.Bid ? a.Bid[i] : id_of(xb)] = make_float4(h0 * 0.5f, h1 * 0.5f, h2 * 0.5f, 0.f);
      if (a.PA) {
        const float2 pb = a.Bp[i], q1 = a.dp1[i], q2 = dp2[i];
        const float g0 = q1.x + q2.x, g1 = q1.y + q2.y;
        pn = make_float2(pb.x + (g0 * 0.5f) * dt, pb.y + (g1 * 0.5f) * dt);
      }
    } else {
      const float e0 = v1.x - c0, e1 = v1.y - c1, e2 = v1.z - c2;
      xn[0] = xb.x + e0 * dt; xn[1] = xb.y + e1 * dt; xn[2] = xb.z + e2 * dt;
      // old_velocities(i) = d1' (euler.hpp:59)
      if (a.old_vel) a.old_vel[a.Bid ? a.Bid[i] : id_of(xb)] = make_float4(e0, e1, e2, 0.f);
      if (a.PA) {
        const float2 pb = a.Bp[i], q1 = a.dp1[i];
        pn = make_float2(pb.x + q1.x * dt, pb.y + q1.y * dt);
      }
    }
    if (D < 3) xn[2] = 0.f;
    const unsigned idb = a.Bid ? a.Bid[i] : id_of(xb);
    a.A[i] = make_float4(xn[0], xn[1], xn[2], __uint_as_float(idb));
    if (a.PA) a.PA[i] = pn;
    // the extra fields: Euler x + d1 dt, Heun x + (d1 + d2) * 0.5 * dt
    for (unsigned k = 0; k < a.E; ++k) {
      const size_t at = k * (size_t)a.capacity + i;
      const bool dbl = (a.ex_dbl >> k) & 1u;
      const float xe = a.EBx[at];
      if (heun) {
        const float h = a.ed1[at] + a.ed2[at];
        a.EA[at] = dbl ? (float)((double)xe + ((double)h * 0.5) * a.dt64) : xe + (h * 0.5f) * dt;
      } else {
        a.EA[at] = ex_update(xe, a.ed1[at], dt, a.dt64, dbl);
      }
    }
    if (a.count_next) count_cell<D>(g, a, i, xn);
    maybe_divide<D>(g, a, n, idb, xn, pn, step, i);
  }
}

}  // namespace tecs
