// common.cuh -- shared device helpers for the TECS cell-step kernels (sm_103a).
//
// Arithmetic that decides which pairs exist (squared distances, midpoints,
// Gabriel radii, bin coordinates) follows the operation order of the
// reference's VectorN code (include/types/vector.hpp) and is compiled with
// -fmad=false, so no multiply-add is contracted and the pair sets agree bit
// for bit with the reference's Serial backend.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <cmath>

namespace tecs {

constexpr float kFltEpsilon = 1.19209290e-7f;  // Kokkos::Experimental::epsilon_v<float>

// Uniform bin grid, include/utils/grid.hpp:71-85 and :201-259.
struct GridP {
  float mn[3];
  float bin_size;   // bin_size_scale * cutoff
  float inv_bin;    // 1 / bin_size
  int ext[3];       // ceil((max - min) / bin_size), 1 for unused dimensions
  int R;            // search radius in bins, ceil(cutoff * inv_bin)
  unsigned nbins;   // product of extents
  uint2 div_x, div_y;  // division of a bin number by ext[0], ext[1] (grid_div)
  int pow2;         // bin_size is a power of two: (p - min) / bin_size == (p - min) * inv_bin exactly
};

// Division of n < 2^31 by an invariant d as a multiplication and a shift
// (Granlund and Montgomery, "Division by Invariant Integers using
// Multiplication", 1994): with s = ceil(log2 d) and m = ceil(2^(31 + s) / d),
// floor(n / d) = (n m) >> (31 + s).
inline uint2 grid_divisor(unsigned d) {
  unsigned s = 0;
  while ((1ull << s) < d) ++s;
  return make_uint2((unsigned)(((1ull << (31 + s)) + d - 1) / d), s);
}
__device__ __forceinline__ unsigned grid_div(unsigned n, uint2 d) { return __umulhi(n << 1, d.x) >> d.y; }

// Sets g.pow2 from g.bin_size and the divisors from the extents (host side,
// after those are set).
// Dividing by 2^k and multiplying by 2^-k round the same real number, so the
// two forms of the bin coordinate agree bit for bit.
inline void grid_set_constants(GridP& g) {
  int e = 0;
  const float m = std::frexp(g.bin_size, &e);
  g.pow2 = (m == 0.5f && g.inv_bin * g.bin_size == 1.0f) ? 1 : 0;
  g.div_x = grid_divisor((unsigned)g.ext[0]);
  g.div_y = grid_divisor((unsigned)g.ext[1]);
}

// Whether float resolves the grid's positions and bins well enough for the
// Gabriel fast path's geometry (kernels.cuh): a witness within 0.95 cutoffs of
// the cell has to be found in cutoff and in the bins around the cell's own.
// Up to 2^18 cutoffs from the origin and 2^18 bins a side, rounding moves a
// midpoint by at most 1/64 of a cutoff and a bin's edges by 1/64 of a bin.
// (At 2^21, five to eleven positions a cutoff, witnesses are missed.)
inline bool grid_resolved(const GridP& g, float cutoff) {
  constexpr float kMost = 262144.0f;
  for (int d = 0; d < 3; ++d) {
    const float hi = g.mn[d] + (float)g.ext[d] * g.bin_size;
    if (!((float)g.ext[d] <= kMost && std::fabs(g.mn[d]) <= kMost * cutoff && std::fabs(hi) <= kMost * cutoff)) return false;
  }
  return true;
}

// Built-in force descriptor plus the pair predicates' constants.
struct ForceP {
  int force;        // tecs_force
  float k_rep, r_rep, k_adh, r_adh, k_pol;
  float rc2;        // cutoff * cutoff
  float gab_factor; // c*c*0.25f  (binned_gabriel.hpp:42)
  float gab_csq;    // c*c        (naive_gabriel.hpp:26)
};

__device__ __forceinline__ int clampi(int v, int hi) { return v < hi ? (v < 0 ? 0 : v) : hi; }

// grid.hpp:222-230: clamp(int((p - min) / bin_size), 0, ext - 1); with a
// power-of-two bin size the division is the (identical) multiplication
template <int D>
__device__ __forceinline__ void bin_coords_div(const GridP& g, const float* p, int* c) {
  if (g.pow2) {
#pragma unroll
    for (int d = 0; d < D; ++d) c[d] = clampi((int)((p[d] - g.mn[d]) * g.inv_bin), g.ext[d] - 1);
  } else {
#pragma unroll
    for (int d = 0; d < D; ++d) c[d] = clampi((int)((p[d] - g.mn[d]) / g.bin_size), g.ext[d] - 1);
  }
}
// binned_all_pairs.hpp:103-109: the same with the inverse bin size
template <int D>
__device__ __forceinline__ void bin_coords_mul(const GridP& g, const float* p, int* c) {
#pragma unroll
  for (int d = 0; d < D; ++d) c[d] = clampi((int)((p[d] - g.mn[d]) * g.inv_bin), g.ext[d] - 1);
}
template <int D>
__device__ __forceinline__ unsigned flatten(const GridP& g, const int* c) {
  unsigned b = (unsigned)c[0];
  if (D >= 2) b += (unsigned)c[1] * (unsigned)g.ext[0];
  if (D >= 3) b += (unsigned)c[2] * ((unsigned)g.ext[0] * (unsigned)g.ext[1]);
  return b;
}

// Two floats in one 64-bit register (the low one first); the packed
// operations round each half as the scalar ones do.
__device__ __forceinline__ unsigned long long f32x2_pack(float lo, float hi) {
  return (unsigned long long)__float_as_uint(lo) | ((unsigned long long)__float_as_uint(hi) << 32);
}
__device__ __forceinline__ float f32x2_lo(unsigned long long v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float f32x2_hi(unsigned long long v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ unsigned long long f32x2_sub(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ unsigned long long f32x2_mul(unsigned long long a, unsigned long long b) {
  unsigned long long r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}

__device__ __forceinline__ unsigned id_of(const float4& v) { return __float_as_uint(v.w); }

// Counter-based RNG keyed by (seed, step, cell id, stream).  SplitMix64's
// finaliser (Steele, Lea & Flood 2014) applied twice.
__host__ __device__ __forceinline__ uint64_t mix64(uint64_t z) {
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
__host__ __device__ __forceinline__ uint64_t hash64(uint64_t seed, uint64_t step, uint64_t cell, uint64_t stream) {
  uint64_t k = step * 0x9E3779B97F4A7C15ull + cell * 0xD1B54A32D192ED03ull + stream * 0x94D049BB133111EBull + 1ull;
  return mix64(seed ^ mix64(k));
}
__host__ __device__ __forceinline__ double u01(uint64_t h) { return (double)(h >> 11) * (1.0 / 9007199254740992.0); }

}  // namespace tecs
