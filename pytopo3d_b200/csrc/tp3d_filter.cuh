// Cone density filter as ring sums marched along z.
//
// The reference builds an explicit sparse H with weights rmin - |d| for
// integer offsets d with rmin - |d| > 1e-9, truncated at the domain boundary
// (pytopo3d/utils/filter.py:122-228).  H is symmetric, so H x and H^T g are the
// same stencil.  Here H is never formed.  The weight of an offset depends on
// dx^2 + dy^2 and |dz| only, so a plane's contribution to the outputs at
// distance a above and below it is the same number
//     S_a = sum over rings c of w(c, a) R_c,   R_c = sum of the plane's values
//     at the (dx, dy) with dx^2 + dy^2 = d2(c),
// and an output is the sum of its planes' S.  A block owns 32 x 8 columns (one
// per thread) and marches along z: it stages one plane of the input with its
// halo in shared memory (double-buffered, the next plane's loads in flight;
// zero outside the domain, which reproduces the boundary truncation), forms
// the ring sums with offsets that are compile-time constants, and adds S_a to
// the 2Z + 1 outputs in progress, which live in registers.
//
// Bound by shared-memory loads (one 8-byte load per column of the disc, output
// and thread) and instruction issue (46-54% busy at 128x64x64, rmin 3).  Per
// output at rmin 4.5 that is 57 loads and 111 FP64 operations; the
// column-by-column stencil it replaces (8 outputs per thread along z) took 178
// loads and 513 multiply-adds.  Filter and projection: 256x128x128 at rmin 4.5
// 285 us before, 160 now; 128x64x64 at rmin 3 21 and 17.  Two outputs per thread
// in y (16-byte loads, half the threads) measured the same at rmin 3 and slower
// from rmin 4.5 on, where its registers spill.
#pragma once

#include <algorithm>
#include <utility>

#include "tp3d_common.cuh"

namespace tp3d {

constexpr int kFilterTY = 32;   // outputs along y per block (one warp)
constexpr int kFilterTX = 8;    // outputs along x per block (warps per block)
constexpr int kFilterThreads = kFilterTY * kFilterTX;
constexpr int kFilterMaxZ = 6;  // supports rmin <= 7

// Largest offset along one axis with a positive cone weight: the largest d with
// rmin - d > 1e-9 (pytopo3d/utils/filter.py:193-206).  -1 for an invalid rmin.
inline int filter_radius_z(double rmin) {
  if (!(rmin > 0.0) || !(rmin < 1.0e6)) return -1;
  int Z = 0;
  for (int d = 1; d <= (int)rmin + 1; ++d)
    if (rmin - sqrt((double)(d * d)) > 1e-9) Z = d;
  return Z;
}

// The radius's Z; TP3D_ERR_ARG (with a message) when it is invalid or too large.
int filter_z_for(double rmin, int* Z);

// Rings of the disc of max offset Z: the distinct d2 = dx^2 + dy^2 below
// (Z + 1)^2 (no offset at that distance or further has a tap), ascending.
constexpr int ring_size(int Z, int d2) {
  int n = 0;
  for (int x = -Z; x <= Z; ++x)
    for (int y = -Z; y <= Z; ++y) n += x * x + y * y == d2;
  return n;
}
constexpr int ring_count(int Z) {
  int n = 0;
  for (int d2 = 0; d2 < (Z + 1) * (Z + 1); ++d2) n += ring_size(Z, d2) > 0;
  return n;
}
constexpr int ring_d2(int Z, int c) {
  for (int d2 = 0; d2 < (Z + 1) * (Z + 1); ++d2)
    if (ring_size(Z, d2) > 0 && c-- == 0) return d2;
  return -1;
}
// offset dx * pitch + dy of the o-th column of the ring
constexpr int ring_offset(int Z, int d2, int o, int pitch) {
  for (int x = -Z; x <= Z; ++x)
    for (int y = -Z; y <= Z; ++y)
      if (x * x + y * y == d2 && o-- == 0) return x * pitch + y;
  return 0;
}

// Weight of ring c at distance a along z (0 without a tap), a kernel parameter.
template <int Z>
struct RingWeights {
  double w[ring_count(Z)][Z + 1];
};
template <int Z>
inline RingWeights<Z> ring_weights(double rmin) {
  RingWeights<Z> r;
  for (int c = 0; c < ring_count(Z); ++c)
    for (int a = 0; a <= Z; ++a) {
      const double wt = rmin - sqrt((double)(ring_d2(Z, c) + a * a));
      r.w[c][a] = wt > 1e-9 ? wt : 0.0;
    }
  return r;
}

constexpr int filter_pitch(int Z) { return kFilterTY + 2 * Z; }
constexpr int filter_plane(int Z) { return filter_pitch(Z) * (kFilterTX + 2 * Z); }

// Split of the outputs into blocks: 32 x 8 columns times kz planes.  A block
// marches 2Z planes more than it writes, so kz is as small as keeps the blocks
// within `slots` (those resident at once) but no smaller than 2Z while there is
// a block for each SM: at 96x48x45, rmin 2.5, the OC update takes 229 us with
// kz = 4 and 260 with kz = 2; grids that cannot fill the SMs want kz = 2.
struct FilterTiles {
  int ty, tx, tz, kz;
  __host__ __device__ long long count() const { return (long long)ty * tx * tz; }
};
inline FilterTiles filter_tiles(const Grid& g, int Z, int nsm, long long slots) {
  FilterTiles t;
  t.ty = (g.ny + kFilterTY - 1) / kFilterTY;
  t.tx = (g.nx + kFilterTX - 1) / kFilterTX;
  auto planes = [&](long long blocks) {  // per block, for about that many blocks
    const long long chunks = std::max<long long>(1, blocks / ((long long)t.ty * t.tx));
    return (int)((g.nz + chunks - 1) / chunks);
  };
  t.kz = std::max({std::min(2, g.nz), planes(slots), std::min(2 * Z, planes(nsm))});
  t.tz = (g.nz + t.kz - 1) / t.kz;
  return t;
}
// blocks per SM that the kernels are compiled for (64 and 80 registers per thread)
constexpr int filter_blocks_per_sm(int Z) { return Z <= 3 ? 4 : 3; }

template <int Z, int C, int... O>
__device__ __forceinline__ double ring_sum(const double* col, std::integer_sequence<int, O...>) {
  return (... + col[std::integral_constant<int, ring_offset(Z, ring_d2(Z, C), O, filter_pitch(Z))>::value]);
}
template <int Z, int C>
__device__ __forceinline__ void ring_add(const RingWeights<Z>& W, const double* col, double* S) {
  constexpr int d2 = ring_d2(Z, C);
  // rings past Z have a tap only where rmin reaches them
  if (d2 > Z * Z && W.w[C][0] == 0.0) return;
  const double R = ring_sum<Z, C>(col, std::make_integer_sequence<int, ring_size(Z, d2)>());
#pragma unroll
  for (int a = 0; a <= Z; ++a)
    if (d2 + a * a < (Z + 1) * (Z + 1)) S[a] = fma(W.w[C][a], R, S[a]);
}
template <int Z, int... C>
__device__ __forceinline__ void ring_adds(const RingWeights<Z>& W, const double* col, double* S,
                                          std::integer_sequence<int, C...>) {
  (ring_add<Z, C>(W, col, S), ...);
}

// Filters tile `t` of the grid.  `src.load(pz, i)` fetches what input element
// pz + i needs (pz: the plane's first element, the same for the block; i: its
// place in the plane) and `src.value(raw)` forms it; `out.load(pz, i)` fetches
// what an output needs ahead of its plane and `out.store(pz, i, pre, value)`
// takes the filtered value.  `s` holds two planes; it is free again when the
// call returns.
template <int Z, class Src, class Out>
__device__ __forceinline__ void filter_march(const Grid& g, const RingWeights<Z>& W, const FilterTiles& tiles,
                                             long long t, double* s, const Src& src, Out& out) {
  constexpr int SY = filter_pitch(Z), NS = filter_plane(Z), NP = (NS + kFilterThreads - 1) / kFilterThreads;
  const int ti = (int)(t % ((long long)tiles.ty * tiles.tx)), tzi = (int)(t / ((long long)tiles.ty * tiles.tx));
  const int y0 = (ti % tiles.ty) * kFilterTY, x0 = (ti / tiles.ty) * kFilterTX;
  const int z0 = tzi * tiles.kz, z1 = min(g.nz, z0 + tiles.kz);
  const int ly = threadIdx.x % kFilterTY, lx = threadIdx.x / kFilterTY;
  const long long plane = (long long)g.nx * g.ny;
  unsigned off[NP];  // this thread's elements of a staged plane
  bool in[NP];       // inside the domain
#pragma unroll
  for (int b = 0; b < NP; ++b) {
    const int i = threadIdx.x + b * kFilterThreads;
    const int gx = x0 + i / SY - Z, gy = y0 + i % SY - Z;
    in[b] = i < NS && gx >= 0 && gx < g.nx && gy >= 0 && gy < g.ny;
    off[b] = in[b] ? gy + (unsigned)g.ny * gx : 0u;
  }
  typename Src::Raw raw[NP];
  auto fetch = [&](int z) {
#pragma unroll
    for (int b = 0; b < NP; ++b)
      if (in[b]) raw[b] = src.load(plane * z, off[b]);
  };
  auto stage = [&](double* d) {
#pragma unroll
    for (int b = 0; b < NP; ++b) {
      const int i = threadIdx.x + b * kFilterThreads;
      if (i < NS) d[i] = in[b] ? src.value(raw[b]) : 0.0;
    }
  };
  const bool live = y0 + ly < g.ny && x0 + lx < g.nx;
  const unsigned e0 = live ? y0 + ly + (unsigned)g.ny * (x0 + lx) : 0u;
  const int zs = max(0, z0 - Z), ze = min(g.nz - 1, z1 - 1 + Z);
  double acc[2 * Z + 1];  // outputs zz - Z .. zz + Z
#pragma unroll
  for (int i = 0; i <= 2 * Z; ++i) acc[i] = 0.0;
  fetch(zs);
  stage(s);
  __syncthreads();
  int buf = 0;
  for (int zz = zs; zz <= ze; ++zz) {
    if (zz < ze) fetch(zz + 1);
    const int k = zz - Z;  // the output this plane completes
    if (live) {
      typename Out::Pre pre;
      if (k >= z0) pre = out.load(plane * k, e0);
      double S[Z + 1];
#pragma unroll
      for (int a = 0; a <= Z; ++a) S[a] = 0.0;
      ring_adds<Z>(W, s + buf * NS + (lx + Z) * SY + ly + Z, S, std::make_integer_sequence<int, ring_count(Z)>());
      acc[Z] += S[0];
#pragma unroll
      for (int a = 1; a <= Z; ++a) {
        acc[Z - a] += S[a];
        acc[Z + a] += S[a];
      }
      if (k >= z0) out.store(plane * k, e0, pre, acc[0]);
#pragma unroll
      for (int i = 0; i < 2 * Z; ++i) acc[i] = acc[i + 1];
      acc[2 * Z] = 0.0;
    }
    buf ^= 1;
    if (zz < ze) stage(s + buf * NS);
    __syncthreads();
  }
  // outputs whose last planes lie past the domain
  if (live) {
#pragma unroll
    for (int i = 0; i < 2 * Z; ++i) {
      const int k = ze + 1 - Z + i;
      if (k >= z0 && k < z1) out.store(plane * k, e0, out.load(plane * k, e0), acc[i]);
    }
  }
}

// Heaviside projection (pytopo3d/utils/filter.py:26-60).
struct Projection {
  double beta, eta, tbe, den;
  __host__ Projection(double b, double e) : beta(b), eta(e) {
    tbe = tanh(b * e);
    den = tanh(b * e) + tanh(b * (1.0 - e));
  }
  // Same operation order as the reference: divide by the denominator.
  __device__ __forceinline__ double value(double rf, double* deriv) const {
    const double t = tanh(beta * (rf - eta));
    if (deriv) *deriv = beta * (1.0 - t * t) / den;
    const double r = (tbe + t) / den;
    return fmin(fmax(r, 0.0), 1.0);
  }
};

// Dispatch a templated launcher on Z at runtime.
#define TP3D_DISPATCH_Z(Zval, ...)                      \
  switch (Zval) {                                       \
    case 0: { constexpr int ZC = 0; __VA_ARGS__; } break; \
    case 1: { constexpr int ZC = 1; __VA_ARGS__; } break; \
    case 2: { constexpr int ZC = 2; __VA_ARGS__; } break; \
    case 3: { constexpr int ZC = 3; __VA_ARGS__; } break; \
    case 4: { constexpr int ZC = 4; __VA_ARGS__; } break; \
    case 5: { constexpr int ZC = 5; __VA_ARGS__; } break; \
    case 6: { constexpr int ZC = 6; __VA_ARGS__; } break; \
    default: return TP3D_ERR_ARG;                       \
  }

}  // namespace tp3d
