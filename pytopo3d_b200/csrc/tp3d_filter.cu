// Density filter, Heaviside projection and the filter transpose (chain rule).
// Reference: pytopo3d/utils/filter.py:26-228.
#include <algorithm>
#include <cmath>

#include "tp3d_filter.cuh"

namespace tp3d {

int filter_z_for(double rmin, int* Z) {
  if (!(rmin > 0.0) || !std::isfinite(rmin)) return TP3D_ERR_ARG;
  *Z = filter_radius_z(rmin);
  if (*Z < 0) return TP3D_ERR_ARG;
  if (*Z > kFilterMaxZ) {
    tp3d_set_last_error("rmin too large for the stencil filter (max 7)");
    return TP3D_ERR_ARG;
  }
  return TP3D_OK;
}

namespace {

constexpr int kNumSMs = 148;

struct Nothing {};

// ones (the input of the row sums)
struct SrcOne {
  using Raw = Nothing;
  __device__ Raw load(long long, unsigned) const { return {}; }
  __device__ double value(Raw) const { return 1.0; }
};
struct SrcVec {
  const double* x;
  using Raw = double;
  __device__ Raw load(long long pz, unsigned i) const { return __ldg(x + pz + i); }
  __device__ double value(Raw r) const { return r; }
};
// g dproj / Hs (g / Hs without dproj)
struct SrcScaled {
  const double *g, *dp, *Hs;
  struct Raw {
    double g, dp, Hs;
  };
  __device__ Raw load(long long pz, unsigned i) const {
    return {__ldg(g + pz + i), dp ? __ldg(dp + pz + i) : 1.0, __ldg(Hs + pz + i)};
  }
  __device__ double value(const Raw& r) const { return (dp ? r.g * r.dp : r.g) / r.Hs; }
};

struct OutPlain {
  double* out;
  using Pre = Nothing;
  __device__ Pre load(long long, unsigned) const { return {}; }
  __device__ void store(long long pz, unsigned i, Pre, double v) const { (out + pz)[i] = v; }
};
// Hs = H 1 (row sums), 0 -> 1 (filter.py:224-226)
struct OutRowsum {
  double* out;
  using Pre = Nothing;
  __device__ Pre load(long long, unsigned) const { return {}; }
  __device__ void store(long long pz, unsigned i, Pre, double v) const { (out + pz)[i] = (v == 0.0) ? 1.0 : v; }
};
// build_physical_density (filter.py:63-100)
struct OutProject {
  const double* Hs;
  Projection pr;
  const uint8_t *solid, *vd;
  double *rf, *rp, *dp;
  struct Pre {
    double Hs;
    bool so, vo;
  };
  __device__ Pre load(long long pz, unsigned i) const {
    return {__ldg(Hs + pz + i), solid && __ldg(solid + pz + i), vd && __ldg(vd + pz + i)};
  }
  __device__ void store(long long pz, unsigned i, const Pre& p, double v) const {
    const double f = v / p.Hs;
    double d;
    double r = pr.value(f, &d);
    if (p.so) r = 1.0;
    if (p.vo) r = 0.0;
    if (p.so || p.vo) d = 0.0;
    if (rf) (rf + pz)[i] = f;
    (rp + pz)[i] = r;
    if (dp) (dp + pz)[i] = d;
  }
};

template <int Z, class Src, class Out>
__global__ void __launch_bounds__(kFilterThreads, filter_blocks_per_sm(Z))
    filter_kernel(Grid g, const __grid_constant__ RingWeights<Z> W, FilterTiles tiles, Src src, Out out) {
  __shared__ __align__(16) double s[2 * filter_plane(Z)];
  filter_march<Z>(g, W, tiles, blockIdx.x, s, src, out);
}

// out = H applied to src on the stream.
template <class Src, class Out>
int filter_launch(const Grid& g, double rmin, cudaStream_t st, const Src& src, const Out& out) {
  int Z = 0;
  if (int rc = filter_z_for(rmin, &Z)) return rc;
  const FilterTiles tiles = filter_tiles(g, Z, kNumSMs, kNumSMs * filter_blocks_per_sm(Z));
  TP3D_DISPATCH_Z(Z, {
    filter_kernel<ZC, Src, Out><<<(unsigned)tiles.count(), kFilterThreads, 0, st>>>(g, ring_weights<ZC>(rmin), tiles,
                                                                                   src, out);
  });
  add_launches(1);
  TP3D_CHECK_LAUNCH();
  return TP3D_OK;
}

__global__ void heaviside_kernel(const double* __restrict__ rf, long long n, Projection pr, double* out,
                                 double* der) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    double d;
    const double r = pr.value(rf[i], &d);
    if (out) out[i] = r;
    if (der) der[i] = d;
  }
}

int check_grid(int nx, int ny, int nz) {
  if (nx < 1 || ny < 1 || nz < 1) {
    tp3d_set_last_error("nelx, nely, and nelz must all be positive");
    return TP3D_ERR_ARG;
  }
  return TP3D_OK;
}

}  // namespace
}  // namespace tp3d

using namespace tp3d;

extern "C" int tp3d_filter_rowsum(int nelx, int nely, int nelz, double rmin, double* Hs, void* stream) {
  if (int rc = check_grid(nelx, nely, nelz)) return rc;
  if (!Hs) return TP3D_ERR_ARG;
  return filter_launch(Grid{nelx, nely, nelz}, rmin, (cudaStream_t)stream, SrcOne{}, OutRowsum{Hs});
}

extern "C" int tp3d_filter_project(int nelx, int nely, int nelz, double rmin, const double* x,
                                   const double* Hs, double beta, double eta, const uint8_t* solid,
                                   const uint8_t* void_, double* rho_filtered, double* rho_physical,
                                   double* dproj, void* stream) {
  if (int rc = check_grid(nelx, nely, nelz)) return rc;
  if (!x || !Hs || !rho_physical) return TP3D_ERR_ARG;
  if (!std::isfinite(beta) || beta <= 0.0) {
    tp3d_set_last_error("beta must be positive");
    return TP3D_ERR_ARG;
  }
  if (!(eta > 0.0 && eta < 1.0)) {
    tp3d_set_last_error("eta must be between 0 and 1");
    return TP3D_ERR_ARG;
  }
  return filter_launch(Grid{nelx, nely, nelz}, rmin, (cudaStream_t)stream, SrcVec{x},
                       OutProject{Hs, Projection(beta, eta), solid, void_, rho_filtered, rho_physical, dproj});
}

extern "C" int tp3d_filter_transpose(int nelx, int nely, int nelz, double rmin, const double* gin,
                                     const double* dproj, const double* Hs, double* out, void* stream) {
  if (int rc = check_grid(nelx, nely, nelz)) return rc;
  if (!gin || !Hs || !out) return TP3D_ERR_ARG;
  return filter_launch(Grid{nelx, nely, nelz}, rmin, (cudaStream_t)stream, SrcScaled{gin, dproj, Hs}, OutPlain{out});
}

extern "C" int tp3d_heaviside(const double* rho_filtered, long long n, double beta, double eta, double* out,
                              double* derivative, void* stream) {
  if (n < 0 || (n > 0 && !rho_filtered)) return TP3D_ERR_ARG;
  if (!std::isfinite(beta) || beta <= 0.0) {
    tp3d_set_last_error("beta must be positive");
    return TP3D_ERR_ARG;
  }
  if (!(eta > 0.0 && eta < 1.0)) {
    tp3d_set_last_error("eta must be between 0 and 1");
    return TP3D_ERR_ARG;
  }
  if (n == 0) return TP3D_OK;
  const Projection pr(beta, eta);
  const int blocks = (int)std::min<long long>((n + 255) / 256, 148 * 16);
  heaviside_kernel<<<blocks, 256, 0, (cudaStream_t)stream>>>(rho_filtered, n, pr, out, derivative);
  add_launches(1);
  TP3D_CHECK_LAUNCH();
  return TP3D_OK;
}
