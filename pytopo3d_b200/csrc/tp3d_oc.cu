// Optimality-criteria update with projected-volume bisection, one cooperative launch.
// Reference: pytopo3d/utils/oc_update.py:25-124 and the change measure of
// pytopo3d/core/optimizer.py:642.
//
// The reference re-filters and re-projects a candidate design for every
// bisection step and syncs the volume to the host.  Here the whole loop runs
// in one persistent kernel: every block owns a set of filter tiles, stages the
// candidate x(lambda) of its tiles (+ halo) in shared memory, filters,
// projects and sums the free volume; per-block partials are combined in a
// fixed order after a (bounded) grid barrier, so every block takes the same
// bisection decision.  Only the best multiplier is kept; the best candidate is
// recomputed from it at the end, so no candidate array is stored.
//
// An evaluation costs a pass over the design and a grid barrier, so the kernel
// makes few of them: the reference's bisection path (about 65 steps) is
// reproduced from about a dozen evaluations (see the kernel), where a search
// over the halvings followed by one evaluation per ordinary step took 34.
#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>
#include <mutex>

#include "tp3d_filter.cuh"

namespace tp3d {
namespace {

constexpr int kOcMaxBlocks = 4096;
constexpr int kOcBatch = 8;  // staged candidates per thread whose loads are in flight together

struct OcArgs {
  Grid g;
  FilterCols fc;
  const double* x;
  const double* dc;
  const double* dv;
  const double* Hs;
  const uint8_t* solid;
  const uint8_t* vd;
  double move, target, tol;
  int max_iter;
  Projection pr;
  double* x_new;
  double* rho_new;
  double* stats;
  double* ratio;     // nele
  double* partA;     // kOcMaxBlocks
  double* partB;     // kOcMaxBlocks
  double* partC;     // kOcMaxBlocks
  GridBarrier bar;
  long long spin_limit;   // polls before a grid-barrier wait gives up
  unsigned int phantom;   // blocks the barrier waits for that never arrive (wait-expiry test only)
};

// Wait-expiry test hook (tp3d_debug_expire_oc_waits): 0 = normal waits.
std::atomic<long long> g_test_spin_limit{0};
std::atomic<int> g_test_phantom{0};

void set_wait_policy(OcArgs& a) {
  const long long lim = g_test_spin_limit.load();
  a.spin_limit = lim > 0 ? lim : kSpinLimit;
  a.phantom = (unsigned int)g_test_phantom.load();
}

// Per-element code written once per call into the ratio scratch: for a free
// element q = sqrt(normalised ratio) >= 0; -1 marks protected solid, -2
// protected void (void wins where both are set, as in the reference).
constexpr double kCodeSolid = -1.0, kCodeVoid = -2.0;

// Candidate value (oc_update.py:76-91): x sqrt(max(r / (lam + 1e-30), 1e-30))
// = x max(q / sqrt(lam + 1e-30), 1e-15), then the move limit and [0, 1].
// `isl` = 1 / sqrt(lam + 1e-30), uniform over the launch.
__device__ __forceinline__ double candidate_q(double xe, double q, double isl, double move) {
  if (q < 0.0) return q == kCodeSolid ? 1.0 : 0.0;
  double c = xe * fmax(q * isl, 1e-15);
  c = fmax(xe - move, fmin(xe + move, c));
  return fmin(fmax(c, 0.0), 1.0);
}

// Projected free volume of the candidate at multiplier lam (oc_update.py:78-111):
// stage candidates of each owned tile (+ halo), filter, project, sum; per-block
// partials go to `part`, and after the grid barrier every block sums them in the
// same order.  Returns false if the barrier wait expired.  (Arrays written
// earlier in this launch are read through L2, __ldcg, never the L1 path.)
template <int Z>
__device__ bool oc_volume(const OcArgs& a, double lam, double* part, double* s, double* red, double* vol) {
  constexpr int SY = kFilterTY + 2 * Z, SX = kFilterTX + 2 * Z, SZ = kFilterKZ + 2 * Z;
  constexpr int NS = SY * SX * SZ;
  const long long ntiles = filter_ntiles(a.g);
  const double isl = 1.0 / sqrt(lam + 1e-30);
  double vpart = 0.0;
  for (long long t = blockIdx.x; t < ntiles; t += gridDim.x) {
    const FilterTile tile = filter_tile_at(a.g, t);
    __syncthreads();
    // kOcBatch elements per thread at a time: all their loads are issued
    // before the first candidate is formed, so they are in flight together
    for (int i0 = threadIdx.x; i0 < NS; i0 += kOcBatch * kFilterThreads) {
      double xv[kOcBatch], qv[kOcBatch];
      unsigned in = 0;
#pragma unroll
      for (int b = 0; b < kOcBatch; ++b) {
        const int i = i0 + b * kFilterThreads;
        xv[b] = 0.0;
        qv[b] = 0.0;
        if (i < NS) {
          const int ly = i % SY, r = i / SY;
          const int lx = r % SX, lz = r / SX;
          const int gx = tile.x0 + lx - Z, gy = tile.y0 + ly - Z, gz = tile.z0 + lz - Z;
          if (gx >= 0 && gx < a.g.nx && gy >= 0 && gy < a.g.ny && gz >= 0 && gz < a.g.nz) {
            const long long e = a.g.eidx(gx, gy, gz);
            xv[b] = __ldg(&a.x[e]);
            qv[b] = __ldcg(&a.ratio[e]);
            in |= 1u << b;
          }
        }
      }
#pragma unroll
      for (int b = 0; b < kOcBatch; ++b) {
        const int i = i0 + b * kFilterThreads;
        if (i < NS) s[i] = ((in >> b) & 1u) ? candidate_q(xv[b], qv[b], isl, a.move) : 0.0;
      }
    }
    __syncthreads();
    filter_apply<Z>(a.g, a.fc, tile, s, [&](long long e, int, int, int, double v) {
      if (__ldcg(&a.ratio[e]) >= 0.0) vpart += a.pr.value(v / __ldg(&a.Hs[e]), nullptr);
    });
  }
  vpart = block_sum(vpart, red);
  if (threadIdx.x == 0) part[blockIdx.x] = vpart;
  if (!grid_sync_flip(a.bar.count, a.bar.err, a.spin_limit, a.phantom)) return false;
  *vol = sum_partials(part, gridDim.x, red);
  return true;
}

// One step of the reference's bisection state: whether [lo, hi] has met its
// stop rule, (hi - lo) / (hi + lo) < tol.  The quotient is formed only near the
// threshold; far above it the product decides the same.
__device__ __forceinline__ bool bisection_done(double lo, double hi, double tol) {
  const double d = hi - lo, m = fmax(hi + lo, DBL_MIN);
  if (d > 2.0 * tol * m) return false;
  return d / m < tol;
}

template <int Z>
__global__ void __launch_bounds__(kFilterThreads) oc_kernel(const __grid_constant__ OcArgs a) {
  extern __shared__ double s[];
  filter_cols_to_smem<Z>(a.fc, s);  // read back after the first barrier
  __shared__ double red[32];
  const long long ntiles = filter_ntiles(a.g);
  const long long nele = a.g.nele();
  const int nblk = gridDim.x;
  auto solid_at = [&](long long e) { return a.solid && a.solid[e]; };
  auto void_at = [&](long long e) { return a.vd && a.vd[e]; };

  // ---- ratio normalisation (oc_update.py:54-68) ----
  double m = 0.0;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nele; e += (long long)nblk * blockDim.x) {
    if (!solid_at(e) && !void_at(e)) {
      const double r = fmax(-__ldg(&a.dc[e]) / fmax(__ldg(&a.dv[e]), 1e-20), 0.0);
      a.ratio[e] = r;
      m = fmax(m, r);
    }
  }
  m = block_max(m, red);
  if (threadIdx.x == 0) a.partC[blockIdx.x] = m;
  if (!grid_sync_flip(a.bar.count, a.bar.err, a.spin_limit, a.phantom)) return;
  double scale = 0.0;
  {
    double t = 0.0;
    for (int i = threadIdx.x; i < nblk; i += blockDim.x) t = fmax(t, a.partC[i]);
    scale = block_max(t, red);
  }
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nele; e += (long long)nblk * blockDim.x) {
    double q;
    if (void_at(e)) q = kCodeVoid;
    else if (solid_at(e)) q = kCodeSolid;
    else q = sqrt(scale > 0.0 ? a.ratio[e] / scale : 1.0);
    a.ratio[e] = q;
  }
  if (!grid_sync_flip(a.bar.count, a.bar.err, a.spin_limit, a.phantom)) return;

  // ---- bisection (oc_update.py:70-122) ----
  // The reference starts from [0, 1e12]; while the projected volume stays at or
  // below the target it only halves the upper bound (midpoints 1e12 / 2^j,
  // j = 1 .. K), then it bisects.  Its steps only compare volumes with the
  // target, and the volume does not increase with the multiplier: a midpoint at
  // or below a multiplier A known to be above the target is above it too, and
  // one at or above a multiplier B known to be at or below the target is at or
  // below it too.  So the crossing is closed in by evaluations of its own, and
  // the path is walked without any:
  //  * a search over the halvings for a first [A, B] (multipliers are around
  //    2^-6 to 2^-12, j = 46 to 52, against ratios of at most 1: probe j = 48,
  //    then outwards in doubling steps);
  //  * secant steps on t = 1 / sqrt(lambda) (a candidate inside its limits is
  //    linear in t), each evaluating an end of the final bisection cell that
  //    holds the estimate; the path is known when both ends of its cell are.
  //    Three evaluations that do not halve [A, B] are followed by the path's own
  //    next midpoint, so their number is bounded whatever the volume's shape.
  // The smallest error along the path is at an end of its last cell (errors fall
  // towards the crossing from either side), and the reference keeps the FIRST
  // step with the smallest error (strict <, oc_update.py:106).  Equal volumes at
  // two multipliers (a plateau, e.g. every candidate held at its move limit),
  // volumes that are not finite, and searches that reach an end of the halvings
  // go to the ordinary steps below instead.  (The path's end before the chosen one
  // is evaluated for this alone: a plateau may lie between two evaluations.)
  // About 11 evaluations in place of the path's 72 to 78 (of which a search over
  // the halvings by bisection and one evaluation per later step took 34):
  // 828 us before and 349 now at 128x64x64, rmin 3; 13.0 and 4.7 ms at
  // 256x128x128, rmin 4.5; 618 and 228 us at 32x16x16.
  double lo = 0.0, hi = 1.0e12;
  double best_err = INFINITY, best_lam = NAN, best_vol = NAN;
  int it = 0, pass = 0;
  bool done = false;
  auto eval = [&](double lam, double* v) {
    return oc_volume<Z>(a, lam, (pass++ & 1) ? a.partB : a.partA, s, red, v);
  };
  auto record = [&](double lam, double vol) {
    const double err = fabs(vol - a.target);
    if (err < best_err) {
      best_err = err;
      best_lam = lam;
      best_vol = vol;
    }
    if (vol > a.target) lo = lam;
    else hi = lam;
    ++it;
    if (bisection_done(lo, hi, a.tol)) done = true;
  };
  int jlo = 0, jhi = a.max_iter + 1;  // halvings known to be at or below the target, and above it
  double vlo = NAN, vhi = NAN;
  constexpr int kProbes = 24;  // the search over j <= 81 keeps at most this many probes
  int pj[kProbes];
  double pv[kProbes];
  int np = 0;
  auto probe = [&](int j) {
    double v;
    if (!eval(ldexp(1.0e12, -j), &v)) return false;
    if (v > a.target) {
      jhi = j;
      vhi = v;
    } else {
      jlo = j;
      vlo = v;
      if (np < kProbes) {
        pj[np] = j;
        pv[np] = v;
        ++np;
      }
    }
    return true;
  };
  bool known = false;  // the path has been walked
  if (a.tol < 1.0) {
    if (a.max_iter > 48 && a.tol > 0.0) {
      if (!probe(48)) return;
      const bool up = jlo > 0;  // the crossing lies at a smaller multiplier
      for (int step = 2; up ? jhi > a.max_iter && jlo + step <= a.max_iter : jlo == 0 && jhi - step >= 1; step *= 2)
        if (!probe(up ? jlo + step : jhi - step)) return;
    }
    bool walk = jlo >= 1 && jhi <= a.max_iter && isfinite(vlo) && isfinite(vhi) && vhi > vlo;
    double A = ldexp(1.0e12, -jhi), VA = vhi, B = ldexp(1.0e12, -jlo), VB = vlo;
    double t0 = 1.0 / sqrt(A), v0 = VA, t1 = 1.0 / sqrt(B), v1 = VB;
    double wlo = 0.0, whi = 1.0e12, width = B - A;  // the walk's own state
    double plo = 0.0, phi = 1.0e12;                  // its ends before the last ones
    int wit = 0, slow = 0;
    __shared__ struct {
      double lo, hi, plo, phi, e;
      int it, done;
    } w;
    while (walk) {
      // one warp walks and picks the next multiplier: the steps are a chain of
      // scalar arithmetic that every warp would repeat
      if (threadIdx.x < 32) {
        bool wdone = false;
        while (!wdone && wit < a.max_iter) {
          const double mid = 0.5 * (wlo + whi);
          if (mid <= A) plo = wlo, wlo = mid;
          else if (mid >= B) phi = whi, whi = mid;
          else break;
          ++wit;
          wdone = bisection_done(wlo, whi, a.tol);
        }
        double e = 0.5 * (wlo + whi);
        if (!wdone && wit < a.max_iter && slow < 3) {
          const double t = t1 + (a.target - v1) * (t0 - t1) / (v0 - v1);
          double r = 1.0 / (t * t);
          if (!(t > 0.0 && r > A && r < B)) r = 0.5 * (A + B);
          double slo = wlo, shi = whi;
          int sit = wit;
          do {
            const double mid = 0.5 * (slo + shi);
            if (mid <= A || (mid < B && mid < r)) slo = mid;
            else shi = mid;
            ++sit;
          } while (sit < a.max_iter && !bisection_done(slo, shi, a.tol));
          if (!(slo > A)) e = shi;
          else if (!(shi < B)) e = slo;
          else e = r - slo < shi - r ? slo : shi;
        }
        if (threadIdx.x == 0) {
          w.lo = wlo, w.hi = whi, w.plo = plo, w.phi = phi, w.e = e;
          w.it = wit, w.done = wdone || wit >= a.max_iter;
        }
      }
      __syncthreads();
      wlo = w.lo, whi = w.hi, plo = w.plo, phi = w.phi, wit = w.it;
      const double e = w.e;
      if (w.done) {
        known = true;
        break;
      }
      double v;
      if (!eval(e, &v)) return;  // its barriers also keep w until every thread has read it
      if (!isfinite(v) || v == VA || v == VB || v == v1) break;
      t0 = t1;
      v0 = v1;
      t1 = 1.0 / sqrt(e);
      v1 = v;
      if (v > a.target) A = e, VA = v;
      else B = e, VB = v;
      if (slow >= 3) slow = 0;
      else if (B - A <= 0.5 * width) slow = 0;
      else ++slow;
      if (slow == 0) width = B - A;
    }
    if (known) {
      // a path that ends among the halvings, or whose first midpoint was the
      // crossing's only neighbour, has no evaluated end there; a path's ends are
      // evaluated except where its cell is wider than a neighbour's
      double vl = VA, vh = VB;
      if (!(wlo > 0.0 && whi < 1.0e12)) known = false;
      if (known && wlo != A && !eval(wlo, &vl)) return;
      if (known && whi != B && !eval(whi, &vh)) return;
      if (known) {
        const double el = fabs(vl - a.target), eh = fabs(vh - a.target);
        const bool low = el < eh;
        // the first of equal errors counts: the end is the answer only if the
        // path's end before it on that side (none: 0 or 1e12) has another volume
        const double prev = low ? plo : phi;
        double v = NAN;
        if (prev > 0.0 && prev < 1.0e12 && !eval(prev, &v)) return;
        if (el == eh || v == (low ? vl : vh)) {
          known = false;
        } else {
          best_err = low ? el : eh;
          best_lam = low ? wlo : whi;
          best_vol = low ? vl : vh;
          lo = wlo;
          hi = whi;
          it = wit;
          done = true;
        }
      }
    }
    if (!known) {
      // The halvings by binary search: K is the number of leading steps at or
      // below the target.  Their volumes do not decrease with j, so the smallest
      // error among them is step K's, and steps 1..K need no evaluation of their
      // own, except for ties: if steps before K have exactly step K's volume,
      // the first of them counts.  Those steps form a range j0..K; j0 is found
      // from the probes (jb: largest probe below K with a smaller volume, jeq:
      // smallest probe with step K's volume), evaluating step K - 1 when no
      // probe decides it and bisecting (jb, jeq] only when a tie is seen.
      if (jhi > 1 && jlo == 0 && !probe(1)) return;  // K = 0 is common here
      while (jhi - jlo > 1)
        if (!probe((jlo + jhi) >> 1)) return;
      if (jlo >= 1) {
        int jb = 0, jeq = jlo;
        for (int i = 0; i < np; ++i) {
          if (pv[i] < vlo) jb = max(jb, pj[i]);
          else if (pv[i] == vlo) jeq = min(jeq, pj[i]);
        }
        if (jeq == jlo && jb < jlo - 1) {
          double v;
          if (!eval(ldexp(1.0e12, -(jlo - 1)), &v)) return;
          if (v == vlo) jeq = jlo - 1;
          else jb = jlo - 1;
        }
        while (jeq - jb > 1) {
          const int jm = (jb + jeq) >> 1;
          double v;
          if (!eval(ldexp(1.0e12, -jm), &v)) return;
          if (v == vlo) jeq = jm;
          else jb = jm;
        }
        best_err = fabs(vlo - a.target);
        best_lam = ldexp(1.0e12, -jeq);
        best_vol = vlo;
        hi = ldexp(1.0e12, -jlo);
        it = jlo;
      }
      if (jhi <= a.max_iter) record(ldexp(1.0e12, -jhi), vhi);  // = 0.5 (lo + hi)
    }
  }
  // the reference's ordinary steps
  while (!done && it < a.max_iter) {
    const double lam = 0.5 * (lo + hi);
    double vol;
    if (!eval(lam, &vol)) return;
    record(lam, vol);
  }

  // ---- best candidate, its density, and change (optimizer.py:642) ----
  const bool have = !isnan(best_lam);
  const double isl = have ? 1.0 / sqrt(best_lam + 1e-30) : 0.0;
  double cmax = 0.0;
  for (long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x; e < nele; e += (long long)nblk * blockDim.x) {
    const double xe = __ldg(&a.x[e]), q = a.ratio[e];
    const double v = have ? candidate_q(xe, q, isl, a.move) : xe;
    a.x_new[e] = v;
    if (q >= 0.0) cmax = fmax(cmax, fabs(v - xe));
  }
  cmax = block_max(cmax, red);
  if (threadIdx.x == 0) a.partC[blockIdx.x] = cmax;
  // x is not read after this barrier: x_new or rho_new may be x
  if (!grid_sync_flip(a.bar.count, a.bar.err, a.spin_limit, a.phantom)) return;
  for (long long t = blockIdx.x; t < ntiles; t += nblk) {
    const FilterTile tile = filter_tile_at(a.g, t);
    __syncthreads();
    filter_stage<Z>(a.g, tile, s, [&](long long e, int, int, int) { return __ldcg(&a.x_new[e]); });
    __syncthreads();
    filter_apply<Z>(a.g, a.fc, tile, s, [&](long long e, int, int, int, double v) {
      double r = a.pr.value(v / __ldg(&a.Hs[e]), nullptr);
      const double q = __ldcg(&a.ratio[e]);
      if (q == kCodeSolid) r = 1.0;
      if (q == kCodeVoid) r = 0.0;
      a.rho_new[e] = r;
    });
  }
  if (blockIdx.x == 0) {
    double t = 0.0;
    for (int i = threadIdx.x; i < nblk; i += blockDim.x) t = fmax(t, __ldcg(&a.partC[i]));
    t = block_max(t, red);
    if (threadIdx.x == 0) {
      a.stats[0] = best_lam;
      a.stats[1] = best_vol;
      a.stats[2] = (double)it;
      a.stats[3] = t;
      a.stats[4] = scale;
      a.stats[5] = lo;
      a.stats[6] = hi;
      a.stats[7] = have ? best_err : NAN;
      a.bar.count[3] = (unsigned int)pass;  // volume evaluations, for tests (cleared with the barrier words)
    }
  }
}

// The cooperative launch: as many blocks as are co-resident, a tile each or more.
template <int Z>
int oc_launch(OcArgs a, cudaStream_t st) {
  auto kern = oc_kernel<Z>;
  const size_t smem = filter_smem_bytes(Z);
  if (int rc = ensure_dynamic_smem(kern, smem)) return rc;
  int dev = 0, nsm = 0, per_sm = 0;
  TP3D_CHECK(cudaGetDevice(&dev));
  TP3D_CHECK(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  TP3D_CHECK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kFilterThreads, smem));
  if (per_sm < 1) {
    tp3d_set_last_error("OC kernel does not fit on an SM");
    return TP3D_ERR_CUDA;
  }
  const long long grid = std::min({(long long)per_sm * nsm, filter_ntiles(a.g), (long long)kOcMaxBlocks});
  void* args[] = {&a};
  TP3D_CHECK(cudaLaunchCooperativeKernel((const void*)kern, dim3((unsigned)grid), dim3(kFilterThreads), args, smem, st));
  return TP3D_OK;
}

}  // namespace
}  // namespace tp3d

using namespace tp3d;

extern "C" size_t tp3d_oc_scratch_bytes(int nelx, int nely, int nelz, double rmin) {
  (void)rmin;
  const long long n = (long long)nelx * nely * nelz;
  return (size_t)(n + 3 * kOcMaxBlocks) * sizeof(double) + 256;
}

extern "C" int tp3d_oc_update(int nelx, int nely, int nelz, double rmin, const double* x, const double* dc_dx,
                              const double* dv_dx, const double* Hs, const uint8_t* solid, const uint8_t* void_,
                              double move, double target_free_volume, double beta, double eta,
                              int max_bisection, double bisection_tol, double* x_new, double* rho_new,
                              double* stats, void* scratch, void* stream) {
  if (nelx < 1 || nely < 1 || nelz < 1 || !x || !dc_dx || !dv_dx || !Hs || !x_new || !rho_new || !stats ||
      !scratch)
    return TP3D_ERR_ARG;
  if (!std::isfinite(move) || move <= 0.0) {
    tp3d_set_last_error("move must be positive");
    return TP3D_ERR_ARG;
  }
  if (max_bisection < 1) {
    tp3d_set_last_error("max_bisection_iterations must be at least 1");
    return TP3D_ERR_ARG;
  }
  if (!std::isfinite(beta) || beta <= 0.0 || !(eta > 0.0 && eta < 1.0)) {
    tp3d_set_last_error("invalid projection parameters");
    return TP3D_ERR_ARG;
  }
  FilterCols fc;
  if (int rc = filter_cols_for(rmin, &fc)) return rc;
  const Grid g{nelx, nely, nelz};
  const long long n = g.nele();
  cudaStream_t st = (cudaStream_t)stream;

  OcArgs a{g, fc, x, dc_dx, dv_dx, Hs, solid, void_, move, target_free_volume, bisection_tol,
           max_bisection, Projection(beta, eta), x_new, rho_new, stats};
  set_wait_policy(a);
  double* base = (double*)scratch;
  a.ratio = base;
  a.partA = base + n;
  a.partB = a.partA + kOcMaxBlocks;
  a.partC = a.partB + kOcMaxBlocks;
  unsigned int* bar = (unsigned int*)(a.partC + kOcMaxBlocks);
  a.bar.count = bar;
  a.bar.gen = bar + 1;
  a.bar.err = (int*)(bar + 2);
  TP3D_CHECK(cudaMemsetAsync(bar, 0, 4 * sizeof(unsigned int), st));
  // NaN stats mark a launch that did not finish (e.g. an expired barrier wait)
  TP3D_CHECK(cudaMemsetAsync(stats, 0xff, 8 * sizeof(double), st));

  TP3D_DISPATCH_Z(fc.Z, if (int rc = oc_launch<ZC>(a, st)) return rc);
  add_launches(1);
  return TP3D_OK;
}

// ---------------------------------------------------------------------------
// OC update without device allocation.
//
// For callers that must not allocate device memory per call: an application
// whose device memory is fully reserved up front by its own allocator, or code
// that cannot accept the implicit device synchronisation that cudaMalloc /
// cudaFree bring.  The scratch of the bisection (normalised ratios, per-block
// partial sums, barrier counters, filter column table) lives in one
// file-scope __device__ array instead.  Every GPU that loads this library
// holds that array (about 2.2 MB) until the process exits.
// ---------------------------------------------------------------------------
namespace tp3d_oc_noalloc {

constexpr long long kNoAllocMaxElements = 1LL << 18;  // e.g. 64x64x64 or 128x64x32
constexpr int kNoAllocMaxCols = (2 * kFilterMaxZ + 1) * (2 * kFilterMaxZ + 1);
constexpr size_t kNoAllocRatioBytes = (size_t)kNoAllocMaxElements * sizeof(double);
constexpr size_t kNoAllocPartBytes = (size_t)3 * kOcMaxBlocks * sizeof(double);
constexpr size_t kNoAllocBarrierBytes = 256;
constexpr size_t kNoAllocDxyBytes = ((kNoAllocMaxCols * sizeof(int2) + 255) / 256) * 256;
constexpr size_t kNoAllocWBytes = (size_t)kNoAllocMaxCols * (2 * kFilterMaxZ + 1) * sizeof(double);
constexpr size_t kNoAllocBytes =
    kNoAllocRatioBytes + kNoAllocPartBytes + kNoAllocBarrierBytes + kNoAllocDxyBytes + kNoAllocWBytes;

static __device__ __align__(256) unsigned char g_oc_noalloc_scratch[kNoAllocBytes];

std::mutex g_noalloc_mu;
void* g_noalloc_addr[64] = {};  // per device: device address of g_oc_noalloc_scratch

// Device address of the static scratch on the current device; looked up once per
// device with that device current.
int noalloc_scratch(void** out) {
  int dev = 0;
  TP3D_CHECK(cudaGetDevice(&dev));
  if (dev < 0 || dev >= 64) {
    tp3d_set_last_error("device ordinal out of range for the static OC scratch");
    return TP3D_ERR_ARG;
  }
  std::lock_guard<std::mutex> lk(g_noalloc_mu);
  if (!g_noalloc_addr[dev]) {
    void* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_oc_noalloc_scratch);
    if (e != cudaSuccess || !p) {
      tp3d_set_last_error(e != cudaSuccess ? cudaGetErrorString(e) : "null symbol address");
      return TP3D_ERR_CUDA;
    }
    g_noalloc_addr[dev] = p;
  }
  *out = g_noalloc_addr[dev];
  return TP3D_OK;
}

// The filter column table of a radius, built in place in the static scratch:
// thread i evaluates candidate column i (filter_column, the same function and
// order as the host-built tables of the allocating path) and writes it at its
// rank among the columns that have a tap.  No host buffer is involved.
__global__ void __launch_bounds__(256) noalloc_columns_kernel(double rmin, int Z, int2* dxy, double* w) {
  __shared__ int has_tap[256];
  const int W = 2 * Z + 1, i = threadIdx.x;
  double col[2 * kFilterMaxZ + 1];
  const bool any = i < W * W && filter_column(rmin, Z, i, col);
  has_tap[i] = any ? 1 : 0;
  __syncthreads();
  if (any) {
    int pos = 0;
    for (int k = 0; k < i; ++k) pos += has_tap[k];
    dxy[pos] = make_int2(i / W - Z, i % W - Z);
    for (int j = 0; j < W; ++j) w[(size_t)pos * W + j] = col[j];
  }
}
static_assert((2 * kFilterMaxZ + 1) * (2 * kFilterMaxZ + 1) <= 256, "one thread per candidate column");

}  // namespace tp3d_oc_noalloc
using namespace tp3d_oc_noalloc;

extern "C" long long tp3d_oc_noalloc_max_elements(void) { return kNoAllocMaxElements; }

extern "C" int tp3d_oc_update_noalloc(int nelx, int nely, int nelz, double rmin, const double* x,
                                      const double* dc_dx, const double* dv_dx, const double* Hs,
                                      const uint8_t* solid, const uint8_t* void_, double move,
                                      double target_free_volume, double beta, double eta, int max_bisection,
                                      double bisection_tol, double* x_new, double* rho_new, double* stats,
                                      void* stream) {
  if (nelx < 1 || nely < 1 || nelz < 1 || !x || !dc_dx || !dv_dx || !Hs || !x_new || !rho_new || !stats)
    return TP3D_ERR_ARG;
  const long long n = (long long)nelx * nely * nelz;
  if (n > kNoAllocMaxElements) {
    tp3d_set_last_error(
        "tp3d_oc_update_noalloc: the grid has more elements than the static scratch holds (max 262144); "
        "use tp3d_oc_update with caller-provided scratch");
    return TP3D_ERR_ARG;
  }
  if (!std::isfinite(move) || move <= 0.0) {
    tp3d_set_last_error("move must be positive");
    return TP3D_ERR_ARG;
  }
  if (max_bisection < 1) {
    tp3d_set_last_error("max_bisection_iterations must be at least 1");
    return TP3D_ERR_ARG;
  }
  if (!std::isfinite(beta) || beta <= 0.0 || !(eta > 0.0 && eta < 1.0)) {
    tp3d_set_last_error("invalid projection parameters");
    return TP3D_ERR_ARG;
  }
  const int Z = filter_radius_z(rmin);
  if (Z < 0 || !std::isfinite(rmin)) return TP3D_ERR_ARG;
  if (Z > kFilterMaxZ) {
    tp3d_set_last_error("rmin too large for the stencil filter (max 7)");
    return TP3D_ERR_ARG;
  }
  void* base_v = nullptr;
  if (int rc = noalloc_scratch(&base_v)) return rc;
  unsigned char* base = (unsigned char*)base_v;
  cudaStream_t st = (cudaStream_t)stream;

  const Grid g{nelx, nely, nelz};
  OcArgs a{g, FilterCols{}, x, dc_dx, dv_dx, Hs, solid, void_, move, target_free_volume, bisection_tol,
           max_bisection, Projection(beta, eta), x_new, rho_new, stats};
  set_wait_policy(a);
  a.ratio = (double*)base;
  a.partA = (double*)(base + kNoAllocRatioBytes);
  a.partB = a.partA + kOcMaxBlocks;
  a.partC = a.partB + kOcMaxBlocks;
  unsigned int* bar = (unsigned int*)(base + kNoAllocRatioBytes + kNoAllocPartBytes);
  a.bar.count = bar;
  a.bar.gen = bar + 1;
  a.bar.err = (int*)(bar + 2);
  int2* d_dxy = (int2*)(base + kNoAllocRatioBytes + kNoAllocPartBytes + kNoAllocBarrierBytes);
  double* d_w = (double*)((unsigned char*)d_dxy + kNoAllocDxyBytes);
  a.fc.dxy = d_dxy;
  a.fc.w = d_w;
  a.fc.ncols = filter_columns_build(rmin, Z, nullptr, nullptr);  // count only
  a.fc.Z = Z;
  // The array keeps the previous call's contents: the column table is
  // rebuilt on the device and the barrier counters cleared on every call.
  noalloc_columns_kernel<<<1, 256, 0, st>>>(rmin, Z, d_dxy, d_w);
  TP3D_CHECK_LAUNCH();
  TP3D_CHECK(cudaMemsetAsync(bar, 0, kNoAllocBarrierBytes, st));
  TP3D_CHECK(cudaMemsetAsync(stats, 0xff, 8 * sizeof(double), st));

  TP3D_DISPATCH_Z(Z, if (int rc = oc_launch<ZC>(a, st)) return rc);
  add_launches(2);
  return TP3D_OK;
}

extern "C" int tp3d_debug_expire_oc_waits(long long spin_limit, int phantom_blocks) {
  if (spin_limit < 0 || phantom_blocks < 0 || phantom_blocks > 1024) return TP3D_ERR_ARG;
  g_test_spin_limit.store(spin_limit);
  g_test_phantom.store(phantom_blocks);
  return TP3D_OK;
}
