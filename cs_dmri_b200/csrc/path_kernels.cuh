// path_kernels.cuh - per-voxel alpha strategies on the device.
//
// AlphaStrategy (src/solver/alpha.rs:195-318) picks alpha per voxel:
//   AlphaMaxRatio   alpha = alpha_max * ratio
//   PathBic         a warm-started descending log path of alphas, keep the
//                   point of minimum BIC (ties to the larger alpha)
//   PathL2Anchored  same path, keep the first (largest-alpha) point whose
//                   RSS <= (1 + slack) RSS_L2, else the point of minimum RSS
// with alpha_max = ||M^T s||_inf / n and the zero result for alpha_max == 0.
// The FP64 fits of radial orders 4, 6 and 8 walk each voxel's path on its own
// slot (k_path_sparse, k_path_dmma); they share path_alpha and path_better with
// the walk below, which serves order 2, the mixed precision and a forced kernel
// shape: one point at a time over the whole volume, each point one FISTA launch
// over the voxels still in play, warm-started in place from the previous point
// (fista.rs:164-178), then one residual pass and the selection update.  Under
// PathL2Anchored a voxel leaves the work list as soon as it is selected: the
// later points of its path cannot change the result, so they are not computed.
#pragma once

#include <cstdint>

namespace csd {

// alpha_max_v = max_k |b_v[k]| / n (src/solver/alpha.rs:47-53); zero flag.
__global__ void k_alpha_max(const double* __restrict__ B, int64_t V, int K, int Kp, int N,
                            double* __restrict__ amax, uint8_t* __restrict__ zero) {
  const int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= V) return;
  double m = 0.0;
  for (int k = 0; k < K; ++k) m = fmax(m, fabs(B[v * Kp + k]));
  const double a = m / static_cast<double>(N);
  amax[v] = a;
  zero[v] = (a == 0.0) ? 1 : 0;
}

// alpha_v = alpha_max_v * ratio (src/solver/alpha.rs:229-236).
__global__ void k_alpha_ratio(const double* __restrict__ amax, int64_t V, double ratio,
                              double* __restrict__ alpha) {
  const int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= V) return;
  alpha[v] = amax[v] * ratio;
}

// Point i of log_path(alpha_max, n, eps) (src/solver/alpha.rs:57-69).
__device__ __forceinline__ double path_alpha(double amax, int i, int n, double eps) {
  const double lmax = log(amax), lmin = log(amax * eps);
  const double t = static_cast<double>(i) / static_cast<double>(n - 1);
  return exp(lmax + t * (lmin - lmax));
}

// Selection at one path point: PathBic keeps the lowest BIC (bic_argmin,
// alpha.rs:107-128), PathL2Anchored the lowest RSS until one is within the
// slack of the Tikhonov fit's, which ends the path (l2_anchored_argmax,
// alpha.rs:140-165).
__device__ __forceinline__ bool path_better(int mode, int N, int nnz, double rss, double rss_limit, double& best,
                                            bool& last) {
  if (mode == 2) {
    const double n = static_cast<double>(N);
    const double bic = n * log(fmax(rss, 2.2250738585072014e-308) / n) + log(n) * static_cast<double>(nnz);
    if (!(bic < best)) return false;
    best = bic;
    return true;
  }
  const bool within = rss <= rss_limit;
  last = last || within;
  if (!within && !(rss < best)) return false;
  best = rss;
  return true;
}

// The alphas of point i for the voxels of `list`.
__global__ void k_path_alpha(const double* __restrict__ amax, const int64_t* __restrict__ list,
                             int64_t n_work, int i, int n, double eps,
                             double* __restrict__ alpha) {
  const int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (w >= n_work) return;
  const int64_t v = list[w];
  alpha[v] = path_alpha(amax[v], i, n, eps);
}

struct PathState {
  double* best;        // V: best BIC (PathBic) or best RSS (L2 fallback)
  uint8_t* selected;   // V: PathL2Anchored point chosen
  uint8_t* active;     // V: still on the path (work-list flag)
  double* alpha_sel;   // V
  uint32_t* it_sel;    // V
  uint8_t* conv_sel;   // V
  double* alpha_fb;    // V
  uint32_t* it_fb;     // V
  uint8_t* conv_fb;    // V
  int8_t* copy_code;   // V: 0 none, 1 -> Xsel, 2 -> Xfb (this point)
};

// Selection update after path point `i` for the voxels of `list` (mode 2 =
// PathBic, mode 3 = PathL2Anchored).
__global__ void k_path_update(int mode, const int64_t* __restrict__ list, int64_t n_work, int N,
                              const double* __restrict__ resid, const int* __restrict__ nnz,
                              const double* __restrict__ alpha, const uint32_t* __restrict__ iters,
                              const uint8_t* __restrict__ conv, const double* __restrict__ rss_l2,
                              double slack, PathState s) {
  const int64_t w = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (w >= n_work) return;
  const int64_t v = list[w];
  const double rss = resid[v] * resid[v];
  int8_t code = 0;
  bool last = false;
  double best = s.best[v];
  if (path_better(mode, N, nnz[v], rss, mode == 3 ? (1.0 + slack) * rss_l2[v] : 0.0, best, last)) {
    s.best[v] = best;
    const bool chosen = mode == 2 || last;  // else PathL2Anchored's fallback, the lowest RSS so far
    code = chosen ? 1 : 2;
    (chosen ? s.alpha_sel : s.alpha_fb)[v] = alpha[v];
    (chosen ? s.it_sel : s.it_fb)[v] = iters[v];
    (chosen ? s.conv_sel : s.conv_fb)[v] = conv[v];
  }
  if (last) {
    s.selected[v] = 1;
    s.active[v] = 0;
  }
  s.copy_code[v] = code;
}

// Copy the coefficients of this path point to the selected / fallback store.
__global__ void k_path_copy(const int64_t* __restrict__ list, int64_t n_work, int Kp,
                            const int8_t* __restrict__ code, const double* __restrict__ X,
                            double* __restrict__ Xsel, double* __restrict__ Xfb) {
  const int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= n_work * Kp) return;
  const int64_t v = list[e / Kp];
  const int k = static_cast<int>(e % Kp);
  const int8_t c = code[v];
  if (c == 1)
    Xsel[v * Kp + k] = X[v * Kp + k];
  else if (c == 2)
    Xfb[v * Kp + k] = X[v * Kp + k];
}

// PathL2Anchored voxels that never met the slack bound take their
// minimum-RSS point; one without any (a residual that is not finite) keeps the
// zero result.
__global__ void k_path_finalize(int64_t V, int Kp, const uint8_t* __restrict__ zero, PathState s,
                                const double* __restrict__ Xfb, double* __restrict__ Xsel) {
  const int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (e >= V * Kp) return;
  const int64_t v = e / Kp;
  const int k = static_cast<int>(e % Kp);
  if (zero[v] || s.selected[v] || !(s.best[v] < INFINITY)) return;
  Xsel[v * Kp + k] = Xfb[v * Kp + k];
  if (k == 0) {
    s.alpha_sel[v] = s.alpha_fb[v];
    s.it_sel[v] = s.it_fb[v];
    s.conv_sel[v] = s.conv_fb[v];
  }
}

// Zero-voxel results (alpha 0, 0 iterations, converged) for the maps.
__global__ void k_zero_voxels(int64_t V, const uint8_t* __restrict__ zero,
                              double* __restrict__ alpha, uint32_t* __restrict__ iters,
                              uint8_t* __restrict__ conv) {
  const int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= V || !zero[v]) return;
  alpha[v] = 0.0;
  iters[v] = 0;
  conv[v] = 1;
}

// Flag array -> list of positions (u8 flags over V), via the mask compaction
// kernels; this builds the u8 "still active" array for them.
__global__ void k_init_active(int64_t V, const uint8_t* __restrict__ zero,
                              uint8_t* __restrict__ active) {
  const int64_t v = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (v >= V) return;
  active[v] = zero[v] ? 0 : 1;
}

}  // namespace csd
