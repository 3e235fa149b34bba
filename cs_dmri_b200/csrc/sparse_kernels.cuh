// sparse_kernels.cuh - FISTA with products over the non-zero entries only, one
// or two voxels per warp, and the alpha path strategies as one kernel.
//
// The iterates of the L1 fit are sparse: over the synthetic CS-DSI volumes a
// momentum point y has 12.5 of 72 non-zero entries (radial order 6, alpha
// 0.01) or 12.8 of 145 (order 8).  A DMMA tile skips a k-step only when its
// four entries vanish for all eight voxels of the warp, so k_fista_v3 still
// executes 52 % (order 6) and 26 % (order 8) of the dense product.  Here the
// non-zero entries are listed by ballots, and G y adds exactly the listed
// columns of G, read from shared memory.
//
// What bounds it: at full load the shared-memory pipe (one voxel per warp,
// order 6: 100 wavefronts of 128 B a voxel-iteration, 85 % of the pipe's
// rate; two per warp read each column of their common list once: 72, at 65 %
// with the issue slots at 63 %); for a few voxels the latency of one
// iteration, 0.3 us for a lone warp and 0.5-0.6 us beside fifteen others,
// against the 1.25-4 us of a DMMA warp.  An SM partition takes 32 B a cycle from
// shared memory, broadcasts included, so a column costs its warp 18 cycles at
// order 6 and 36 at order 8 besides 12 for its list entry: dense iterates belong
// on DMMA slots (PassChoice, k_choose_by_alpha).  Volume fits, N = 259, alpha
// 0.01, against the DMMA kernel alone: 108 voxels 1.64 -> 0.42 ms, 4,000 voxels
// 3.55 -> 0.84 ms, 32,000 voxels at order 8 11.4 -> 3.5 ms (with the residual pass
// that no output reads dropped there).
#pragma once

#include <cstdint>

namespace csd {

// Shared-memory accesses by 32-bit address, so that a column costs one add per
// base.  The list accesses are ordered by __syncwarp (memory clobber); G does
// not change after it is staged.
__device__ __forceinline__ double2 sp_ld_g2(uint32_t a) {
  double2 v;
  asm("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a));
  return v;
}
__device__ __forceinline__ void sp_ld_g1(double& v, uint32_t a, bool on) {  // v keeps its value where off
  asm("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q ld.shared.f64 %0, [%1];\n}" : "+d"(v) : "r"(a), "r"(static_cast<int>(on)));
}
__device__ __forceinline__ double2 sp_ld_v2(uint32_t a) {
  double2 v;
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ int4 sp_ld_i4(uint32_t a) {
  int4 v;
  asm volatile("ld.shared.v4.s32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ int2 sp_ld_i2(uint32_t a) {
  int2 v;
  asm volatile("ld.shared.v2.s32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void sp_st_f64(uint32_t a, double v, bool on) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q st.shared.f64 [%0], %1;\n}" ::"r"(a), "d"(v), "r"(static_cast<int>(on)) : "memory");
}
__device__ __forceinline__ void sp_st_2f64(uint32_t a, double v, double w, bool on) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %3, 0;\n @q st.shared.v2.f64 [%0], {%1, %2};\n}" ::"r"(a), "d"(v), "d"(w), "r"(static_cast<int>(on)) : "memory");
}
__device__ __forceinline__ void sp_st_s32(uint32_t a, int v, bool on) {
  asm volatile("{\n .reg .pred q;\n setp.ne.s32 q, %2, 0;\n @q st.shared.s32 [%0], %1;\n}" ::"r"(a), "r"(v), "r"(static_cast<int>(on)) : "memory");
}

// Rows of a K-vector over a warp: lane l holds rows 64 i + 2 l and
// 64 i + 2 l + 1 of each full pair block i (one 16-byte load of a column), and
// row 64 PAIRS + l of the remainder (lanes < REM; the others load nothing and
// their threshold is infinite, so their entries stay 0).
template <int K, int P>
struct SparseShape {
  static constexpr int PAIRS = K / 64;
  static constexpr int REM = K % 64;
  static constexpr int NR = 2 * PAIRS + 1;          // rows per lane
  static constexpr int KP = 8 * ((K + 7) / 8);      // row stride of B and X
  static constexpr int LD = (K + 1) & ~1;           // column stride in shared memory (16-byte columns)
  static constexpr int CAP = (K + 3) / 4 * 4 + 4;   // list entries of a warp (with the padding of the last group)
  static constexpr size_t G_BYTES = sizeof(double) * K * LD;
  static constexpr size_t WARP_BYTES = (P * sizeof(double) + sizeof(int)) * CAP;
  static_assert(REM > 0 && REM <= 32, "one remainder row per lane");
  static_assert(G_BYTES % 16 == 0 && WARP_BYTES % 16 == 0 && P * sizeof(double) * CAP % 16 == 0, "16-byte slices");
  __device__ static constexpr int row(int i, int lane) {
    return i < 2 * PAIRS ? 64 * (i / 2) + 2 * lane + (i & 1) : 64 * PAIRS + lane;
  }
};

// The states of a warp's P voxel slots and one FISTA iteration of them all
// (src/solver/fista.rs:89-128).
// WIDE: groups of eight columns while more than four are left (a group's chain
// is two shared-memory latencies and its dependent FMAs, so fewer, wider groups
// shorten an iteration where registers allow: 4,000 voxels at order 6, 128
// registers and 16 warps per SM, 0.84 ms; groups of four, 64 registers and 32
// warps, 0.99 ms).
template <int K, int P, bool NONNEG, bool WIDE>
struct SparseFista {
  using S = SparseShape<K, P>;
  double x[P][S::NR], y[P][S::NR], b[P][S::NR];
  double thr[P];                  // step * alpha
  double sx[P], sd[P];            // scales of the stopping filter
  unsigned fl[P];
  int it[P];                      // iterations done; -1: the slot is empty
  uint32_t gp, gr;                // this lane's pair rows and remainder row of column 0
  uint32_t lv, li;                // the warp's list: values (P per entry), column offsets in bytes
  int lane;

  // G (KP x KP, row-major) into shared memory, columns of stride LD; the
  // caller synchronises the CTA.
  __device__ __forceinline__ void init(const double* __restrict__ G, unsigned char* smem) {
    double* g = reinterpret_cast<double*>(smem);
    for (int e = threadIdx.x; e < K * S::LD; e += blockDim.x) {
      const int j = e / S::LD, r = e - j * S::LD;
      g[e] = r < K ? __ldg(G + j * S::KP + r) : 0.0;
    }
    attach(g, smem + S::G_BYTES + (threadIdx.x >> 5) * S::WARP_BYTES, threadIdx.x & 31);
  }

  // The warp's states over a matrix already in shared memory (columns of
  // stride LD) and its list (WARP_BYTES), every slot empty.
  __device__ __forceinline__ void attach(const double* g, void* list, int l) {
    lane = l;
    const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(g));
    gp = base + 16u * lane;
    gr = base + 8u * (64 * S::PAIRS + (lane < S::REM ? lane : 0));
    lv = static_cast<uint32_t>(__cvta_generic_to_shared(list));
    li = lv + static_cast<uint32_t>(P * sizeof(double) * S::CAP);
#pragma unroll
    for (int p = 0; p < P; ++p) clear(p);
  }

  // An empty slot: every entry 0 and kept there by an infinite threshold.
  __device__ __forceinline__ void clear(int p) {
#pragma unroll
    for (int i = 0; i < S::NR; ++i) x[p][i] = y[p][i] = b[p][i] = 0.0;
    thr[p] = INFINITY;
    it[p] = -1;
    start(p);
  }

  // The slot's fit starts (or restarts): its first stopping test is exact.
  __device__ __forceinline__ void start(int p) {
    sx[p] = sd[p] = 0.0;
    fl[p] = 0u;
  }

  __device__ __forceinline__ void list_row(int row, int i, bool e, int pos) {
    if constexpr (P == 1)
      sp_st_f64(lv + 8u * pos, y[0][i], e);
    else
      sp_st_2f64(lv + 16u * pos, y[0][i], y[P - 1][i], e);
    sp_st_s32(li + 4u * pos, row * static_cast<int>(sizeof(double) * S::LD), e);
  }

  static constexpr int U = P == 1 ? 4 : 2;  // columns per group

  // acc += the C columns of list entries t .. t + C - 1.
  template <int C>
  __device__ __forceinline__ void group(int t, double (&acc)[P][S::NR]) const {
    uint32_t off[C];
    double yv[C][P];
    if constexpr (C == 2) {
      const int2 id = sp_ld_i2(li + 4u * t);
      off[0] = id.x, off[1] = id.y;
    } else {
#pragma unroll
      for (int c = 0; c < C; c += 4) {
        const int4 id = sp_ld_i4(li + 4u * (t + c));
        off[c] = id.x, off[c + 1] = id.y, off[c + 2] = id.z, off[c + 3] = id.w;
      }
    }
#pragma unroll
    for (int e = 0; e < C * P; e += 2) {
      const double2 v = sp_ld_v2(lv + 8u * (P * t + e));
      yv[e / P][e % P] = v.x;
      yv[(e + 1) / P][(e + 1) % P] = v.y;
    }
    double2 g2[C][S::PAIRS > 0 ? S::PAIRS : 1];
    double g1[C];
#pragma unroll
    for (int c = 0; c < C; ++c) {
      g1[c] = 0.0;
#pragma unroll
      for (int i = 0; i < S::PAIRS; ++i) g2[c][i] = sp_ld_g2(gp + off[c] + 512u * i);
      sp_ld_g1(g1[c], gr + off[c], lane < S::REM);
    }
#pragma unroll
    for (int c = 0; c < C; ++c)
#pragma unroll
      for (int p = 0; p < P; ++p) {
#pragma unroll
        for (int i = 0; i < S::PAIRS; ++i) {
          acc[p][2 * i] = fma(g2[c][i].x, yv[c][p], acc[p][2 * i]);
          acc[p][2 * i + 1] = fma(g2[c][i].y, yv[c][p], acc[p][2 * i + 1]);
        }
        acc[p][S::NR - 1] = fma(g1[c], yv[c][p], acc[p][S::NR - 1]);
      }
  }

  // acc = G y for every slot.  The rows with a non-zero y in any slot are
  // listed in increasing order (ballots), padded to whole groups with zero
  // entries, and their columns added in that order, one FMA per row and slot:
  // the sums of the dense product without its zero terms.
  __device__ __forceinline__ void product(double (&acc)[P][S::NR]) {
    const unsigned lt = (1u << lane) - 1u;
    int n = 0;
    auto live = [&](int i) {
      bool e = y[0][i] != 0.0;
#pragma unroll
      for (int p = 1; p < P; ++p) e = e || y[p][i] != 0.0;
      return e;
    };
#pragma unroll
    for (int i = 0; i < S::PAIRS; ++i) {
      const bool e = live(2 * i), o = live(2 * i + 1);
      const unsigned me = __ballot_sync(kFull, e), mo = __ballot_sync(kFull, o);
      const int pos = n + __popc(me & lt) + __popc(mo & lt);
      list_row(64 * i + 2 * lane, 2 * i, e, pos);
      list_row(64 * i + 2 * lane + 1, 2 * i + 1, o, pos + (e ? 1 : 0));
      n += __popc(me) + __popc(mo);
    }
    {
      const bool e = live(S::NR - 1);
      const unsigned me = __ballot_sync(kFull, e);
      list_row(64 * S::PAIRS + lane, S::NR - 1, e, n + __popc(me & lt));
      n += __popc(me);
    }
    {
      const bool pad = lane < U - 1;
      if constexpr (P == 1)
        sp_st_f64(lv + 8u * (n + lane), 0.0, pad);
      else
        sp_st_2f64(lv + 16u * (n + lane), 0.0, 0.0, pad);
      sp_st_s32(li + 4u * (n + lane), 0, pad);
    }
    __syncwarp();
#pragma unroll
    for (int p = 0; p < P; ++p)
#pragma unroll
      for (int i = 0; i < S::NR; ++i) acc[p][i] = 0.0;
    int t = 0;
    if constexpr (WIDE)
#pragma unroll 1
      for (; n - t > 4; t += 8) group<8>(t, acc);
#pragma unroll 1
    for (; t < n; t += U) group<U>(t, acc);
    __syncwarp();
  }

  // The update of slot p with the momentum mom; true when the relative change
  // sqrt(dx2) / max(sqrt(xn2), 1e-12) is below tol.
  __device__ __forceinline__ bool update(int p, const double (&acc)[S::NR], double mom, double c, double tol) {
    double dx2 = 0.0, xn2 = 0.0;
#pragma unroll
    for (int i = 0; i < S::NR; ++i) {
      const double th = (i == S::NR - 1 && lane >= S::REM) ? INFINITY : thr[p];
      const double xn = fista_prox<NONNEG>(acc[i], b[p][i], y[p][i], c, th);
      const double d = __dsub_rn(xn, x[p][i]);
      y[p][i] = fma(mom, d, xn);
      dx2 = fma(d, d, dx2);
      xn2 = fma(xn, xn, xn2);
      x[p][i] = xn;
    }
    // Filter: dx2 and xn2 summed over the warp as integers in units of
    // 4 tol^2 X / 2^20 (rounded down) and X / 2^20 (rounded up), X the norm of
    // the last exact test.  A larger dx2 sum means a ratio above 2 tol, far
    // outside rounding (fl covers the 1e-12 floor of the norm; a sum that
    // outgrew the scale never passes).
    const unsigned ud = min(__double2uint_rd(dx2 * sd[p]), 1u << 20);
    const unsigned ux = min(__double2uint_ru(xn2 * sx[p]), 1u << 26);
    if (__reduce_add_sync(kFull, ud) > __reduce_add_sync(kFull, ux) + fl[p]) return false;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      dx2 += __shfl_xor_sync(kFull, dx2, o);
      xn2 += __shfl_xor_sync(kFull, xn2, o);
    }
    const double X = fmax(xn2, 1e-24);
    const double s = 1048576.0 / X;
    sx[p] = s;
    sd[p] = s / (4.0 * tol * tol);
    fl[p] = __double2uint_ru(1e-24 * s);
    if (dx2 > 4.0 * tol * tol * X) return false;
    return sqrt(dx2) / fmax(sqrt(xn2), 1e-12) < tol;
  }
};

// FISTA over a work queue, P voxels per warp (FistaParams as for k_fista_v3;
// with `resume` the voxels continue from the parked state X, Y at iteration
// `cap`).
template <int K, int P, int MAXWARPS, int MINCTAS, bool NONNEG>
__global__ void __launch_bounds__(32 * MAXWARPS, MINCTAS) k_fista_sparse(FistaParams p) {
  using S = SparseShape<K, P>;
  constexpr bool WIDE = P == 1 && K == 72;
  extern __shared__ __align__(16) unsigned char sp_smem[];
  const unsigned long long n_work = p.n_work_dev ? *p.n_work_dev : static_cast<unsigned long long>(p.n_work);
  if (n_work == 0) return;
  SparseFista<K, P, NONNEG, WIDE> f;
  f.init(p.G, sp_smem);
  __syncthreads();
  const int it0 = p.resume ? p.cap : 0;
  const double c = p.step * p.n_inv;
  unsigned long long executed = 0;
  int64_t vid[P];
  bool need[P];
#pragma unroll
  for (int s = 0; s < P; ++s) {
    vid[s] = -1;
    need[s] = true;
  }
  while (true) {
#pragma unroll
    for (int s = 0; s < P; ++s) {
      if (!need[s]) continue;
      need[s] = false;
      unsigned long long w = 0;
      if (f.lane == 0) w = atomicAdd(p.queue, 1ull);
      w = __shfl_sync(kFull, w, 0);
      if (w >= n_work) {
        vid[s] = -1;
        f.clear(s);
        continue;
      }
      const int64_t v = p.list ? p.list[w] : static_cast<int64_t>(w);
      vid[s] = v;
#pragma unroll
      for (int i = 0; i < S::NR; ++i) {
        const int row = S::row(i, f.lane);
        const bool in = row < K;
        f.b[s][i] = in ? p.B[v * S::KP + row] : 0.0;
        if (p.resume) {
          f.x[s][i] = in ? p.X[v * S::KP + row] : 0.0;
          f.y[s][i] = in ? p.Y[v * S::KP + row] : 0.0;
        } else {
          f.x[s][i] = (in && p.warm) ? p.warm[v * S::KP + row] : 0.0;
          f.y[s][i] = f.x[s][i];
        }
      }
      f.thr[s] = p.alpha_v ? __dmul_rn(p.step, p.alpha_v[v]) : p.thr;
      f.it[s] = it0;
      f.start(s);
    }
    bool any = false;
#pragma unroll
    for (int s = 0; s < P; ++s) any = any || vid[s] >= 0;
    if (!any) break;
    double mom[P];
#pragma unroll
    for (int s = 0; s < P; ++s) mom[s] = vid[s] >= 0 ? __ldg(p.mom + f.it[s]) : 0.0;
    double acc[P][S::NR];
    f.product(acc);
#pragma unroll
    for (int s = 0; s < P; ++s) {
      if (vid[s] < 0) continue;
      const bool conv = f.update(s, acc[s], mom[s], c, p.tol);
      const int it = ++f.it[s];
      if (!conv && it < p.max_iter) continue;
      const int64_t v = vid[s];
#pragma unroll
      for (int i = 0; i < S::NR; ++i) {
        const int row = S::row(i, f.lane);
        if (row < S::KP) p.X[v * S::KP + row] = f.x[s][i];
      }
      if (f.lane == 0) {
        p.iters[v] = static_cast<uint32_t>(it);
        p.conv[v] = conv ? 1 : 0;
      }
      executed += static_cast<unsigned long long>(it - it0);
      need[s] = true;
    }
  }
  if (p.iter_total && f.lane == 0 && executed) atomicAdd(p.iter_total, executed);
}

// ------------------------------------------------------- alpha path, fused

// A voxel in mid-path: where it stands, its x and y in rows v of Xp and Yp.
struct PathPark {
  double best;
  int v, point, it, pad;
};

struct PathParams {
  FistaParams f;         // B, X (the chosen point's coefficients), iters, conv, step, n_inv, tol, max_iter, queue
  const double* amax;    // V: alpha_max
  const double* rss_l2;  // V: the Tikhonov fit's RSS (PathL2Anchored), or nullptr
  double* alpha;         // V out
  const float* data;     // signals: row vox[v] of `data`, or row v of `sig`
  const int64_t* vox;
  const float* sig;
  const double* Mt;      // KP x N, transposed design
  int N, n_alphas, mode; // mode 2 = PathBic, 3 = PathL2Anchored
  double eps, slack;
  // k_path_dmma leaves the voxels of its last warps here for k_path_sparse
  PathPark* park;
  unsigned long long* n_park;
  double *Xp, *Yp;       // V x KP
  int resume;            // take the parked voxels (*n_park of them) instead of 0 .. n_work-1
};

// ||s - M c||^2 of one voxel on a warp, c sparse (listed in increasing row as
// values, every P-th double, and rows): four samples a lane and
// four coefficients at a time, so 16 loads are in flight; the columns of M are
// read from M^T (coalesced, L1 / L2).
template <int P>
__device__ __forceinline__ double sparse_rss(const float* __restrict__ sig, const double* __restrict__ Mt, int N,
                                             const double* val, const int* row, int nnz, int lane) {
  double rss = 0.0;
  for (int n0 = lane; n0 < N; n0 += 128) {
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    int off[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) off[u] = n0 + 32 * u < N ? n0 + 32 * u : N - 1;
#pragma unroll 4
    for (int e = 0; e < nnz; ++e) {
      const double c = val[P * e];
      const double* col = Mt + static_cast<size_t>(row[e]) * N;
#pragma unroll
      for (int u = 0; u < 4; ++u) acc[u] = fma(__ldg(col + off[u]), c, acc[u]);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (n0 + 32 * u < N) {
        const double r = static_cast<double>(__ldg(sig + n0 + 32 * u)) - acc[u];
        rss = fma(r, r, rss);
      }
  }
  for (int o = 16; o > 0; o >>= 1) rss += __shfl_xor_sync(kFull, rss, o);
  return rss;
}

// The whole alpha path of a voxel on its slot (src/solver/alpha.rs:249-318):
// FISTA at each alpha from the previous point's answer, the residual and the
// selection between them, no pass over the volume per alpha.  A point's
// coefficients are written to X when they are the best so far (PathBic: lower
// BIC; PathL2Anchored: lower RSS, or the first within the slack, which ends the
// path); alpha_max == 0 gives the zero result.
//
// Point by point over the volume (one FISTA launch, residual pass, selection
// and compaction with a host round trip per alpha) every alpha waits for its
// slowest voxel: 15 tails a fit.  Here a voxel's slot goes on to its next
// alpha alone and the fit has one tail.
template <int K, int P, int MAXWARPS, int MINCTAS, bool NONNEG>
__global__ void __launch_bounds__(32 * MAXWARPS, MINCTAS) k_path_sparse(PathParams q) {
  using S = SparseShape<K, P>;
  extern __shared__ __align__(16) unsigned char sp_smem[];
  const FistaParams& p = q.f;
  SparseFista<K, P, NONNEG, (P == 1 && K == 72)> f;
  f.init(p.G, sp_smem);
  __syncthreads();
  const double c = p.step * p.n_inv;
  unsigned long long executed = 0;
  int64_t vid[P];
  bool need[P];
  int point[P];
  double best[P], alpha[P];
#pragma unroll
  for (int s = 0; s < P; ++s) {
    vid[s] = -1;
    need[s] = true;
    point[s] = 0;
    best[s] = alpha[s] = 0.0;
  }
  const unsigned long long n_work = q.resume ? *q.n_park : static_cast<unsigned long long>(p.n_work);
  auto set_alpha = [&](int s, int it) {
    alpha[s] = path_alpha(q.amax[vid[s]], point[s], q.n_alphas, q.eps);
    f.thr[s] = __dmul_rn(p.step, alpha[s]);
    f.it[s] = it;
    f.start(s);
  };
  auto store = [&](int s, int it, bool conv, double a) {
    const int64_t v = vid[s];
#pragma unroll
    for (int i = 0; i < S::NR; ++i) {
      const int row = S::row(i, f.lane);
      if (row < S::KP) p.X[v * S::KP + row] = f.x[s][i];
    }
    if (f.lane == 0) {
      p.iters[v] = static_cast<uint32_t>(it);
      p.conv[v] = conv ? 1 : 0;
      q.alpha[v] = a;
    }
  };
  while (true) {
#pragma unroll
    for (int s = 0; s < P; ++s) {
      while (need[s]) {
        unsigned long long w = 0;
        if (f.lane == 0) w = atomicAdd(p.queue, 1ull);
        w = __shfl_sync(kFull, w, 0);
        f.clear(s);
        if (w >= n_work) {
          vid[s] = -1;
          need[s] = false;
          break;
        }
        if (q.resume) {
          const PathPark k = q.park[w];
          vid[s] = k.v;
          point[s] = k.point;
          best[s] = k.best;
          need[s] = false;
#pragma unroll
          for (int i = 0; i < S::NR; ++i) {
            const int row = S::row(i, f.lane);
            const bool in = row < K;
            f.b[s][i] = in ? p.B[vid[s] * S::KP + row] : 0.0;
            f.x[s][i] = in ? q.Xp[vid[s] * S::KP + row] : 0.0;
            f.y[s][i] = in ? q.Yp[vid[s] * S::KP + row] : 0.0;
          }
          set_alpha(s, k.it);
          break;
        }
        vid[s] = static_cast<int64_t>(w);
        store(s, 0, true, 0.0);  // the zero result: kept when alpha_max == 0 or no point is ever better
        if (q.amax[vid[s]] == 0.0) continue;
        need[s] = false;
#pragma unroll
        for (int i = 0; i < S::NR; ++i) {
          const int row = S::row(i, f.lane);
          f.b[s][i] = row < K ? p.B[vid[s] * S::KP + row] : 0.0;
        }
        point[s] = 0;
        best[s] = INFINITY;
        set_alpha(s, 0);
      }
    }
    bool any = false;
#pragma unroll
    for (int s = 0; s < P; ++s) any = any || vid[s] >= 0;
    if (!any) break;
    double mom[P];
#pragma unroll
    for (int s = 0; s < P; ++s) mom[s] = vid[s] >= 0 ? __ldg(p.mom + f.it[s]) : 0.0;
    double acc[P][S::NR];
    f.product(acc);
#pragma unroll
    for (int s = 0; s < P; ++s) {
      if (vid[s] < 0) continue;
      const bool conv = f.update(s, acc[s], mom[s], c, p.tol);
      const int it = ++f.it[s];
      if (!conv && it < p.max_iter) continue;
      executed += static_cast<unsigned long long>(it);
      // residual of this point: list its non-zero coefficients
      const int64_t v = vid[s];
      const unsigned lt = (1u << f.lane) - 1u;
      int nnz = 0;
      auto put = [&](int i, int row, bool e, int pos) {
        sp_st_f64(f.lv + 8u * P * pos, f.x[s][i], e);
        sp_st_s32(f.li + 4u * pos, row, e);
      };
#pragma unroll
      for (int i = 0; i < S::PAIRS; ++i) {
        const bool e = f.x[s][2 * i] != 0.0, o = f.x[s][2 * i + 1] != 0.0;
        const unsigned me = __ballot_sync(kFull, e), mo = __ballot_sync(kFull, o);
        const int pos = nnz + __popc(me & lt) + __popc(mo & lt);
        put(2 * i, 64 * i + 2 * f.lane, e, pos);
        put(2 * i + 1, 64 * i + 2 * f.lane + 1, o, pos + (e ? 1 : 0));
        nnz += __popc(me) + __popc(mo);
      }
      {
        const bool e = f.x[s][S::NR - 1] != 0.0;
        const unsigned me = __ballot_sync(kFull, e);
        put(S::NR - 1, 64 * S::PAIRS + f.lane, e, nnz + __popc(me & lt));
        nnz += __popc(me);
      }
      __syncwarp();
      const float* sig = q.sig ? q.sig + v * q.N : q.data + q.vox[v] * q.N;
      const double resid = sqrt(sparse_rss<P>(sig, q.Mt, q.N, static_cast<const double*>(__cvta_shared_to_generic(f.lv)),
                                            static_cast<const int*>(__cvta_shared_to_generic(f.li)), nnz, f.lane));
      __syncwarp();
      const double rss = resid * resid;
      bool last = point[s] + 1 >= q.n_alphas;
      const double limit = q.mode == 3 ? (1.0 + q.slack) * q.rss_l2[v] : 0.0;
      if (path_better(q.mode, q.N, nnz, rss, limit, best[s], last)) store(s, it, conv, alpha[s]);
      if (last) {
        need[s] = true;
        continue;
      }
      ++point[s];
#pragma unroll
      for (int i = 0; i < S::NR; ++i) f.y[s][i] = f.x[s][i];
      set_alpha(s, 0);
    }
  }
  if (p.iter_total && f.lane == 0 && executed) atomicAdd(p.iter_total, executed);
}

// The fused path on the DMMA slots of k_fista_v3: eight voxels to a warp, each
// slot on its own alpha.  Along a path the iterates fill up - a voxel spends
// most of its ~2,300 iterations at the last five of the 14 points it visits,
// with 30-60 % of y non-zero - so the product is a dense one there and the
// tensor cores carry it (118 SM cycles a voxel-iteration dense, against ~250
// of k_path_sparse).  A warp whose queue is empty and whose active slots are
// down to `park_at` leaves them to k_path_sparse, where an iteration takes a
// third of the time: the slowest voxels would otherwise finish alone.
template <int MT>
constexpr int kPathWarpDoubles = 2 * (8 * MT) * 8 + (8 * MT) + (8 * MT) / 2 + 8 + 8 + 4;

template <int MT, int WARPS, bool NONNEG>
__global__ void __launch_bounds__(32 * WARPS) k_path_dmma(PathParams pp, int park_at) {
  constexpr int KP = 8 * MT, KT = 2 * MT;
  static_assert(KT <= 32, "one word of live k-steps");
  extern __shared__ __align__(16) double smem_pd[];
  const FistaParams& p = pp.f;
  const double* sG = smem_pd;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  double* ybuf = smem_pd + MT * KT * 32 + warp * kPathWarpDoubles<MT>;  // KP x 8 [k][voxel]
  double* bbuf = ybuf + KP * 8;                                           // thread-private [mt][lane][2]
  double* lval = bbuf + KP * 8;                                           // a point's coefficients: values ...
  int* lrow = reinterpret_cast<int*>(lval + KP);                          // ... and rows
  double* s_best = lval + KP + KP / 2;                                    // per slot
  double* s_alpha = s_best + 8;
  int* s_point = reinterpret_cast<int*>(s_alpha + 8);
  for (int i = threadIdx.x; i < MT * KT * 32; i += blockDim.x) smem_pd[i] = p.gfrag[i];
  __syncthreads();

  const int g = lane >> 2, q = lane & 3;
  const double tol2x4 = 4.0 * p.tol * p.tol;
  const double c = p.step * p.n_inv;
  const unsigned long long n_work = static_cast<unsigned long long>(p.n_work);
  double x[MT][2];
  int64_t vid[2] = {-1, -1};
  int it[2] = {0, 0};
  double thr[2] = {INFINITY, INFINITY};
  bool need[2] = {true, true};
  bool exhausted = false;
  unsigned executed = 0, ksteps = 0;
  unsigned live[1] = {kFull};
  auto columns = [&](bool f0, bool f1) {  // the slots whose lanes set a flag
    const unsigned n0 = __ballot_sync(kFull, lane < 4 && f0), n1 = __ballot_sync(kFull, lane < 4 && f1);
    unsigned cols = 0;
#pragma unroll
    for (int l = 0; l < 4; ++l) cols |= (((n0 >> l) & 1u) << (2 * l)) | (((n1 >> l) & 1u) << (2 * l + 1));
    return cols;
  };

  while (true) {
    // ---- refill; a voxel with alpha_max == 0 has its zero result and its slot is filled again
    bool refilled = false;
    while (__any_sync(kFull, need[0] || need[1])) {
      refilled = true;
      const unsigned cols = columns(need[0], need[1]);
      unsigned long long base = n_work;
      if (!exhausted) {
        if (lane == 0) base = atomicAdd(p.queue, static_cast<unsigned long long>(__popc(cols)));
        base = __shfl_sync(kFull, base, 0);
        if (base + __popc(cols) >= n_work) exhausted = true;
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (!need[j]) continue;
        const int col = 2 * q + j;
        const unsigned long long cand = base + __popc(cols & ((1u << col) - 1u));
        const bool some = cand < n_work;
        const int64_t v = static_cast<int64_t>(cand);
        const double am = some ? pp.amax[v] : 0.0;
        const bool run = some && am != 0.0;
        need[j] = some && !run;
        vid[j] = run ? v : -1;
        it[j] = 0;
        const double a = run ? path_alpha(am, 0, pp.n_alphas, pp.eps) : 0.0;
        thr[j] = run ? __dmul_rn(p.step, a) : INFINITY;
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) {
          const int row = 8 * mt + g;
          x[mt][j] = 0.0;
          bbuf[(mt * 32 + lane) * 2 + j] = run ? p.B[v * KP + row] : 0.0;
          ybuf[row * 8 + col] = 0.0;
          if (some) p.X[v * KP + row] = 0.0;  // kept when alpha_max == 0 or no point is ever better
        }
        if (g == 0) {
          s_best[col] = INFINITY;
          s_alpha[col] = a;
          s_point[col] = 0;
          if (some) {
            p.iters[v] = 0;
            p.conv[v] = 1;
            pp.alpha[v] = 0.0;
          }
        }
      }
      __syncwarp();
    }
    if (refilled && exhausted) {
      const unsigned cols = columns(vid[0] >= 0, vid[1] >= 0);
      if (__popc(cols) <= park_at) {
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          if (vid[j] < 0) continue;
          const int64_t v = vid[j];
          const int col = 2 * q + j;
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) {
            const int row = 8 * mt + g;
            pp.Xp[v * KP + row] = x[mt][j];
            pp.Yp[v * KP + row] = ybuf[row * 8 + col];
          }
          if (g == 0) {
            const unsigned long long slot = atomicAdd(pp.n_park, 1ull);
            pp.park[slot] = PathPark{s_best[col], static_cast<int>(v), s_point[col], it[j], 0};
          }
        }
        break;
      }
    }
    if (!__any_sync(kFull, vid[0] >= 0 || vid[1] >= 0)) break;

    double mom[2], dx2[2], xn2[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) mom[j] = vid[j] >= 0 ? p.mom[it[j]] : 0.0;
    ksteps += dmma_fista_step<MT, NONNEG>(sG, ybuf, bbuf, live, x, mom, thr, c, lane, dx2, xn2);

    // ---- per-voxel stopping rule (fista.rs:115-127)
    bool conv[2] = {false, false}, fin[2] = {false, false};
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      if (vid[j] < 0) continue;
      it[j] += 1;
      if (!(dx2[j] > tol2x4 * fmax(xn2[j], 1e-24))) conv[j] = sqrt(dx2[j]) / fmax(sqrt(xn2[j]), 1e-12) < p.tol;
      fin[j] = conv[j] || it[j] >= p.max_iter;
    }
    __syncwarp();
    if (!__any_sync(kFull, fin[0] || fin[1])) continue;

    // ---- finished points: residual, selection, next alpha
    for (unsigned cols = columns(fin[0], fin[1]); cols != 0; cols &= cols - 1) {
      const int col = __ffs(static_cast<int>(cols)) - 1, odd = col & 1;
      const bool own = q == (col >> 1);
      const int64_t v = __shfl_sync(kFull, odd ? vid[1] : vid[0], col >> 1);
      int nnz = 0;  // its non-zero coefficients, in increasing row
#pragma unroll
      for (int mt = 0; mt < MT; ++mt) {
        const double xv = odd ? x[mt][1] : x[mt][0];
        const bool e = own && xv != 0.0;
        const unsigned m = __ballot_sync(kFull, e);
        if (e) {
          const int pos = nnz + __popc(m & ((1u << lane) - 1u));
          lval[pos] = xv;
          lrow[pos] = 8 * mt + g;
        }
        nnz += __popc(m);
      }
      __syncwarp();
      const float* sig = pp.sig ? pp.sig + v * pp.N : pp.data + pp.vox[v] * pp.N;
      const double resid =
          sqrt(sparse_rss<1>(sig, pp.Mt, pp.N, lval, lrow, nnz, lane));
      const double limit = pp.mode == 3 ? (1.0 + pp.slack) * pp.rss_l2[v] : 0.0;
      const int point = s_point[col];
      double best = s_best[col];
      const double a = s_alpha[col];
      bool last = point + 1 >= pp.n_alphas;
      const bool better = path_better(pp.mode, pp.N, nnz, resid * resid, limit, best, last);
      const double next = last ? 0.0 : path_alpha(pp.amax[v], point + 1, pp.n_alphas, pp.eps);
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (!own || j != odd) continue;
        if (better) {
#pragma unroll
          for (int mt = 0; mt < MT; ++mt) p.X[v * KP + 8 * mt + g] = x[mt][j];
        }
        if (g == 0) {
          executed += it[j];
          if (better) {
            p.iters[v] = static_cast<uint32_t>(it[j]);
            p.conv[v] = conv[j] ? 1 : 0;
            pp.alpha[v] = a;
            s_best[col] = best;
          }
          s_point[col] = point + 1;
          s_alpha[col] = next;
        }
        need[j] = last;
        if (last) vid[j] = -1;
        it[j] = 0;
        thr[j] = last ? INFINITY : __dmul_rn(p.step, next);
#pragma unroll
        for (int mt = 0; mt < MT; ++mt) ybuf[(8 * mt + g) * 8 + col] = x[mt][j];  // y = x
      }
      __syncwarp();
    }
    live[0] = kFull;
  }
  if (p.iter_total) {
    for (int o = 16; o > 0; o >>= 1) executed += __shfl_xor_sync(kFull, executed, o);
    if (lane == 0) atomicAdd(p.iter_total, static_cast<unsigned long long>(executed));
  }
  if (p.kstep_total && lane == 0) atomicAdd(p.kstep_total, static_cast<unsigned long long>(ksteps));
}

}  // namespace csd
