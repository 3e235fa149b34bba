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
// iteration, 0.3 us against the 1.25-2 us of a DMMA warp.  Volume fits, N =
// 259, against the DMMA kernel alone: 108 voxels 1.64 -> 0.47 ms, 4,000
// voxels 3.55 -> 0.99 ms, 32,000 voxels at order 8 11.4 -> 3.5 ms (with the
// residual pass that no output reads dropped there).
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
template <int K, int P, bool NONNEG>
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
    lane = threadIdx.x & 31;
    const uint32_t base = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
    gp = base + 16u * lane;
    gr = base + 8u * (64 * S::PAIRS + (lane < S::REM ? lane : 0));
    lv = base + static_cast<uint32_t>(S::G_BYTES + (threadIdx.x >> 5) * S::WARP_BYTES);
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
    constexpr int U = P == 1 ? 4 : 2;  // columns per group
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
    double g1[U];
#pragma unroll
    for (int c = 0; c < U; ++c) g1[c] = 0.0;
    const bool rem = lane < S::REM;
#pragma unroll 1
    for (int t = 0; t < n; t += U) {
      uint32_t off[U];
      double yv[U][P];
      if constexpr (U == 4) {
        const int4 id = sp_ld_i4(li + 4u * t);
        off[0] = id.x, off[1] = id.y, off[2] = id.z, off[3] = id.w;
      } else {
        const int2 id = sp_ld_i2(li + 4u * t);
        off[0] = id.x, off[1] = id.y;
      }
#pragma unroll
      for (int e = 0; e < U * P; e += 2) {
        const double2 v = sp_ld_v2(lv + 8u * (P * t + e));
        yv[e / P][e % P] = v.x;
        yv[(e + 1) / P][(e + 1) % P] = v.y;
      }
      double2 g2[U][S::PAIRS > 0 ? S::PAIRS : 1];
#pragma unroll
      for (int c = 0; c < U; ++c) {
#pragma unroll
        for (int i = 0; i < S::PAIRS; ++i) g2[c][i] = sp_ld_g2(gp + off[c] + 512u * i);
        sp_ld_g1(g1[c], gr + off[c], rem);
      }
#pragma unroll
      for (int c = 0; c < U; ++c)
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
  extern __shared__ __align__(16) unsigned char sp_smem[];
  SparseFista<K, P, NONNEG> f;
  f.init(p.G, sp_smem);
  __syncthreads();
  const unsigned long long n_work = p.n_work_dev ? *p.n_work_dev : static_cast<unsigned long long>(p.n_work);
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

}  // namespace csd
