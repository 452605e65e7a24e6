// finalize.cuh -- the last step of every matrix build: units, MIJ_CUTOFF and the clamped
// spline of one matrix element (its column of nR radial values), by one warp.
//
//  (a) the column, already in Hartree, is written to Mat_el(:,k);
//  (b) MIJ_CUTOFF at R~r_cut1/r_cut2 (MQCT_SOURCE_CODES/matrix_ini.f:1969-1997): the
//      column is zeroed and flagged when max(|M(ir1)|, |M(ir2)|) < cut;
//  (c) the clamped cubic spline with finite-difference end slopes
//      (MQCT_SOURCE_CODES/matrix_ini.f:2005-2016; recurrence of
//      MQCT_SOURCE_CODES/suppl_routines.f:914-965).  With both end slopes equal to the end
//      differences, u_0 = 0 and u_n = 0; the remaining recurrences
//        u_i = t_i - s_i u_{i-1},   y2_i = f_i y2_{i+1} + u_i
//      have grid-only s_i, f_i and data terms t_i = c_i (d_i - d_{i-1}),
//      d_i = (y_{i+1} - y_i) / h_i.
//
// What bounds it: the output (16 B per value) where there are many columns, else the
// latency of the two recurrences.  Both are compositions of affine maps x -> a x + b: each
// lane composes the maps of a contiguous segment of the column, a shuffle scan composes
// the segments, each lane replays its segment from the value that enters it.  The a parts
// depend on the grid alone, so a warp forms the products its scan steps need once and
// keeps them for all of its columns: a scan moves one double per step.  One warp per
// column and no block barrier: the earlier form (one CTA of 128 threads per column, one of
// its warps scanning) spent most of a column's time with three warps waiting.  Measured on
// a B200: 31 977 columns of 300 points from three partial sums 135 -> 92 us (0.35 GB of DRAM
// traffic); 301 204 columns of 101 points with the expansion's contraction 2 150 -> 555 us.
#pragma once
#include "common.cuh"

namespace mqct {

// A lane's segment is an odd number of points, so that the 16 lanes of a half warp, L
// doubles apart, read 16 different 8-byte banks.
__host__ __device__ __forceinline__ int fin_seg(int nR) { return nR > 2 ? ((nR + 29) / 32) | 1 : 1; }
__host__ __device__ __forceinline__ int fin_len(int nR) { return (nR + 1) & ~1; }

// What every column of a build shares.
struct FinGrid {
  int nR, ir1, ir2;
  double cut;          // Hartree
  const double* gc;    // 5 x nR: 1/h_i, c_i, s_i, f_i, and the factor of y2_{n-1} at [4 nR]
  double* mat;
  int* skipped;        // may be null
  double* y2;          // may be null
};

// Register-resident segments of at most LM points; LM = 0: any nR, segments in shared memory.
template <int LM>
struct FinLane {
  int i0, n;           // first interior point of the lane's segment, its length
  int last;            // the lane that holds point nR - 2
  const double* mul;   // shared: forward [k][lane], backward [5 + k][lane] scan multipliers,
                       // [10][lane] the product of the f of all later segments
  double ylf;          // y2_{n-1} = ylf * u_{n-2}
};
constexpr int kFinMul = 11 * 32;

// Shared memory of one CTA: the scan multipliers, the grid coefficients (four rows),
// then per warp its column (and for LM = 0 a second row).
template <int LM>
__host__ __device__ __forceinline__ size_t fin_smem(int nR, int warps) {
  return sizeof(double) * (kFinMul + (size_t)fin_len(nR) * (4 + (size_t)warps * (LM ? 1 : 2)));
}

// Grid coefficients into shared memory (all threads of the CTA; ends with a barrier) and
// the scan multipliers of the lanes' segments (the same in every warp).
template <int LM>
__device__ __forceinline__ void fin_init(const FinGrid& g, double* sm, FinLane<LM>& f) {
  const int nR = g.nR, ld = fin_len(nR);
  double* coef = sm + kFinMul;
  for (int q = threadIdx.x; q < 4 * nR; q += blockDim.x) {
    const int a = q / nR, i = q - a * nR;
    coef[a * ld + i] = g.gc[q];
  }
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int m = nR - 2;                       // interior points 1 .. nR - 2
  const int L = fin_seg(nR);
  f.i0 = 1 + lane * L;
  f.n = max(0, min(L, m - lane * L));
  f.last = m > 0 ? (m - 1) / L : 0;
  f.ylf = g.gc[4 * (size_t)nR];
  f.mul = sm;
  if (threadIdx.x < 32) {
    double a = 1.0, b = 1.0;
    for (int e = 0; e < f.n; ++e) {
      a *= -coef[2 * ld + f.i0 + e];
      b *= coef[3 * ld + f.i0 + e];
    }
    const unsigned full = 0xffffffffu;
#pragma unroll
    for (int k = 0; k < 5; ++k) {
      const int o = 1 << k;
      sm[32 * k + lane] = a;
      sm[32 * (5 + k) + lane] = b;
      const double pa = __shfl_up_sync(full, a, o), pb = __shfl_down_sync(full, b, o);
      if (lane >= o) a *= pa;
      if (lane + o < 32) b *= pb;
    }
    const double bx = __shfl_down_sync(full, b, 1);
    sm[320 + lane] = lane == 31 ? 1.0 : bx;
  }
  __syncthreads();
}

// Q columns k[q] (k < 0: none), their values in Hartree in the warp's shared rows cols +
// q ld: Mat_el, the flags and y2.  The recurrences of the Q columns run interleaved (a column
// alone is a chain of dependent FP64 operations and shuffles) and share the reads of the
// grid's coefficients.  NC: groups of 32 points that hold a register-resident column; tb:
// scratch rows of the LM = 0 form (Q = 1).
template <int LM, int NC, int Q>
__device__ __forceinline__ void fin_columns(const FinGrid& g, const FinLane<LM>& f,
                                            const double* coef, double* cols, double* tb,
                                            const int64_t (&k)[Q]) {
  static_assert(LM > 0 || Q == 1, "the shared-memory form takes one column");
  const unsigned full = 0xffffffffu;
  const int lane = threadIdx.x & 31, nR = g.nR, ld = fin_len(nR);
  bool drop[Q];
  bool work = false;
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    const double* col = cols + q * ld;
    drop[q] = fmax(fabs(col[g.ir1]), fabs(col[g.ir2])) < g.cut;
    if (k[q] < 0) continue;
    work |= !drop[q];
    double* out = g.mat + (size_t)k[q] * nR;
    if constexpr (LM > 0) {
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (lane + 32 * c < nR) out[lane + 32 * c] = drop[q] ? 0.0 : col[lane + 32 * c];
    } else {
      for (int i = lane; i < nR; i += 32) out[i] = drop[q] ? 0.0 : col[i];
    }
    if (lane == 0 && g.skipped) g.skipped[k[q]] = drop[q] ? 1 : 0;
  }
  if (!g.y2) return;
  if (!work || nR < 3) {
#pragma unroll
    for (int q = 0; q < Q; ++q)
      if (k[q] >= 0)
        for (int i = lane; i < nR; i += 32) g.y2[(size_t)k[q] * nR + i] = 0.0;
    return;
  }
  const double* invh = coef + f.i0;
  const double* cfac = invh + ld;
  const double* sfac = cfac + ld;
  const double* ffac = sfac + ld;
  double* seg = cols + f.i0;   // the lane's points of column 0
  double* ts = tb + f.i0;
  double tv[LM ? LM : 1][Q], be[Q], u[Q], y[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) be[q] = 0.0;
  // data terms and the composed forward map of the segment
  if (f.n > 0) {
    double ym[Q], d0[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      ym[q] = seg[q * ld];
      d0[q] = (ym[q] - seg[q * ld - 1]) * invh[-1];
    }
    auto point = [&](int e, double (&t)[Q]) {
      const double ih = invh[e], cf = cfac[e], sf = -sfac[e];
#pragma unroll
      for (int q = 0; q < Q; ++q) {
        const double yr = seg[q * ld + e + 1];
        const double d1 = (yr - ym[q]) * ih;
        t[q] = cf * (d1 - d0[q]);
        be[q] = fma(sf, be[q], t[q]);
        ym[q] = yr;
        d0[q] = d1;
      }
    };
    if constexpr (LM > 0) {
#pragma unroll
      for (int e = 0; e < LM; ++e)
        if (e < f.n) point(e, tv[e]);
    } else {
      for (int e = 0; e < f.n; ++e) {
        point(e, tv[0]);
        ts[e] = tv[0][0];
      }
    }
  }
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const double m = f.mul[32 * s + lane];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const double p = __shfl_up_sync(full, be[q], 1 << s);
      if (lane >= (1 << s)) be[q] = fma(m, p, be[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    u[q] = __shfl_up_sync(full, be[q], 1);  // the value entering the segment; u_0 = 0
    if (lane == 0) u[q] = 0.0;
  }
  // replay
  if constexpr (LM > 0) {
#pragma unroll
    for (int e = 0; e < LM; ++e)
      if (e < f.n) {
        const double sf = -sfac[e];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          u[q] = fma(sf, u[q], tv[e][q]);
          tv[e][q] = u[q];
        }
      }
  } else {
    for (int e = 0; e < f.n; ++e) {
      u[0] = fma(-sfac[e], u[0], ts[e]);
      ts[e] = u[0];
    }
  }
  // the composed backward map (from the segment's top down)
  double yl[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    yl[q] = f.ylf * __shfl_sync(full, u[q], f.last);
    be[q] = 0.0;
  }
  if constexpr (LM > 0) {
#pragma unroll
    for (int e = LM - 1; e >= 0; --e)
      if (e < f.n) {
        const double ff = ffac[e];
#pragma unroll
        for (int q = 0; q < Q; ++q) be[q] = fma(ff, be[q], tv[e][q]);
      }
  } else {
    for (int e = f.n - 1; e >= 0; --e) be[0] = fma(ffac[e], be[0], ts[e]);
  }
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const double m = f.mul[32 * (5 + s) + lane];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      const double p = __shfl_down_sync(full, be[q], 1 << s);
      if (lane + (1 << s) < 32) be[q] = fma(m, p, be[q]);
    }
  }
  {
    const double m = f.mul[320 + lane];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      y[q] = __shfl_down_sync(full, be[q], 1);
      if (lane == 31) y[q] = 0.0;
      y[q] = fma(m, yl[q], y[q]);          // y2 at the point above the segment
    }
  }
  __syncwarp();                            // every lane has read the columns' values
  if constexpr (LM > 0) {
#pragma unroll
    for (int e = LM - 1; e >= 0; --e)
      if (e < f.n) {
        const double ff = ffac[e];
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          y[q] = fma(ff, y[q], tv[e][q]);
          seg[q * ld + e] = y[q];
        }
      }
  } else {
    for (int e = f.n - 1; e >= 0; --e) {
      y[0] = fma(ffac[e], y[0], ts[e]);
      seg[e] = y[0];
    }
  }
  if (lane == 0) {
    const double f0 = coef[3 * ld];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      cols[q * ld + nR - 1] = yl[q];
      cols[q * ld] = f0 * y[q];            // lane 0 ends at point 1; u_0 = 0
    }
  }
  __syncwarp();
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    if (k[q] < 0) continue;
    const double* col = cols + q * ld;
    double* oy = g.y2 + (size_t)k[q] * nR;
    if constexpr (LM > 0) {
#pragma unroll
      for (int c = 0; c < NC; ++c)
        if (lane + 32 * c < nR) oy[lane + 32 * c] = drop[q] ? 0.0 : col[lane + 32 * c];
    } else {
      for (int i = lane; i < nR; i += 32) oy[i] = drop[q] ? 0.0 : col[i];
    }
  }
}

}  // namespace mqct
