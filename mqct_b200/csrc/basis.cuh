// basis.cuh -- tables of a direct build: rotor wavefunctions on the angular grid and the
// PES times the quadrature weights, from small per-rotor tables.
#pragma once
#include "common.cuh"
#include "pes.cuh"

namespace mqct {

// Where a basis row goes: the FP64 table psi[row][G2] of the FP64 contraction, or the FP32
// images of the tensor-core contraction (per m-block and 64-point chunk, the block's rows of
// 66 values; the padding stays as it was cleared).
struct BasisOut {
  double2* psi;
  float2* img;
  const int64_t* row_off;  // image place of the row's chunk 0
  const int* row_step;     // distance of the row's places in consecutive chunks
  int G2;
};
template <bool IMG>
__device__ __forceinline__ void basis_put(const BasisOut& o, int row, int64_t off, int step, int g,
                                          double re, double im) {
  if constexpr (IMG) o.img[off + (int64_t)(g >> 6) * step + (g & 63)] = make_float2((float)re, (float)im);
  else o.psi[(size_t)row * o.G2 + g] = make_double2(re, im);
}

// ------------------------------------------------------------------ rotor + atom (type 4)
// psi(beta, gamma) = sum_K (c_K d^j_{Km}(beta)) e^{iK gamma}, one CTA per basis row.  The
// products c_K d of the row's nonzero K (half of them for an asymmetric top) are formed once
// per beta in shared memory; a thread then takes one gamma and four betas, so that a phase
// read serves four sums.  Formed value by value from the tables (one thread per grid point,
// two table reads per K) it was bound by those reads: 70 us at 969 rows x 2 304 points, and
// 18 us more to convert the FP64 table into the FP32 images that this kernel writes itself;
// now 18 us.  The sum over K runs in the same order.
constexpr int kCdMax = 2048;  // products in shared memory (a tile of betas)
template <bool IMG>
__global__ void __launch_bounds__(256)
basis_top_kernel(const int* __restrict__ row_state, const int* __restrict__ st_chan,
                 const int* __restrict__ st_m, const int* __restrict__ ch_j,
                 const double* __restrict__ vec, int ldv, int n_beta, int n_gamma,
                 const double* __restrict__ dtab, const double2* __restrict__ phase, int jmax,
                 BasisOut out) {
  __shared__ double cd[kCdMax];
  __shared__ int nz[96];
  __shared__ int n_nz;
  const int r = blockIdx.x, st = row_state[r], ch = st_chan[st], j = ch_j[ch], m = st_m[st];
  const double* c = vec + (size_t)ch * ldv;
  const int nk = 2 * j + 1;
  if (threadIdx.x < 32) {
    int cnt = 0;
    for (int i0 = 0; i0 < nk; i0 += 32) {
      const int i = i0 + threadIdx.x;
      const bool use = i < nk && c[i] != 0.0;
      const unsigned b = __ballot_sync(0xffffffffu, use);
      if (use) nz[cnt + __popc(b & ((1u << threadIdx.x) - 1u))] = i;
      cnt += __popc(b);
    }
    if (threadIdx.x == 0) n_nz = cnt;
  }
  __syncthreads();
  const int n = n_nz;
  const double* dj = dtab + (size_t)(j * (2 * j - 1) * (2 * j + 1) / 3 + (m + j)) * n_beta;
  const double2* pk = phase + (size_t)(jmax - j) * n_gamma;
  const int64_t off = IMG ? out.row_off[r] : 0;
  const int step = IMG ? out.row_step[r] : 0;
  const int bt = max(4, min((n_beta + 3) & ~3, (n ? kCdMax / n : kCdMax) & ~3));
  for (int b0 = 0; b0 < n_beta; b0 += bt) {
    __syncthreads();
    for (int q = threadIdx.x; q < bt * n; q += blockDim.x) {
      const int k = q / bt, b = q - k * bt;  // betas fastest: coalesced table reads
      cd[b * n + k] = b0 + b < n_beta ? c[nz[k]] * dj[(size_t)nz[k] * nk * n_beta + b0 + b] : 0.0;
    }
    __syncthreads();
    for (int it = threadIdx.x; it < n_gamma * (bt / 4); it += blockDim.x) {
      const int bq = it / n_gamma, ig = it - bq * n_gamma;
      const double* cq = cd + 4 * bq * n;
      double re[4] = {0.0, 0.0, 0.0, 0.0}, im[4] = {0.0, 0.0, 0.0, 0.0};
      for (int k = 0; k < n; ++k) {
        const double2 e = __ldg(pk + (size_t)nz[k] * n_gamma + ig);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const double d = cq[u * n + k];
          re[u] += d * e.x;
          im[u] += d * e.y;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int b = b0 + 4 * bq + u;
        if (b < n_beta) basis_put<IMG>(out, r, off, step, b * n_gamma + ig, re[u], im[u]);
      }
    }
  }
}

// ------------------------------------------------------------------ two rotors (type 0)
// Per-rotor tables: psi1(level, m1; beta1, gamma1), psi2(level, m2; beta2, gamma2), the
// phases e^{i m2 alpha2}, and the rotated interaction sites of both rotors.
struct PairTab {
  int n_lm1, n_lm2;                        // (level, m) of rotor 1 and 2
  const int *lm1_ch, *lm1_m, *lm2_ch, *lm2_m;  // a channel with that level, and m
  const int *ch_lm1, *ch_lm2;              // per channel: place of (its level, m = -j)
  int J2;                                  // largest j2
  int n_s1, n_s2;                          // sites (0: no site surface)
  const double *s1, *s2;
  double2 *psi1, *psi2, *ph2;
  double *x1, *x2;
};

// psi for SYS_TYPE 0: sum_{m1} CG(j1 m1 j2 m2 | j12 m12) psi1_{m1}(beta1, gamma1)
// psi2_{m2}(beta2, gamma2) e^{i m2 alpha2} on the 5-D grid (WF_ASYM_TOP_ASYM_TOP,
// MQCT_SOURCE_CODES/basis_wave_functions.f:1-41).  A thread keeps its grid point's place in
// the tables for a run of rows.  Bound by its output (8 B a value as an FP32 image); with
// both rotors' Wigner functions evaluated at every grid point it took 1 625 us for 100 rows
// x 72 900 points, now 58 us.
constexpr int kRowRun = 16;
template <bool IMG>
__global__ void __launch_bounds__(256)
basis_pair_kernel(int n_rows, const int* __restrict__ row_state, const int* __restrict__ st_chan,
                  const int* __restrict__ st_m, const int* __restrict__ ch_j1,
                  const int* __restrict__ ch_j2, const double* __restrict__ cg, int cg_ld, int nb1,
                  int ng1, int nbb, int naa, int ngg, PairTab t, BasisOut out) {
  const int g = blockIdx.x * blockDim.x + threadIdx.x;
  if (g >= out.G2) return;
  unsigned q = (unsigned)g;
  const int ig2 = q % (unsigned)ngg;
  q /= (unsigned)ngg;
  const int ig1 = q % (unsigned)ng1;
  q /= (unsigned)ng1;
  const int ib2 = q % (unsigned)nbb;
  q /= (unsigned)nbb;
  const int ib1 = q % (unsigned)nb1, ia2 = q / (unsigned)nb1;
  const int np1 = nb1 * ng1, np2 = nbb * ngg;
  const double2* a1 = t.psi1 + ib1 * ng1 + ig1;
  const double2* a2 = t.psi2 + ib2 * ngg + ig2;
  const double2* ap = t.ph2 + ia2;
  const int r1 = min(n_rows, (int)(blockIdx.y + 1) * kRowRun);
  for (int r = blockIdx.y * kRowRun; r < r1; ++r) {
    const int st = row_state[r], ch = st_chan[st], m = st_m[st];
    const int j1 = ch_j1[ch], j2 = ch_j2[ch];
    const double* cgs = cg + (size_t)st * cg_ld;
    const double2* b1 = a1 + (size_t)(t.ch_lm1[ch] + j1) * np1;
    const double2* b2 = a2 + (size_t)(t.ch_lm2[ch] + j2) * np2;
    double re = 0.0, im = 0.0;
    for (int m1 = max(-j1, m - j2); m1 <= min(j1, m + j2); ++m1) {
      const double w = cgs[m1 + j1];
      if (w == 0.0) continue;
      const int m2 = m - m1;
      const double2 p1 = b1[(int64_t)m1 * np1], v = b2[(int64_t)m2 * np2];
      const double2 e = ap[(m2 + t.J2) * naa];
      const double2 p2 = make_double2(v.x * e.x - v.y * e.y, v.x * e.y + v.y * e.x);
      re += w * (p1.x * p2.x - p1.y * p2.y);
      im += w * (p1.x * p2.y + p1.y * p2.x);
    }
    basis_put<IMG>(out, r, IMG ? out.row_off[r] : 0, IMG ? out.row_step[r] : 0, g, re, im);
  }
}

// ------------------------------------------------------------------ site surfaces
// A site-site surface in the form the weight kernel reads: the distinct site (pairs) u, the
// terms in the order of their u (u0[u] .. u0[u + 1]), five values per term: a, re, D, C6,
// 1 / rd^2.
struct SiteTerms {
  int n_terms, n_u;
  const int* u0;
  const int* us1;   // site of rotor 1 (the rotor)
  const int* us2;   // site of rotor 2 (two rotors)
  const double* q;
};
constexpr int kSiteMax = 512;      // terms and distinct sites of this form
constexpr int kGeoMax = 1536;      // (grid point, site) places of one CTA

// W[g][i] = wt[g] V(R_i, g) for SITES1 (rotor + atom) and SITES2 (two rotors).  The distance
// of a site (pair) is r^2 = rho^2 + (R + z)^2 with rho and z functions of the angles alone:
// they are formed once per grid point and site in shared memory, r and 1/r^6 once per site
// (by one reciprocal square root), and the dispersion damping 1 - e^{-(r/rd)^6} only below
// (r/rd)^6 = 40, where it is 1 to double precision.  FP64-bound: per term one exp (two near the
// well) and about twenty FP64 operations; with the rotations of both rotors, a square root
// and two divisions in every term of every radial point it took 10 900 us at 72 900 points x
// 101 R x 81 terms and 69 us at 2 304 x 300 x 12; now 3 170 and 49 us.
// SYS 4: the PES arguments are (-beta, -gamma), SYS 0: rotor 1 at (0, beta1, gamma1), rotor 2
// at (alpha2, beta2, gamma2) (MQCT_SOURCE_CODES/pes_sys_type.f:32-37, 90-97), SYS 1: beta.
template <int SYS>
__global__ void __launch_bounds__(128)
pes_sites_kernel(SiteTerms ps, int G2, int nR, int GB, const double* __restrict__ R,
                 const double* __restrict__ beta, const double* __restrict__ gamma, int n_gamma,
                 const double* __restrict__ sites, int nb1, int ng1, int nbb, int ngg, int n_s1,
                 int n_s2, const double* __restrict__ x1, const double* __restrict__ x2,
                 const double* __restrict__ wt, double* __restrict__ W, int ldw) {
  __shared__ double2 geo[kGeoMax];
  extern __shared__ double site_sm[];
  double* sq = site_sm;                                       // 5 per term
  int* su = reinterpret_cast<int*>(sq + 5 * ps.n_terms);      // n_u + 1
  const int g0 = blockIdx.x * GB, ng = min(GB, G2 - g0);
  for (int q = threadIdx.x; q < 5 * ps.n_terms; q += blockDim.x) sq[q] = ps.q[q];
  for (int q = threadIdx.x; q <= ps.n_u; q += blockDim.x) su[q] = ps.u0[q];
  for (int q = threadIdx.x; q < ng * ps.n_u; q += blockDim.x) {
    const int gl = q / ps.n_u, u = q - gl * ps.n_u, g = g0 + gl;
    double rho2, z;
    if constexpr (SYS == 0) {
      unsigned p = (unsigned)g;
      const int ig2 = p % (unsigned)ngg;
      p /= (unsigned)ngg;
      const int ig1 = p % (unsigned)ng1;
      p /= (unsigned)ng1;
      const int ib2 = p % (unsigned)nbb;
      p /= (unsigned)nbb;
      const int ib1 = p % (unsigned)nb1, ia2 = p / (unsigned)nb1;
      const double* a = x1 + 3 * ((size_t)(ib1 * ng1 + ig1) * n_s1 + ps.us1[u]);
      const double* b = x2 + 3 * ((size_t)((ia2 * nbb + ib2) * ngg + ig2) * n_s2 + ps.us2[u]);
      const double dx = b[0] - a[0], dy = b[1] - a[1];
      rho2 = dx * dx + dy * dy;
      z = b[2] - a[2];
    } else {
      const int ib = SYS == 4 ? g / n_gamma : g;
      double sb, cb, sg = 0.0, c2 = 1.0;
      sincos(SYS == 4 ? -beta[ib] : beta[ib], &sb, &cb);
      if (SYS == 4) sincos(-gamma[g - ib * n_gamma], &sg, &c2);
      const double dx = sb * c2, dy = sb * sg, dz = cb;   // the atom's direction
      const double* s = sites + 3 * ps.us1[u];
      const double t = dx * s[0] + dy * s[1] + dz * s[2];
      const double px = s[0] - t * dx, py = s[1] - t * dy, pz = s[2] - t * dz;
      rho2 = px * px + py * py + pz * pz;
      z = -t;
    }
    geo[q] = make_double2(rho2, z);
  }
  __syncthreads();
  for (int it = threadIdx.x; it < ng * nR; it += blockDim.x) {
    const int gl = it / nR, i = it - gl * nR;
    const double Ri = R[i];
    const double2* ge = geo + gl * ps.n_u;
    double v = 0.0;
    for (int u = 0; u < ps.n_u; ++u) {
      const double z = Ri + ge[u].y;
      const double r2 = z * z + ge[u].x;
      const double ir = rsqrt(r2), r = r2 * ir;
      const double i2 = ir * ir, i6 = i2 * i2 * i2;
      for (int t = su[u]; t < su[u + 1]; ++t) {
        const double* q = sq + 5 * t;
        const double e = exp(-q[0] * (r - q[1]));
        const double x2v = r2 * q[4], x6 = x2v * x2v * x2v;
        const double damp = x6 > 40.0 ? 1.0 : 1.0 - exp(-x6);
        v += q[2] * (e * e - 2.0 * e) - q[3] * damp * i6;
      }
    }
    W[(size_t)(g0 + gl) * ldw + i] = wt[g0 + gl] * v;
  }
}

// ------------------------------------------------------------------ Legendre surface
// W[g][i] = wt[g] sum_l (A_l e^{-b_l R} - C_l / R^6) P_l(cos beta): the radial factors once
// per CTA (a block of 128 R) and the polynomials once per beta instead of per value.
constexpr int kLegMax = 40, kLegG = 8;
__global__ void __launch_bounds__(128)
pes_legendre_kernel(int n, const double* __restrict__ p, int G2, int nR,
                    const double* __restrict__ R, const double* __restrict__ beta, int n_gamma,
                    const double* __restrict__ wt, double* __restrict__ W, int ldw) {
  __shared__ double f[kLegMax][128];
  __shared__ double P[kLegG][kLegMax];
  const int i = blockIdx.x * 128 + threadIdx.x, g0 = blockIdx.y * kLegG;
  if (i < nR) {
    const double r = R[i], r2 = r * r, r6 = r2 * r2 * r2;
    for (int l = 0; l < n; ++l) f[l][threadIdx.x] = p[l] * exp(-p[n + l] * r) - p[2 * n + l] / r6;
  }
  if (threadIdx.x < kLegG && g0 + (int)threadIdx.x < G2) {
    const double x = cos(beta[(g0 + threadIdx.x) / n_gamma]);
    double pm = 1.0, pc = x;  // P_l(x) by Bonnet's recurrence
    for (int l = 0; l < n; ++l) {
      double pl;
      if (l == 0) pl = 1.0;
      else if (l == 1) pl = x;
      else {
        pl = ((2.0 * l - 1.0) * x * pc - (l - 1.0) * pm) / l;
        pm = pc;
        pc = pl;
      }
      P[threadIdx.x][l] = pl;
    }
  }
  __syncthreads();
  if (i >= nR) return;
  for (int gl = 0; gl < kLegG && g0 + gl < G2; ++gl) {
    double v = 0.0;
    for (int l = 0; l < n; ++l) v += f[l][threadIdx.x] * P[gl][l];
    W[(size_t)(g0 + gl) * ldw + i] = wt[g0 + gl] * v;
  }
}

}  // namespace mqct
