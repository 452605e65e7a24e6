// contract_tc.cu -- split-precision tensor-core contraction of the matrix build
// on sm_100a: tcgen05.mma kind::f16 with FP32 accumulators in TMEM, drained into
// sums of two FP32 parts (48 bits) after every short accumulation.
//
//   M[row, i] = w sum_{c, alpha} sum_{g in chunk c} X[row, g] W[g, i]
//   X = X_hi + X_lo, W = W_hi + W_lo (16-bit parts),
//   D = X_hi W_hi + X_hi W_lo + X_lo W_hi          (FP32, one K-chunk of 64 points)
//   S + E += D                                      (S the FP32 sum, E its rounding errors)
//
// Two 16-bit formats: BF16x3 (8 significant bits per part, ~16 bits kept) and
// F16x3 (11 bits per part, ~22 bits kept; the products of FP16 parts are exact
// in FP32).  FP16's range is narrow, so in F16x3 X is scaled by 2^14 and every
// radial column of W by the power of two that brings its largest entry to
// [2^13, 2^14); the exact inverse is applied to the sums.
//
// Accuracy: the tensor core adds the products of one MMA into its FP32
// accumulator with a rounding relative to the largest addend, so a long
// accumulation loses bits in proportion to its length and to how much its terms
// cancel.  Here an accumulator lives for one K-chunk of one group of alpha points (3 x 4 MMAs
// of K = 16 a point) and is then added to the pair S + E by TwoSum, whose S is exact up to E:
// against sums in FP64 a build's elements move by 1e-12 (2-norm; the FP32 partials carry 6e-8, the
// split 5e-6), its error against 64 bits is the same 5.3e-6 (7.0e-6 with an alpha axis).  E is
// folded back into S after every chunk of several groups (48 bits); with one group a chunk it
// grows to half an ulp of S for each of the n chunks of a unit, so that its own rounding stays below
// n^2 2^-49 of the largest sum: 2e-12 for 36 chunks, 2e-9 for 1 000 (a fold every 16 chunks spills:
// 612 -> 639 us).  S has FP32's range: W is scaled in F16x3; BF16x3 sums overflow at 3.4e38.  The
// ranges of a split axis and the alpha weight (the same for every point of the midpoint grid) are
// FP64.  The tensor-core operand of a K-chunk is the same for every alpha point of a same-m pair
// (the e^{i m alpha} phases of the two states cancel, so the integrand at every alpha point is
// w Re(psi_a^* psi_b) exactly), and the tensor cores contract it once per alpha point.
//
// What bounds it, and what the forms before measured (B200; asymmetric top + atom, j <= 8, 31 977
// pairs, 48 x 48 points, 300 R, whole build after a pause; builds that follow one another run at
// 0.92 of these rates under the power cap: 5.6 ms; with the 48-point alpha axis):
//   * FP64 instructions beside MMAs: a drain of converted values into FP64 sums and the MMAs slowed
//     one another down to half (3 100 clocks a group of two alpha points against 1 750 for its
//     MMAs alone; the same without the TMEM loads).  In packed FP32 adds: 7.9 -> 5.1 ms;
//   * the operand X in shared memory was read again by every MMA, 60 clocks of shared-memory
//     bandwidth for 56 of tensor work.  In TMEM: 5.1 -> 4.9 ms (4.7 of them this kernel), and 64 KB
//     of shared memory free;
//   * with one group a chunk (no alpha axis), forming X and the drains alternate in the same
//     warps: 903 -> 612 us, by the cheaper drain, X through TMEM, accesses that stay in the
//     shared address space (no spills in this form; 76 to 80 bytes in those of several groups), and
//     sums stored as whole sectors.
// The rest is the MMAs (58 to 62 clocks of N = 96 to 112 issued in order by one thread), about 300
// clocks between two groups, and, without the alpha axis, X.
//
// Work unit = one 128-row tile of pair rows (one m-block) x one column part (at
// most 112 radial points) x one range of K-chunks.  Two FP32 accumulators of a part in TMEM
// (double buffering: the tensor cores fill one while the epilogue drains the other) and the
// sums of a part in registers.
// Warp roles (64 + 32 PE threads; PE = 16 epilogue warps when a K-chunk has several
// accumulation groups, 8 when it has one):
//   warp 0      bulk-copy (TMA) producer: per K-chunk the pre-arranged W image of
//               the part (hi and lo planes, K-major core-matrix layout) and the
//               block's rotor-basis slice, one cp.async.bulk each, mbarrier
//               complete_tx, double-buffered where shared memory allows;
//   warp 1      TMEM allocator + single-thread MMA issuer;
//   warps 2..   X producers and epilogue: per K-chunk X = Re(psi_a^* psi_b) in FP32
//               from the staged basis, split to 16-bit hi/lo parts in TMEM (lane = row, PE / 4
//               threads per tile row); then, for every group of the chunk, tcgen05.ld of the
//               accumulator and the update of the sums (PE / 4 warps per TMEM lane quarter, each
//               a share of the part's columns); at the end of a unit the sums go to global
//               memory in FP64, one array per K range.
// W uses the K-major SWIZZLE_NONE canonical layout: 8 rows x
// 16 B core matrices, K-adjacent core matrices LBO apart, 8-row groups SBO =
// 128 B apart.  Every mbarrier wait is bounded; on timeout the CTA records an
// error code, drains, frees its TMEM and returns.
#include <cfloat>
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>

#include "matrix_plan.cuh"
#include "ptx.cuh"

namespace mqct {

constexpr int TC_M = 128;        // rows per tile
constexpr int TC_KC = 64;        // K elements per chunk (8 core-matrix columns of 8 x 16 bit)
constexpr int TC_PSI_LD = 66;    // float2 per staged basis row (64 + pad)
constexpr int TC_NC_MAX = 112;   // columns of one part (TMEM buffer width)
constexpr int TC_MAX_PARTS = 8;
constexpr int TC_NLD = 16;       // columns of one TMEM read of the epilogue
// Tensor memory: two accumulators, then two A stages, each a hi and a lo plane of 16-bit pairs.
constexpr int TC_A_PLANE = TC_KC / 2;
constexpr int TC_TMEM_A = 2 * TC_NC_MAX;
constexpr int TC_TMEM_COLS = 512;  // allocation (a power of two)
static_assert(TC_TMEM_A + 4 * TC_A_PLANE <= TC_TMEM_COLS, "accumulators and A stages must fit");
// Epilogue warps: a template parameter of the kernel, 8 (two per TMEM lane quarter) or 16.
template <int PE>
struct TcShape {
  static constexpr int THREADS = 64 + 32 * PE;
  static constexpr int PRODUCERS = 32 * PE;           // X-producer / epilogue threads
  static constexpr int WPQ = PE / 4;                  // epilogue warps per TMEM lane quarter
  static constexpr int NCH_MAX = TC_NC_MAX * 4 / PE;  // columns drained by one epilogue thread
};
constexpr uint32_t TC_SPIN_LIMIT = kSpinLimit;  // bounded mbarrier waits

// Shared-memory matrix descriptor: K-major, SWIZZLE_NONE, version 1.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  uint64_t d = 0;
  d |= (uint64_t)((addr >> 4) & 0x3FFF);
  d |= (uint64_t)((lbo >> 4) & 0x3FFF) << 16;
  d |= (uint64_t)((sbo >> 4) & 0x3FFF) << 32;
  d |= (uint64_t)1 << 46;  // descriptor version (sm_100)
  return d;                // base offset 0, lbo mode 0, layout SWIZZLE_NONE (0)
}
// Instruction descriptor, kind::f16: BF16 A/B, FP32 D, both K-major.
// a/b format 1 = BF16, 0 = F16 (A and B always of the same type).
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) |
         ((uint32_t)(M >> 4) << 24);
}
__host__ __device__ constexpr uint32_t idesc_f16(int M, int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
// A from tensor memory (lane = row, two K elements per 32-bit column), B from shared memory.
__device__ __forceinline__ void mma_f16(uint32_t tmem_d, uint32_t a, uint64_t b, uint32_t idesc,
                                        uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(tmem_d),
      "r"(a), "l"(b), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}
// One accumulation group: Q slices x three split products x four K-steps, in the order
// small products first ((A_hi, B_lo), (A_lo, B_hi), then (A_hi, B_hi)).  The descriptors are
// the chunk's base descriptors plus compile-time or per-chunk offsets (a descriptor holds the
// shared-memory address >> 4 in its low bits), so that the issuing thread does little more
// than issue: the tensor cores consume a group as fast as one thread issues it.
template <int Q>
__device__ __forceinline__ void mma_group(uint32_t td, uint32_t ad0, uint64_t bd0, uint32_t bpl16,
                                          uint32_t bkk16, uint32_t idesc, int nsl) {
  uint32_t acc = 0u;
#pragma unroll
  for (int pr = 1; pr <= 3; ++pr) {
    const int prod = pr % 3;
    const uint32_t ap = (prod == 2) ? 1u : 0u, bp = (prod == 1) ? 1u : 0u;
    const uint32_t adp = ad0 + ap * TC_A_PLANE;
    const uint64_t bdp = bd0 + bp * bpl16;
#pragma unroll
    for (int sl = 0; sl < (Q > 0 ? Q : 1); ++sl) {
      if (Q == 0 && sl >= nsl) break;
#pragma unroll
      for (int kk = 0; kk < TC_KC / 16; ++kk) {
        mma_f16(td, adp + kk * 8, bdp + (uint64_t)(kk * bkk16), idesc, acc);
        acc = 1u;
      }
    }
    if (Q == 0) {  // a group whose size is not a compile-time case: the remaining slices
      for (int sl = 1; sl < nsl; ++sl)
#pragma unroll
        for (int kk = 0; kk < TC_KC / 16; ++kk)
          mma_f16(td, adp + kk * 8, bdp + (uint64_t)(kk * bkk16), idesc, 1u);
    }
  }
}
// 16, 8 or 4 consecutive TMEM columns of this warp's lane quarter (one 32-bit value per lane
// each); the values are valid after tmem_wait().
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,"
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
        "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
        "=r"(r[7])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
__device__ __forceinline__ void tmem_st4(uint32_t taddr, const uint4& v) {
  asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1,%2,%3,%4};" ::"r"(taddr), "r"(v.x),
               "r"(v.y), "r"(v.z), "r"(v.w)
               : "memory");
}
__device__ __forceinline__ void tmem_wait_st() {
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_wait() {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}
// (no use of x moves ahead of a wait before it)
__device__ __forceinline__ void tmem_landed(uint32_t& x) { asm volatile("" : "+r"(x)); }

// Two columns' sums as FP32 pairs, value S + E: TwoSum (Knuth) of S and the drained value x,
// with the rounding error of S, which it gives exactly, added to E.
struct F32x2 {
  unsigned long long v;
};
__device__ __forceinline__ F32x2 add2(F32x2 a, F32x2 b) {
  F32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F32x2 sub2(F32x2 a, F32x2 b) {
  F32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F32x2 pack2(uint32_t a, uint32_t b) {
  return F32x2{(unsigned long long)b << 32 | a};
}
__device__ __forceinline__ void two_sum(F32x2& S, F32x2& E, F32x2 x) {
  const F32x2 t = add2(S, x), z = sub2(t, S);
  E = add2(E, add2(sub2(S, sub2(t, z)), sub2(x, z)));
  S = t;
}
// E back into S, what does not fit S's 24 bits left in E.  (An infinite S has a NaN in E: fmaxf
// takes the number, and S stays.)
__device__ __forceinline__ void fold(F32x2& S, F32x2& E) {
  const F32x2 e = pack2(
      __float_as_uint(fmaxf(__uint_as_float((uint32_t)E.v), -FLT_MAX)),
      __float_as_uint(fmaxf(__uint_as_float((uint32_t)(E.v >> 32)), -FLT_MAX)));
  const F32x2 t = add2(S, e);
  E = sub2(e, sub2(t, S));
  S = t;
}
// S + E in FP64; an infinite or NaN sum stays what it is.
__device__ __forceinline__ double pair_value(uint32_t s, uint32_t e) {
  const float f = __uint_as_float(s);
  return isfinite(f) ? (double)f + (double)__uint_as_float(e) : (double)f;
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
  __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
__device__ __forceinline__ uint32_t pack_f16(float a, float b) {
  __half2 h = __floats2half2_rn(a, b);
  return *reinterpret_cast<uint32_t*>(&h);
}
// Split of 8 FP32 values into hi and lo 16-bit parts (packed pairs).
template <bool kF16>
__device__ __forceinline__ void split8(const float (&x)[8], uint4& h, uint4& l) {
  float r[8];
  if (kF16) {
    h.x = pack_f16(x[0], x[1]);
    h.y = pack_f16(x[2], x[3]);
    h.z = pack_f16(x[4], x[5]);
    h.w = pack_f16(x[6], x[7]);
    const __half2* hb = reinterpret_cast<const __half2*>(&h);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float2 f = __half22float2(hb[e]);
      r[2 * e] = x[2 * e] - f.x;
      r[2 * e + 1] = x[2 * e + 1] - f.y;
    }
    l.x = pack_f16(r[0], r[1]);
    l.y = pack_f16(r[2], r[3]);
    l.z = pack_f16(r[4], r[5]);
    l.w = pack_f16(r[6], r[7]);
  } else {
    h.x = pack_bf16(x[0], x[1]);
    h.y = pack_bf16(x[2], x[3]);
    h.z = pack_bf16(x[4], x[5]);
    h.w = pack_bf16(x[6], x[7]);
    const __nv_bfloat162* hb = reinterpret_cast<const __nv_bfloat162*>(&h);
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      float2 f = __bfloat1622float2(hb[e]);
      r[2 * e] = x[2 * e] - f.x;
      r[2 * e + 1] = x[2 * e + 1] - f.y;
    }
    l.x = pack_bf16(r[0], r[1]);
    l.y = pack_bf16(r[2], r[3]);
    l.z = pack_bf16(r[4], r[5]);
    l.w = pack_bf16(r[6], r[7]);
  }
}

// F16x3 column scaling: max_g |W[g, i]| of every radial column (its bits; non-negative doubles
// order as integers), lanes along R over a slice of the grid.  The exponent s_i brings it to
// [2^13, 2^14); 2^-(s_i + kXScaleExp) undoes both scalings (tc_bimage_kernel).
constexpr int kXScaleExp = 14;
__global__ void __launch_bounds__(256)
tc_wmax_kernel(const double* __restrict__ W, int ldw, int G2, int nR, int rows,
               unsigned long long* __restrict__ wmax) {
  __shared__ double red[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
  const int g1 = min(G2, (int)(blockIdx.y + 1) * rows);
  double m = 0.0;
  if (i < nR)
#pragma unroll 8
    for (int g = blockIdx.y * rows + w; g < g1; g += 8) m = fmax(m, fabs(__ldg(W + (size_t)g * ldw + i)));
  red[w][lane] = m;
  __syncthreads();
  if (w == 0 && i < nR) {
#pragma unroll
    for (int q = 1; q < 8; ++q) m = fmax(m, red[q][lane]);
    atomicMax(wmax + i, (unsigned long long)__double_as_longlong(m));
  }
}
__device__ __forceinline__ int tc_wexp(unsigned long long bits) {
  const double m = __longlong_as_double((long long)bits);
  if (!(m > 0.0)) return 0;
  int e = 0;
  frexp(m, &e);  // m = f 2^e, f in [0.5, 1)
  return 14 - e;
}

// Column parts of the radial axis: part p covers columns [c0[p], c0[p] + nc[p]).
struct TcParts {
  int n;
  int c0[TC_MAX_PARTS];
  int nc[TC_MAX_PARTS];
};

// ---------------------------------------------------------------- operand images
// W (FP64, [g][ldw]) -> per column part p and chunk c: [plane hi/lo][kg 0..7][ng 0..nc/8-1]
// [8 rows][8 x 16 bit] at part_off(p) + c * 2 * TC_KC * nc(p), part_off(p) = n_chunks * 2 *
// TC_KC * c0(p); F16x3 scales column n by the power of two of tc_wexp first (exact).  A
// thread takes one column and eight grid points, one 16-byte core-matrix row per plane:
// reads are coalesced along R, writes along the rows (a thread per value, grid points
// fastest, read a sector per value).
template <bool kF16>
__global__ void __launch_bounds__(256)
tc_bimage_kernel(const double* __restrict__ W, int ldw, int G2, int nR, int npad, int n_chunks,
                 TcParts parts, const unsigned long long* __restrict__ wmax,
                 double* __restrict__ col_scale, unsigned short* __restrict__ img) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)npad * 8 * n_chunks) return;
  const int n = (int)(idx % npad);
  const int64_t q = idx / npad;
  const int kg = (int)(q & 7), c = (int)(q >> 3);
  int p = 0;
  while (p + 1 < parts.n && parts.c0[p + 1] <= n) ++p;
  const int nl = n - parts.c0[p], nc = parts.nc[p];
  const int g0 = c * TC_KC + kg * 8;
  const int s = kF16 && n < nR ? tc_wexp(wmax[n]) : 0;
  if (kF16 && q == 0) col_scale[n] = n < nR ? ldexp(1.0, -(s + kXScaleExp)) : 0.0;
  double w[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) w[e] = (g0 + e < G2 && n < nR) ? __ldg(W + (size_t)(g0 + e) * ldw + n) : 0.0;
  unsigned short hi[8], lo[8];
#pragma unroll
  for (int e = 0; e < 8; ++e) {
    if (kF16) {
      const double x = ldexp(w[e], s);
      const __half h = __double2half(x);
      hi[e] = __half_as_ushort(h);
      lo[e] = __half_as_ushort(__double2half(x - (double)__half2float(h)));
    } else {
      const __nv_bfloat16 h = __double2bfloat16(w[e]);
      hi[e] = __bfloat16_as_ushort(h);
      lo[e] = __bfloat16_as_ushort(__double2bfloat16(w[e] - (double)__bfloat162float(h)));
    }
  }
  auto pack = [](const unsigned short (&v)[8]) {
    return make_uint4(v[0] | (unsigned)v[1] << 16, v[2] | (unsigned)v[3] << 16,
                      v[4] | (unsigned)v[5] << 16, v[6] | (unsigned)v[7] << 16);
  };
  const size_t plane = (size_t)TC_KC * nc;
  const size_t off = (size_t)n_chunks * 2 * TC_KC * parts.c0[p] + (size_t)c * 2 * plane +
                     (((size_t)kg * (nc / 8) + (nl >> 3)) * 8 + (nl & 7)) * 8;
  *reinterpret_cast<uint4*>(img + off) = pack(hi);
  *reinterpret_cast<uint4*>(img + off + plane) = pack(lo);
}

// psi (FP64, [basis row][G2]) -> per (block, chunk): [local state][TC_PSI_LD] float2, for the
// bases that are not written as images at once (SYS_TYPE 1).
__global__ void tc_psiimage_kernel(const double2* __restrict__ psi, int G2, int n_chunks,
                                   const int* __restrict__ blk_row0, const int* __restrict__ blk_n,
                                   const int64_t* __restrict__ blk_img_off, int n_blocks,
                                   float2* __restrict__ img, int n_basis_rows) {
  int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  int64_t per_row = (int64_t)n_chunks * TC_PSI_LD;
  if (idx >= per_row * n_basis_rows) return;
  int row = (int)(idx / per_row);
  int rem = (int)(idx % per_row);
  int c = rem / TC_PSI_LD, k = rem % TC_PSI_LD;
  int b = 0;
  while (b + 1 < n_blocks && blk_row0[b + 1] <= row) ++b;
  int ls = row - blk_row0[b];
  int g = c * TC_KC + k;
  double2 v = (k < TC_KC && g < G2) ? psi[(size_t)row * G2 + g] : make_double2(0.0, 0.0);
  img[blk_img_off[b] + ((int64_t)c * blk_n[b] + ls) * TC_PSI_LD + k] =
      make_float2((float)v.x, (float)v.y);
}

// ---------------------------------------------------------------- main kernel
struct TcArgs {
  int n_units, n_parts, n_ks, n_chunks, chunks_per_ks, n_alpha_it;
  int slices_per_drain;           // alpha points accumulated in FP32 between two drains
  int nbuf;                       // B / basis-slice buffers (1 or 2)
  uint32_t b_stage, psi_stage;    // bytes of one B / basis-slice buffer
  TcParts parts;
  const int* tile_block;          // per tile
  const int* blk_row0;            // basis row offset per block
  const int* blk_n;
  const int64_t* blk_img_off;     // float2 offset of the block's psi image
  const int* rowa;                // basis row of st1 / st2 per GEMM row
  const int* rowb;
  const float2* psi_img;
  const unsigned short* b_img;    // hi/lo planes of W, BF16 or F16 bits, per column part
  const double* walpha;           // the weight of every alpha point, or null (weight 1)
  const double* col_scale;        // per radial column: factor applied to the FP64 sums
  double* part;                   // n_ks x n_rows x ldp FP64 sums
  int64_t part_stride;
  int ldp;
  int* status;
};

// Use k of a resource with nb buffers: buffer k % nb; its "full" barrier completes
// for the (k / nb)-th time, its "empty" barrier (before reuse, k >= nb) completed
// (k / nb - 1) times before.
__device__ __forceinline__ uint32_t full_parity(uint32_t k, uint32_t nb) { return (k / nb) & 1u; }
__device__ __forceinline__ uint32_t empty_parity(uint32_t k, uint32_t nb) {
  return ((k / nb) + 1u) & 1u;
}

// kMulti: several accumulation groups a chunk are possible (its code costs the eight-warp form
// registers: 613 -> 650 us of the j <= 8 build).
template <bool kF16, int PE, bool kMulti>
__global__ void __launch_bounds__(TcShape<PE>::THREADS, 1) tc_contract_kernel(TcArgs a) {
  constexpr int TC_THREADS = TcShape<PE>::THREADS, TC_PRODUCERS = TcShape<PE>::PRODUCERS;
  constexpr int TC_KSPLIT = TC_PRODUCERS / TC_M;  // threads per tile row in X production
  constexpr int TC_WPQ = TcShape<PE>::WPQ, TC_NCH_MAX = TcShape<PE>::NCH_MAX;
  static_assert(TC_PRODUCERS % TC_M == 0 && (TC_KC / 8) % TC_KSPLIT == 0, "X production split");
  static_assert(TC_NC_MAX <= TC_WPQ * TC_NCH_MAX && 16 % TC_WPQ == 0, "drain split");
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // (an offset, not a rounded integer: the accesses stay in the shared address space)
  unsigned char* sB = smem_raw + ((0u - smem_u32(smem_raw)) & 1023u);    // nbuf x b_stage
  unsigned char* sPsi = sB + a.nbuf * a.b_stage;                         // nbuf x psi_stage
  uint64_t* bars = reinterpret_cast<uint64_t*>(sPsi + a.nbuf * a.psi_stage);
  uint64_t* B_full = bars;          // [2]
  uint64_t* B_empty = bars + 2;     // [2]
  uint64_t* P_full = bars + 4;      // [2]
  uint64_t* P_empty = bars + 6;     // [2]
  uint64_t* A_full = bars + 8;      // [2]
  uint64_t* A_empty = bars + 10;    // [2]
  uint64_t* ACC_full = bars + 12;   // [2]
  uint64_t* ACC_empty = bars + 14;  // [2]
  uint64_t* DONE = bars + 16;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 18);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(bars + 19);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < 2; ++s) {
      mbar_init(&B_full[s], 1);
      mbar_init(&B_empty[s], 1);
      mbar_init(&P_full[s], 1);
      mbar_init(&P_empty[s], PE);  // one arrival per warp: 512 on one barrier took 1 000 clocks
      mbar_init(&A_full[s], PE);
      mbar_init(&A_empty[s], 1);
      mbar_init(&ACC_full[s], 1);
      mbar_init(&ACC_empty[s], PE);
    }
    mbar_init(DONE, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_u32(tmem_slot)),
                 "r"(TC_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t nbuf = (uint32_t)a.nbuf;

  if (warp == 0) {
    // ---------------- bulk-copy producer
    if (lane == 0) {
      uint32_t k = 0;  // chunk uses so far (B and basis slices move together)
      for (int u = blockIdx.x; u < a.n_units && !*abort_flag; u += gridDim.x) {
        const int ks = u % a.n_ks, pt = (u / a.n_ks) % a.n_parts, tile = u / (a.n_ks * a.n_parts);
        const int blk = a.tile_block[tile];
        const int nb = a.blk_n[blk];
        const int nc = a.parts.nc[pt];
        const uint32_t psi_bytes = (uint32_t)nb * TC_PSI_LD * 8u;
        const uint32_t b_bytes = 2u * TC_KC * (uint32_t)nc * 2u;
        const unsigned short* bsrc = a.b_img + (size_t)a.n_chunks * 2 * TC_KC * a.parts.c0[pt];
        const int c0 = ks * a.chunks_per_ks, c1 = min(a.n_chunks, c0 + a.chunks_per_ks);
        for (int c = c0; c < c1; ++c, ++k) {
          const uint32_t s = k % nbuf;
          if (k >= nbuf) {
            if (!mbar_wait(&B_empty[s], empty_parity(k, nbuf), abort_flag, a.status, 11)) break;
            if (!mbar_wait(&P_empty[s], empty_parity(k, nbuf), abort_flag, a.status, 12)) break;
          }
          mbar_expect_tx(&B_full[s], b_bytes);
          bulk_g2s(sB + s * a.b_stage, bsrc + (size_t)c * 2 * TC_KC * nc, b_bytes, &B_full[s]);
          mbar_expect_tx(&P_full[s], psi_bytes);
          bulk_g2s(sPsi + s * a.psi_stage,
                   a.psi_img + a.blk_img_off[blk] + (int64_t)c * nb * TC_PSI_LD, psi_bytes,
                   &P_full[s]);
        }
      }
      // the copies issued last must have landed before the CTA exits
      for (uint32_t j = (k > nbuf ? k - nbuf : 0); j < k; ++j) {
        const uint32_t s = j % nbuf;
        for (uint32_t it = 0; it < TC_SPIN_LIMIT && !mbar_try_wait(&B_full[s], full_parity(j, nbuf)); ++it) {}
        for (uint32_t it = 0; it < TC_SPIN_LIMIT && !mbar_try_wait(&P_full[s], full_parity(j, nbuf)); ++it) {}
      }
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer
    if (lane == 0) {
      uint32_t kc = 0, ka = 0, kacc = 0;  // chunk uses, A-stage uses, accumulator uses
      const uint32_t sB0 = smem_u32(sB);
      for (int u = blockIdx.x; u < a.n_units && !*abort_flag; u += gridDim.x) {
        const int ks = u % a.n_ks, pt = (u / a.n_ks) % a.n_parts;
        const int nc = a.parts.nc[pt];
        const uint32_t idesc = kF16 ? idesc_f16(TC_M, nc) : idesc_bf16(TC_M, nc);
        const uint32_t lbo_b = (uint32_t)(nc / 8) * 128, bplane = (uint32_t)TC_KC * nc * 2;
        const int c0 = ks * a.chunks_per_ks, c1 = min(a.n_chunks, c0 + a.chunks_per_ks);
        bool ok = true;
        for (int c = c0; c < c1 && ok; ++c, ++kc, ++ka) {
          const uint32_t sb = kc % nbuf, sa = ka & 1u;
          ok = mbar_wait(&B_full[sb], full_parity(kc, nbuf), abort_flag, a.status, 21) &&
               mbar_wait(&A_full[sa], full_parity(ka, 2), abort_flag, a.status, 22);
          if (!ok) break;
          tc_fence_after();
          const uint32_t ad0 = tmem + TC_TMEM_A + sa * (2 * TC_A_PLANE);
          const uint32_t boff0 = sB0 + sb * a.b_stage;
          const uint64_t bd0 = smem_desc(boff0, lbo_b, 128);
          const uint32_t bpl16 = bplane >> 4, bkk16 = (2 * lbo_b) >> 4;
          for (int al = 0; al < a.n_alpha_it; ++al, ++kacc) {
            const uint32_t sc = kacc & 1u;
            if (kacc >= 2) {  // the epilogue must have drained this accumulator
              if (!mbar_wait(&ACC_empty[sc], empty_parity(kacc, 2), abort_flag, a.status, 23)) {
                ok = false;
                break;
              }
              tc_fence_after();
            }
            const uint32_t td = tmem + sc * TC_NC_MAX;
            const int ns_grp = min(a.slices_per_drain, a.n_alpha_it - al);
            switch (ns_grp) {
              case 1: mma_group<1>(td, ad0, bd0, bpl16, bkk16, idesc, 1); break;
              case 2: mma_group<2>(td, ad0, bd0, bpl16, bkk16, idesc, 2); break;
              case 4: mma_group<4>(td, ad0, bd0, bpl16, bkk16, idesc, 4); break;
              case 8: mma_group<8>(td, ad0, bd0, bpl16, bkk16, idesc, 8); break;
              default: mma_group<0>(td, ad0, bd0, bpl16, bkk16, idesc, ns_grp); break;
            }
            mma_commit(&ACC_full[sc]);  // the epilogue may read once these MMAs complete
            al += ns_grp - 1;
          }
          mma_commit(&A_empty[sa]);  // A and B may be overwritten once the chunk's MMAs complete
          mma_commit(&B_empty[sb]);
        }
      }
      // every MMA issued by this thread has completed before TMEM is released
      mma_commit(DONE);
      for (uint32_t it = 0; it < TC_SPIN_LIMIT && !mbar_try_wait(DONE, 0); ++it) {}
    }
  } else {
    // ---------------- X producers (warps 2 to PE + 1) and epilogue
    const int q = warp & 3;        // TMEM lane quarter accessible to this warp
    const int h = (warp - 2) >> 2; // its share of a chunk's K groups and of a part's columns
    const int p = q * 32 + lane;   // the thread's tile row
    uint32_t kc = 0, ka = 0, kacc = 0;
    const double wa = a.walpha ? a.walpha[0] : 1.0;  // every alpha point's weight
    F32x2 S[TC_NCH_MAX / 2], E[TC_NCH_MAX / 2];
    for (int u = blockIdx.x; u < a.n_units && !*abort_flag; u += gridDim.x) {
      const int ks = u % a.n_ks, pt = (u / a.n_ks) % a.n_parts, tile = u / (a.n_ks * a.n_parts);
      const int blk = a.tile_block[tile];
      const int row = tile * TC_M + p;
      const int la = a.rowa[row] - a.blk_row0[blk], lb = a.rowb[row] - a.blk_row0[blk];
      // the part's columns (a multiple of 16) split over the warps of a lane quarter
      const int nch = a.parts.nc[pt] / TC_WPQ, coff = h * nch, col0 = a.parts.c0[pt] + coff;
      const int c0 = ks * a.chunks_per_ks, c1 = min(a.n_chunks, c0 + a.chunks_per_ks);
#pragma unroll
      for (int i = 0; i < TC_NCH_MAX / 2; ++i) S[i].v = E[i].v = 0;
      // produce the operand of chunk use kcu into A stage (kau & 1) from basis slice
      // (kcu % nbuf)
      auto produce = [&](uint32_t kcu, uint32_t kau) -> bool {
        const uint32_t sp = kcu % nbuf, sa = kau & 1u;
        if (!mbar_wait(&P_full[sp], full_parity(kcu, nbuf), abort_flag, a.status, 31)) return false;
        if (kau >= 2 && !mbar_wait(&A_empty[sa], empty_parity(kau, 2), abort_flag, a.status, 32))
          return false;
        tc_fence_after();
        __syncwarp();
        const float2* ps = reinterpret_cast<const float2*>(sPsi + sp * a.psi_stage);
        const float2* pa = ps + la * TC_PSI_LD;
        const float2* pb = ps + lb * TC_PSI_LD;
        const uint32_t ta = tmem + ((uint32_t)(q * 32) << 16) + TC_TMEM_A + sa * (2 * TC_A_PLANE);
#pragma unroll
        for (int kq = 0; kq < TC_KC / 8 / TC_KSPLIT; ++kq) {
          const int kg = h * (TC_KC / 8 / TC_KSPLIT) + kq;
          float x[8];
#pragma unroll
          for (int e = 0; e < 8; e += 2) {
            const float4 va = *reinterpret_cast<const float4*>(pa + kg * 8 + e);
            const float4 vb = *reinterpret_cast<const float4*>(pb + kg * 8 + e);
            x[e] = va.x * vb.x + va.y * vb.y;
            x[e + 1] = va.z * vb.z + va.w * vb.w;
          }
          if (kF16) {
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] *= (float)(1 << kXScaleExp);  // exact
          }
          uint4 hv, lv;
          split8<kF16>(x, hv, lv);
          tmem_st4(ta + kg * 4, hv);
          tmem_st4(ta + TC_A_PLANE + kg * 4, lv);
        }
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(&A_full[sa]);
          mbar_arrive(&P_empty[sp]);
        }
        return true;
      };
      // With two B / basis buffers the next chunk's operand is formed before this chunk
      // is drained, so the tensor cores go on while the epilogue works.  With one, the
      // next copy waits for this chunk's MMAs, which wait for its drains: form it after.
      const bool ahead = nbuf == 2;
      bool ok = c0 < c1 ? produce(kc, ka) : true;
      for (int c = c0; c < c1 && ok; ++c, ++kc, ++ka) {
        if (ahead && c + 1 < c1 && !produce(kc + 1, ka + 1)) {
          ok = false;
          break;
        }
        for (int al = 0; al < a.n_alpha_it; al += a.slices_per_drain, ++kacc) {
          const uint32_t sc = kacc & 1u;
          if (!mbar_wait(&ACC_full[sc], full_parity(kacc, 2), abort_flag, a.status, 33)) {
            ok = false;
            break;
          }
          tc_fence_after();
          __syncwarp();
          const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + sc * TC_NC_MAX + (uint32_t)coff;
          // batches of columns; after the last load the accumulator is free
#pragma unroll
          for (int b0 = 0; b0 < TC_NCH_MAX; b0 += TC_NLD) {  // conditions alike for the warp
            uint32_t r[TC_NLD];
            const int m = nch - b0;
            if (m > 0) {
              if (b0 + 16 <= TC_NCH_MAX && m >= 16) {
                tmem_ld16(taddr + b0, r);
              } else {
                if (m >= 8) tmem_ld8(taddr + b0, r);
                if (m >= 12) tmem_ld4(taddr + b0 + 8, r + 8);
                else if (m == 4) tmem_ld4(taddr + b0, r);
              }
              tmem_wait();
            }
            if (b0 + TC_NLD >= TC_NCH_MAX) {
              tc_fence_before();
              __syncwarp();
              if (lane == 0) mbar_arrive(&ACC_empty[sc]);
            }
#pragma unroll
            for (int i = 0; i < TC_NLD && b0 + i < TC_NCH_MAX; i += 4) {
              if (i >= m) break;
#pragma unroll
              for (int e = i; e < i + 4; ++e) tmem_landed(r[e]);
              two_sum(S[(b0 + i) / 2], E[(b0 + i) / 2], pack2(r[i], r[i + 1]));
              two_sum(S[(b0 + i) / 2 + 1], E[(b0 + i) / 2 + 1], pack2(r[i + 2], r[i + 3]));
            }
          }
        }
        if (kMulti && a.n_alpha_it > a.slices_per_drain) {  // E goes back below an ulp of S
#pragma unroll
          for (int i = 0; i < TC_NCH_MAX / 2; ++i) fold(S[i], E[i]);
        }
        if (ok && !ahead && c + 1 < c1 && !produce(kc + 1, ka + 1)) ok = false;
      }
      if (!ok) break;
      // the unit's sums in FP64, with the alpha weight and the exact column factors
      double* dst = a.part + (int64_t)ks * a.part_stride + (int64_t)row * a.ldp;
#pragma unroll
      for (int i = 0; i < TC_NCH_MAX; i += 4)
        if (i < nch) {
          double v[4];
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int h32 = 32 * (e & 1), j = (i + e) / 2;
            v[e] = wa * pair_value((uint32_t)(S[j].v >> h32), (uint32_t)(E[j].v >> h32)) *
                   __ldg(a.col_scale + col0 + i + e);
          }
          // whole 32-byte sectors: 16-byte stores took 11 000 clocks of a 128 x 112 unit
          asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(dst + col0 + i), "d"(v[0]),
                       "d"(v[1]), "d"(v[2]), "d"(v[3])
                       : "memory");
        }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(TC_TMEM_COLS));
  }
}

// ---------------------------------------------------------------- host side
static const void* tc_kernel(bool f16, bool many, bool multi) {
  if (many)
    return f16 ? (const void*)tc_contract_kernel<true, 16, true>
               : (const void*)tc_contract_kernel<false, 16, true>;
  if (multi)
    return f16 ? (const void*)tc_contract_kernel<true, 8, true>
               : (const void*)tc_contract_kernel<false, 8, true>;
  return f16 ? (const void*)tc_contract_kernel<true, 8, false>
             : (const void*)tc_contract_kernel<false, 8, false>;
}
int MatrixPlan::tc_init() {
  MQCT_ARG_CHECK(nR <= TC_NC_MAX * TC_MAX_PARTS, "tensor-core contraction supports nR <= %d (got %d)",
                 TC_NC_MAX * TC_MAX_PARTS, nR);
  int dev = 0, cc_major = 0, cc_minor = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&cc_major, cudaDevAttrComputeCapabilityMajor, dev);
  cudaDeviceGetAttribute(&cc_minor, cudaDevAttrComputeCapabilityMinor, dev);
  if (cc_major != 10) {
    set_error("the tcgen05 contraction needs an sm_100 device (got sm_%d%d)", cc_major, cc_minor);
    return MQCT_E_NODEV;
  }
  tc = std::make_unique<TcInfo>();
  TcInfo& t = *tc;
  t.npad = (nR + 15) / 16 * 16;
  // column parts: as few as the TMEM buffer width allows, balanced, widths multiples of 16
  const int n16 = t.npad / 16;
  t.n_parts = (t.npad + TC_NC_MAX - 1) / TC_NC_MAX;
  for (int p = 0, c = 0; p < t.n_parts; ++p) {
    const int w = (n16 / t.n_parts + (p < n16 % t.n_parts ? 1 : 0)) * 16;
    t.part_c0[p] = c;
    t.part_nc[p] = w;
    c += w;
  }
  t.n_chunks = (G2 + TC_KC - 1) / TC_KC;
  std::vector<int> row0(h_block_row0), nb(h_block_n);
  t.n_blocks = (int)row0.size();
  t.nbmax = 0;
  std::vector<int64_t> off(t.n_blocks);
  int64_t acc = 0;
  for (int b = 0; b < t.n_blocks; ++b) {
    off[b] = acc;
    acc += (int64_t)nb[b] * t.n_chunks * TC_PSI_LD;
    t.nbmax = std::max(t.nbmax, nb[b]);
  }
  // shared memory: B buffers, basis-slice buffers, barriers
  int ncmax = 0;
  for (int p = 0; p < t.n_parts; ++p) ncmax = std::max(ncmax, t.part_nc[p]);
  auto up = [](size_t x) { return (x + 1023) & ~size_t(1023); };
  t.b_stage = (uint32_t)up(2ull * TC_KC * ncmax * 2);
  t.psi_stage = (uint32_t)up((size_t)t.nbmax * TC_PSI_LD * 8);
  int dev_smem = 0;
  cudaDeviceGetAttribute(&dev_smem, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  for (t.nbuf = 2; t.nbuf >= 1; --t.nbuf) {
    t.smem = 1024 + (size_t)t.nbuf * (t.b_stage + t.psi_stage) + 256;
    if (t.smem <= (size_t)dev_smem) break;
  }
  MQCT_ARG_CHECK(t.nbuf >= 1, "shared memory too small for the tcgen05 tiles (nR=%d, block %d)",
                 nR, t.nbmax);
  // one CTA per SM (the TMEM buffers and the register sums are sized for it)
  t.smem = std::max(t.smem, (size_t)dev_smem / 2 + 1024);
  MQCT_CUDA_TRY(t.blk_row0.upload(row0, stream));
  MQCT_CUDA_TRY(t.blk_n.upload(nb, stream));
  MQCT_CUDA_TRY(t.blk_img_off.upload(off, stream));
  // alpha points per drain: 2 keeps the drains under the MMA time.  The weight is applied to the
  // sums: it is the same for every point of the midpoint grid, the only alpha grid there is.
  t.slices_per_drain = n_alpha > 1 ? 2 : 1;
  // K ranges: split the chunks only to fill the last wave of units, or the SMs when the units of
  // one range are fewer (the FP64 sums of every range are written once and added by the
  // finalize).  The cost of ks ranges, in accumulation groups: a chunk's groups and its X, and 15
  // for a unit's start, its sums and their way through the finalize (asymmetric top, j <= 8,
  // 771 units a range: 636, 649, 690 and 766 us for 1 to 4 ranges; with 24 groups a chunk 5 394,
  // 5 077, 4 922 and 5 120; two tops, 13 units: 5 555, 4 027, 3 662 and 3 497 for 1, 4, 8, 11).
  cudaDeviceGetAttribute(&t.n_sm, cudaDevAttrMultiProcessorCount, dev);
  const int64_t units1 = (int64_t)n_tiles * t.n_parts;
  const int ks_max = std::min(units1 < t.n_sm ? 16 : 4, t.n_chunks);
  const int groups = (std::max(1, n_alpha) + t.slices_per_drain - 1) / t.slices_per_drain;
  int best_ks = 1;
  double best = 0.0;
  for (int ks = 1; ks <= ks_max; ++ks) {
    const int cps = (t.n_chunks + ks - 1) / ks, ns = (t.n_chunks + cps - 1) / cps;
    const double cost = (double)((units1 * ns + t.n_sm - 1) / t.n_sm) * (cps * (groups + 1) + 15);
    if (ks == 1 || cost < best) {
      best = cost;
      best_ks = ks;
    }
  }
  t.chunks_per_split = (t.n_chunks + best_ks - 1) / best_ks;
  tc_splits = (t.n_chunks + t.chunks_per_split - 1) / t.chunks_per_split;
  tc_ldp = t.npad;
  MQCT_CUDA_TRY(d_part.alloc((size_t)tc_splits * n_rows * tc_ldp));
  MQCT_CUDA_TRY(d_bimg.alloc((size_t)t.n_chunks * 2 * TC_KC * t.npad));
  MQCT_CUDA_TRY(d_psi32.alloc((size_t)acc));
  {
    // (the images' padding, two values a row and the grid points past G2, stays zero)
    MQCT_CUDA_TRY(cudaMemsetAsync(d_psi32.p, 0, sizeof(float2) * (size_t)acc, stream));
    std::vector<int64_t> ro(n_basis_rows);
    std::vector<int> rs(n_basis_rows);
    for (int b = 0; b < t.n_blocks; ++b)
      for (int l = 0; l < nb[b]; ++l) {
        ro[row0[b] + l] = off[b] + (int64_t)l * TC_PSI_LD;
        rs[row0[b] + l] = nb[b] * TC_PSI_LD;
      }
    MQCT_CUDA_TRY(t.row_off.upload(ro, stream));
    MQCT_CUDA_TRY(t.row_step.upload(rs, stream));
    MQCT_CUDA_TRY(cudaStreamSynchronize(stream));  // the host arrays end here
  }
  MQCT_CUDA_TRY(d_status.alloc(1));
  MQCT_CUDA_TRY(cudaMemsetAsync(d_status.p, 0, sizeof(int), stream));
  MQCT_CUDA_TRY(d_col_scale.alloc((size_t)t.npad));
  if (precision == MQCT_PREC_F16X3) {
    MQCT_CUDA_TRY(t.wmax.alloc((size_t)nR));
    MQCT_CUDA_TRY(cudaMemsetAsync(d_col_scale.p, 0, sizeof(double) * t.npad, stream));
  } else {
    std::vector<double> ones(t.npad, 1.0);
    MQCT_CUDA_TRY(d_col_scale.upload(ones, stream));
  }
  return tc_pick();
}

// The kernel form for the plan's settings, with its shared-memory limit (only a form that the plan
// launches is loaded: the first one of a process takes most of a millisecond).
int MatrixPlan::tc_pick() {
  TcInfo& t = *tc;
  const int n_alpha_it = std::max(1, n_alpha);
  const bool multi = n_alpha_it > t.slices_per_drain;
  // sixteen epilogue warps when a K-chunk has several accumulation groups (the drains then
  // dominate: the as-written alpha grid), eight when it has one (the drain of a chunk then
  // alternates with its X production, and eight warps with more registers are faster)
  const bool many = t.pe_force ? t.pe_force == 16 : multi;
  t.pe_warps = many ? 16 : 8;
  const void* fn = tc_kernel(precision == MQCT_PREC_F16X3, many, multi);
  if (fn == t.fn) return MQCT_OK;
  const int rc = allow_max_smem(fn);
  if (rc == MQCT_OK) t.fn = fn;
  return rc;
}

int MatrixPlan::tc_execute() {
  TcInfo& t = *tc;
  const int thr = 256;
  const bool f16 = precision == MQCT_PREC_F16X3;
  TcParts parts{};
  parts.n = t.n_parts;
  for (int p = 0; p < t.n_parts; ++p) {
    parts.c0[p] = t.part_c0[p];
    parts.nc[p] = t.part_nc[p];
  }
  const int64_t nb_img = (int64_t)t.n_chunks * 8 * t.npad;
  const unsigned nbb = (unsigned)((nb_img + thr - 1) / thr);
  if (f16) {
    MQCT_CUDA_TRY(cudaMemsetAsync(t.wmax.p, 0, sizeof(unsigned long long) * nR, stream));
    const int nx = (nR + 31) / 32;
    const int rows = std::max(64, (int)(((int64_t)G2 * nx + 4 * t.n_sm - 1) / (4 * t.n_sm)));
    tc_wmax_kernel<<<dim3(nx, (G2 + rows - 1) / rows), 256, 0, stream>>>(d_W.p, ldw, G2, nR, rows,
                                                                         t.wmax.p);
    MQCT_CUDA_TRY(cudaGetLastError());
    tc_bimage_kernel<true><<<nbb, thr, 0, stream>>>(d_W.p, ldw, G2, nR, t.npad, t.n_chunks, parts,
                                                    t.wmax.p, d_col_scale.p, d_bimg.p);
  } else {
    tc_bimage_kernel<false><<<nbb, thr, 0, stream>>>(d_W.p, ldw, G2, nR, t.npad, t.n_chunks, parts,
                                                     nullptr, nullptr, d_bimg.p);
  }
  MQCT_CUDA_TRY(cudaGetLastError());
  if (sys_type == 1) {
    const int64_t np_img = (int64_t)n_basis_rows * t.n_chunks * TC_PSI_LD;
    tc_psiimage_kernel<<<(unsigned)((np_img + thr - 1) / thr), thr, 0, stream>>>(
        d_psi.p, G2, t.n_chunks, t.blk_row0.p, t.blk_n.p, t.blk_img_off.p, t.n_blocks, d_psi32.p,
        n_basis_rows);
    MQCT_CUDA_TRY(cudaGetLastError());
  }
  TcArgs a{};
  a.n_parts = t.n_parts;
  a.n_ks = tc_splits;
  a.n_units = n_tiles * t.n_parts * tc_splits;
  a.n_chunks = t.n_chunks;
  a.chunks_per_ks = t.chunks_per_split;
  a.n_alpha_it = n_alpha > 0 ? n_alpha : 1;
  a.slices_per_drain = std::max(1, std::min(t.slices_per_drain, a.n_alpha_it));
  a.nbuf = t.nbuf;
  a.b_stage = t.b_stage;
  a.psi_stage = t.psi_stage;
  a.parts = parts;
  a.tile_block = d_tile_block.p;
  a.blk_row0 = t.blk_row0.p;
  a.blk_n = t.blk_n.p;
  a.blk_img_off = t.blk_img_off.p;
  a.rowa = d_rowa.p;
  a.rowb = d_rowb.p;
  a.psi_img = d_psi32.p;
  a.b_img = d_bimg.p;
  a.walpha = n_alpha > 0 ? d_walpha.p : nullptr;
  a.col_scale = d_col_scale.p;
  a.part = d_part.p;
  a.part_stride = (int64_t)n_rows * tc_ldp;
  a.ldp = tc_ldp;
  a.status = d_status.p;
  int grid = std::min(a.n_units, t.n_sm);
  const int rc = tc_pick();
  if (rc) return rc;
  void* args[] = {&a};
  MQCT_CUDA_TRY(cudaLaunchKernel(t.fn, dim3(grid),
                                 dim3(t.pe_warps == 16 ? TcShape<16>::THREADS : TcShape<8>::THREADS),
                                 args, t.smem, stream));
  MQCT_CUDA_TRY(cudaGetLastError());
  return MQCT_OK;
}

int MatrixPlan::tc_check_status() {
  if (!tc) return MQCT_OK;
  int st = 0;
  MQCT_CUDA_TRY(cudaMemcpyAsync(&st, d_status.p, sizeof(int), cudaMemcpyDeviceToHost, stream));
  MQCT_CUDA_TRY(cudaStreamSynchronize(stream));
  if (st) {
    set_error("tcgen05 contraction aborted: a pipeline wait timed out (code %d)", st);
    cudaMemsetAsync(d_status.p, 0, sizeof(int), stream);
    return MQCT_E_DEVICE;
  }
  return MQCT_OK;
}

int MatrixPlan::error_report(const double*, mqct_err_report_t* err) {
  if (err) err->n_sampled = 0;
  return MQCT_OK;
}

}  // namespace mqct
