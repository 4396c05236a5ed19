// Complex x real FP64 products on the tensor cores (tcgen05), exact digit slices.
//
// This GPU's FP64 pipe retires two FMAs per clock and SM (about 1.2 TFLOP/s), so a contraction on
// it is bound by that pipe whatever its tiling.  Here both operands are written as integer digits
// and multiplied on the FP16 tensor cores, about forty times the rate, at FP64 accuracy:
//
//  * a row x[0..K) (a row of A: real or imaginary part; a column of B) is x ~= 2^e sum_{t<6} q_t 2^-(9 + 9 t)
//    with integers |q_0| <= 512, |q_t| <= 256 (exact in FP16), one exponent e per row: 54 bits below the row's
//    largest element;
//  * products q_t q_u of equal order d = t + u <= 6 (26 of the 36) share one FP32 accumulator in TMEM.  Over a slab
//    of 64 k every partial sum of the orders d <= 3 stays below 2^24, so it is an exact integer (a row whose |q_0|
//    would sum past 8192 over 32 k gets e + 1: then |q_0| <= 256); the orders above carry 2^-54 of the row maxima
//    and less, where the last bit does not matter;
//  * after each slab the seven sums are added into one 64-bit integer per output, which is converted to FP64 once.
//
// The slices are those of the error-free transformation of Ozaki, Ogita, Oishi and Rump (Numer. Algorithms 59, 2012), with
// digits of fixed width instead of rounded remainders.
//
// The error is relative to the maxima of the two rows, about 2^-54 of their product per term, not to the terms as in an
// FP64 sum: rows whose large elements meet zeros or small elements of the other operand lose what the FP64 sum keeps (a
// factor of 10^s against 10^-s, K = 120: 2.4e-15 of the result at s = 2, 2.3e-11 at s = 6).  The operands here have
// no such rows but for the step adjoint's, which are balanced first (adjoint_dg_gv).  On the force bias, exchange, VHS and
// CISD operands of systems of 24 to 135 orbitals (K = 24 ... 2160), against a long-double product: 1.0e-16 ... 6.1e-16 of
// the result, an FP64 sum over k 1.7e-16 ... 1.5e-15 (0.2 to 0.86 of it; five digits, or orders d <= 5 only, are worse
// than FP64 where one element dominates its row).  The result does not depend on the tiling or on the other rows.
//
// Rate (1024 x 7260, K = 600, the VHS of 120 orbitals): 0.455 ms + 0.040 ms for the digits = 36 TFLOP/s, against
// 14.5 ms on the FP64 pipe; bound by the MMAs' operand reads from shared memory (about 50 cycles per MMA and 0.75 per
// column and K16 step).  (1024 x 7200, K = 120): 0.123 ms, where the epilogue's conversions take half of the time.
//
// One persistent CTA per SM: MMA rows are the columns of B (128 per tile), MMA columns the rows of A in tiles of 32
// (16 complex rows: re, im).  Per K16 step six (seven in a slab's first) MMAs: digit plane t of B against planes
// 0..min(5, 6 - t) of A stacked along the MMA's N.  Two TMEM accumulators (7 x 32 columns) let the tensor core run
// the next slab while 16 epilogue warps empty this one.  Keeping a 128-row tile in shared memory for two or four 32-row
// tiles saves loads but not time (VHS 0.460 ms, K = 120 0.117 / 0.125 against 0.442 and 0.112 ms: the outputs of
// several tiles come in a burst that the two accumulators cannot hide, and small products leave CTAs without work).
#include <cooperative_groups.h>
#include <cuda_fp16.h>

#include <algorithm>
#include <cmath>

#include "digits.h"
#include "step_tail.cuh"
#include "tc.cuh"

namespace trot {

static constexpr int kDgS = 6;           // digit planes
static constexpr int kDgGroups = 7;      // orders d = 0..6
static constexpr int kDgTop = 9, kDgLow = 9;
static constexpr int kDgBits = kDgTop + kDgLow * (kDgS - 1);  // 54
static constexpr int kDgP = 32;          // real rows of A per tile
static constexpr int kDgSlab = 4;        // K16 steps per slab
static constexpr uint32_t kDgAStep = kDgS * 128 * 32;    // 24576 B: one K16 step of a 128-row tile
static constexpr uint32_t kDgBStep = kDgS * kDgP * 32;   // 6144 B: one K16 step of a 32-row tile
static constexpr int kDgASlots = 6, kDgBSlots = 3;
static constexpr int kDgEpi = 512;
static constexpr int kDgThreads = kDgEpi + 3 * 32;       // 16 epilogue warps, MMA warp, two loader warps
static constexpr size_t kDgOffB = (size_t)kDgASlots * kDgAStep;
static constexpr size_t kDgOffBar = kDgOffB + (size_t)kDgBSlots * kDgSlab * kDgBStep;
static constexpr size_t kDgSmem = kDgOffBar + 256 + 128;  // + base alignment
static_assert(kDgSmem <= 232448, "digit product: shared memory");
static constexpr int kDgNonFinite = 0x4000;               // exponent code of a row with inf or NaN

// 16-bit index of element (r, k) of a [rows x 16] block (8 x 8 core matrices, K-adjacent ones
// 128 B apart, 8-row groups 256 B apart)
TROT_HD uint32_t dg_idx(int r, int k) { return (uint32_t)((r >> 3) * 128 + (k >> 3) * 64 + (r & 7) * 8 + (k & 7)); }

// ------------------------------------------------------------------ digits
// Digit planes of eight consecutive k of one row, w[t] = 16 B of FP16: q = rint(|x| 2^(54 - e)) <= 2^54 (half away
// from zero; subnormal x gives 0) split by 32-bit operations into five balanced 9-bit digits (mod 512, in
// [-256, 256)) and the leading one (<= 512), the sign of x flipped in afterwards.  A digit d becomes FP16 as the bits
// 0x6600 + d of 1536 + d less 1536, two at a time: the conversion instructions run at a quarter of the rate.
TROT_D void dg_split8(const double* x, int e, uint4* w) {
  const __half2 off = __half2half2(__ushort_as_half((unsigned short)0x6600));
  uint32_t h[kDgS][4];
#pragma unroll
  for (int i = 0; i < 8; i += 2) {
    int d[2][kDgS];
    uint32_t sign[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
      const unsigned long long u = (unsigned long long)__double_as_longlong(x[i + c]);
      const unsigned uh = (unsigned)(u >> 32);
      const int ex = (int)((uh >> 20) & 0x7FFu);
      sign[c] = uh & 0x80000000u;
      const unsigned long long M = (u & 0xFFFFFFFFFFFFFull) | 0x10000000000000ull;
      const int sh = 1075 - kDgBits + e - ex;  // |x| 2^(54 - e) = M 2^-sh; |x| < 2^e: sh >= -1
      unsigned long long q = (2 * M + (1ull << (sh + 1 < 63 ? sh + 1 : 63)) / 2) >> (sh + 1 < 63 ? sh + 1 : 63);
      if (ex == 0) q = 0;
      int lo = (int)((unsigned)q & 0x7FFFFFFu), hi = (int)(unsigned)(q >> 27);
#pragma unroll
      for (int t = kDgS - 1; t >= 3; --t) {
        d[c][t] = (lo << 23) >> 23;
        lo = (lo - d[c][t]) >> kDgLow;
      }
      hi += lo;  // the carry out of the low three digits
      d[c][2] = (hi << 23) >> 23;
      hi = (hi - d[c][2]) >> kDgLow;
      d[c][1] = (hi << 23) >> 23;
      d[c][0] = (hi - d[c][1]) >> kDgLow;
    }
    const uint32_t sg = (sign[0] >> 16) | sign[1];
#pragma unroll
    for (int t = 0; t < kDgS; ++t) {
      const uint32_t b = (uint32_t)((0x6600 + d[0][t]) & 0xFFFF) | ((uint32_t)(0x6600 + d[1][t]) << 16);
      const __half2 v = __hsub2(*reinterpret_cast<const __half2*>(&b), off);
      h[t][i >> 1] = *reinterpret_cast<const uint32_t*>(&v) ^ sg;
    }
  }
#pragma unroll
  for (int t = 0; t < kDgS; ++t) w[t] = make_uint4(h[t][0], h[t][1], h[t][2], h[t][3]);
}

// the same as stores of the six planes, `plane` entries apart
TROT_D void dg_store8(const double* x, int e, uint16_t* o, size_t plane) {
  uint4 w[kDgS];
  dg_split8(x, e, w);
#pragma unroll
  for (int t = 0; t < kDgS; ++t) *reinterpret_cast<uint4*>(o + t * plane) = w[t];
}

// x 2^k by its exponent bits (below the normal range: 0)
TROT_D double dg_shift(double x, int k) {
  const int hi = __double2hiint(x), e = (hi >> 20) & 0x7FF;
  if (e == 0x7FF) return x;
  if (e == 0 || e + k <= 0) return 0.0;
  if (e + k >= 0x7FF) return __hiloint2double(0x7FF00000, 0);
  return __hiloint2double(hi + k * (1 << 20), __double2loint(x));
}

TROT_D double dg_neg(double x) { return __hiloint2double(__double2hiint(x) ^ (int)0x80000000u, __double2loint(x)); }

// high word of the largest |x| so far, and sum of |x| as a float from its high word (the range only matters near
// the row maximum)
TROT_D void dg_row_max(double x, unsigned& mx, float& s) {
  const unsigned b = (unsigned)__double2hiint(x) & 0x7FFFFFFFu;
  mx = b > mx ? b : mx;
  const unsigned f = b - (896u << 20);
  s += f < (254u << 20) ? __uint_as_float(f << 3) : 0.f;
}

// exponent e (max |x| < 2^e) of a row from the high words of its largest |x| and its largest sum of |x| over 32 k
TROT_D int dg_exponent(unsigned mx, float l1) {
  const int E = (int)(mx >> 20);
  if (E == 0x7FF) return kDgNonFinite;
  if (E == 0) return 0;  // zero (or subnormal: dropped)
  int e = E - 1022;
  // sum |q_0| <= l1 2^(9 - e) + 16 over 32 k: keep it at 8192 or below
  // (rows outside FP32's range, whose sum is not known: always)
  if (e <= -110 || e >= 110 || l1 > ldexpf(8160.f, e - kDgTop)) ++e;
  return e;
}

// Real rows (complex A: row 2 m + c = real / imaginary part of row m; real B: a row or, with kst = ldb, a column) as
// digit images [tile][K16][plane][R][16].  A CTA takes one group of eight rows, lane = (row, k group), so a warp
// writes 128 B runs.  A cluster of KS CTAs (grid.x) shares one row group along K and exchanges the row maxima through
// distributed shared memory, so that long rows fill the chip; with K <= 256 KS every element is read once.
// The integer work (about 100 instructions per element) bounds it: 4.4M elements (7260 x 600) take 74 us with one CTA
// per 32 columns, 20 us like this.
struct DgSrc {
  const double* p;
  int K, nk16, R;        // R = 32 or 128 rows per tile
  int cplx, conj;        // conj: imaginary rows change sign
  // image row -> block (of bstride doubles) row / rpad, row r = row % rpad of it; rows r >= rpb and blocks
  // >= nblk are padding
  int rpb, rpad, nblk;
  long long bstride, rst, kst;  // strides in doubles (rst: of a complex row)
  // complex rows r >= split come from a second array (the other spin's walkers)
  int split;
  const double* p2;
  long long bstride2, kst2;
  uint16_t* img;
  int16_t* ex;
  // balanced sums (mode 2): element k of block b times 2^(ksign kexp[b kld + k])
  const int16_t* kexp;
  int kld, ksign;
  // exponent of the larger part of complex row r of block b at cexp[b cld + r] (mode 1; null: not wanted)
  int16_t* cexp;
  int cld;
};
static constexpr int kDgZeroTerm = -0x4000;  // exponent of a zero row: 2^e of it makes anything 0
static constexpr int kDgOneBlock = 1 << 30;
// `rows` rows of stride rst (complex ones count twice), one block
static DgSrc dg_src(const double* p, int cplx, int rows, int K, int R, long long rst, long long kst, uint16_t* img,
                    int16_t* ex) {
  return DgSrc{p, K, (K + 15) / 16, R, cplx, 0, rows, kDgOneBlock, 1, 0, rst, kst, kDgOneBlock, nullptr, 0, 0, img, ex,
               nullptr, 0, 0, nullptr, 0};
}

// Up to four sources of the same K in one launch: most are small (3 to 10 us, half of it the launch and the tail), and
// the operands of a product do not depend on one another.  FP64 energy of 67 orbitals, 200 walkers: 7 launches -> 4.
struct DgRows {
  static constexpr int kMax = 4;
  DgSrc s[kMax];
  int first[kMax + 1];  // first group of eight rows of each
  int count, ks;        // ks: CTAs of a cluster, one after the other in the grid
};

// MODE 1: a source may write cexp; 2: use kexp (in the plain kernel their tests alone cost 3 % of an FP64 step)
template <int MODE>
__global__ void __launch_bounds__(256) dg_rows_kernel(const __grid_constant__ DgRows q) {
  const int KS = q.ks, rank = (int)blockIdx.x % KS;
  int src = 0, group = (int)blockIdx.x / KS;
  while (src + 1 < q.count && group >= q.first[src + 1]) ++src;
  group -= q.first[src];
  const DgSrc& a = q.s[src];
  __shared__ unsigned smx[8][8], cmx[8];
  __shared__ float sl1[8][8], cl1[8];
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rl = lane & 7, kg = lane >> 3;
  const int row = group * 8 + rl;
  const int blk = row / a.rpad, rr = row - blk * a.rpad;
  const bool valid = blk < a.nblk && rr < a.rpb, flip = a.conj && (rr & 1);
  const double* p = a.p;
  long long kst = a.kst;
  if (valid) {
    if (rr >= a.split) {
      p = a.p2 + blk * a.bstride2 + ((rr - a.split) >> 1) * a.rst + (rr & 1);
      kst = a.kst2;
    } else if (a.cplx) {
      p += blk * a.bstride + (rr >> 1) * a.rst + (rr & 1);
    } else {
      p += blk * a.bstride + rr * a.rst;
    }
  }
  const int16_t* kexp = MODE == 2 ? a.kexp + (size_t)(valid ? blk : 0) * a.kld : nullptr;
  const int nwarp = (int)blockDim.x >> 5, kpad = a.nk16 * 16, kstep = nwarp * 32 * KS;
  unsigned mx = 0;
  float l1 = 0.f;
  double x[8];
  for (int k0 = (rank * nwarp + warp) * 32; k0 < kpad; k0 += kstep) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = k0 + kg * 8 + i;
      x[i] = (valid && k < a.K) ? p[k * kst] : 0.0;
      if (flip) x[i] = dg_neg(x[i]);
      if (MODE == 2 && k < a.K) x[i] = dg_shift(x[i], a.ksign * kexp[k]);
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) dg_row_max(x[i], mx, s);
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    s += __shfl_xor_sync(0xffffffffu, s, 16);
    l1 = fmaxf(l1, s);
  }
#pragma unroll
  for (int o = 8; o < 32; o <<= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane < 8) {
    smx[warp][lane] = mx;
    sl1[warp][lane] = l1;
  }
  __syncthreads();
  for (int w = 0; w < nwarp; ++w) {
    mx = max(mx, smx[w][rl]);
    l1 = fmaxf(l1, sl1[w][rl]);
  }
  if (KS > 1) {
    if (threadIdx.x < 8) {
      cmx[rl] = mx;
      cl1[rl] = l1;
    }
    cl.sync();
    for (int c = 0; c < KS; ++c) {
      mx = max(mx, cl.map_shared_rank(cmx, c)[rl]);
      l1 = fmaxf(l1, cl.map_shared_rank(cl1, c)[rl]);
    }
  }
  const int e = dg_exponent(mx, l1);
  if (rank == 0 && warp == 0 && lane < 8) a.ex[row] = (int16_t)e;
  if (MODE == 1 && a.cexp && rank == 0 && warp == 0) {
    const unsigned both = max(mx, __shfl_xor_sync(0xffffffffu, mx, 1));  // real and imaginary part
    if (lane < 8 && !(lane & 1) && valid)
      a.cexp[(size_t)blk * a.cld + (rr >> 1)] = (int16_t)(both >> 20 ? (int)(both >> 20) - 1022 : kDgZeroTerm);
  }
  const bool live = valid && e != kDgNonFinite;
  const int r = row % a.R;
  uint16_t* out = a.img + (size_t)(row / a.R) * a.nk16 * kDgS * a.R * 16;
  const bool once = kpad <= kstep;
  for (int k0 = (rank * nwarp + warp) * 32; k0 < kpad; k0 += kstep) {
    const int kb = k0 + kg * 8;
    if (kb >= kpad) continue;
    if (!once) {
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        x[i] = (live && kb + i < a.K) ? p[(kb + i) * kst] : 0.0;
        if (flip) x[i] = dg_neg(x[i]);
        if (MODE == 2 && kb + i < a.K) x[i] = dg_shift(x[i], a.ksign * kexp[kb + i]);
      }
    }
    if (!live) {
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = 0.0;
    }
    dg_store8(x, live ? e : 0, out + (size_t)(kb >> 4) * kDgS * a.R * 16 + dg_idx(r, kb & 15), a.R * 16);
  }
  if (KS > 1) cl.sync();  // the maxima stay readable until every CTA of the cluster has them
}

// a warp per 32 k, eight at most
static int dg_row_threads(int nk16) { return 32 * std::min(8, (nk16 + 1) / 2); }

static int dg_rows_launch(DgRows q, cudaStream_t st, int mode = 0) {
  const int groups = q.first[q.count], nk16 = q.s[0].nk16;
  if (groups == 0) return TROT_OK;
  int ks = 1;
  while (ks < 8 && nk16 * 16 > 256 * ks && groups * ks < 304) ks *= 2;
  cudaLaunchConfig_t cfg{};
  q.ks = ks;
  cfg.gridDim = dim3((unsigned)ks * (unsigned)groups);
  cfg.blockDim = dim3(dg_row_threads(nk16));
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = ks;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = ks > 1 ? 1 : 0;
  const cudaError_t rc = cudaLaunchKernelEx(
      &cfg, mode == 0 ? dg_rows_kernel<0> : mode == 1 ? dg_rows_kernel<1> : dg_rows_kernel<2>, q);
  if (rc != cudaSuccess) return cuda_status(rc, "dg_rows_kernel");
  TROT_CHECK_LAUNCH("dg_rows_kernel");
  return TROT_OK;
}
static void dg_rows_add(DgRows& q, const DgSrc& a, int groups) {
  q.s[q.count] = a;
  q.first[q.count + 1] = q.first[q.count] + groups;
  ++q.count;
}
static int dg_rows_launch(const DgSrc& a, int groups, cudaStream_t st, int mode = 0) {
  DgRows q{};
  dg_rows_add(q, a, groups);
  return dg_rows_launch(q, st, mode);
}

// ------------------------------------------------------------------ product
struct DgArgs {
  const uint16_t* imgB;  // MMA rows: columns n of B, [rt][nk16][6][128][16]
  const int16_t* exB;
  const uint16_t* imgA;  // MMA columns: rows of A, [tile][nk16][6][32][16]
  const int16_t* exA;
  int Nn, M;             // outputs: n < Nn, complex rows m < M
  int nrt, ntile;        // 128-row tiles and 32-row tiles (per batch)
  int nbatch, bB;        // batches: ntile 32-row tiles each, bB 128-row tiles (0: all share them)
  long long cstride;     // and cstride complex outputs
  // PAIR: outputs p >= psplit (0: none) go to C2 (row stride ldc2, batches cstride2 apart), column p - psplit; rows m
  // are stored at (m % perm) permn + m / perm (perm = 0: at m)
  int psplit, perm, permn;
  double2* C2;
  long long ldc2, cstride2;
  int nk16, shift;       // K16 steps; the outputs' integers are in units 2^(eA + eB - 54 + shift)
  double2* C;
  long long ldc;
  int salpha, ealpha, accumulate;  // alpha = salpha 2^ealpha, salpha = +-1
  int* status;
  int test_timeout_polls;          // TEST: the MMA thread's first wait is on a barrier nothing arrives on
};

// q 2^(ex - 1075) for results next to or outside the normal range
__device__ __noinline__ double dg_ldexp(unsigned long long q, unsigned sign, int ex) {
  const double d = ldexp((double)q, ex - 1075);
  return sign ? -d : d;
}

// v 2^E rounded to a double (ties away from zero), by integer operations (conversions and FP64 additions run on the
// narrow FP64 pipe: two of them per output took longer than the output's 26 products)
TROT_D double dg_double(long long v, int E) {
  const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
  const unsigned hi = (unsigned)(a >> 32);
  const int lz = __clz((int)(hi ? hi : (unsigned)a)) + (hi ? 0 : 32);  // 64 for v = 0
  const unsigned long long m = a << (lz & 63);              // 2^63 <= m < 2^64
  const unsigned long long q = ((m >> 10) + 1) >> 1;        // 53 bits; 2^53 carries into the exponent
  const int ex = 1023 + 63 - lz + E;                        // of the unrounded value
  const unsigned sign = (unsigned)((unsigned long long)v >> 32) & 0x80000000u;
  double d = __hiloint2double((int)(((unsigned)(ex - 1) << 20) + (unsigned)(q >> 32) + sign), (int)(unsigned)q);
  if (ex <= 0 || ex >= 0x7FE) d = dg_ldexp(q, sign, ex);
  return v == 0 ? 0.0 : d;
}

// out of line, so that its FP64 instructions are not issued (predicated off) for plain stores
__device__ __noinline__ void dg_add(double2* o, double2 v) { *o = cadd(*o, v); }

// PAIR: the 128-row tiles hold complex rows (row 2 p = real, 2 p + 1 = imaginary part of V[p]) and the product is the
// complex V T: C[m][p] = V_p . A_m.  Lanes 2 p and 2 p + 1 exchange the cross terms; each stores its part.
// TEST: the kernel of the timeout switch (its test in the MMA loop's function made every product 6 % slower)
template <bool PAIR, bool TEST>
__global__ void __launch_bounds__(kDgThreads, 1) dg_gemm_kernel(DgArgs a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char* base = smem_raw + ((128 - (tc::smem_u32(smem_raw) & 127)) & 127);
  unsigned char* sA = base;             // B's 128-row tile, K16 steps (kDgASlots)
  unsigned char* sB = base + kDgOffB;   // A's 32-row tiles, slabs (kDgBSlots)
  uint64_t* bars = reinterpret_cast<uint64_t*>(base + kDgOffBar);
  uint64_t* a_full = bars;
  uint64_t* a_free = a_full + kDgASlots;
  uint64_t* b_full = a_free + kDgASlots;
  uint64_t* b_free = b_full + kDgBSlots;
  uint64_t* acc_full = b_free + kDgBSlots;   // [2]
  uint64_t* acc_empty = acc_full + 2;        // [2]
  uint64_t* drain = acc_empty + 2;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(drain + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(drain + 2);
  static_assert((2 * kDgASlots + 2 * kDgBSlots + 4 + 3) * 8 <= 256, "barrier table");
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int n_items = a.nrt * a.ntile * a.nbatch, nk = a.nk16;
  const int nslab = (nk + kDgSlab - 1) / kDgSlab;
  if (warp == 16) tc::tmem_alloc(tslot, 512);
  if (tid == kDgEpi) {
    for (int k = 0; k < kDgASlots; ++k) {
      tc::mbar_init(&a_full[k], 1);
      tc::mbar_init(&a_free[k], 1);
    }
    for (int k = 0; k < kDgBSlots; ++k) {
      tc::mbar_init(&b_full[k], 1);
      tc::mbar_init(&b_free[k], 1);
    }
    for (int k = 0; k < 2; ++k) {
      tc::mbar_init(&acc_full[k], 1);
      tc::mbar_init(&acc_empty[k], 16);
    }
    tc::mbar_init(drain, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t taddr = *tslot;
  // item -> (batch, 32-row tile, 128-row tile), the last fastest
  if (warp == 16) {
    if (lane == 0) {
      bool ok = true;
      const uint64_t ad0 = tc::smem_desc(tc::smem_u32(sA), 128, 256);
      const uint64_t bd0 = tc::smem_desc(tc::smem_u32(sB), 128, 256);
      const uint32_t adlo = (uint32_t)ad0, bdlo = (uint32_t)bd0, dhi = (uint32_t)(ad0 >> 32);
      int ca = 0, cs = 0;  // K16 step and slab counters of this CTA
      if (TEST) ok = tc::mbar_wait(drain, 0u, (uint32_t)a.test_timeout_polls);
      for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
        for (int s = 0; s < nslab && ok; ++s, ++cs) {
          const int ks = min(kDgSlab, nk - s * kDgSlab), buf = cs & 1, bs = cs % kDgBSlots;
          if (cs >= 2) ok = tc::mbar_wait(&acc_empty[buf], (uint32_t)(((cs >> 1) - 1) & 1));
          if (ok) ok = tc::mbar_wait(&b_full[bs], (uint32_t)((cs / kDgBSlots) & 1));
          if (!ok) break;
          const uint32_t dcol = taddr + (uint32_t)(buf * 256);
          for (int k = 0; k < ks; ++k, ++ca) {
            const int slot = ca % kDgASlots;
            ok = tc::mbar_wait(&a_full[slot], (uint32_t)((ca / kDgASlots) & 1));
            if (!ok) break;
            tc::fence_after_sync();
            const uint32_t alo = adlo + (uint32_t)((slot * kDgAStep) >> 4);
            const uint32_t blo = bdlo + (uint32_t)((bs * kDgSlab * kDgBStep + k * kDgBStep) >> 4);
#pragma unroll
            for (int t = 0; t < kDgS; ++t) {
              const int np = t < 1 ? kDgS : kDgGroups - t;  // planes 0 .. np - 1
              if (t == 1 && k == 0) {  // order 6 starts here: its columns are overwritten
                tc::mma_bf16_lo(dcol + 32, alo + 256, blo, dhi, tc::idesc_f16_f32(128, 160), 1u);
                tc::mma_bf16_lo(dcol + 192, alo + 256, blo + (5 * kDgP * 32) / 16, dhi, tc::idesc_f16_f32(128, 32), 0u);
              } else {
                tc::mma_bf16_lo(dcol + (uint32_t)(t * kDgP), alo + (uint32_t)(t * 256), blo, dhi,
                                tc::idesc_f16_f32(128, np * kDgP), (k > 0 || t > 0) ? 1u : 0u);
              }
            }
            tc::mma_commit(&a_free[slot]);
          }
          if (ok) {
            tc::mma_commit(&b_free[bs]);
            tc::mma_commit(&acc_full[buf]);
          }
        }
      }
      if (!ok) {
        if (a.status) report_timeout(a.status);
        *abort_flag = 1;
        tc::mma_commit(drain);  // the MMAs already issued complete before the epilogue is released
        tc::mbar_wait(drain, 0u, 1000000u);
        tc::mbar_arrive(&acc_full[0]);
        tc::mbar_arrive(&acc_full[1]);
      }
    }
    __syncwarp();
  } else if (warp > 16) {
    if (lane == 0) {
      const bool la = warp == 17;  // loader of the 128-row tile; the other one loads the 32-row tiles
      const int slots = la ? kDgASlots : kDgBSlots;
      uint64_t* full = la ? a_full : b_full;
      uint64_t* free_ = la ? a_free : b_free;
      bool ok = !TEST;
      int c = 0;
      for (int item = blockIdx.x; item < n_items && ok; item += gridDim.x) {
        const int bt = item / (a.nrt * a.ntile);
        const int rt = item % a.nrt + bt * a.bB, tile = (item / a.nrt) % a.ntile + bt * a.ntile;
        for (int s = 0; s < nslab && ok; ++s) {
          const int ks = min(kDgSlab, nk - s * kDgSlab);
          const int nc = la ? ks : 1;
          for (int j = 0; j < nc; ++j, ++c) {
            const int slot = c % slots;
            if (c >= slots) {  // the MMAs that read the slot's previous contents are done
              const uint32_t par = (uint32_t)(((c / slots) - 1) & 1);
              uint32_t polls = 0;
              while (!tc::mbar_try_wait(&free_[slot], par))
                if (*abort_flag || ++polls > 20000000u) {
                  ok = false;
                  break;
                }
              if (!ok) break;
            }
            if (la) {
              tc::mbar_expect_tx(&full[slot], kDgAStep);
              tc::bulk_g2s(sA + (size_t)slot * kDgAStep,
                           a.imgB + ((size_t)rt * nk + s * kDgSlab + j) * (kDgAStep / 2), kDgAStep, &full[slot]);
            } else {
              tc::mbar_expect_tx(&full[slot], ks * kDgBStep);
              tc::bulk_g2s(sB + (size_t)slot * kDgSlab * kDgBStep,
                           a.imgA + ((size_t)tile * nk + s * kDgSlab) * (kDgBStep / 2), ks * kDgBStep,
                           &full[slot]);
            }
          }
        }
      }
      if (!ok) {
        if (!*abort_flag && a.status && !TEST) report_timeout(a.status);
        for (int u = c - 1; u >= 0 && u >= c - slots; --u)  // bounded drain of the copies in flight
          tc::mbar_wait(&full[u % slots], (uint32_t)((u / slots) & 1), 1000000u);
      }
    }
    __syncwarp();
  } else {
    const int q = warp & 3, h = warp >> 2;
    const uint32_t tl = taddr + ((uint32_t)(q * 32) << 16) + (uint32_t)(h * 8);
    const int sh = a.shift;
    // digit weights in the accumulator's units (sh >= 1, so that the largest stays an int32)
    const int m0 = 1 << (31 - sh), m1 = 1 << (27 - sh), m2 = 1 << (18 - sh), m3 = 1 << (9 - sh);
    const float lscale = __int_as_float((127 - sh) << 23);
    int cs = 0;
    bool ok = true;
    for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
      const int rt = item % a.nrt, ct = (item / a.nrt) % a.ntile, bt = item / (a.nrt * a.ntile);
      const int n = rt * 128 + q * 32 + lane;
      // exponents of this column and of the warp's eight rows (int16), loaded before the first wait
      int eb = n < a.Nn ? a.exB[(size_t)bt * a.bB * 128 + n] : 0;
      const uint4 ea = __ldg(reinterpret_cast<const uint4*>(a.exA + (size_t)(bt * a.ntile + ct) * kDgP + h * 8));
      long long acc[8];
#pragma unroll
      for (int x = 0; x < 8; ++x) acc[x] = 0;
      for (int s = 0; s < nslab; ++s, ++cs) {
        const int buf = cs & 1;
        if (ok && (!tc::mbar_wait(&acc_full[buf], (uint32_t)((cs >> 1) & 1)) || *abort_flag)) {
          if (!*abort_flag && a.status && lane == 0) report_timeout(a.status);
          ok = false;
        }
        ok = __all_sync(0xffffffffu, ok);
        if (!ok) continue;
        tc::fence_after_sync();
        uint32_t raw[kDgGroups][8];
#pragma unroll
        for (int d = 0; d < kDgGroups; ++d) tc::tmem_ld8_raw(tl + (uint32_t)(buf * 256 + d * kDgP), raw[d]);
        tc::tmem_wait_ld();
        tc::fence_before_sync();
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(&acc_empty[buf]);
#pragma unroll
        for (int x = 0; x < 8; ++x) {
          float f[kDgGroups];
#pragma unroll
          for (int d = 0; d < kDgGroups; ++d) {
            uint32_t v = raw[d][x];
            asm volatile("" : "+r"(v));  // consume after tcgen05.wait::ld
            f[d] = __uint_as_float(v);
          }
          // sum_d S_d 2^(-9 d) in units 2^(sh - 36): orders 0-3 exactly, the rest rounded once
          const float f4 = fmaf(fmaf(f[6], 1.953125e-03f, f[5]), 1.953125e-03f, f[4]) * lscale;
          long long v = acc[x];
          v += (long long)(__float2int_rn(f[0]) << 5) * m0;
          v += (long long)__float2int_rn(f[1]) * m1;
          v += (long long)__float2int_rn(f[2]) * m2;
          v += (long long)__float2int_rn(f[3]) * m3;
          v += (long long)__float2int_rn(f4);
          acc[x] = v;
        }
      }
      // outputs: lane = column n of C, register pairs = (re, im) of four complex rows
      if (!ok) eb = kDgNonFinite;
      const bool bad = eb == kDgNonFinite;
      eb += sh - kDgBits + a.ealpha;
      const int m0r = ct * (kDgP / 2) + h * 4;
      double2* o = a.C + bt * a.cstride + (long long)m0r * a.ldc + (PAIR ? n >> 1 : n);
      const uint32_t ew[4] = {ea.x, ea.y, ea.z, ea.w};
#pragma unroll
      for (int y = 0; y < 4; ++y, o += a.ldc) {
        const int e0 = (int)(int16_t)(ew[y] & 0xFFFFu), e1 = (int)(int16_t)(ew[y] >> 16);
        const double nan = __longlong_as_double(0x7FF8000000000000ll);
        double2 v = cmk(dg_double(a.salpha < 0 ? -acc[2 * y] : acc[2 * y], e0 + eb),
                        dg_double(a.salpha < 0 ? -acc[2 * y + 1] : acc[2 * y + 1], e1 + eb));
        if (bad || e0 == kDgNonFinite) v.x = nan;
        if (bad || e1 == kDgNonFinite) v.y = nan;
        if (PAIR) {
          const double w = __shfl_xor_sync(0xffffffffu, v.y, 1);
          if (m0r + y < a.M && n < a.Nn) {
            double* od = reinterpret_cast<double*>(o);
            if (a.perm | a.psplit) {
              const int m = m0r + y, pp = n >> 1;
              const long long mm = a.perm ? (long long)(m % a.perm) * a.permn + m / a.perm : m;
              od = reinterpret_cast<double*>(a.psplit && pp >= a.psplit
                                                 ? a.C2 + bt * a.cstride2 + mm * a.ldc2 + (pp - a.psplit)
                                                 : a.C + bt * a.cstride + mm * a.ldc + pp);
            }
            if (n & 1) od[1] = v.x + w;
            else od[0] = v.x - w;
          }
        } else if (m0r + y < a.M && n < a.Nn) {
          if (a.accumulate) dg_add(o, v);
          else *o = v;
        }
      }
    }
  }
  tc::fence_before_sync();
  __syncthreads();
  if (warp == 16) tc::tmem_dealloc(taddr, 512);
}

// ------------------------------------------------------------------ host
static constexpr size_t kDgRowBytes(size_t nk16) { return nk16 * 16 * kDgS * 2; }
// rows of A per pass are limited so that their image stays in L2
static constexpr size_t kDgImageCap = size_t(64) << 20;

static size_t dg_chunk_rows(size_t M, size_t K) {
  const size_t nk16 = (K + 15) / 16, per = 2 * kDgRowBytes(nk16);
  size_t mc = kDgImageCap / per / 64 * 64;
  if (mc < 64) mc = 64;
  return mc < M ? mc : (M + 15) / 16 * 16;
}

size_t dg_scratch_bytes(size_t M, size_t Nn, size_t K) {
  const size_t nk16 = (K + 15) / 16, mc = dg_chunk_rows(M, K), nb = (Nn + 127) / 128 * 128;
  return nb * kDgRowBytes(nk16) + 2 * mc * kDgRowBytes(nk16) + nb * 2 + 2 * mc * 2 + 5 * 256;
}

template <bool PAIR>
static int dg_gemm(DgArgs a, cudaStream_t st) {
  a.test_timeout_polls = tune_get(TROT_TUNE_TEST_TIMEOUT);
  const auto kernel = a.test_timeout_polls > 0 ? dg_gemm_kernel<PAIR, true> : dg_gemm_kernel<PAIR, false>;
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDgSmem);
  const int items = a.nrt * a.ntile * a.nbatch;
  kernel<<<items < 152 ? items : 152, kDgThreads, kDgSmem, st>>>(a);
  TROT_CHECK_LAUNCH("dg_gemm_kernel");
  return TROT_OK;
}

int launch_zgemm_dg(int M, int Nn, int K, double alpha, const double2* A, int lda, const double* B, int ldb,
                    bool b_is_nk, double2* C, long long ldc, bool accumulate, const DgScratch& s, cudaStream_t st) {
  if (M <= 0 || Nn <= 0) return TROT_OK;
  if (K <= 0 || K > (1 << 17) || s.bytes < dg_scratch_bytes(M, Nn, K)) {
    set_error("digit product: K=%d, scratch %zu < %zu", K, s.bytes, dg_scratch_bytes(M, Nn, K));
    return TROT_ERR_WORKSPACE_TOO_SMALL;
  }
  const int nk16 = (K + 15) / 16, nrt = (Nn + 127) / 128;
  const size_t mc = dg_chunk_rows(M, K);
  char* p = reinterpret_cast<char*>(((uintptr_t)s.p + 255) & ~(uintptr_t)255);
  auto take = [&](size_t n) {
    char* r = p;
    p += (n + 255) & ~(size_t)255;
    return r;
  };
  DgArgs a{};
  uint16_t* imgB = reinterpret_cast<uint16_t*>(take((size_t)nrt * 128 * kDgRowBytes(nk16)));
  uint16_t* imgA = reinterpret_cast<uint16_t*>(take(2 * mc * kDgRowBytes(nk16)));
  int16_t* exB = reinterpret_cast<int16_t*>(take((size_t)nrt * 128 * 2));
  int16_t* exA = reinterpret_cast<int16_t*>(take(2 * mc * 2));
  int lk = 0;
  while ((1 << lk) < K) ++lk;
  a.imgB = imgB; a.exB = exB; a.imgA = imgA; a.exA = exA;
  a.Nn = Nn; a.nrt = nrt; a.nk16 = nk16; a.nbatch = 1;
  // |sum| <= K 2^17 2^36 2^-shift <= 2^62 (the leading digits of a row average 256 at most); at most 8 (K <= 2^17)
  a.shift = lk > 10 ? lk - 9 : 1;
  int ea = 0;
  const double fa = frexp(alpha, &ea);  // alpha = fa 2^ea
  if (fa != 0.5 && fa != -0.5) { set_error("digit product: alpha %g is not a power of two", alpha); return TROT_ERR_UNSUPPORTED; }
  a.salpha = fa < 0 ? -1 : 1;
  a.ealpha = ea - 1;
  a.ldc = ldc; a.accumulate = accumulate ? 1 : 0; a.status = s.status;
  for (size_t m0 = 0; m0 < (size_t)M; m0 += mc) {
    const int mm = (int)std::min(mc, (size_t)M - m0);
    a.ntile = (2 * mm + kDgP - 1) / kDgP;
    DgRows rows{};
    dg_rows_add(rows, dg_src(reinterpret_cast<const double*>(A + (long long)m0 * lda), 1, 2 * mm, K, kDgP, 2ll * lda, 2,
                             imgA, exA), a.ntile * 4);
    if (m0 == 0) dg_rows_add(rows, dg_src(B, 0, Nn, K, 128, b_is_nk ? ldb : 1, b_is_nk ? 1 : ldb, imgB, exB), nrt * 16);
    TROT_TRY(dg_rows_launch(rows, st));
    a.M = mm;
    a.C = C + (long long)m0 * ldc;
    TROT_TRY(dg_gemm<false>(a, st));
  }
  return TROT_OK;
}

// ------------------------------------------------------------------ squares of real matrices
static size_t square_dg_each(size_t N) {  // scratch of one matrix
  const size_t rows = (2 * ((N + 1) / 2) + kDgP - 1) / kDgP * kDgP + (N + 127) / 128 * 128;
  return rows * (kDgRowBytes((N + 15) / 16) + 2) + (N + 1) / 2 * N * sizeof(double2);
}
int square_dg_count(size_t N, size_t G) {
  return (int)std::max<size_t>(1, std::min<size_t>({G, (size_t(128) << 20) / square_dg_each(N), 65535}));
}
size_t square_dg_bytes(size_t N, size_t count) { return count * square_dg_each(N) + 6 * 256; }

int launch_square_dg(int N, int count, const double* L, const DgScratch& s, double2** C, cudaStream_t st) {
  if (s.bytes < square_dg_bytes(N, count)) { set_error("squares: scratch %zu", s.bytes); return TROT_ERR_WORKSPACE_TOO_SMALL; }
  char* p = reinterpret_cast<char*>(((uintptr_t)s.p + 255) & ~(uintptr_t)255);
  auto take = [&](size_t n) {
    char* r = p;
    p += (n + 255) & ~(size_t)255;
    return r;
  };
  const int mh = (N + 1) / 2, tiles = (2 * mh + kDgP - 1) / kDgP, nrt = (N + 127) / 128;
  const size_t ra = (size_t)count * tiles * kDgP, rb = (size_t)count * nrt * 128, bytes = kDgRowBytes((N + 15) / 16);
  DgArgs a{};
  uint16_t* ia = reinterpret_cast<uint16_t*>(take(ra * bytes));
  uint16_t* ib = reinterpret_cast<uint16_t*>(take(rb * bytes));
  int16_t* ea = reinterpret_cast<int16_t*>(take(ra * 2));
  int16_t* eb = reinterpret_cast<int16_t*>(take(rb * 2));
  *C = reinterpret_cast<double2*>(take((size_t)count * mh * N * sizeof(double2)));
  DgSrc sa = dg_src(L, 0, N, N, kDgP, N, 1, ia, ea);
  sa.rpad = tiles * kDgP; sa.nblk = count; sa.bstride = (long long)N * N;
  DgRows rows{};
  dg_rows_add(rows, sa, (int)(ra / 8));
  DgSrc sb = dg_src(L, 0, N, N, 128, 1, N, ib, eb);
  sb.rpad = nrt * 128; sb.nblk = count; sb.bstride = (long long)N * N;
  dg_rows_add(rows, sb, (int)(rb / 8));
  TROT_TRY(dg_rows_launch(rows, st));
  a.imgA = ia; a.exA = ea; a.imgB = ib; a.exB = eb;
  a.Nn = N; a.M = mh; a.nrt = a.bB = nrt; a.ntile = tiles; a.nbatch = count; a.cstride = (long long)mh * N;
  a.nk16 = (N + 15) / 16; a.shift = 1; a.C = *C; a.ldc = N; a.salpha = 1; a.status = s.status;
  return dg_gemm<false>(a, st);
}

// ------------------------------------------------------------------ exchange
// f_g[i][j] = sum_p rot_chol_g[i][p] G[j][p] of a chunk of walkers as one product F (rows (b, j), columns (g, i)), then
// per walker sum_g sum_ij f_gij f_gji and the traces tr f_g (trot/meas/rhf.py:33-60,119-125).  F of a chunk stays in
// L2 (96 MB cap), so only the products cost: padding every walker's 2 n columns to the 32 of a tile, for sums
// in the product's own epilogue, would cost more than writing and reading F (n = 10: 38 % idle columns).
//
// exchange_pairs_kernel, one CTA per (64 Cholesky vectors, walker): the vectors' n x n blocks in shared memory, row i
// takes the pairs (i, i + k mod n), k <= n / 2, each product once (weight 2 off the diagonal), four FP64 FMAs each:
// 0.6 ms of the FP64 pipe at 120 orbitals, 12 + 10 electrons, 600 vectors, 1024 walkers, which bounds it.  The CTA's
// own reduction (8 FP64 additions in a row) costs as much as 6 vectors' products, hence 64 vectors per CTA.
static constexpr int kExgChunk = 64;     // vectors per partial sum
static constexpr int kExgThreads = 128;  // a thread per (vector, i) of the vectors in shared memory

int exchange_dg_chunks(int G) { return (G + kExgChunk - 1) / kExgChunk; }

__global__ void __launch_bounds__(kExgThreads)
exchange_pairs_kernel(int n, int G, int gsub, int nchunks, int mult, int add, const double2* __restrict__ F,
                      double2* __restrict__ partial, double2* __restrict__ fb) {
  extern __shared__ double2 sm[];
  __shared__ double2 red[32];
  const int b = blockIdx.y, chunk = blockIdx.x, tid = threadIdx.x;
  const int g0 = chunk * kExgChunk, g1 = min(G, g0 + kExgChunk);
  const size_t ld = (size_t)G * n;
  const double2* Fb = F + (size_t)b * n * ld;
  const int lds = gsub * n, g = tid / n, i = tid - g * n;
  double2 once = cmk(0.0, 0.0), twice = cmk(0.0, 0.0);
  for (int gs = g0; gs < g1; gs += gsub) {
    const int ng = min(gsub, g1 - gs), cols = ng * n;
    __syncthreads();
    if (tid < cols) {
      const double2* src = Fb + (size_t)gs * n + tid;
#pragma unroll 4
      for (int j = 0; j < n; ++j) sm[j * lds + tid] = src[(size_t)j * ld];
    }
    __syncthreads();
    if (tid < cols) {
      const double2* row = sm + (size_t)i * lds + g * n;  // f_{., i} of this thread's vector: element j is f[j][i]
      double2 x = sm[i * lds + tid];
      cfma(once, x, x);
      int j = i;
      for (int k = 1; 2 * k < n; ++k) {
        j = j + 1 == n ? 0 : j + 1;
        cfma(twice, sm[j * lds + tid], row[j]);
      }
      if ((n & 1) == 0) {  // both rows of an antipodal pair visit it
        j = j + 1 == n ? 0 : j + 1;
        cfma(once, sm[j * lds + tid], row[j]);
      }
    }
    // the traces, a thread per vector and component (a thread per vector issued twice the FP64 instructions of one warp,
    // which the others waited for: 54 us a chunk of 12-electron walkers, 50 like this)
    for (int q = tid; q < 2 * ng; q += kExgThreads) {
      const double* d = reinterpret_cast<const double*>(sm + (q >> 1) * n) + (q & 1);
      double t = 0.0;
      for (int r = 0; r < n; ++r) t += d[2 * r * (lds + 1)];
      if (mult == 2) t += t;
      double* o = reinterpret_cast<double*>(fb + (size_t)b * G + gs) + q;
      *o = add ? *o + t : t;
    }
  }
  once = cadd(once, cadd(twice, twice));
  once = block_sum2(once, red);
  if (tid == 0) {
    if (mult == 2) once = cadd(once, once);
    double2* o = partial + (size_t)b * nchunks + chunk;
    *o = add ? cadd(*o, once) : once;
  }
}

static size_t exg_chunk(size_t W, size_t n, size_t G) {  // walkers per pass, a multiple of 16 (whole 32-row tiles)
  size_t wc = (size_t(96) << 20) / (n * n * G * sizeof(double2)) / 16 * 16;
  if (wc < 16) wc = 16;
  return std::min(wc, (W + 15) / 16 * 16);
}

size_t exchange_dg_bytes(const Spins& sp, size_t W, size_t N, size_t G) {
  const size_t rb = kDgRowBytes((N + 15) / 16);
  size_t rows = 0, brows = 0, f = 0;
  for (int q = 0; q < sp.nspin; ++q) {
    const size_t n = sp.n[q];
    rows = std::max(rows, (2 * W * n + 31) / 32 * 32);
    brows = std::max(brows, (G * n + 127) / 128 * 128);
    f = std::max(f, exg_chunk(W, n, G) * n * n * G * sizeof(double2));
  }
  return (rows + brows) * (rb + 2) + f + 6 * 256;
}

int launch_exchange_dg(const Spins& sp, int W, int N, int G, const double2* green, double2* partial, double2* fb,
                       const DgScratch& s, cudaStream_t st) {
  const int nk16 = (N + 15) / 16, nchunks = exchange_dg_chunks(G);
  const size_t rb = kDgRowBytes(nk16);
  if (s.bytes < exchange_dg_bytes(sp, W, N, G)) { set_error("exchange: scratch %zu", s.bytes); return TROT_ERR_WORKSPACE_TOO_SMALL; }
  const int nmax = std::max(sp.n[0], sp.nspin == 2 ? sp.n[1] : 0);
  const size_t rows = ((size_t)2 * W * nmax + 31) / 32 * 32, brows = ((size_t)G * nmax + 127) / 128 * 128;
  char* p = reinterpret_cast<char*>(((uintptr_t)s.p + 255) & ~(uintptr_t)255);
  auto take = [&](size_t n) {
    char* r = p;
    p += (n + 255) & ~(size_t)255;
    return r;
  };
  DgArgs a{};
  uint16_t* imgB = reinterpret_cast<uint16_t*>(take(brows * rb));
  uint16_t* imgA = reinterpret_cast<uint16_t*>(take(rows * rb));
  int16_t* exB = reinterpret_cast<int16_t*>(take(brows * 2));
  int16_t* exA = reinterpret_cast<int16_t*>(take(rows * 2));
  double2* F = reinterpret_cast<double2*>(p);
  for (int q = 0; q < sp.nspin; ++q) {
    const int n = sp.n[q], Gn = G * n;
    a.nrt = (Gn + 127) / 128;
    DgRows rows{};
    if (q == 0 || sp.rot_chol[q] != sp.rot_chol[0] || n != sp.n[0])
      dg_rows_add(rows, dg_src(sp.rot_chol[q], 0, Gn, N, 128, N, 1, imgB, exB), a.nrt * 16);
    const int tiles = (2 * W * n + kDgP - 1) / kDgP;
    DgSrc sa = dg_src(reinterpret_cast<const double*>(green + (size_t)sp.off[q] * N), 1, 2 * n, N, kDgP, 2ll * N, 2, imgA, exA);
    sa.rpad = 2 * n;
    sa.nblk = W;
    sa.bstride = 2ll * sp.ntot * N;
    dg_rows_add(rows, sa, tiles * 4);
    TROT_TRY(dg_rows_launch(rows, st));
    a.imgB = imgB; a.exB = exB;
    a.Nn = Gn; a.nk16 = nk16; a.nbatch = 1; a.shift = 1;  // N <= 1024
    a.C = F; a.ldc = Gn; a.salpha = 1; a.ealpha = 0; a.accumulate = 0; a.status = s.status;
    const int wc = (int)exg_chunk(W, n, G);
    const int gsub = kExgThreads / n;  // n <= 64
    const size_t smem = (size_t)n * n * gsub * sizeof(double2);
    if (smem > 40 * 1024) cudaFuncSetAttribute(exchange_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    for (int w0 = 0; w0 < W; w0 += wc) {
      const int wn = std::min(wc, W - w0);
      const size_t t0 = (size_t)w0 * 2 * n / kDgP;
      a.imgA = imgA + t0 * kDgP * (rb / 2);
      a.exA = exA + t0 * kDgP;
      a.M = wn * n;
      a.ntile = (2 * wn * n + kDgP - 1) / kDgP;
      TROT_TRY(dg_gemm<false>(a, st));
      exchange_pairs_kernel<<<dim3(nchunks, wn), kExgThreads, smem, st>>>(n, G, gsub, nchunks, sp.mult[q], q > 0, F,
                                                                  partial + (size_t)w0 * nchunks, fb + (size_t)w0 * G);
      TROT_CHECK_LAUNCH("exchange_pairs_kernel");
    }
  }
  return TROT_OK;
}

// The traces alone, for a force bias without an energy: the diagonal elements f_gii of every occupied orbital i as one
// batch (rows: walkers, columns: vectors), then the sums over i in exchange_pairs_kernel's order, so that a step moves its
// walkers by the same bits whether or not it reports their energy.  The sums are left to the kernel that forms the fields
// (FbParts) where all f_gii fit a cap; they are FP64 additions, 43 us of that pipe at 22 columns, 600 vectors, 1024 walkers.
// One product over (i, p), of other roundings, takes about as long: its K is n times as long and its tiles are fewer (N =
// 135, n = 16, 540 vectors, 128 walkers leave 112 SMs without one).
static constexpr size_t kFbCap = size_t(256) << 20;
static size_t fb_chunk(const Spins& sp, size_t W, size_t G) {  // walkers per pass, a multiple of 16
  size_t wc = kFbCap / (sp.ntot * G * sizeof(double2)) / 16 * 16;
  if (wc < 16) wc = 16;
  return std::min(wc, (W + 15) / 16 * 16);
}

size_t fb_dg_bytes(const Spins& sp, size_t W, size_t N, size_t G) {
  const size_t rb = kDgRowBytes((N + 15) / 16), wc = fb_chunk(sp, W, G);
  const size_t nmax = std::max(sp.n[0], sp.nspin == 2 ? sp.n[1] : 0);
  return nmax * ((2 * wc + 31) / 32 * 32 + (G + 127) / 128 * 128) * (rb + 2) + sp.ntot * wc * G * sizeof(double2) + 6 * 256;
}

__global__ void __launch_bounds__(256) fb_traces_kernel(FbParts f, double2* __restrict__ fb) {
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < f.len; e += (size_t)gridDim.x * blockDim.x)
    fb[e] = fb_trace(f, e);
}

int launch_fb_dg(const Spins& sp, int W, int N, int G, const double2* green, double2* fb, FbParts* parts,
                 const DgScratch& s, cudaStream_t st) {
  if (s.bytes < fb_dg_bytes(sp, W, N, G)) { set_error("force bias: scratch %zu", s.bytes); return TROT_ERR_WORKSPACE_TOO_SMALL; }
  const size_t rb = kDgRowBytes((N + 15) / 16);
  const int gpad = (G + 127) / 128 * 128, wc = (int)fb_chunk(sp, W, G), nmax = std::max(sp.n[0], sp.nspin == 2 ? sp.n[1] : 0);
  const size_t rows = (size_t)nmax * ((2 * wc + 31) / 32 * 32);
  char* p = reinterpret_cast<char*>(((uintptr_t)s.p + 255) & ~(uintptr_t)255);
  auto take = [&](size_t n) {
    char* r = p;
    p += (n + 255) & ~(size_t)255;
    return r;
  };
  DgArgs a{};
  uint16_t* imgB = reinterpret_cast<uint16_t*>(take((size_t)nmax * gpad * rb));
  uint16_t* imgA = reinterpret_cast<uint16_t*>(take(rows * rb));
  int16_t* exB = reinterpret_cast<int16_t*>(take((size_t)nmax * gpad * 2));
  int16_t* exA = reinterpret_cast<int16_t*>(take(rows * 2));
  double2* F = reinterpret_cast<double2*>(p);
  const double* held = nullptr;  // whose digits imgB holds
  int held_n = 0;
  for (int w0 = 0; w0 < W; w0 += wc) {
    const int wn = std::min(wc, W - w0), apad = (2 * wn + kDgP - 1) / kDgP * kDgP;
    FbParts f{};
    f.nspin = sp.nspin;
    f.len = (size_t)wn * G;
    for (int q = 0; q < sp.nspin; ++q) {
      const int n = sp.n[q];
      DgRows r{};
      if (sp.rot_chol[q] != held || n != held_n) {
        held = sp.rot_chol[q];
        held_n = n;
        DgSrc sb = dg_src(sp.rot_chol[q], 0, G, N, 128, (long long)n * N, 1, imgB, exB);
        sb.rpad = gpad; sb.nblk = n; sb.bstride = N;
        dg_rows_add(r, sb, n * (gpad / 8));
      }
      DgSrc sa = dg_src(reinterpret_cast<const double*>(green + ((size_t)w0 * sp.ntot + sp.off[q]) * N), 1, 2 * wn, N,
                        kDgP, 2ll * sp.ntot * N, 2, imgA, exA);
      sa.rpad = apad; sa.nblk = n; sa.bstride = 2ll * N;
      dg_rows_add(r, sa, n * (apad / 8));
      TROT_TRY(dg_rows_launch(r, st));
      a.imgB = imgB; a.exB = exB; a.imgA = imgA; a.exA = exA;
      a.Nn = G; a.M = wn; a.nrt = a.bB = gpad / 128; a.ntile = apad / kDgP; a.nbatch = n;
      a.cstride = (long long)f.len; a.nk16 = (N + 15) / 16; a.shift = 1;  // N <= 1024
      a.C = F + sp.off[q] * f.len; a.ldc = G; a.salpha = 1; a.status = s.status;
      TROT_TRY(dg_gemm<false>(a, st));
      f.F[q] = a.C;
      f.n[q] = n;
      f.mult[q] = sp.mult[q];
    }
    if (parts && wc >= W) {
      *parts = f;
      return TROT_OK;
    }
    fb_traces_kernel<<<(unsigned)std::min<size_t>((f.len + 255) / 256, 152 * 8), 256, 0, st>>>(f, fb + (size_t)w0 * G);
    TROT_CHECK_LAUNCH("fb_traces_kernel");
  }
  return TROT_OK;
}

// ------------------------------------------------------------------ Trotter propagation
// w' = E sum_k ((i sqrt(dt))^k / k!) V^k E w of every walker (trot/prop/chol_afqmc_ops.py:198-222,
// trot/prop/utils.py:20-30) as a chain of batched digit products: per walker V (2 N rows, re / im interleaved) against
// the 2 nc columns (j, re / im) of U_k = V^k E w, U_{k+1}[j][p] = sum_q V[p][q] U_k[j][q] (PAIR).  Between two products
// dg_taylor_kernel adds the term to the sum O and rewrites U_k as digits.  U and O are kept transposed (walker, j, p), so
// that the products' rows are contiguous.  Bound by the products (0.11 ms per term at 120 orbitals, 22 columns, 1024
// walkers, with the digit image of V, 0.4 GB, streaming from HBM at half its rate).
struct DgTaylor {
  int W, N, nc, rpad;       // rpad: 32-row-tile rows per walker
  int k, last;              // term k of the sum; last: the digits are those of O (the operand of the final E)
  double coef;              // sqrt(dt)^k / k!
  const double* U;          // (W, nc, N) complex
  double* O;                // (W, nc, N) complex
  uint16_t* img;
  int16_t* ex;
};

// rows r = 2 j + c of a walker as in dg_rows_kernel; each thread also updates component c of O[j][k]
__global__ void __launch_bounds__(256) dg_taylor_kernel(DgTaylor a) {
  __shared__ unsigned smx[8][8];
  __shared__ float sl1[8][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rl = lane & 7, kg = lane >> 3;
  const int row = blockIdx.x * 8 + rl;
  const int b = row / a.rpad, r = row - b * a.rpad, c = r & 1;
  const bool valid = (r >> 1) < a.nc;
  const size_t base = valid ? 2 * ((size_t)(b * a.nc + (r >> 1)) * a.N) + c : 0;
  const int nk16 = (a.N + 15) / 16, kpad = nk16 * 16, nwarp = (int)blockDim.x >> 5, kstep = nwarp * 32;
  // i^k = 1, i, -1, -i: component c of i^k U is +- component c ^ (k & 1) of U
  const int flip = (a.k & 1) ? 1 - 2 * c : 0;  // offset of the other component
  const int q = a.k & 3;
  const double cf = (q == 2 || (q == 1 && c == 0) || (q == 3 && c == 1)) ? -a.coef : a.coef;
  unsigned mx = 0;
  float l1 = 0.f;
  double x[8];
  for (int k0 = warp * 32; k0 < kpad; k0 += kstep) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
      const int k = k0 + kg * 8 + i;
      x[i] = 0.0;
      if (valid && k < a.N) {
        const size_t e = base + 2 * (size_t)k;
        // both components in one load: the loads, 16 bytes apart from lane to lane, bound this pass
        const double2 uc = reinterpret_cast<const double2*>(a.U)[e >> 1];
        const double u = c ? uc.y : uc.x;
        double o = flip ? (c ? uc.x : uc.y) : u;
        o = a.k == 0 ? o : fma(cf, o, a.O[e]);
        a.O[e] = o;
        x[i] = a.last ? o : u;
      }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) dg_row_max(x[i], mx, s);
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    s += __shfl_xor_sync(0xffffffffu, s, 16);
    l1 = fmaxf(l1, s);
  }
#pragma unroll
  for (int o = 8; o < 32; o <<= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane < 8) {
    smx[warp][lane] = mx;
    sl1[warp][lane] = l1;
  }
  __syncthreads();
  for (int w = 0; w < nwarp; ++w) {
    mx = max(mx, smx[w][rl]);
    l1 = fmaxf(l1, sl1[w][rl]);
  }
  const int e = dg_exponent(mx, l1);
  if (warp == 0 && lane < 8) a.ex[row] = (int16_t)e;
  const bool live = valid && e != kDgNonFinite;
  uint16_t* out = a.img + (size_t)(row / kDgP) * nk16 * kDgS * kDgP * 16;
  const double* src = a.last ? a.O : a.U;
  for (int k0 = warp * 32; k0 < kpad; k0 += kstep) {
    const int kb = k0 + kg * 8;
    if (kb >= kpad) continue;
    if (kpad > kstep) {  // more than one run per thread: read again
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = (live && kb + i < a.N) ? src[base + 2 * (size_t)(kb + i)] : 0.0;
    }
    if (!live) {
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = 0.0;
    }
    dg_store8(x, live ? e : 0, out + (size_t)(kb >> 4) * kDgS * kDgP * 16 + dg_idx(row % kDgP, kb & 15), kDgP * 16);
  }
}

// propagated walkers from the transposed w'[j][p]; in step mode their overlap and weight
__global__ void __launch_bounds__(256) dg_trotter_tail_kernel(Spins sp, TrotterArgs a, const double2* __restrict__ wt) {
  extern __shared__ double2 smem[];
  const int b = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
  const int N = a.N, nc = sp.ntot;
  double2* W2 = smem;           // N x nc
  double2* Ms = W2 + N * nc;    // n x n
  const double2* src = wt + (size_t)b * nc * N;
  for (int e = tid; e < N * nc; e += nt) W2[(e % N) * nc + e / N] = src[e];
  __syncthreads();
  for (int s = 0; s < sp.nspin; ++s) {
    const int n = sp.n[s];
    double2* w = (s == 0 ? a.out_a : a.out_b) + (size_t)b * N * n;
    for (int e = tid; e < N * n; e += nt) w[e] = W2[(e / n) * nc + sp.off[s] + e % n];
  }
  if (a.overlaps == nullptr) return;
  overlap_and_weight(sp, a, N, nc, W2, Ms);
}

struct DgTrotterPlan {
  int nk16, vtiles, tiles, rpad;  // K16 steps; 128-row tiles of V, 32-row tiles and rows of U per walker
  int wc;                         // walkers per pass
  size_t rb, bytes;
};
// The digits of V are 1.5 times the size of V and more (rows up to a multiple of 128), so they are kept for a pass of
// walkers only, 1 GB of them (1800 walkers of 120 orbitals: many times what fills the chip).
static constexpr size_t kDgTrotterCap = size_t(1) << 30;
static DgTrotterPlan dg_trotter_plan(const Spins& sp, size_t W, size_t N) {
  DgTrotterPlan p{};
  p.nk16 = (int)((N + 15) / 16);
  p.vtiles = (int)((2 * N + 127) / 128);
  p.tiles = (2 * sp.ntot + kDgP - 1) / kDgP;
  p.rpad = p.tiles * kDgP;
  p.rb = kDgRowBytes(p.nk16);
  const size_t erows = (N + 127) / 128 * 128;
  const size_t rows = p.vtiles * 128 + p.rpad, each = rows * (p.rb + 2) + 2 * sp.ntot * N * sizeof(double2);
  const size_t wc = std::max<size_t>(1, std::min<size_t>(W, kDgTrotterCap / each));
  p.wc = (int)((W + (W + wc - 1) / wc - 1) / ((W + wc - 1) / wc));  // passes of equal size
  p.bytes = p.wc * each + erows * (p.rb + 2) + 10 * 256;
  return p;
}

size_t trotter_dg_bytes(const Spins& sp, size_t W, size_t N) { return dg_trotter_plan(sp, W, N).bytes; }

int launch_trotter_dg(const Spins& sp, const TrotterArgs& t, const DgScratch& s, cudaStream_t st) {
  const int N = t.N, nc = sp.ntot;
  const DgTrotterPlan pl = dg_trotter_plan(sp, t.W, N);
  if (s.bytes < pl.bytes) { set_error("trotter: scratch %zu < %zu", s.bytes, pl.bytes); return TROT_ERR_WORKSPACE_TOO_SMALL; }
  char* p = reinterpret_cast<char*>(((uintptr_t)s.p + 255) & ~(uintptr_t)255);
  auto take = [&](size_t n) {
    char* r = p;
    p += (n + 255) & ~(size_t)255;
    return r;
  };
  const size_t vrows = (size_t)pl.wc * pl.vtiles * 128, urows = (size_t)pl.wc * pl.rpad, erows = (size_t)(N + 127) / 128 * 128;
  uint16_t* vimg = reinterpret_cast<uint16_t*>(take(vrows * pl.rb));
  uint16_t* uimg = reinterpret_cast<uint16_t*>(take(urows * pl.rb));
  uint16_t* eimg = reinterpret_cast<uint16_t*>(take(erows * pl.rb));
  int16_t* vex = reinterpret_cast<int16_t*>(take(vrows * 2));
  int16_t* uex = reinterpret_cast<int16_t*>(take(urows * 2));
  int16_t* eex = reinterpret_cast<int16_t*>(take(erows * 2));
  double2* U = reinterpret_cast<double2*>(take((size_t)pl.wc * nc * N * sizeof(double2)));
  double2* O = reinterpret_cast<double2*>(take((size_t)pl.wc * nc * N * sizeof(double2)));
  const int nmax = std::max(sp.n[0], sp.nspin == 2 ? sp.n[1] : 0);
  const size_t smem = (size_t)(N * nc + nmax * nmax) * sizeof(double2);
  for (int w0 = 0; w0 < t.W; w0 += pl.wc) {
    const int W = std::min(pl.wc, t.W - w0);
    TrotterArgs a = t;  // of this pass
    a.W = W;
    a.vhs += (size_t)w0 * N * N;
    for (int q = 0; q < sp.nspin; ++q) {
      const size_t off = (size_t)w0 * N * sp.n[q];
      (q ? a.in_b : a.in_a) += off;
      (q ? a.out_b : a.out_a) += off;
    }
    if (a.overlaps) {
      a.overlaps += w0;
      a.weights += w0;
      a.shift_term += w0;
      a.fb_term += w0;
      a.node_flag += w0;
    }
    // digits of V (walker, 2 p + c), of E and of the walkers (walker, 2 j + c; K along the orbitals)
    DgSrc sv = dg_src(reinterpret_cast<const double*>(a.vhs), 1, 2 * N, N, 128, 2ll * N, 2, vimg, vex);
    sv.rpad = pl.vtiles * 128;
    sv.nblk = W;
    sv.bstride = 2ll * N * N;
    DgRows rows{};
    if (t.nterms > 0) dg_rows_add(rows, sv, W * pl.vtiles * 16);
    if (w0 == 0) dg_rows_add(rows, dg_src(t.expH, 0, N, N, 128, N, 1, eimg, eex), (int)erows / 8);
    DgSrc sw = dg_src(reinterpret_cast<const double*>(a.in_a), 1, 2 * nc, N, kDgP, 2, 2ll * sp.n[0], uimg, uex);
    sw.rpad = pl.rpad;
    sw.nblk = W;
    sw.bstride = 2ll * N * sp.n[0];
    if (sp.nspin == 2) {
      sw.split = 2 * sp.n[0];
      sw.p2 = reinterpret_cast<const double*>(a.in_b);
      sw.bstride2 = 2ll * N * sp.n[1];
      sw.kst2 = 2ll * sp.n[1];
    }
    dg_rows_add(rows, sw, W * pl.tiles * 4);
    TROT_TRY(dg_rows_launch(rows, st));
    DgArgs e{};  // E x
    e.imgB = eimg; e.exB = eex; e.imgA = uimg; e.exA = uex;
    e.Nn = N; e.M = nc; e.nrt = (N + 127) / 128; e.ntile = pl.tiles; e.nk16 = pl.nk16; e.shift = 1;
    e.nbatch = W; e.bB = 0; e.cstride = (long long)nc * N;
    e.C = U; e.ldc = N; e.salpha = 1; e.status = s.status;
    DgArgs v = e;  // V x
    v.imgB = vimg; v.exB = vex; v.Nn = 2 * N; v.nrt = v.bB = pl.vtiles;
    TROT_TRY(dg_gemm<false>(e, st));
    DgTaylor ty{W, N, nc, pl.rpad, 0, t.nterms == 0, 1.0, (const double*)U, (double*)O, uimg, uex};
    for (int k = 0;; ++k) {
      ty.k = k;
      ty.last = k == t.nterms;
      dg_taylor_kernel<<<W * pl.tiles * 4, dg_row_threads(pl.nk16), 0, st>>>(ty);
      TROT_CHECK_LAUNCH("dg_taylor_kernel");
      if (k == t.nterms) break;
      TROT_TRY(dg_gemm<true>(v, st));
      ty.coef *= t.sqrt_dt / (double)(k + 1);
    }
    TROT_TRY(dg_gemm<false>(e, st));
    if (smem > 40 * 1024)
      cudaFuncSetAttribute(dg_trotter_tail_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    dg_trotter_tail_kernel<<<W, 256, smem, st>>>(sp, a, U);
    TROT_CHECK_LAUNCH("dg_trotter_tail_kernel");
  }
  return TROT_OK;
}

// ------------------------------------------------------------------ step adjoint
static size_t adj_rows(size_t rows, size_t tile) { return (rows + tile - 1) / tile * tile; }

size_t adjoint_dg_bytes(size_t W, size_t N, size_t nc, size_t K2) {
  DgAdjoint d{};
  DgScratch s{};
  adjoint_dg_carve(d, (int)W, (int)N, (int)nc, (int)K2, s);
  return (size_t)((char*)d.cexp - (char*)nullptr) + W * K2 * 2 + 512;
}

// (with s.p null the pointers are offsets from the start, for the size)
void adjoint_dg_carve(DgAdjoint& d, int W, int N, int nc, int K2, const DgScratch& s) {
  d.W = W; d.N = N; d.nc = nc; d.K2 = K2; d.status = s.status;
  char* p = reinterpret_cast<char*>(((uintptr_t)s.p + 255) & ~(uintptr_t)255);
  auto take = [&](size_t n) {
    char* r = p;
    p += (n + 255) & ~(size_t)255;
    return r;
  };
  const size_t rb = kDgRowBytes((N + 15) / 16), rb2 = kDgRowBytes((K2 + 15) / 16);
  const size_t vr = (size_t)W * adj_rows(2 * N, 128), ur = (size_t)W * adj_rows(2 * nc, kDgP);
  const size_t gr = (size_t)W * adj_rows(2 * N, kDgP), er = adj_rows(N, 128);
  d.vimg = reinterpret_cast<uint16_t*>(take(vr * std::max(rb, rb2)));
  d.uimg = reinterpret_cast<uint16_t*>(take(std::max(ur * rb, gr * rb2)));
  d.eimg = reinterpret_cast<uint16_t*>(take(er * rb));
  d.etimg = reinterpret_cast<uint16_t*>(take(er * rb));
  d.vex = reinterpret_cast<int16_t*>(take(vr * 2));
  d.uex = reinterpret_cast<int16_t*>(take(std::max(ur, gr) * 2));
  d.eex = reinterpret_cast<int16_t*>(take(er * 2));
  d.etex = reinterpret_cast<int16_t*>(take(er * 2));
  d.cexp = reinterpret_cast<int16_t*>(take((size_t)W * K2 * 2));
}

int adjoint_dg_e(const DgAdjoint& d, const double* E, cudaStream_t st) {
  const int groups = (int)adj_rows(d.N, 128) / 8;
  DgRows rows{};
  dg_rows_add(rows, dg_src(E, 0, d.N, d.N, 128, d.N, 1, d.eimg, d.eex), groups);
  dg_rows_add(rows, dg_src(E, 0, d.N, d.N, 128, 1, d.N, d.etimg, d.etex), groups);
  return dg_rows_launch(rows, st);
}

int adjoint_dg_v(const DgAdjoint& d, const double2* V, bool transposed, cudaStream_t st) {
  const int N = d.N, rpad = (int)adj_rows(2 * N, 128);
  DgSrc s = dg_src(reinterpret_cast<const double*>(V), 1, 2 * N, N, 128, transposed ? 2 : 2ll * N,
                   transposed ? 2ll * N : 2, d.vimg, d.vex);
  s.rpad = rpad;
  s.nblk = d.W;
  s.bstride = 2ll * N * N;
  return dg_rows_launch(s, d.W * (rpad / 8), st);
}

__global__ void dg_clear_flags_kernel(int W, int rpad, const int* __restrict__ act, int16_t* __restrict__ ex) {
  const size_t total = (size_t)W * rpad;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x)
    if (!act[e / rpad] && ex[e] == kDgNonFinite) ex[e] = 0;  // such a row's digits are zeros
}

int adjoint_dg_v_active(const DgAdjoint& d, const int* act, cudaStream_t st) {
  const int rpad = (int)adj_rows(2 * d.N, 128);
  const size_t total = (size_t)d.W * rpad;
  dg_clear_flags_kernel<<<(int)std::min<size_t>((total + 255) / 256, 1024), 256, 0, st>>>(d.W, rpad, act, d.vex);
  TROT_CHECK_LAUNCH("dg_clear_flags_kernel");
  return TROT_OK;
}

static int adj_apply(const DgAdjoint& d, DgOperand op, DgSrc s, double2* out, long long ostride, cudaStream_t st) {
  const int rpad = (int)adj_rows(2 * d.nc, kDgP);
  s.rpad = rpad;
  s.nblk = d.W;
  TROT_TRY(dg_rows_launch(s, d.W * (rpad / 8), st, s.cexp ? 1 : 0));
  DgArgs a{};
  a.imgA = d.uimg; a.exA = d.uex;
  a.imgB = op == kDgV ? d.vimg : op == kDgE ? d.eimg : d.etimg;
  a.exB = op == kDgV ? d.vex : op == kDgE ? d.eex : d.etex;
  a.Nn = op == kDgV ? 2 * d.N : d.N; a.M = d.nc;
  a.nrt = (a.Nn + 127) / 128; a.bB = op == kDgV ? a.nrt : 0;
  a.ntile = rpad / kDgP; a.nbatch = d.W; a.cstride = ostride;
  a.nk16 = (d.N + 15) / 16; a.shift = 1;
  a.C = out; a.ldc = d.N; a.salpha = 1; a.status = d.status;
  return op == kDgV ? dg_gemm<true>(a, st) : dg_gemm<false>(a, st);
}

int adjoint_dg_from_walkers(const DgAdjoint& d, DgOperand op, const double2* wa, int na, const double2* wb, int nb,
                            bool conj, double2* out, long long ostride, cudaStream_t st) {
  DgSrc s = dg_src(reinterpret_cast<const double*>(wa), 1, 2 * d.nc, d.N, kDgP, 2, 2ll * na, d.uimg, d.uex);
  s.conj = conj;
  s.bstride = 2ll * d.N * na;
  if (wb) {
    s.split = 2 * na;
    s.p2 = reinterpret_cast<const double*>(wb);
    s.bstride2 = 2ll * d.N * nb;
    s.kst2 = 2ll * nb;
  }
  return adj_apply(d, op, s, out, ostride, st);
}

int adjoint_dg_from_rows(const DgAdjoint& d, DgOperand op, const double2* src, long long sstride, double2* out,
                         long long ostride, cudaStream_t st, int term) {
  DgSrc s = dg_src(reinterpret_cast<const double*>(src), 1, 2 * d.nc, d.N, kDgP, 2ll * d.N, 2, d.uimg, d.uex);
  s.bstride = 2 * sstride;
  if (term >= 0) {
    s.cexp = d.cexp + term * d.nc;
    s.cld = d.K2;
  }
  return adj_apply(d, op, s, out, ostride, st);
}

// A term k = (l, j) of the sum is column j of V^l E w times one of its cotangent: the first grows like |V|^l, the second
// falls like sqrt(dt)^(l + 1) / (l + 1)!, and their columns' scales are each other's inverse.  A digit row has one
// exponent, so as they stand the large l of U (at the small l of S) would leave the leading terms few digits: with
// sqrt(dt) |V| = 1.4 (80 orbitals) the error was 7.7e-12 of the largest element, 1.9e-9 with 2.8 (120 orbitals).
// Therefore U_k 2^-e and S_k 2^e with e the exponent of column k of U: all columns of U peak at 1/2 to 1, and the row
// maxima of S are those of the terms (2e-16 at both).
int adjoint_dg_gv(const DgAdjoint& d, const double2* S, long long sstride, const double2* U, long long ustride,
                  double2* gv, cudaStream_t st) {
  const int N = d.N, rpad = (int)adj_rows(2 * N, kDgP), vpad = (int)adj_rows(2 * N, 128);
  DgSrc s = dg_src(reinterpret_cast<const double*>(S), 1, 2 * N, d.K2, kDgP, 2, 2ll * N, d.uimg, d.uex);
  s.rpad = rpad;
  s.nblk = d.W;
  s.bstride = 2 * sstride;
  s.kexp = d.cexp;
  s.kld = d.K2;
  s.ksign = 1;
  DgRows rows{};
  dg_rows_add(rows, s, d.W * (rpad / 8));
  DgSrc u = dg_src(reinterpret_cast<const double*>(U), 1, 2 * N, d.K2, 128, 2, 2ll * N, d.vimg, d.vex);
  u.rpad = vpad;
  u.nblk = d.W;
  u.bstride = 2 * ustride;
  u.kexp = d.cexp;
  u.kld = d.K2;
  u.ksign = -1;
  dg_rows_add(rows, u, d.W * (vpad / 8));
  TROT_TRY(dg_rows_launch(rows, st, 2));
  DgArgs a{};
  a.imgA = d.uimg; a.exA = d.uex; a.imgB = d.vimg; a.exB = d.vex;
  a.Nn = 2 * N; a.M = N; a.nrt = a.bB = vpad / 128; a.ntile = rpad / kDgP; a.nbatch = d.W;
  a.cstride = (long long)N * N; a.nk16 = (d.K2 + 15) / 16; a.shift = 1;  // K2 <= 7 x 64
  a.C = gv; a.ldc = N; a.salpha = 1; a.status = d.status;
  return dg_gemm<true>(a, st);
}

// ------------------------------------------------------------------ CISD per-vector terms
// Per walker and Cholesky vector (L = chol_g, R = L[:n, :]): lg1 = R G^T, B = G lci1_g, gl = G L, glgp = gl gp and
// sum gl o lci2_green = <lg1, gl P2> (lci2_green = lg1 P2^T).  For a chunk of walkers: three products of the rows of G
// (all vectors), then gl's rows against [gp | P2] (N columns per walker), so that no contraction over orbitals is left on
// the FP64 pipe; cisd_pairs_kernel sums what is left, 4 n^2 (n + 3) FMAs per vector.  Chunks keep gl (64 MB) in L2.
// 41 orbitals, 6 + 6 electrons, 164 vectors, 96 walkers: 1.74 ms with every contraction on the FP64 pipe (per vector, in
// shared memory), 0.38 ms like this.
static constexpr int kPairsChunk = 64;

int cisd_gamma_dg_chunks(int G) { return (G + kPairsChunk - 1) / kPairsChunk; }

// Q[b][i][c]: gp (c < v: rows i < n hold x[i][c] = G[i][n + c], row n + c holds -1) and P2 (c >= v)
__global__ void cisd_q_kernel(int N, int n, int v, const double2* __restrict__ green, const double2* __restrict__ p2,
                              double2* __restrict__ Q) {
  const int b = blockIdx.y;
  for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < N * N; e += gridDim.x * blockDim.x) {
    const int i = e / N, c = e - i * N;
    double2 x = cmk(0.0, 0.0);
    if (c >= v) x = p2[((size_t)b * N + i) * n + c - v];
    else if (i < n) x = green[((size_t)b * n + i) * N + n + c];
    else if (i - n == c) x = cmk(-1.0, 0.0);
    Q[(size_t)b * N * N + e] = x;
  }
}

// F1[(b, q)][(g, p)] = lg1[p][q], F2[(b, p)][(g, q)] = B[p][q], F3[b][g][p][k] = (gl P2)[p][k]:
// [0] sum lg1 o lg1^T, [1] tr(lg1 lg1 ci1g1), [2] sum B o lg1, [3] sum F3 o lg1
__global__ void __launch_bounds__(128)
cisd_pairs_kernel(int n, int G, int gsub, int nchunk, const double2* __restrict__ F1, const double2* __restrict__ F2,
                  const double2* __restrict__ F3, const double2* __restrict__ ci1g1, double2* __restrict__ gpart) {
  extern __shared__ double2 sm[];
  __shared__ double2 red[32];
  const int chunk = blockIdx.x, b = blockIdx.y, tid = threadIdx.x, nt = blockDim.x, nn = n * n;
  double2* C1 = sm;       // n x n
  double2* A = C1 + nn;   // gsub x n x n
  for (int e = tid; e < nn; e += nt) C1[e] = ci1g1[(size_t)b * nn + e];
  const size_t ld = (size_t)G * n;
  const double2* f1 = F1 + (size_t)b * n * ld;
  const double2* f2 = F2 + (size_t)b * n * ld;
  const double2* f3 = F3 + (size_t)b * G * nn;
  double2 s0 = cmk(0.0, 0.0), s1 = cmk(0.0, 0.0), s2 = cmk(0.0, 0.0), s3 = cmk(0.0, 0.0);
  const int g0 = chunk * kPairsChunk, g1 = min(G, g0 + kPairsChunk);
  for (int gs = g0; gs < g1; gs += gsub) {
    const int cols = min(gsub, g1 - gs) * n, items = cols * n;
    __syncthreads();
    for (int e = tid; e < items; e += nt) {  // (q, g, p), p fastest
      const int q = e / cols, r = e - q * cols, g = r / n, p = r - g * n;
      A[g * nn + p * n + q] = f1[(size_t)q * ld + (size_t)gs * n + r];
    }
    __syncthreads();
    for (int e = tid; e < items; e += nt) {
      const int g = e / nn, pq = e - g * nn, p = pq / n, q = pq - p * n;
      const double2* Ag = A + g * nn;
      const double2 apq = Ag[pq];
      double2 t = cmk(0.0, 0.0);
      for (int a = 0; a < n; ++a) cfma(t, Ag[q * n + a], C1[a * n + p]);
      cfma(s0, apq, Ag[q * n + p]);
      cfma(s1, apq, t);
      cfma(s2, apq, f2[(size_t)p * ld + (size_t)(gs + g) * n + q]);
      cfma(s3, apq, f3[(size_t)(gs + g) * nn + pq]);
    }
  }
  s0 = block_sum2(s0, red);
  s1 = block_sum2(s1, red);
  s2 = block_sum2(s2, red);
  s3 = block_sum2(s3, red);
  if (tid == 0) {
    double2* o = gpart + ((size_t)b * nchunk + chunk) * 4;
    o[0] = s0; o[1] = s1; o[2] = s2; o[3] = s3;
  }
}

static void cisd_lg_rows(DgRows& rows, const CisdGammaArgs& c, uint16_t* irow, int16_t* erow, uint16_t* ilc,
                         int16_t* elc);

static size_t cgd_chunk(size_t W, size_t N, size_t n, size_t G) {
  const size_t wc = std::max<size_t>(1, (size_t(64) << 20) / (n * G * N * sizeof(double2)));
  return std::min(wc, W);
}

struct CgdBuffers {
  uint16_t *icol, *irow, *ilc, *ig, *igl, *iq;
  int16_t *ecol, *erow, *elc, *eg, *egl, *eq;
  double2 *gl, *F1, *F2, *F3, *Q;
};
static size_t cgd_carve(CgdBuffers& b, size_t wc, size_t N, size_t n, size_t G, void* base) {
  char* p0 = reinterpret_cast<char*>(((uintptr_t)base + 255) & ~(uintptr_t)255);
  char* p = p0;
  auto take = [&](size_t k) {
    char* r = p;
    p += (k + 255) & ~(size_t)255;
    return r;
  };
  const size_t rb = kDgRowBytes((N + 15) / 16);
  const size_t col = adj_rows(G * N, 128), row = adj_rows(G * n, 128), g = adj_rows(2 * wc * n, kDgP);
  const size_t gl = wc * adj_rows(2 * G * n, kDgP), q = wc * adj_rows(2 * N, 128);
  b.icol = (uint16_t*)take(col * rb); b.irow = (uint16_t*)take(row * rb); b.ilc = (uint16_t*)take(row * rb);
  b.ig = (uint16_t*)take(g * rb); b.igl = (uint16_t*)take(gl * rb); b.iq = (uint16_t*)take(q * rb);
  b.ecol = (int16_t*)take(col * 2); b.erow = (int16_t*)take(row * 2); b.elc = (int16_t*)take(row * 2);
  b.eg = (int16_t*)take(g * 2); b.egl = (int16_t*)take(gl * 2); b.eq = (int16_t*)take(q * 2);
  b.gl = (double2*)take(wc * n * G * N * sizeof(double2));
  b.F1 = (double2*)take(wc * n * n * G * sizeof(double2));
  b.F2 = (double2*)take(wc * n * n * G * sizeof(double2));
  b.F3 = (double2*)take(wc * n * n * G * sizeof(double2));
  b.Q = (double2*)take(wc * N * N * sizeof(double2));
  return (size_t)(p - p0) + 256;
}

size_t cisd_gamma_dg_bytes(size_t W, size_t N, size_t n, size_t G) {
  CgdBuffers b;
  return cgd_carve(b, cgd_chunk(W, N, n, G), N, n, G, nullptr);
}

int launch_cisd_gamma_dg(const CisdGammaArgs& c, const DgScratch& s, cudaStream_t st) {
  const int W = c.W, N = c.N, n = c.n, v = c.v, G = c.G, nn = n * n;
  const int wc = (int)cgd_chunk(W, N, n, G);
  CgdBuffers b;
  if (s.bytes < cgd_carve(b, wc, N, n, G, s.p)) { set_error("CISD terms: scratch %zu", s.bytes); return TROT_ERR_WORKSPACE_TOO_SMALL; }
  // rows (g, i) = columns of L_g; (g, p) = rows p < n of L_g; (g, a) = columns of lci1_g
  DgSrc sc = dg_src(c.chol, 0, N, N, 128, 1, N, b.icol, b.ecol);
  sc.rpad = N; sc.nblk = G; sc.bstride = (long long)N * N;
  DgRows first{};
  dg_rows_add(first, sc, (int)(adj_rows((size_t)G * N, 128) / 8));
  cisd_lg_rows(first, c, b.irow, b.erow, b.ilc, b.elc);
  const int gsub = std::max(1, std::min(kPairsChunk, 256 / nn)), nchunk = cisd_gamma_dg_chunks(G);
  const size_t smem = (size_t)(gsub + 1) * nn * sizeof(double2);
  if (smem > 40 * 1024) cudaFuncSetAttribute(cisd_pairs_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  const int qpad = (int)adj_rows(2 * N, 128), glpad = (int)adj_rows((size_t)2 * G * n, kDgP);
  for (int w0 = 0; w0 < W; w0 += wc) {
    const int wn = std::min(wc, W - w0);
    const double2* gr = c.green + (size_t)w0 * n * N;
    const int tiles = (2 * wn * n + kDgP - 1) / kDgP;
    DgRows rows = w0 == 0 ? first : DgRows{};
    dg_rows_add(rows, dg_src(reinterpret_cast<const double*>(gr), 1, 2 * wn * n, N, kDgP, 2ll * N, 2, b.ig, b.eg), tiles * 4);
    TROT_TRY(dg_rows_launch(rows, st));
    DgArgs a{};
    a.imgA = b.ig; a.exA = b.eg; a.M = wn * n; a.ntile = tiles; a.nbatch = 1;
    a.nk16 = (N + 15) / 16; a.shift = 1; a.salpha = 1; a.status = s.status;
    a.imgB = b.irow; a.exB = b.erow; a.Nn = G * n; a.nrt = (G * n + 127) / 128; a.C = b.F1; a.ldc = (long long)G * n;
    TROT_TRY(dg_gemm<false>(a, st));
    a.imgB = b.ilc; a.exB = b.elc; a.C = b.F2;
    TROT_TRY(dg_gemm<false>(a, st));
    a.imgB = b.icol; a.exB = b.ecol; a.Nn = G * N; a.nrt = (G * N + 127) / 128; a.C = b.gl; a.ldc = (long long)G * N;
    TROT_TRY(dg_gemm<false>(a, st));
    // gl rows (p, g) of each walker against the columns of [gp | P2]
    cisd_q_kernel<<<dim3((N * N + 255) / 256, wn), 256, 0, st>>>(N, n, v, gr, c.p2 + (size_t)w0 * N * n, b.Q);
    TROT_CHECK_LAUNCH("cisd_q_kernel");
    DgSrc sq = dg_src(reinterpret_cast<const double*>(b.Q), 1, 2 * N, N, 128, 2, 2ll * N, b.iq, b.eq);
    sq.rpad = qpad; sq.nblk = wn; sq.bstride = 2ll * N * N;
    DgRows pair{};
    dg_rows_add(pair, sq, wn * (qpad / 8));
    DgSrc s2 = dg_src(reinterpret_cast<const double*>(b.gl), 1, 2 * G * n, N, kDgP, 2ll * N, 2, b.igl, b.egl);
    s2.rpad = glpad; s2.nblk = wn; s2.bstride = 2ll * n * G * N;
    dg_rows_add(pair, s2, wn * (glpad / 8));
    TROT_TRY(dg_rows_launch(pair, st));
    DgArgs q{};
    q.imgA = b.igl; q.exA = b.egl; q.imgB = b.iq; q.exB = b.eq;
    q.M = G * n; q.ntile = glpad / kDgP; q.Nn = 2 * N; q.nrt = q.bB = qpad / 128; q.nbatch = wn;
    q.nk16 = (N + 15) / 16; q.shift = 1; q.salpha = 1; q.status = s.status;
    q.C = c.xg + (size_t)w0 * G * n * v; q.ldc = v; q.cstride = (long long)G * n * v;
    q.C2 = b.F3; q.ldc2 = n; q.cstride2 = (long long)G * nn; q.psplit = v;
    q.perm = G; q.permn = n;
    TROT_TRY(dg_gemm<true>(q, st));
    cisd_pairs_kernel<<<dim3(nchunk, wn), 128, smem, st>>>(n, G, gsub, nchunk, b.F1, b.F2, b.F3,
                                                           c.ci1g1 + (size_t)w0 * nn, c.gpart + (size_t)w0 * nchunk * 4);
    TROT_CHECK_LAUNCH("cisd_pairs_kernel");
  }
  return TROT_OK;
}

struct ClgBuffers {
  uint16_t *irow, *ilc, *ig;
  int16_t *erow, *elc, *eg;
  double2 *F1, *F2;
};
static size_t clg_carve(ClgBuffers& b, size_t W, size_t N, size_t n, size_t G, void* base) {
  char* p0 = reinterpret_cast<char*>(((uintptr_t)base + 255) & ~(uintptr_t)255);
  char* p = p0;
  auto take = [&](size_t k) {
    char* r = p;
    p += (k + 255) & ~(size_t)255;
    return r;
  };
  const size_t rb = kDgRowBytes((N + 15) / 16), row = adj_rows(G * n, 128), g = adj_rows(2 * W * n, kDgP);
  b.irow = (uint16_t*)take(row * rb); b.ilc = (uint16_t*)take(row * rb); b.ig = (uint16_t*)take(g * rb);
  b.erow = (int16_t*)take(row * 2); b.elc = (int16_t*)take(row * 2); b.eg = (int16_t*)take(g * 2);
  b.F1 = (double2*)take(W * n * n * G * sizeof(double2));
  b.F2 = (double2*)take(W * n * n * G * sizeof(double2));
  return (size_t)(p - p0) + 256;
}

size_t cisd_lg_dg_bytes(size_t W, size_t N, size_t n, size_t G) {
  ClgBuffers b;
  return clg_carve(b, W, N, n, G, nullptr);
}

// digits of the rows p < n of every L_g and of the columns of every lci1_g
static void cisd_lg_rows(DgRows& rows, const CisdGammaArgs& c, uint16_t* irow, int16_t* erow, uint16_t* ilc,
                         int16_t* elc) {
  const int N = c.N, n = c.n, G = c.G, groups = (int)(adj_rows((size_t)G * n, 128) / 8);
  DgSrc sr = dg_src(c.chol, 0, n, N, 128, N, 1, irow, erow);
  sr.rpad = n; sr.nblk = G; sr.bstride = (long long)N * N;
  dg_rows_add(rows, sr, groups);
  DgSrc sl = dg_src(c.lci1, 0, n, N, 128, 1, n, ilc, elc);
  sl.rpad = n; sl.nblk = G; sl.bstride = (long long)N * n;
  dg_rows_add(rows, sl, groups);
}

int launch_cisd_lg_dg(const CisdGammaArgs& c, const DgScratch& s, double2** F1, double2** F2, cudaStream_t st) {
  const int W = c.W, N = c.N, n = c.n, G = c.G;
  ClgBuffers b;
  if (s.bytes < clg_carve(b, W, N, n, G, s.p)) { set_error("CISD terms: scratch %zu", s.bytes); return TROT_ERR_WORKSPACE_TOO_SMALL; }
  DgRows rows{};
  cisd_lg_rows(rows, c, b.irow, b.erow, b.ilc, b.elc);
  const int tiles = (2 * W * n + kDgP - 1) / kDgP;
  dg_rows_add(rows, dg_src(reinterpret_cast<const double*>(c.green), 1, 2 * W * n, N, kDgP, 2ll * N, 2, b.ig, b.eg),
              tiles * 4);
  TROT_TRY(dg_rows_launch(rows, st));
  DgArgs a{};
  a.imgA = b.ig; a.exA = b.eg; a.M = W * n; a.ntile = tiles; a.nbatch = 1;
  a.nk16 = (N + 15) / 16; a.shift = 1; a.salpha = 1; a.status = s.status;
  a.imgB = b.irow; a.exB = b.erow; a.Nn = G * n; a.nrt = (G * n + 127) / 128; a.C = b.F1; a.ldc = (long long)G * n;
  TROT_TRY(dg_gemm<false>(a, st));
  a.imgB = b.ilc; a.exB = b.elc; a.C = b.F2;
  TROT_TRY(dg_gemm<false>(a, st));
  *F1 = b.F1;
  *F2 = b.F2;
  return TROT_OK;
}

}  // namespace trot

extern "C" size_t trot_zgemm_digits_workspace(int M, int N, int K) {
  return M > 0 && N > 0 && K > 0 ? trot::dg_scratch_bytes(M, N, K) + 512 : 0;
}

extern "C" int trot_zgemm_digits(int M, int N, int K, double alpha, const double* A, int lda, const double* B, int ldb,
                                 int b_is_nk, double* C, int ldc, int accumulate, void* ws, size_t ws_bytes,
                                 void* stream) {
  using namespace trot;
  if (!A || !B || !C || !ws) { set_error("null digit product buffer"); return TROT_ERR_NULL_PTR; }
  if (M <= 0 || N <= 0 || K <= 0 || lda < K || ldc < N || ldb < (b_is_nk ? K : N)) {
    set_error("zgemm_digits: bad sizes M=%d N=%d K=%d lda=%d ldb=%d ldc=%d", M, N, K, lda, ldb, ldc);
    return TROT_ERR_BAD_SHAPE;
  }
  Carver c(ws, ws_bytes);
  DgScratch s;
  s.bytes = dg_scratch_bytes(M, N, K);
  s.p = c.take<char>(s.bytes);
  s.status = c.status();
  if (!c.ok) { set_error("workspace too small: %zu < %zu", ws_bytes, c.used); return TROT_ERR_WORKSPACE_TOO_SMALL; }
  const cudaError_t e = cudaMemsetAsync(s.status, 0, sizeof(int), (cudaStream_t)stream);
  if (e != cudaSuccess) return cuda_status(e, "trot_zgemm_digits memset");
  return launch_zgemm_dg(M, N, K, alpha, (const double2*)A, lda, B, ldb, b_is_nk != 0, (double2*)C, ldc,
                         accumulate != 0, s, (cudaStream_t)stream);
}
