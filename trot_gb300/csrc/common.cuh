// Shared device helpers for the trot_gb300 kernels.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>
#include "trot_gb300.h"

#define TROT_HD __host__ __device__ __forceinline__
#define TROT_D __device__ __forceinline__

// ---------------------------------------------------------------- device status words
// A workspace starts with int[4] status words: [0] the status of the current call
// (reset when the call begins), [3] a sticky copy that only trot_workspace_timeouts
// clears.  A tensor-core kernel whose bounded wait ran out records
// TROT_ERR_DEVICE_TIMEOUT in both, skips its outputs (digit products: makes them NaN)
// and returns; the kernels that combine its results then write NaN instead of numbers.
TROT_D void report_timeout(int* status) {
  atomicExch(status, (int)TROT_ERR_DEVICE_TIMEOUT);
  atomicExch(status + 3, (int)TROT_ERR_DEVICE_TIMEOUT);
}
// The NaN of those results.  A walker's own NaN energy costs it its weight and no more (block_energy_kernel); an energy
// with this one means that the whole call gave no numbers.
static constexpr long long kTimeoutNan = 0x7FF8000074696D65ll;
TROT_D double timeout_nan() { return __longlong_as_double(kTimeoutNan); }

// ---------------------------------------------------------------- complex (double2)
TROT_HD double2 cmk(double r, double i) { return make_double2(r, i); }
TROT_HD double2 cadd(double2 a, double2 b) { return cmk(a.x + b.x, a.y + b.y); }
TROT_HD double2 csub(double2 a, double2 b) { return cmk(a.x - b.x, a.y - b.y); }
TROT_HD double2 cmul(double2 a, double2 b) { return cmk(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x); }
TROT_HD double2 cscale(double2 a, double s) { return cmk(a.x * s, a.y * s); }
// a += b * c (complex)
TROT_HD void cfma(double2& a, double2 b, double2 c) {
  a.x = fma(b.x, c.x, a.x);
  a.x = fma(-b.y, c.y, a.x);
  a.y = fma(b.x, c.y, a.y);
  a.y = fma(b.y, c.x, a.y);
}
// a += s * c (real times complex)
TROT_HD void crfma(double2& a, double s, double2 c) {
  a.x = fma(s, c.x, a.x);
  a.y = fma(s, c.y, a.y);
}
TROT_HD double cabs2(double2 a) { return a.x * a.x + a.y * a.y; }
// complex division a / b, scaled to avoid overflow (Smith's method)
TROT_HD double2 cdiv(double2 a, double2 b) {
  if (fabs(b.x) >= fabs(b.y)) {
    double r = b.y / b.x, d = b.x + b.y * r;
    return cmk((a.x + a.y * r) / d, (a.y - a.x * r) / d);
  } else {
    double r = b.x / b.y, d = b.y + b.x * r;
    return cmk((a.x * r + a.y) / d, (a.y * r - a.x) / d);
  }
}
TROT_HD double2 cexp(double2 a) {
  double s, c;
  sincos(a.y, &s, &c);
  double e = exp(a.x);
  return cmk(e * c, e * s);
}

// ---------------------------------------------------------------- reductions
TROT_D double warp_sum(double v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Block-wide sum in a fixed order (deterministic).  `red` holds >= 32 double2.  The halves of a warp take one component
// each after the first exchange: 5 + 3 dependent FP64 additions for 256 threads instead of 20, at about 60 cycles each.
TROT_D double2 block_sum2(double2 v, double2* red) {
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  const bool im = lane & 16;
  double a = (im ? v.y : v.x) + __shfl_xor_sync(0xffffffffu, im ? v.x : v.y, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
  double* rd = reinterpret_cast<double*>(red) + (im ? 1 : 0);
  __syncthreads();
  if ((lane & 15) == 0) rd[2 * wid] = a;
  __syncthreads();
  if (nw > 1) {
    if (wid == 0) {
      const int k = lane & 15;
      a = k < nw ? rd[2 * k] : 0.0;
      if (nw > 16) a += k + 16 < nw ? rd[2 * (k + 16)] : 0.0;
#pragma unroll 1
      for (int o = 8; o > 0; o >>= 1)
        if (nw > o) a += __shfl_xor_sync(0xffffffffu, a, o);
      __syncwarp();
      if (k == 0) rd[0] = a;
    }
    __syncthreads();
  }
  const double2 t = red[0];
  __syncthreads();
  return t;
}

// Sums of eight doubles over a block of 256 threads, into out[0..7] (shared, visible to all on return; red: 64 doubles).
// Each step of the exchange halves the values a lane carries: 9 additions a warp instead of 40.
TROT_D void block_sum8(double (&v)[8], double* red, double* out) {
  const int t = threadIdx.x, l = t & 31;
#pragma unroll
  for (int o = 16, n = 4; n >= 1; o >>= 1, n >>= 1)
#pragma unroll
    for (int i = 0; i < n; ++i) {
      const double keep = (l & o) ? v[i + n] : v[i], give = (l & o) ? v[i] : v[i + n];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 2);
  v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
  if ((l & 3) == 0) red[(t >> 5) * 8 + (l >> 2)] = v[0];  // lane l holds value l >> 2
  __syncthreads();
  if (t < 32) {
    double s = red[t] + red[t + 32];
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    s += __shfl_xor_sync(0xffffffffu, s, 16);
    if (t < 8) out[t] = s;
  }
  __syncthreads();
}

// ---------------------------------------------------------------- spin layout
// Per-system spin description used by every kernel: up to two spins; a
// restricted walker has one spin with multiplicity 2.
struct Spins {
  int nspin;        // 1 (restricted) or 2
  int n[2];         // columns per spin
  int mult[2];      // 2 for restricted, 1 otherwise
  int off[2];       // offset of spin s in the concatenated (n_a + n_b) column space
  int ntot;         // n[0] + n[1] (concatenated columns)
  const double* mo[2];
  const double* rot_h1[2];
  const double* rot_chol[2];
};

// Small complex matrices A (n x n <= kGjMax, row stride n) in shared memory, partial pivoting (the first largest
// |A[i][k]| wins, by integer reductions of the squares' words: five shuffles of FP64 comparisons took longer than the
// elimination).  Threads 0..127 of the block call gauss_jordan, which returns det(A) to thread 0.  With `inverse`, A is
// overwritten by its inverse (in-place Gauss-Jordan: each pivot step updates the n x n array once, half the work of
// eliminating [A | I]; the row interchanges are undone as column interchanges at the end); without it, A holds its LU
// factors.  Each quarter of an SM has an FP64 pipe of its own that takes an instruction of a warp every 64 cycles (72
// for a dependent one, 405 for a division), so a pivot costs one warp about 2 divisions + 6 n^2 / 32 instructions in a
// row.  The inverse (and the factors from kGjQuadLu on) updates on four warps and the serial part of a pivot (search,
// interchange, reciprocal) moves from warp to warp (quad_gauss_jordan); smaller factors stay in one warp without
// barriers (warp_lu).  FP64 instructions that are predicated off take the pipe as well: the loops are not unrolled.
// Cycles per pivot, one block: inverse, n = 5 / 12 / 16: 4850 / 7940 / 10070 (one warp, divisions) -> 2870 / 3320 /
// 3420; factors, n = 5 / 12 / 16: 3190 / 3900 / 4570 -> 2360 / 2980 / 3580 (one warp), 2470 / 2650 / 2820 (four); with
// the SMs full of blocks one warp stays ahead up to n = 13 (N = 120, n = 12, W = 1024: 95 against 97 us).
// float-float Green's functions, N = 97, n = 12, W = 128: 65 -> 39 us.
static constexpr int kGjMax = 64, kGjQuadLu = 14;
struct GjScratch {
  double2 rp, piv, det, col[kGjMax];
  int perm[kGjMax];
};
// e / m for e < m^2 <= kGjMax^2 by a product (an integer division takes as long as two FP64 instructions)
TROT_D unsigned gj_magic(int m) { return m > 0 ? ((1u << 20) + m - 1) / m : 0u; }
TROT_D int gj_div(int e, unsigned magic) { return (int)(((unsigned)e * magic) >> 20); }
// 1/u for 2^-300 <= |u| <= 2^300 to about 2^-46: an FP32 reciprocal of the leading 24 bits of the mantissa, one
// second-order Newton step in FP32 over all its 53 bits, joined as a fixed-point number
TROT_D double gj_seed(double u) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(u), m = b & 0xFFFFFFFFFFFFFull;
  const float h = __int_as_float(0x3F800000 | (int)(m >> 29));
  const float l = __fmul_rn(__uint2float_rn((unsigned)m & 0x1FFFFFFFu), 0x1p-52f);
  const float r = __fdividef(1.0f, h);
  const float e = fmaf(-r, l, fmaf(-r, h, 1.0f));
  const int lo = __float2int_rn(__fmul_rn(__fmul_rn(r, fmaf(e, e, e)), 0x1p53f));
  const long long f = ((long long)__float2int_rn(__fmul_rn(r, 0x1p24f)) << 29) + lo;  // 2^53 / mantissa
  const long long ex = (long long)((b >> 52) & 0x7FF) - 1023;
  return __longlong_as_double((long long)(b & 0x8000000000000000ull) | (f + ((1021ll - ex) << 52)));
}
// a / u from that: Markstein's correction by the residual, the rounded quotient but for about one case in 2^39
TROT_D double gj_div_by(double a, double u, double ru) {
  const double q = a * ru;
  return fma(fma(-q, u, a), ru, q);
}
static __device__ __noinline__ double2 gj_rcp_general(double2 p) { return cdiv(cmk(1.0, 0.0), p); }
// Re (part = 0) or Im (part = 1) of 1/p by Smith's two steps, every lane alike but for the last numerator.  (The
// division routine takes 600 to 750 cycles; three in a row were half of a pivot.)
TROT_D double gj_reciprocal(double2 p, int part) {
  const unsigned long long mx = (unsigned long long)__double_as_longlong(p.x) << 1,
                           my = (unsigned long long)__double_as_longlong(p.y) << 1;
  const bool c = mx >= my;  // |Re p| >= |Im p|
  const double u = c ? p.x : p.y, o = c ? p.y : p.x;
  const int eu = (int)((c ? mx : my) >> 53) - 1023, eo = (int)((c ? my : mx) >> 53) - 1023;
  if (eu > 300 || eu < -300 || (eo < -300 && (c ? my : mx) != 0)) {
    const double2 r = gj_rcp_general(p);
    return part ? r.y : r.x;
  }
  const double r = gj_div_by(o, u, gj_seed(u)), d = u + o * r;
  return gj_div_by(part ? (c ? -r : -1.0) : (c ? 1.0 : r), d, gj_seed(d));
}
TROT_D void gj_sync() { asm volatile("bar.sync 1, 128;" ::: "memory"); }
TROT_D double2 warp_lu(double2* A, int n) {
  const int lane = threadIdx.x & 31;
  double2 det = cmk(1.0, 0.0);
  for (int k = 0; k < n; ++k) {
    unsigned long long best = 0;  // bits of the square, with one added to the high word (0: no row)
    int bi = k;
#pragma unroll 1
    for (int i = k + lane; i < n; i += 32) {
      const unsigned long long a = (unsigned long long)__double_as_longlong(cabs2(A[i * n + k])) + (1ull << 32);
      if (a > best) { best = a; bi = i; }
    }
    const unsigned th = __reduce_max_sync(0xffffffffu, (unsigned)(best >> 32));
    const bool cand = (unsigned)(best >> 32) == th;
    const unsigned tl = __reduce_max_sync(0xffffffffu, cand ? (unsigned)best : 0u);
    bi = (int)__reduce_min_sync(0xffffffffu, cand && (unsigned)best == tl ? (unsigned)bi : 0x7fffffffu);
    if (bi != k) {
#pragma unroll 1
      for (int j = lane; j < n; j += 32) {
        const double2 t = A[k * n + j];
        A[k * n + j] = A[bi * n + j];
        A[bi * n + j] = t;
      }
      det = cmk(-det.x, -det.y);
    }
    __syncwarp();
    const double2 piv = A[k * n + k];
    const double v = k + 1 < n ? gj_reciprocal(piv, lane & 1) : 0.0;
    if (lane == 0) det = cmul(det, piv);
    const double2 rp = cmk(__shfl_sync(0xffffffffu, v, 0), __shfl_sync(0xffffffffu, v, 1));
#pragma unroll 1
    for (int i = k + 1 + lane; i < n; i += 32) A[i * n + k] = cmul(A[i * n + k], rp);
    __syncwarp();
    const int m = n - k - 1;
    const unsigned im = gj_magic(m);
#pragma unroll 1
    for (int e = lane; e < m * m; e += 32) {
      const int r = gj_div(e, im), i = k + 1 + r, j = k + 1 + e - r * m;
      A[i * n + j] = csub(A[i * n + j], cmul(A[i * n + k], A[k * n + j]));
    }
    __syncwarp();
  }
  return det;
}

TROT_D double2 quad_gauss_jordan(double2* A, int n, bool inverse, GjScratch& S, int turn) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const unsigned in = gj_magic(n);
  if (t == 0) S.det = cmk(1.0, 0.0);
  for (int k = 0; k < n; ++k) {
    const int role = (warp - k - turn) & 3;
    if (role == 0) {
      unsigned long long best = 0;  // bits of the square, with one added to the high word (0: no row)
      int bi = k;
#pragma unroll 1
      for (int i = k + lane; i < n; i += 32) {
        const unsigned long long a = (unsigned long long)__double_as_longlong(cabs2(A[i * n + k])) + (1ull << 32);
        if (a > best) { best = a; bi = i; }
      }
      const unsigned th = __reduce_max_sync(0xffffffffu, (unsigned)(best >> 32));
      const bool cand = (unsigned)(best >> 32) == th;
      const unsigned tl = __reduce_max_sync(0xffffffffu, cand ? (unsigned)best : 0u);
      bi = (int)__reduce_min_sync(0xffffffffu, cand && (unsigned)best == tl ? (unsigned)bi : 0x7fffffffu);
      const double2 p = A[bi * n + k];
      __syncwarp();
      if (bi != k) {
#pragma unroll 1
        for (int j = lane; j < n; j += 32) {
          const double2 x = A[k * n + j];
          A[k * n + j] = A[bi * n + j];
          A[bi * n + j] = x;
        }
      }
      if (lane == 0) {
        S.perm[k] = bi;
        S.piv = p;
      }
      if (inverse || k + 1 < n) {
        const double v = gj_reciprocal(p, lane & 1);
        if (lane < 2) (lane == 0 ? S.rp.x : S.rp.y) = v;
      }
    }
    gj_sync();
    if (role == 1) {
      const double2 rp = S.rp;
      if (inverse) {
#pragma unroll 1
        for (int j = lane; j < n; j += 32) {
          const double2 x = A[k * n + j];
          A[k * n + j] = j == k ? rp : cmk(fma(x.x, rp.x, -__dmul_rn(x.y, rp.y)), fma(x.x, rp.y, __dmul_rn(x.y, rp.x)));
        }
      } else {
#pragma unroll 1
        for (int i = k + 1 + lane; i < n; i += 32) A[i * n + k] = cmul(A[i * n + k], rp);
      }
    } else if (role == 2) {
      if (inverse)
#pragma unroll 1
        for (int i = lane; i < n; i += 32)
          if (i != k) S.col[i] = A[i * n + k];
    } else if (role == 3 && lane == 0) {
      const double2 d = S.det;
      S.det = cmul(S.perm[k] != k ? cmk(-d.x, -d.y) : d, S.piv);
    }
    gj_sync();
    // A[i][j] -= A[i][k] A[k][j] for i != k; in column k the old value counts as 0.  Which of two products is rounded
    // first is spelled out (and differs in column k): results that are rounded to FP32 later must not move.
    if (inverse) {
#pragma unroll 1
      for (int e = t; e < (n - 1) * n; e += 128) {
        int i = gj_div(e, in);
        const int j = e - i * n;
        i += i >= k;
        const bool pc = j == k;
        const double2 c = S.col[i], b = A[k * n + j], o = pc ? cmk(0.0, 0.0) : A[i * n + j];
        double x = fma(pc ? c.y : c.x, pc ? b.y : b.x, -__dmul_rn(pc ? c.x : c.y, pc ? b.x : b.y));
        if (pc) x = -x;
        A[i * n + j] = cmk(__dsub_rn(o.x, x), __dsub_rn(o.y, fma(c.y, b.x, __dmul_rn(c.x, b.y))));
      }
    } else {
      const int m = n - k - 1;
      const unsigned im = gj_magic(m);
#pragma unroll 1
      for (int e = t; e < m * m; e += 128) {
        const int r = gj_div(e, im), i = k + 1 + r, j = k + 1 + e - r * m;
        A[i * n + j] = csub(A[i * n + j], cmul(A[i * n + k], A[k * n + j]));
      }
    }
    gj_sync();
  }
  if (inverse) {
    if (t < n)
      for (int k = n - 1; k >= 0; --k) {
        const int p = S.perm[k];
        if (p != k) {
          const double2 x = A[t * n + k];
          A[t * n + k] = A[t * n + p];
          A[t * n + p] = x;
        }
      }
    gj_sync();
  }
  return S.det;
}

TROT_D double2 gauss_jordan(double2* A, int n, bool inverse, GjScratch& S, int turn) {
  if (inverse || n >= kGjQuadLu) return quad_gauss_jordan(A, n, inverse, S, turn);
  return threadIdx.x < 32 ? warp_lu(A, n) : cmk(0.0, 0.0);
}

// ---------------------------------------------------------------- errors
namespace trot {
void set_error(const char* fmt, ...);
int cuda_status(cudaError_t e, const char* where);
void prof_count_launch();  // profile.cu: counts launches while the timers are enabled
}  // namespace trot

#define TROT_CHECK_LAUNCH(where)                                      \
  do {                                                                \
    trot::prof_count_launch();                                        \
    cudaError_t _e = cudaGetLastError();                              \
    if (_e != cudaSuccess) return trot::cuda_status(_e, where);       \
  } while (0)
