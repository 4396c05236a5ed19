// Walker QR orthonormalisation and stochastic reconfiguration (FP64).
#include <algorithm>

#include "ff.cuh"
#include "kernels.h"

namespace trot {

// x 2^k for a normal x whose exponent stays at or below that of 1 (results below 2^-1022 become 0)
TROT_D double qr_scale(double x, int k) {
  const int hi = __double2hiint(x), e = (hi >> 20) & 0x7FF;
  return (e == 0 || e + k <= 0) ? 0.0 : __hiloint2double(hi + k * (1 << 20), __double2loint(x));
}


// ------------------------------------------------------------------ QR
// Reduced QR of one walker spin block (N x n) with diag(R) real non-negative (trot/walkers.py:137-148): the matrix the
// phase-fixed Householder QR returns.  One CTA per walker, both spins in turn.
//
// Two Cholesky factorisations instead of Gram-Schmidt, whose dot products of one column at a time spend as much on
// reductions and barriers as on products:
//   1. w = v D (D: the columns' power-of-two scales), S = v^H v in float-float on the FP32 pipe (about 2^-44),
//      S = R1^H R1, R1^-1 in FP64 by one warp;
//   2. Q1 = v R1^-1 in FP64: Q1^H Q1 = I + E with E the float-float error (about 1e-13);
//   3. E by the FP64 Gram matrix of Q1; R2 = I + X, X = upper(E) with half its diagonal (X^H X is below 1e-19), and
//      Q = Q1 - Q1 X, whose correction needs only FP32;  diag(R) = (1 + X_jj) R1_jj D_jj.
// FP64 work: 4 N n^2 FMAs (products 2 and 3) against 8 N n^2 of twice-iterated Gram-Schmidt; that pipe bounds it (88 %
// busy): 0.39 ms for 1024 walkers of 120 x (12 + 10), Gram-Schmidt with a CTA per spin 1.31 ms.
// A walker whose columns are too close to dependent for step 1 (a pivot below 1e-4 of its column, E above 2e-10) or not
// finite takes twice-iterated classical Gram-Schmidt, as do all where the two n x n matrices do not fit beside the walker
// (gs_only).
// A thread per row, 128 at least (fewer rows leave the dot products and pairs to more warps) and 256 at most: 135 rows on 128
// threads were two rounds of every column.
static int qr_threads(int N) { return std::min(256, std::max(128, (N + 31) / 32 * 32)); }

// Twice-iterated classical Gram-Schmidt in shared memory (row stride ld); returns prod ||v||.  Bound by its FP64
// instructions and the waits between them: four fused multiply-adds per complex product and five additions per dot product
// (six and ten before) pay for the first pass of a walker that ends here: condition 1e6, 1024 walkers of 120 x (12 + 10) 1290
// -> 875 us, of 160 x (24 + 24) 6958 -> 4239.  Out of line, so that its registers are not the fast route's.
static __device__ __noinline__ double qr_gram_schmidt(int N, int n, int ld, double2* Q, double2* coef, double2* red) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, wid = tid >> 5, nw = nt >> 5;
  double prod = 1.0;
  for (int j = 0; j < n; ++j) {
    for (int pass = 0; pass < 2; ++pass) {
      // coef[i] = -<Q_i, v> for i < j  (one warp per i)
      for (int i = wid; i < j; i += nw) {
        double2 acc = cmk(0.0, 0.0);
        for (int p = lane; p < N; p += 32) {
          const double2 q = Q[p * ld + i], v = Q[p * ld + j];
          cfma(acc, cmk(q.x, -q.y), v);
        }
        // a half warp per component after the first exchange
        const bool im = lane & 16;
        double a = (im ? acc.y : acc.x) + __shfl_xor_sync(0xffffffffu, im ? acc.x : acc.y, 16);
#pragma unroll
        for (int o = 8; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
        if ((lane & 15) == 0) (im ? coef[i].y : coef[i].x) = -a;
      }
      __syncthreads();
      for (int p = tid; p < N; p += nt) {
        double2 v = Q[p * ld + j];
        for (int i = 0; i < j; ++i) cfma(v, Q[p * ld + i], coef[i]);
        Q[p * ld + j] = v;
      }
      __syncthreads();
    }
    double2 nn = cmk(0.0, 0.0);
    for (int p = tid; p < N; p += nt) nn.x += cabs2(Q[p * ld + j]);
    nn = block_sum2(nn, red);
    const double nrm = sqrt(nn.x);
    prod *= nrm;
    const double inv = 1.0 / nrm;
    for (int p = tid; p < N; p += nt) Q[p * ld + j] = cscale(Q[p * ld + j], inv);
    __syncthreads();
  }
  return prod;
}

// Cholesky S = R^H R of the Hermitian n x n S (its upper triangle is read) and X = R^-1 (upper) by one warp; rdiag[j] (1 +
// rcorr[j].x) = 1 / X_jj, the R_jj that belongs to v X (d rsqrt(d) alone is off by twice the error of rsqrt(d), which the
// norm's product collects over the columns: 1.07e-15 RMS at n = 12).  Returns false (in every lane) where a pivot is not
// above 1e-4 S_jj.
__device__ bool warp_cholesky_inverse(double2* S, double2* X, int n, double* rdiag, double2* rcorr) {
  const int lane = threadIdx.x & 31;
  bool ok = true;
  for (int k = 0; k < n; ++k) {
    // row k of R: the pivot's square root and reciprocal by one lane (FP64 divisions are slow)
    double rk = 0.0;
    if (lane == 0) {
      const double d = S[k * n + k].x;
      ok = d > 1e-4 * rdiag[k];  // rdiag[k] holds S_kk until the pivot is known
      rk = rsqrt(d);
      const double r = d * rk;
      S[k * n + k] = cmk(r, 0.0);
      rdiag[k] = r;
      rcorr[k].x = fma(-r, rk, 1.0);
    }
    ok = __shfl_sync(0xffffffffu, ok, 0);
    if (!ok) return false;
    rk = __shfl_sync(0xffffffffu, rk, 0);
    for (int j = k + 1 + lane; j < n; j += 32) S[k * n + j] = cscale(S[k * n + j], rk);
    __syncwarp();
    const int m = n - k - 1;
    for (int e = lane; e < m * m; e += 32) {  // S[i][j] -= conj(R[k][i]) R[k][j], i <= j
      const int i = k + 1 + e / m, j = k + 1 + e % m;
      if (j < i) continue;
      const double2 a = S[k * n + i];
      S[i * n + j] = csub(S[i * n + j], cmul(cmk(a.x, -a.y), S[k * n + j]));
    }
    if (lane == 0) X[k * n + k] = cmk(rk, 0.0);
    __syncwarp();
  }
  // column j of R^-1 by lane j (mod 32): x_i = -(sum_{i < k <= j} R[i][k] x_k) / R_ii
  for (int j = lane; j < n; j += 32)
    for (int i = j - 1; i >= 0; --i) {
      double2 acc = cmk(0.0, 0.0);
      for (int k = i + 1; k <= j; ++k) cfma(acc, S[i * n + k], X[k * n + j]);
      X[i * n + j] = cscale(acc, -X[i * n + i].x);
    }
  __syncwarp();
  return true;
}

// x truncated to a float, and back, by integer operations (below the normal range: 0; x finite and below 2^127).  The
// general conversions carry an FP64-pipe instruction for their special cases, which is issued even when predicated off.
TROT_D float qr_f32(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), t = (hi & 0x7FFFFFFFu) - (896u << 20);
  const unsigned f = (t << 3) | ((unsigned)__double2loint(x) >> 29);
  return __uint_as_float(t - (1u << 20) < (253u << 20) ? f | (hi & 0x80000000u) : 0u);
}
TROT_D double qr_f64(float x) {
  const unsigned v = __float_as_uint(x), t = v & 0x7FFFFFFFu;
  return t < 0x00800000u ? 0.0 : __hiloint2double((int)((v & 0x80000000u) | ((t >> 3) + (896u << 20))), (int)(t << 29));
}

// (i, j) of the e-th pair i <= j < n, row-major
TROT_D void qr_pair(int e, int n, int& i, int& j) {
  i = 0;
  while (e >= n - i) {
    e -= n - i;
    ++i;
  }
  j = i + e;
}

__global__ void __launch_bounds__(256)
qr_kernel(Spins sp, int N, double2* __restrict__ wa, double2* __restrict__ wb, double2* __restrict__ norm, int write_q,
          int gs_only) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ double2 red[32];
  __shared__ double2 coef[64];
  __shared__ double rdiag[64];
  __shared__ int cexp[64], bad;
  const int b = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
  const int quad = tid >> 2, part = tid & 3, nq = nt >> 2;    // four lanes per pair (float-float)
  const int oct = tid >> 3, opart = tid & 7, no = nt >> 3;    // eight (FP64: fewer idle lanes in the last round)
  double prod_all = 1.0;
  for (int s = 0; s < sp.nspin; ++s) {
    const int n = s ? sp.n[1] : sp.n[0], ld = gs_only ? n : n | 1, np = n * (n + 1) / 2;
    double2* Q = reinterpret_cast<double2*>(smem_raw);  // N x ld, first as float-float
    ffc* Vf = reinterpret_cast<ffc*>(smem_raw);
    double2* S = Q + (size_t)N * ld;                     // n x n
    double2* X = S + n * n;                              // n x n: R1^-1, then X
    double2* gw = (s ? wb : wa) + (size_t)b * N * n;
    __syncthreads();
    if (tid == 0) bad = gs_only;
    for (int j = tid; j < n; j += nt) cexp[j] = 0;
    __syncthreads();
    // columns' largest exponents
    for (int e = gs_only ? N * n : tid; e < N * n; e += nt) {
      const double2 x = gw[e];
      const unsigned hx = (unsigned)__double2hiint(x.x) & 0x7FFFFFFFu, hy = (unsigned)__double2hiint(x.y) & 0x7FFFFFFFu;
      atomicMax(&cexp[e % n], (int)(max(hx, hy) >> 20));
    }
    __syncthreads();
    for (int j = tid; j < n; j += nt)
      if (cexp[j] == 0 || cexp[j] == 0x7FF) bad = 1;  // a zero or non-finite column
    for (int e = gs_only ? N * n : tid; e < N * n; e += nt) {
      const double2 x = gw[e];
      const int k = 1023 - cexp[e % n];
      Vf[(e / n) * ld + e % n] = ffc{ff_from_d(qr_scale(x.x, k)), ff_from_d(qr_scale(x.y, k))};
    }
    __syncthreads();
    if (!bad) {
      // S[i][j] = sum_p conj(v[p][i]) v[p][j], four lanes per pair
      for (int e0 = 0; e0 < np; e0 += nq) {
        const int e = e0 + quad;
        ff re{0.f, 0.f}, im{0.f, 0.f};
        int i = 0, j = 0;
        if (e < np) {
          qr_pair(e, n, i, j);
          for (int p = part; p < N; p += 4) {
            const ffc x = Vf[p * ld + i], y = Vf[p * ld + j];
            ff_mad(re, x.re, y.re);
            ff_mad(re, x.im, y.im);
            ff_mad(im, x.re, y.im);
            ff_mad(im, ff{-x.im.hi, -x.im.lo}, y.re);
          }
          re = ff_fast(re.hi, re.lo);
          im = ff_fast(im.hi, im.lo);
        }
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
          re = ff_add(re, ff_shfl_xor(re, o));
          im = ff_add(im, ff_shfl_xor(im, o));
        }
        if (e < np && part == 0) {
          S[i * n + j] = cmk(ff_d(re), i == j ? 0.0 : ff_d(im));
          if (i == j) rdiag[i] = ff_d(re);
        }
      }
      __syncthreads();
      if (tid < 32) {
        const bool ok = warp_cholesky_inverse(S, X, n, rdiag, coef);
        if (tid == 0 && !ok) bad = 1;
      }
      __syncthreads();
    }
    if (!bad) {
      // Q1 = v R1^-1: a thread per row, columns from the last (row p is its own)
      for (int p = tid; p < N; p += nt) {
        double2* row = Q + (size_t)p * ld;
        const double2* src = gw + (size_t)p * n;
        for (int j = 0; j < n; ++j) {
          const double2 x = src[j];
          row[j] = cmk(qr_scale(x.x, 1023 - cexp[j]), qr_scale(x.y, 1023 - cexp[j]));
        }
        for (int j = n - 1; j >= 0; --j) {
          double2 acc = cmk(0.0, 0.0);
          for (int i = 0; i <= j; ++i) cfma(acc, row[i], X[i * n + j]);
          row[j] = acc;
        }
      }
      __syncthreads();
      // X = upper(Q1^H Q1 - I), half its diagonal; in FP32 over the dead S
      float2* Xf = reinterpret_cast<float2*>(S);
      for (int e0 = 0; e0 < np; e0 += no) {
        const int e = e0 + oct;
        double2 acc = cmk(0.0, 0.0);
        int i = 0, j = 0;
        if (e < np) {
          qr_pair(e, n, i, j);
          if (i == j) acc.x = -0.125;  // the eight lanes' shares of - I: the sums end near 0 and round little
          for (int p = opart; p < N; p += 8) {
            const double2 x = Q[p * ld + i];
            cfma(acc, cmk(x.x, -x.y), Q[p * ld + j]);
          }
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) {
          acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
          acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
        }
        if (e < np && opart == 0) {
          if (i == j) {
            acc = cmk(0.5 * acc.x, 0.0);
            X[i * n + i] = acc;
          }
          const float2 xf = make_float2(qr_f32(acc.x), qr_f32(acc.y));
          Xf[i * n + j] = xf;
          if (!(fabsf(xf.x) + fabsf(xf.y) < 2e-10f) || !isfinite(acc.x + acc.y)) bad = 1;
        }
      }
      __syncthreads();
    }
    double prod = 1.0;
    if (!bad) {
      const float2* Xf = reinterpret_cast<const float2*>(S);
      for (int p = tid; p < N; p += nt) {
        double2* row = Q + (size_t)p * ld;
        for (int j = n - 1; j >= 0; --j) {
          float cr = 0.f, ci = 0.f;
          for (int i = 0; i <= j; ++i) {
            const double2 q = row[i];
            const float2 x = Xf[i * n + j];
            const float qr = qr_f32(q.x), qi = qr_f32(q.y);
            cr = fmaf(qr, x.x, fmaf(-qi, x.y, cr));
            ci = fmaf(qr, x.y, fmaf(qi, x.x, ci));
          }
          row[j] = csub(row[j], cmk(qr_f64(cr), qr_f64(ci)));
        }
      }
      if (tid == 0)
        for (int j = 0; j < n; ++j) prod *= ldexp(fma(rdiag[j], X[j * n + j].x + coef[j].x, rdiag[j]), cexp[j] - 1023);
      __syncthreads();
    } else {
      __syncthreads();
      for (int e = tid; e < N * n; e += nt) Q[(e / n) * ld + e % n] = gw[e];
      __syncthreads();
      prod = qr_gram_schmidt(N, n, ld, Q, coef, red);
    }
    if (write_q)
      for (int e = tid; e < N * n; e += nt) gw[e] = Q[(e / n) * ld + e % n];
    prod_all *= sp.mult[s] == 2 ? prod * prod : prod;
  }
  // prod_j R_jj of both spins (restricted walkers: squared)
  if (tid == 0 && norm) norm[b] = cmk(prod_all, 0.0);
}

int launch_qr(const Spins& sp, int W, int N, double2* wa, double2* wb, double2* norm_out, cudaStream_t st,
              bool write_q) {
  int nmax = sp.n[0] > sp.n[1] ? sp.n[0] : sp.n[1];
  if (nmax > 64) {
    set_error("qr: nocc %d > 64 unsupported", nmax);
    return TROT_ERR_UNSUPPORTED;
  }
  if ((size_t)N * nmax * sizeof(double2) > 200 * 1024) {
    set_error("qr: walker tile of %zu bytes exceeds shared memory", (size_t)N * nmax * sizeof(double2));
    return TROT_ERR_UNSUPPORTED;
  }
  size_t smem = ((size_t)N * (nmax | 1) + 2 * (size_t)nmax * nmax) * sizeof(double2);
  const bool gs_only = smem > 220 * 1024;
  if (gs_only) smem = (size_t)N * nmax * sizeof(double2);
  if (smem > 40 * 1024) cudaFuncSetAttribute(qr_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  qr_kernel<<<W, qr_threads(N), smem, st>>>(sp, N, wa, wb, norm_out, write_q ? 1 : 0, gs_only ? 1 : 0);
  TROT_CHECK_LAUNCH("qr_kernel");
  return TROT_OK;
}

// ------------------------------------------------------------------ SR
// Comb resampling (trot/walkers.py:249-293): cw = cumsum|w| (sequential, same
// order as numpy), z_k = cw[-1] (k + zeta) / W, idx_k = first i with cw[i] >= z_k.
// The sums are one chain of W dependent FP64 additions, which bounds the kernel; the weights come to it, and the sums
// go to the searches, through shared memory (4096 at a time), so that nothing else waits between two additions.
static constexpr int kSrTile = 4096;

__global__ void __launch_bounds__(1024)
sr_index_kernel(int W, const double* __restrict__ weights, const double* __restrict__ zeta_dev, double zeta,
                double* __restrict__ cw, long long* __restrict__ idx, double* __restrict__ weights_out) {
  __shared__ double c_s[kSrTile];
  if (zeta_dev) zeta = zeta_dev[0];
  double c = 0.0;  // thread 0's running sum
  for (int t0 = 0; t0 < W; t0 += kSrTile) {
    const int m = min(kSrTile, W - t0);
    __syncthreads();
    for (int i = threadIdx.x; i < m; i += blockDim.x) c_s[i] = fabs(weights[t0 + i]);
    __syncthreads();
    if (threadIdx.x == 0) {
      int i = 0;
      for (; i + 16 <= m; i += 16) {
        double v[16];
#pragma unroll
        for (int u = 0; u < 16; ++u) v[u] = c_s[i + u];
#pragma unroll
        for (int u = 0; u < 16; ++u) {
          c += v[u];
          c_s[i + u] = c;
        }
      }
      for (; i < m; ++i) {
        c += c_s[i];
        c_s[i] = c;
      }
    }
    __syncthreads();
    if (W > kSrTile)
      for (int i = threadIdx.x; i < m; i += blockDim.x) cw[t0 + i] = c_s[i];
  }
  __syncthreads();
  const double* cum = W > kSrTile ? cw : c_s;
  const double tot = cum[W - 1], per = tot / (double)W;
  for (int k = threadIdx.x; k < W; k += blockDim.x) {
    const double z = tot * ((double)k + zeta) / (double)W;
    int lo = 0, hi = W;  // first i in [0, W) with cw[i] >= z; W if none
    while (lo < hi) {
      int mid = (lo + hi) >> 1;
      if (cum[mid] < z) lo = mid + 1; else hi = mid;
    }
    idx[k] = lo < W ? lo : W - 1;
    weights_out[k] = per;
  }
}

__global__ void gather_kernel(int W, size_t per, const double2* __restrict__ in, double2* __restrict__ out,
                              const long long* __restrict__ idx) {
  const int k = blockIdx.y;
  const double2* src = in + (size_t)idx[k] * per;
  double2* dst = out + (size_t)k * per;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < per; e += (size_t)gridDim.x * blockDim.x)
    dst[e] = src[e];
}

int launch_sr(const Spins& sp, int W, int N, const double* weights, const double* zeta_dev, double zeta,
              const double2* ina,
              const double2* inb, double2* outa, double2* outb, double* weights_out, long long* idx,
              double* cw, cudaStream_t st) {
  sr_index_kernel<<<1, 1024, 0, st>>>(W, weights, zeta_dev, zeta, cw, idx, weights_out);
  TROT_CHECK_LAUNCH("sr_index_kernel");
  for (int s = 0; s < sp.nspin; ++s) {
    size_t per = (size_t)N * sp.n[s];
    int gx = (int)((per + 255) / 256);
    if (gx > 8) gx = 8;
    dim3 grid(gx, W);
    gather_kernel<<<grid, 256, 0, st>>>(W, per, s == 0 ? ina : inb, s == 0 ? outa : outb, idx);
    TROT_CHECK_LAUNCH("gather_kernel");
  }
  return TROT_OK;
}

// ------------------------------------------------------------------ block energy
// Block tail of trot/prop/blocks.py:236-257 on the device: E = Re(E_L); walkers
// with non-finite E get weight 0; E is clamped to e_ref when |E - e_ref| >
// sqrt(2/dt); e_block = sum w E / sum w (e_ref if sum w == 0);
// e_estimate <- (1 - ema) e_estimate + ema e_block.  obs = [e_block, sum w].  Energies of a call that timed out
// (timeout_nan): weights, e_estimate and obs become NaN too.
__global__ void __launch_bounds__(1024)
block_energy_kernel(int W, const double2* __restrict__ energy, double* __restrict__ weights,
                    double* __restrict__ scalars, double dt, double ema, double* __restrict__ obs) {
  __shared__ double2 red[32];
  const double e_ref = scalars[1];
  const double thresh = sqrt(2.0 / dt);
  double2 acc = cmk(0.0, 0.0);  // (sum w E, sum w)
  bool timed_out = false;
  for (int i = threadIdx.x; i < W; i += blockDim.x) {
    double e = energy[i].x;
    const bool bad = !isfinite(e);
    timed_out |= __double_as_longlong(e) == kTimeoutNan;
    if (bad || fabs(e - e_ref) > thresh) e = e_ref;
    double w = weights[i];
    if (bad) { w = 0.0; weights[i] = 0.0; }
    acc.x += w * e;
    acc.y += w;
  }
  if (__syncthreads_or(timed_out)) {  // the energies are no numbers (report_timeout): nor is the block
    for (int i = threadIdx.x; i < W; i += blockDim.x) weights[i] = timeout_nan();
    if (threadIdx.x == 0) scalars[1] = obs[0] = obs[1] = timeout_nan();
    return;
  }
  acc = block_sum2(acc, red);
  if (threadIdx.x == 0) {
    const double wsum = acc.y;
    const double eb = wsum == 0.0 ? e_ref : acc.x / wsum;
    scalars[1] = (1.0 - ema) * scalars[1] + ema * eb;
    obs[0] = eb;
    obs[1] = wsum;
  }
}

}  // namespace trot

extern "C" int trot_block_energy(int n_walkers, const double* energy, double* weights, double* scalars,
                                 double dt, double shift_ema, double* obs_out, void* stream) {
  using namespace trot;
  if (!energy || !weights || !scalars || !obs_out) { set_error("null block-energy buffer"); return TROT_ERR_NULL_PTR; }
  if (n_walkers <= 0 || !(dt > 0.0)) { set_error("bad block-energy arguments"); return TROT_ERR_BAD_SHAPE; }
  block_energy_kernel<<<1, 1024, 0, (cudaStream_t)stream>>>(n_walkers, (const double2*)energy, weights, scalars,
                                                            dt, shift_ema, obs_out);
  TROT_CHECK_LAUNCH("block_energy_kernel");
  return TROT_OK;
}
