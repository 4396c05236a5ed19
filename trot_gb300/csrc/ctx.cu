// One-time propagation and measurement constants on the device.
//
// Propagation context (trot/runtime_layout.py:125-197, the host twin of
// trot/prop/chol_afqmc_ops.py:103-127), with rho the spin-summed trial 1-RDM:
//   t_g        = sum_ij L_g[i][j] rho[j][i]          (mf_shifts = i t_g)
//   h0_prop    = -h0 - 1/2 sum_g mf_g^2 = -h0 + 1/2 sum_g t_g^2
//   h1_eff     = h1 - 1/2 sum_g L_g L_g + sum_g t_g L_g
//   exp_h1_half = expm(-dt/2 h1_eff)
// The matrix exponential is scaling and squaring of a degree-16 Taylor
// polynomial: s = the smallest power of two with ||A||_1 / 2^s <= 1/2, the
// Taylor sum of B = A / 2^s by Horner's rule (remainder < 0.5^17 / 17! ~ 2e-20
// relative), then s squarings, all in one cooperative kernel (s is chosen on the
// device, no host round trip).
//
// Half rotation (trot/runtime_layout.py:200-245; trot/meas/rhf.py:308-319):
//   rot_h1 = C^T h1 (n, N),  rot_chol[g] = C^T L_g (n, N)   for a real trial C (N, n).
// CISD (trot/runtime_layout.py:248-292; trot/meas/cisd.py:92-110):
//   lci1[g][i][p] = sum_t L_g[i][nocc + t] ci1[p][t]   (G, N, nocc).
#include <cooperative_groups.h>

#include <algorithm>

#include "digits.h"
#include "kernels.h"

namespace trot {

static constexpr int kCtxT = 32;        // output tile of the FP64 matrix products
static constexpr int kTaylorDeg = 16;
static constexpr int kMaxSquarings = 40;

struct CtxBuffers {
  int* status;   // [0] status, [1] number of squarings s
  double *a, *p0, *p1, *part;
};

static void ctx_slices(int N, int G, int& S, int& gper) {
  const int tiles = ((N + kCtxT - 1) / kCtxT) * ((N + kCtxT - 1) / kCtxT);
  S = (2 * 152 + tiles - 1) / tiles;
  if (S > G) S = G;
  if (S < 1) S = 1;
  gper = (G + S - 1) / S;
  S = (G + gper - 1) / gper;
}

static size_t carve_ctx(int N, int G, Carver& c, CtxBuffers& b) {
  int S, gper;
  ctx_slices(N, G, S, gper);
  const size_t nn = (size_t)N * N;
  b.status = c.status();  // 64 ints
  b.a = c.take<double>(nn);
  b.p0 = c.take<double>(nn);
  b.p1 = c.take<double>(nn);
  b.part = c.take<double>((size_t)S * nn);
  return c.used;
}

// t_g = sum_ij L_g[i][j] rho[j][i]; one block per g, fixed-order reduction
__global__ void ctx_mf_kernel(int N, const double* __restrict__ chol, const double* __restrict__ rho,
                              double* __restrict__ t) {
  __shared__ double2 red[32];
  const int g = blockIdx.x;
  const double* L = chol + (size_t)g * N * N;
  double acc = 0.0;
  for (int e = threadIdx.x; e < N * N; e += blockDim.x) {
    const int i = e / N, j = e - i * N;
    acc = fma(L[e], rho[(size_t)j * N + i], acc);
  }
  const double2 s = block_sum2(cmk(acc, 0.0), red);
  if (threadIdx.x == 0) t[g] = s.x;
}

// h0_prop = -h0 + 1/2 sum_g t_g^2
__global__ void ctx_h0_kernel(int G, double h0, const double* __restrict__ t, double* __restrict__ h0_prop) {
  __shared__ double2 red[32];
  double acc = 0.0;
  for (int g = threadIdx.x; g < G; g += blockDim.x) acc = fma(t[g], t[g], acc);
  const double2 s = block_sum2(cmk(acc, 0.0), red);
  if (threadIdx.x == 0) *h0_prop = -h0 + 0.5 * s.x;
}

// part[s][i][j] = sum_{g in slice s} (t_g L_g[i][j] - 1/2 sum_k L_g[i][k] L_g[k][j]);
// grid (j tiles, i tiles, slices), 256 threads: thread (ty, tx) owns rows ty + 8r of column tx.
__global__ void __launch_bounds__(256) ctx_v_partial_kernel(int N, int G, int gper, const double* __restrict__ chol,
                                                            const double* __restrict__ t, double* __restrict__ part) {
  __shared__ double As[kCtxT][kCtxT + 1], Bs[kCtxT][kCtxT + 1];
  const int j0 = blockIdx.x * kCtxT, i0 = blockIdx.y * kCtxT, sl = blockIdx.z;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  double quad[4] = {0.0, 0.0, 0.0, 0.0}, lin[4] = {0.0, 0.0, 0.0, 0.0};
  const int g0 = sl * gper, g1 = min(G, g0 + gper);
  for (int g = g0; g < g1; ++g) {
    const double* L = chol + (size_t)g * N * N;
    for (int k0 = 0; k0 < N; k0 += kCtxT) {
#pragma unroll
      for (int r = ty; r < kCtxT; r += 8) {
        const int i = i0 + r, k = k0 + tx, kk = k0 + r, j = j0 + tx;
        As[r][tx] = (i < N && k < N) ? L[(size_t)i * N + k] : 0.0;
        Bs[r][tx] = (kk < N && j < N) ? L[(size_t)kk * N + j] : 0.0;
      }
      __syncthreads();
#pragma unroll 8
      for (int k = 0; k < kCtxT; ++k) {
        const double bv = Bs[k][tx];
#pragma unroll
        for (int r = 0; r < 4; ++r) quad[r] = fma(As[ty + 8 * r][k], bv, quad[r]);
      }
      __syncthreads();
    }
    const double tg = t[g];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const int i = i0 + ty + 8 * r, j = j0 + tx;
      if (i < N && j < N) lin[r] = fma(tg, L[(size_t)i * N + j], lin[r]);
    }
  }
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int i = i0 + ty + 8 * r, j = j0 + tx;
    if (i < N && j < N) part[((size_t)sl * N + i) * N + j] = lin[r] - 0.5 * quad[r];
  }
}

// A = -dt/2 (h1 + sum_s part[s]) in slice order
__global__ void ctx_heff_kernel(int N, int S, double dt, const double* __restrict__ h1, const double* __restrict__ part,
                                double* __restrict__ A) {
  const size_t nn = (size_t)N * N;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < nn; e += (size_t)gridDim.x * blockDim.x) {
    double v = h1[e];
    for (int s = 0; s < S; ++s) v += part[(size_t)s * nn + e];
    A[e] = -0.5 * dt * v;
  }
}

// part[s][i][j] (+)= sum of t_g L_g[i][j] - 1/2 (L_g L_g)[i][j] over every S-th of the `count` vectors from s on, with
// the squares given as pairs of rows (launch_square_dg)
__global__ void ctx_v_sum_kernel(int N, int count, int add, const double* __restrict__ chol, const double* __restrict__ t,
                                 const double2* __restrict__ sq, double* __restrict__ part) {
  const size_t nn = (size_t)N * N, ld = (size_t)((N + 1) / 2) * N;
  const int S = gridDim.y, s = blockIdx.y;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < nn; e += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / N), j = (int)(e - (size_t)i * N);
    double v = add ? part[s * nn + e] : 0.0;
    const double* q = reinterpret_cast<const double*>(sq + (size_t)(i >> 1) * N + j) + (i & 1);
    for (int g = s; g < count; g += S) v = fma(t[g], chol[g * nn + e], fma(-0.5, q[2 * (size_t)g * ld], v));
    part[s * nn + e] = v;
  }
}

// out = expm(A).  One cooperative launch: the 16 Horner products and the squarings were 56 launches, most of them
// squarings past s that only returned, and a 32 x 32 tile per CTA left all but 9 to 25 SMs idle at N = 80 (1.54 ms of two
// exponentials of N = 80 and 2 N = 160, 0.36 ms like this; the 32 products and 5 squarings of FP64 0.15).  Tiles of 8 x 8, two halves of K: a CTA's four
// warps are one per FP64 pipe of its SM.  Products of other CTAs are read past L1.
// The sums are kept as R = T - I (R <- (B + B R) / k, R <- 2 R + R^2), rounded relative to R and not to I, which the
// squarings would amplify; I is added at the end.
static constexpr int kExpmK = 64;
// Z = (by X + X Y) scale (+ I)
__device__ __forceinline__ void expm_product(int n, const double* X, const double* Y, double scale, double by, bool last, double* Z) {
  __shared__ double As[8][kExpmK + 1], Bs[kExpmK][9], half[64];
  const int tid = threadIdx.x, h = tid >> 6, r = (tid & 63) >> 3, c = tid & 7, nt = (n + 7) / 8;
  for (int tile = blockIdx.x; tile < nt * nt; tile += gridDim.x) {
    const int i0 = tile / nt * 8, j0 = tile % nt * 8;
    double acc[2] = {0.0, 0.0}, xa[4], xb[4];
    auto fetch = [&](int k0) {
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int e = tid + q * 128, i = i0 + e / kExpmK, ka = k0 + e % kExpmK, kb = k0 + e / 8, j = j0 + e % 8;
        xa[q] = i < n && ka < n ? __ldcg(X + (size_t)i * n + ka) : 0.0;
        xb[q] = kb < n && j < n ? __ldcg(Y + (size_t)kb * n + j) : 0.0;
      }
    };
    fetch(0);
    for (int k0 = 0; k0 < n; k0 += kExpmK) {
      __syncthreads();
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int e = tid + q * 128;
        As[e / kExpmK][e % kExpmK] = xa[q];
        Bs[e / 8][e % 8] = xb[q];
      }
      __syncthreads();
      if (k0 + kExpmK < n) fetch(k0 + kExpmK);
#pragma unroll 8
      for (int k = h * (kExpmK / 2); k < (h + 1) * (kExpmK / 2); k += 2) {
        acc[0] = fma(As[r][k], Bs[k][c], acc[0]);
        acc[1] = fma(As[r][k + 1], Bs[k + 1][c], acc[1]);
      }
    }
    if (h) half[tid & 63] = acc[0] + acc[1];
    __syncthreads();
    const int i = i0 + r, j = j0 + c;
    if (!h && i < n && j < n)
      Z[(size_t)i * n + j] = fma(by, __ldcg(X + (size_t)i * n + j), acc[0] + acc[1] + half[tid]) * scale +
                             (last && i == j ? 1.0 : 0.0);
  }
}

__global__ void __launch_bounds__(128) ctx_expm_kernel(int n, const double* A, double* out, double* P0, double* P1,
                                                       int* status) {
  namespace cg = cooperative_groups;
  cg::grid_group grid = cg::this_grid();
  __shared__ unsigned long long top;
  const int tid = threadIdx.x, lane = tid & 31;
  // ||A||_1, the largest column sum (columns into P0): NaN and infinity are the largest words
  for (int j = blockIdx.x * 4 + (tid >> 5); j < n; j += gridDim.x * 4) {
    double s = 0.0;
    for (int i = lane; i < n; i += 32) s += fabs(A[(size_t)i * n + j]);
    s = warp_sum(s);
    if (lane == 0) P0[j] = s;
  }
  if (tid == 0) top = 0;
  grid.sync();
  unsigned long long m = 0;
  for (int j = tid; j < n; j += 128)
    m = max(m, (unsigned long long)__double_as_longlong(__ldcg(P0 + j)) & 0x7FFFFFFFFFFFFFFFull);
  atomicMax(&top, m);
  __syncthreads();
  double nrm = __longlong_as_double((long long)top);
  int s = 0;
  bool bad = !(nrm <= 1.7e308);
  if (!bad) {
    while (nrm > 0.5 && s < kMaxSquarings) { nrm *= 0.5; ++s; }
    bad = nrm > 0.5;
  }
  if (blockIdx.x == 0 && tid == 0) {
    if (bad && status[0] == TROT_OK) status[0] = TROT_ERR_NUMERIC_GUARD;  // (a timed-out product's NaN: its own status)
    status[1] = s;
  }
  grid.sync();
  // R <- (B + B R) / k for k = 16 .. 1 (the first with R = 0), B = A / 2^s
  const double b = ldexp(1.0, -s);
  const size_t nn = (size_t)n * n;
  for (size_t e = blockIdx.x * (size_t)128 + tid; e < nn; e += (size_t)gridDim.x * 128) P0[e] = A[e] * (b / kTaylorDeg);
  double *from = P0, *to = P1;
  for (int k = kTaylorDeg - 1; k >= 1 - s; --k) {  // k <= 0: squarings
    grid.sync();
    const bool last = k == 1 - s;
    double* z = last ? out : to;
    if (k >= 1) expm_product(n, A, from, b / k, 1.0, last, z);
    else expm_product(n, from, from, 1.0, 2.0, last, z);
    to = from;
    from = z;
  }
}

// out[g][p][j] = sum_i C[i][p] M_g[i][j] for p in [p0, p0 + 16): grid (G, ceil(n / 16)), 128 threads
// over j; C rows staged in shared memory 128 at a time.
__global__ void __launch_bounds__(128) ctx_rotate_kernel(int N, int n, const double* __restrict__ C,
                                                         const double* __restrict__ M, double* __restrict__ out) {
  __shared__ double Cs[128][16];
  const int g = blockIdx.x, p0 = blockIdx.y * 16;
  const int np = min(16, n - p0);
  const double* Mg = M + (size_t)g * N * N;
  double* og = out + (size_t)g * n * N;
  for (int jb = 0; jb < N; jb += 128) {
    const int j = jb + threadIdx.x;
    double acc[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) acc[q] = 0.0;
    for (int ib = 0; ib < N; ib += 128) {
      const int ni = min(128, N - ib);
      __syncthreads();
      for (int e = threadIdx.x; e < 128 * 16; e += 128) {
        const int r = e >> 4, q = e & 15;
        Cs[r][q] = (r < ni && q < np) ? C[(size_t)(ib + r) * n + p0 + q] : 0.0;
      }
      __syncthreads();
      if (j < N) {
        for (int r = 0; r < ni; ++r) {
          const double m = Mg[(size_t)(ib + r) * N + j];
#pragma unroll
          for (int q = 0; q < 16; ++q) acc[q] = fma(Cs[r][q], m, acc[q]);
        }
      }
    }
    if (j < N) {
#pragma unroll
      for (int q = 0; q < 16; ++q)
        if (q < np) og[(size_t)(p0 + q) * N + j] = acc[q];
    }
  }
}

// lci1[g][i][p] = sum_t L_g[i][nocc + t] ci1[p][t]; one block per g, threads over (i, p)
__global__ void ctx_lci1_kernel(int N, int nocc, const double* __restrict__ ci1, const double* __restrict__ chol,
                                double* __restrict__ lci1) {
  const int g = blockIdx.x, nv = N - nocc;
  const double* L = chol + (size_t)g * N * N;
  for (int e = threadIdx.x; e < N * nocc; e += blockDim.x) {
    const int i = e / nocc, p = e - i * nocc;
    double acc = 0.0;
    for (int t = 0; t < nv; ++t) acc = fma(L[(size_t)i * N + nocc + t], ci1[(size_t)p * nv + t], acc);
    lci1[((size_t)g * N + i) * nocc + p] = acc;
  }
}

// M (2N x 2N) = [[A^T, Gb], [0, A^T]]: expm(M)'s upper-right block is the
// adjoint of the Frechet derivative of expm at A applied to Gb (for the
// Frobenius inner product the adjoint of L(A, .) is L(A^T, .); Higham,
// "Functions of Matrices", 2008, Thm. 3.6 and sec. 3.2).
// The upper-right block is linear in Gb: it is scaled to max |Gb| = 1 (keeping
// ||M||_1 and so the number of squarings small) and scaled back on the way out.
__global__ void ctx_absmax_kernel(size_t n, const double* __restrict__ x, double* __restrict__ out) {
  __shared__ double red[256];
  double m = 0.0;
  for (size_t e = threadIdx.x; e < n; e += blockDim.x) m = fmax(m, fabs(x[e]));
  red[threadIdx.x] = m;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] = fmax(red[threadIdx.x], red[threadIdx.x + o]);
    __syncthreads();
  }
  if (threadIdx.x == 0) *out = red[0] > 0.0 ? red[0] : 1.0;
}

__global__ void ctx_frechet_build_kernel(int N, const double* __restrict__ A, const double* __restrict__ Gb,
                                         const double* __restrict__ gscale, double* __restrict__ M) {
  const int n2 = 2 * N;
  const double inv = 1.0 / *gscale;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < (size_t)n2 * n2;
       e += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / n2), j = (int)(e % n2);
    double v = 0.0;
    if (i < N && j < N) v = A[(size_t)j * N + i];
    else if (i < N) v = Gb[(size_t)i * N + (j - N)] * inv;
    else if (j >= N) v = A[(size_t)(j - N) * N + (i - N)];
    M[e] = v;
  }
}

// g_h1[i][j] += scale * gscale * E[i][N + j]
__global__ void ctx_frechet_take_kernel(int N, const double* __restrict__ E, double scale,
                                        const double* __restrict__ gscale, double* __restrict__ g) {
  const double sc = scale * *gscale;
  for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < (size_t)N * N;
       e += (size_t)gridDim.x * blockDim.x) {
    const int i = (int)(e / N), j = (int)(e % N);
    g[e] += sc * E[(size_t)i * 2 * N + N + j];
  }
}

// out = expm(A) for a real n x n matrix on the device; status[0] is set to
// TROT_ERR_NUMERIC_GUARD on a non-finite or huge norm, status[1] receives s.
// p0, p1: n x n scratch.  Used by the propagation context and its adjoint.
int launch_expm(int n, const double* A, double* out, double* p0, double* p1, int* status, cudaStream_t st) {
  int dev = 0, sms = 0, per = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, ctx_expm_kernel, 128, 0);
  const long long nt = (n + 7) / 8, tiles = nt * nt;
  const int grid = (int)std::min<long long>(tiles, (long long)sms * std::max(1, std::min(per, 4)));
  void* args[] = {&n, &A, &out, &p0, &p1, &status};
  const cudaError_t e = cudaLaunchCooperativeKernel((const void*)ctx_expm_kernel, dim3(grid), dim3(128), args, 0, st);
  if (e != cudaSuccess) return cuda_status(e, "ctx_expm_kernel");
  TROT_CHECK_LAUNCH("ctx_expm_kernel");
  return TROT_OK;
}

// Scratch of the squares' digit products, at the end of a workspace (none for sizes that keep the FP64 kernel, or where
// the rest of a caller's workspace is too small for it)
static DgScratch carve_squares(int N, int G, Carver& c, int* status) {
  DgScratch d;
  if (!dg_takes(N) || N > 1024) return d;
  const Carver before = c;
  const size_t bytes = square_dg_bytes(N, square_dg_count(N, G));
  d.p = c.take<char>(bytes);
  if (before.base && before.ok && !c.ok) {
    c = before;
    return DgScratch{};
  }
  d.bytes = bytes;
  d.status = status;
  return d;
}

// part[s] for S slices: sum_g t_g L_g - 1/2 L_g L_g.  400 vectors of 80 orbitals: 880 us with FP64 tiles, 110 us from the
// digit products.
static int launch_v(int N, int G, int S, int gper, const double* chol, const double* t, double* part, const DgScratch& d,
                    cudaStream_t st) {
  if (!d.p) {
    const int nt = (N + kCtxT - 1) / kCtxT;
    ctx_v_partial_kernel<<<dim3(nt, nt, S), 256, 0, st>>>(N, G, gper, chol, t, part);
    TROT_CHECK_LAUNCH("ctx_v_partial_kernel");
    return TROT_OK;
  }
  const int per = square_dg_count(N, G);
  const size_t nn = (size_t)N * N;
  for (int g = 0; g < G; g += per) {
    const int count = std::min(per, G - g);
    double2* sq = nullptr;
    TROT_TRY(launch_square_dg(N, count, chol + g * nn, d, &sq, st));
    ctx_v_sum_kernel<<<dim3((unsigned)((nn + 255) / 256), S), 256, 0, st>>>(N, count, g > 0, chol + g * nn, t + g, sq, part);
    TROT_CHECK_LAUNCH("ctx_v_sum_kernel");
  }
  return TROT_OK;
}

}  // namespace trot

using namespace trot;

extern "C" {

static size_t ctx_workspace(int norb, int nchol, bool digits) {
  if (norb < 1 || nchol < 1) { set_error("bad shape: norb %d, nchol %d", norb, nchol); return 0; }
  Carver c(nullptr, 0);
  CtxBuffers b;
  carve_ctx(norb, nchol, c, b);
  if (digits) carve_squares(norb, nchol, c, b.status);
  return c.used + 256;
}
size_t trot_prop_ctx_workspace_size(int norb, int nchol) { return ctx_workspace(norb, nchol, false); }
size_t trot_prop_ctx_workspace_size_digits(int norb, int nchol) { return ctx_workspace(norb, nchol, true); }

int trot_build_prop_ctx(int norb, int nchol, double h0, double dt, const double* h1, const double* chol,
                        const double* rdm1, double* mf_im, double* h0_prop, double* exp_h1_half, void* ws,
                        size_t ws_bytes, void* stream) {
  if (!h1 || !chol || !rdm1 || !mf_im || !h0_prop || !exp_h1_half || !ws) {
    set_error("null input, output or workspace");
    return TROT_ERR_NULL_PTR;
  }
  if (norb < 1 || nchol < 1) { set_error("bad shape: norb %d, nchol %d", norb, nchol); return TROT_ERR_BAD_SHAPE; }
  if (!(dt > 0.0) || !(dt < 1e300)) { set_error("bad time step %g", dt); return TROT_ERR_BAD_SHAPE; }
  const int N = norb, G = nchol;
  Carver c(ws, ws_bytes);
  CtxBuffers b;
  carve_ctx(N, G, c, b);
  const DgScratch dg = carve_squares(N, G, c, b.status);
  if (!c.ok) { set_error("workspace too small: %zu < %zu", ws_bytes, c.used); return TROT_ERR_WORKSPACE_TOO_SMALL; }
  int S, gper;
  ctx_slices(N, G, S, gper);
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(b.status, 0, 2 * sizeof(int), st);
  if (e != cudaSuccess) return cuda_status(e, "trot_build_prop_ctx memset");
  ctx_mf_kernel<<<G, 256, 0, st>>>(N, chol, rdm1, mf_im);
  TROT_CHECK_LAUNCH("ctx_mf_kernel");
  ctx_h0_kernel<<<1, 256, 0, st>>>(G, h0, mf_im, h0_prop);
  TROT_CHECK_LAUNCH("ctx_h0_kernel");
  TROT_TRY(launch_v(N, G, S, gper, chol, mf_im, b.part, dg, st));
  const size_t nn = (size_t)N * N;
  const int eb = (int)((nn + 255) / 256 < 1024 ? (nn + 255) / 256 : 1024);
  ctx_heff_kernel<<<eb, 256, 0, st>>>(N, S, dt, h1, b.part, b.a);
  TROT_CHECK_LAUNCH("ctx_heff_kernel");
  TROT_TRY(launch_expm(N, b.a, exp_h1_half, b.p0, b.p1, b.status, st));
  return TROT_OK;
}

static size_t ctx_vjp_workspace(int norb, int nchol, bool digits) {
  if (norb < 1 || nchol < 1) { set_error("bad shape: norb %d, nchol %d", norb, nchol); return 0; }
  Carver c(nullptr, 0);
  CtxBuffers b;
  carve_ctx(norb, nchol, c, b);
  const size_t m = (size_t)4 * norb * norb;
  c.take<double>(nchol);      // mean-field traces
  for (int k = 0; k < 4; ++k) c.take<double>(m);  // M, P0, P1, expm(M)
  if (digits) carve_squares(norb, nchol, c, b.status);
  return c.used + 256;
}
size_t trot_prop_ctx_vjp_workspace_size(int norb, int nchol) { return ctx_vjp_workspace(norb, nchol, false); }
size_t trot_prop_ctx_vjp_workspace_size_digits(int norb, int nchol) { return ctx_vjp_workspace(norb, nchol, true); }

int trot_prop_ctx_vjp(int norb, int nchol, double dt, const double* h1, const double* chol, const double* rdm1,
                      const double* g_exp_h1_half, double* g_h1, void* ws, size_t ws_bytes, void* stream) {
  if (!h1 || !chol || !rdm1 || !g_exp_h1_half || !g_h1 || !ws) {
    set_error("null input, output or workspace");
    return TROT_ERR_NULL_PTR;
  }
  if (norb < 1 || nchol < 1) { set_error("bad shape: norb %d, nchol %d", norb, nchol); return TROT_ERR_BAD_SHAPE; }
  if (!(dt > 0.0) || !(dt < 1e300)) { set_error("bad time step %g", dt); return TROT_ERR_BAD_SHAPE; }
  const int N = norb, G = nchol;
  Carver c(ws, ws_bytes);
  CtxBuffers b;
  carve_ctx(N, G, c, b);
  const size_t m = (size_t)4 * N * N;
  double* t = c.take<double>(G);
  double* M = c.take<double>(m);
  double* q0 = c.take<double>(m);
  double* q1 = c.take<double>(m);
  double* E = c.take<double>(m);
  const DgScratch dg = carve_squares(N, G, c, b.status);
  if (!c.ok) { set_error("workspace too small: %zu < %zu", ws_bytes, c.used); return TROT_ERR_WORKSPACE_TOO_SMALL; }
  int S, gper;
  ctx_slices(N, G, S, gper);
  cudaStream_t st = (cudaStream_t)stream;
  cudaError_t e = cudaMemsetAsync(b.status, 0, 2 * sizeof(int), st);
  if (e != cudaSuccess) return cuda_status(e, "trot_prop_ctx_vjp memset");
  ctx_mf_kernel<<<G, 256, 0, st>>>(N, chol, rdm1, t);
  TROT_CHECK_LAUNCH("ctx_mf_kernel");
  TROT_TRY(launch_v(N, G, S, gper, chol, t, b.part, dg, st));
  const size_t nn = (size_t)N * N;
  const int eb = (int)((nn + 255) / 256 < 1024 ? (nn + 255) / 256 : 1024);
  ctx_heff_kernel<<<eb, 256, 0, st>>>(N, S, dt, h1, b.part, b.a);
  TROT_CHECK_LAUNCH("ctx_heff_kernel");
  const int eb2 = (int)((m + 255) / 256 < 1024 ? (m + 255) / 256 : 1024);
  double* gscale = reinterpret_cast<double*>(b.status + 8);
  ctx_absmax_kernel<<<1, 256, 0, st>>>(nn, g_exp_h1_half, gscale);
  TROT_CHECK_LAUNCH("ctx_absmax_kernel");
  ctx_frechet_build_kernel<<<eb2, 256, 0, st>>>(N, b.a, g_exp_h1_half, gscale, M);
  TROT_CHECK_LAUNCH("ctx_frechet_build_kernel");
  TROT_TRY(launch_expm(2 * N, M, E, q0, q1, b.status, st));
  // A = -dt/2 h1_eff and h1_eff = h1 + (terms without h1): dJ/dh1 = -dt/2 dJ/dA
  ctx_frechet_take_kernel<<<eb, 256, 0, st>>>(N, E, -0.5 * dt, gscale, g_h1);
  TROT_CHECK_LAUNCH("ctx_frechet_take_kernel");
  return TROT_OK;
}

int trot_half_rotate(int norb, int nchol, int nocc, const double* mo, const double* h1, const double* chol,
                     double* rot_h1, double* rot_chol, void* stream) {
  if (!mo || (!h1 && !chol) || (h1 && !rot_h1) || (chol && !rot_chol)) {
    set_error("null input or output");
    return TROT_ERR_NULL_PTR;
  }
  if (norb < 1 || nocc < 1 || nocc > norb || (chol && nchol < 1)) {
    set_error("bad shape: norb %d, nchol %d, nocc %d", norb, nchol, nocc);
    return TROT_ERR_BAD_SHAPE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const unsigned pb = (unsigned)((nocc + 15) / 16);
  if (h1) {
    ctx_rotate_kernel<<<dim3(1, pb), 128, 0, st>>>(norb, nocc, mo, h1, rot_h1);
    TROT_CHECK_LAUNCH("ctx_rotate_kernel");
  }
  if (chol) {
    ctx_rotate_kernel<<<dim3(nchol, pb), 128, 0, st>>>(norb, nocc, mo, chol, rot_chol);
    TROT_CHECK_LAUNCH("ctx_rotate_kernel");
  }
  return TROT_OK;
}

int trot_cisd_lci1(int norb, int nchol, int nocc, const double* ci1, const double* chol, double* lci1, void* stream) {
  if (!ci1 || !chol || !lci1) { set_error("null input or output"); return TROT_ERR_NULL_PTR; }
  if (norb < 2 || nchol < 1 || nocc < 1 || nocc >= norb) {
    set_error("bad shape: norb %d, nchol %d, nocc %d", norb, nchol, nocc);
    return TROT_ERR_BAD_SHAPE;
  }
  ctx_lci1_kernel<<<nchol, 256, 0, (cudaStream_t)stream>>>(norb, nocc, ci1, chol, lci1);
  TROT_CHECK_LAUNCH("ctx_lci1_kernel");
  return TROT_OK;
}

}  // extern "C"
