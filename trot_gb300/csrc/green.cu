// Half Green's functions, trial overlaps and one-body energy per walker (FP64).
//
// For each walker b and spin s (trot/meas/rhf.py:21-25, trot/trial/rhf.py:45-54):
//   M_s   = C_s^T w_s                     (n_s x n_s)
//   G_s   = (w_s M_s^{-1})^T              (n_s x N)   half Green's function
//   ovlp  = prod_s det(M_s)^mult_s
//   e1    = sum_s mult_s sum_{i,p} G_s[i][p] rot_h1_s[i][p]
// A CTA per (walker, spin), the spins of a walker in a cluster: the first one combines the determinants and energies.
// The walker tile and M (then M^{-1}, in place by one warp) live in shared memory.  FP64 pipe: 2 N n^2 FMAs for M (four
// lanes per element) and 4 N n^2 for G per spin; at 120 orbitals, 12 + 10 electrons, 1024 walkers these take 0.31 ms of
// it.  One CTA per walker with the elimination of [M | I] by all its threads took 0.55 ms there (0.28 ms for overlaps
// only), now 0.50 and 0.19; at 67 orbitals, 9 + 9 electrons, 200 walkers, where the elimination's barriers bound it, 0.108
// -> 0.052 ms.
#include <cooperative_groups.h>

#include "kernels.h"

namespace trot {

static constexpr int kGreenThreads = 128;
static constexpr int kMaxOcc = 64;

__global__ void __launch_bounds__(kGreenThreads)
green_kernel(Spins sp, int N, int padded, const double2* __restrict__ wa, const double2* __restrict__ wb,
             double2* __restrict__ green, double2* __restrict__ ovlp_out, double2* __restrict__ e1_out,
             int* __restrict__ status) {
  extern __shared__ double2 smem[];
  __shared__ double2 red[32];
  __shared__ double2 sums[2];  // det^mult, mult e1 of this spin
  __shared__ GjScratch gj;
  namespace cg = cooperative_groups;
  cg::cluster_group cl = cg::this_cluster();
  const int s = sp.nspin == 2 ? blockIdx.x & 1 : 0, b = sp.nspin == 2 ? blockIdx.x >> 1 : blockIdx.x;
  const int tid = threadIdx.x, nt = blockDim.x;
  if (status && blockIdx.x == 0 && tid == 0) *status = 0;  // this call's status word (the sticky one persists)
  const bool want_green = green != nullptr || e1_out != nullptr;
  const int n = s ? sp.n[1] : sp.n[0], ld = padded ? n | 1 : n;
  const double2* w = (s ? wb : wa) + (size_t)b * N * n;
  const double* C = s ? sp.mo[1] : sp.mo[0];
  double2* Ws = smem;                     // N x ld
  double2* Ms = Ws + (size_t)N * ld;      // n x n
  for (int e = tid; e < N * n; e += nt) Ws[(e / n) * ld + e % n] = w[e];
  __syncthreads();
  // M[i][j] = sum_p C[p][i] w[p][j], four lanes per element
  for (int e0 = 0; e0 < n * n; e0 += nt >> 2) {
    const int e = e0 + (tid >> 2), i = e / n, j = e - i * n;
    double2 acc = cmk(0.0, 0.0);
    if (e < n * n)
      for (int p = tid & 3; p < N; p += 4) crfma(acc, C[(size_t)p * n + i], Ws[p * ld + j]);
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
      acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    }
    if (e < n * n && (tid & 3) == 0) Ms[e] = acc;
  }
  __syncthreads();
  const int mult = s ? sp.mult[1] : sp.mult[0];
  const double2 det = gauss_jordan(Ms, n, want_green, gj, b);
  if (tid == 0) sums[0] = mult == 2 ? cmul(det, det) : det;
  __syncthreads();
  if (want_green) {
    // G[i][p] = sum_j w[p][j] Minv[j][i]
    double2 e1 = cmk(0.0, 0.0);
    const double* H = s ? sp.rot_h1[1] : sp.rot_h1[0];
    double2* gout = green ? green + (size_t)b * sp.ntot * N + (size_t)(s ? sp.off[1] : 0) * N : nullptr;
    for (int e = tid; e < n * N; e += nt) {
      const int i = e / N, p = e - i * N;
      double2 acc = cmk(0.0, 0.0);
      for (int j = 0; j < n; ++j) cfma(acc, Ws[p * ld + j], Ms[j * n + i]);
      if (gout) gout[e] = acc;
      if (H) crfma(e1, H[e], acc);
    }
    if (e1_out) {
      e1 = block_sum2(e1, red);
      if (tid == 0) sums[1] = mult == 2 ? cadd(e1, e1) : e1;
    }
  }
  if (sp.nspin == 2) cl.sync();
  if (s == 0 && tid == 0) {
    double2 d = cmul(cmk(1.0, 0.0), sums[0]), e1 = cadd(cmk(0.0, 0.0), sums[1]);
    if (sp.nspin == 2) {
      const double2* other = cl.map_shared_rank(sums, 1);
      d = cmul(d, other[0]);
      if (e1_out) e1 = cadd(e1, other[1]);
    }
    if (ovlp_out) ovlp_out[b] = d;
    if (e1_out) e1_out[b] = e1;
  }
  if (sp.nspin == 2) cl.sync();  // the other CTA's sums stay readable until here
}

int launch_green(const Spins& sp, int W, int N, const double2* wa, const double2* wb, double2* green,
                 double2* ovlp_out, double2* e1_out, cudaStream_t st, int* status) {
  int nmax = sp.n[0] > sp.n[1] ? sp.n[0] : sp.n[1];
  if (nmax > kMaxOcc) {
    set_error("green: nocc %d > %d unsupported", nmax, kMaxOcc);
    return TROT_ERR_UNSUPPORTED;
  }
  const size_t limit = (size_t)(N * nmax + 2 * nmax * nmax) * sizeof(double2);
  if (limit > 200 * 1024) {
    set_error("green: walker tile of %zu bytes exceeds shared memory", limit);
    return TROT_ERR_UNSUPPORTED;
  }
  // odd row stride against bank conflicts where it fits
  const size_t padded = ((size_t)N * (nmax | 1) + (size_t)nmax * nmax) * sizeof(double2);
  const bool pad = padded <= 220 * 1024;
  const size_t smem = pad ? padded : (size_t)(N * nmax + nmax * nmax) * sizeof(double2);
  if (smem > 40 * 1024)
    cudaFuncSetAttribute(green_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3(W * sp.nspin);
  cfg.blockDim = dim3(kGreenThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = sp.nspin;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = sp.nspin == 2 ? 1 : 0;
  const cudaError_t rc = cudaLaunchKernelEx(&cfg, green_kernel, sp, N, pad ? 1 : 0, wa, wb, green, ovlp_out, e1_out,
                                            status);
  if (rc != cudaSuccess) return cuda_status(rc, "green_kernel");
  TROT_CHECK_LAUNCH("green_kernel");
  return TROT_OK;
}

}  // namespace trot
