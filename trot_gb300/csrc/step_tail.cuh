// Shared tail of the Trotter kernels: overlap of the propagated walker with
// the trial (FP64 LU determinant) and the phaseless importance weight.
#pragma once
#include "kernels.h"

namespace trot {

// Phaseless importance weight of walker b given its new trial overlap
// (trot/prop/afqmc.py:111-130): weights, overlaps and node flag are updated in place.
//   imp_ph = |e^(u) rho| cos(arg(e^(v) rho)),  rho = new / old overlap, v = -sqrt(dt) shift, u = v + fb term + ...
// Away from overflow that is e^(Re u) Re(rho e^(i Im v)): one exponential and one sine / cosine pair instead of two of
// each, an arc tangent, another cosine and a square root, all of which wait on one another in the FP64 pipe (10 us for
// one warp, however few walkers).  Beyond the bounds, the formula as it stands.
static __device__ __noinline__ double phaseless_factor_general(double2 ratio, double2 expo, double2 v) {
  const double2 imp = cmul(cexp(expo), ratio);
  const double2 ph = cmul(cexp(v), ratio);
  const double theta = atan2(ph.y, ph.x);
  return hypot(imp.x, imp.y) * cos(theta);
}
__device__ __forceinline__ int exponent_of(double x) { return ((__double2hiint(x) >> 20) & 0x7FF) - 1023; }
__device__ __forceinline__ void phaseless_update(const TrotterArgs& a, int b, double2 ov_new) {
  const double2 ov_old = a.overlaps[b];
  const double2 ratio = cdiv(ov_new, ov_old);
  const double2 shift = a.shift_term[b];
  const double2 fbt = a.fb_term[b];
  const double e_shift = a.scalars[0];
  const double2 v = cscale(shift, -a.sqrt_dt);
  const double2 expo = cadd(cadd(v, fbt), cmk(a.dt * (e_shift + a.h0_prop), 0.0));
  const int er = max(exponent_of(ratio.x), exponent_of(ratio.y));
  double imp_ph;
  if (exponent_of(expo.x) < 8 && exponent_of(expo.y) < 8 && exponent_of(v.x) < 8 && exponent_of(v.y) < 8 && er < 100 &&
      er > -100) {
    double s, c;
    sincos(v.y, &s, &c);
    imp_ph = exp(expo.x) * (ratio.x * c - ratio.y * s);
  } else {
    imp_ph = phaseless_factor_general(ratio, expo, v);
  }
  if (!isfinite(imp_ph) || imp_ph < a.w_floor) imp_ph = 0.0;
  a.node_flag[b] = imp_ph <= 0.0 ? 1 : 0;
  if (imp_ph > a.w_cap) imp_ph = 0.0;
  double wn = a.weights[b] * imp_ph;
  if (wn > a.w_cap) wn = 0.0;
  a.weights[b] = wn;
  a.overlaps[b] = ov_new;
}

// W2: propagated walker columns (N x nc, FP64, shared memory); Ms: n x n scratch.
__device__ __forceinline__ void overlap_and_weight(const Spins& sp, const TrotterArgs& a, int N, int nc,
                                                   const double2* W2, double2* Ms) {
  __shared__ GjScratch gj;
  const int b = blockIdx.x, tid = threadIdx.x, nt = blockDim.x;
  // new overlap: prod_s det(C_s^T w'_s)^mult  (trot/trial/rhf.py:45-54, trot/trial/uhf.py:54-58)
  double2 det_all = cmk(1.0, 0.0);
  for (int s = 0; s < sp.nspin; ++s) {
    const int n = sp.n[s];
    const double* C = sp.mo[s];
    __syncthreads();
    for (int e = tid; e < n * n; e += nt) {
      const int i = e / n, j = e % n;
      double2 acc = cmk(0.0, 0.0);
      for (int p = 0; p < N; ++p) crfma(acc, C[p * n + i], W2[p * nc + sp.off[s] + j]);
      Ms[e] = acc;
    }
    __syncthreads();
    double2 det = cmk(0.0, 0.0);
    if (tid < 128) det = gauss_jordan(Ms, n, false, gj, b);  // n <= kGjMax: the step's Green's functions take no more
    det_all = cmul(det_all, sp.mult[s] == 2 ? cmul(det, det) : det);
  }
  if (tid == 0) phaseless_update(a, b, det_all);
}

}  // namespace trot
