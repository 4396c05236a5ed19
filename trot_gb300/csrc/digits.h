// FP64-accurate products on the tensor cores by exact digit slices (digits.cu).
// Shorter rows than 20 stay on the FP64 pipe: the digits' error does not fall with K (1.05e-16 of the result at K = 3,
// 1.1e-16 at 16, 1.2e-16 at 135), that of an FP64 sum does (0.8e-16, 1.5e-16, 3.9e-16).  Past 2^17 the 64-bit sums
// would overflow.  There is no limit on the other sizes: one 64 x 64 x 16 step of the FP64 kernel takes 34 us on its
// SM, a whole small product here 20 us.
#pragma once
#include "kernels.h"

namespace trot {

static constexpr int kDgMinK = 20, kDgMaxK = 1 << 17;
inline bool dg_takes(int K) { return K >= kDgMinK && K <= kDgMaxK; }

// Bytes that launch_zgemm_dg wants for C (M x Nn) = alpha A (M x K complex) B (K x Nn real).
size_t dg_scratch_bytes(size_t M, size_t Nn, size_t K);

// C[m][n] (+)= alpha sum_k A[m][k] B(k, n) as launch_zgemm_cr, with both operands as six
// FP16 digit planes per row and 26 exact tensor-core products.
int launch_zgemm_dg(int M, int Nn, int K, double alpha, const double2* A, int lda, const double* B, int ldb,
                    bool b_is_nk, double2* C, long long ldc, bool accumulate, const DgScratch& s, cudaStream_t st);


// Exchange sums and force bias of all walkers from one set of digit products f_g = rot_chol_g G^T (N >= kDgMinK
// orbitals): partial[b][chunk] as launch_exchange but exchange_dg_chunks(G) of them (fewer), fb[b][g] = sum_s mult_s tr f_sg.
int exchange_dg_chunks(int G);
size_t exchange_dg_bytes(const Spins& sp, size_t W, size_t N, size_t G);
int launch_exchange_dg(const Spins& sp, int W, int N, int G, const double2* green, double2* partial, double2* fb,
                       const DgScratch& s, cudaStream_t st);

// Trotter propagation (with overlaps and weights in step mode) by digit products; same results as launch_trotter.
size_t trotter_dg_bytes(const Spins& sp, size_t W, size_t N);
int launch_trotter_dg(const Spins& sp, const TrotterArgs& a, const DgScratch& s, cudaStream_t st);

}  // namespace trot
