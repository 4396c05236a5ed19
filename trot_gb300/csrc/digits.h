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

// C[m][n] (+)= alpha sum_k A[m][k] B(k, n) as launch_zgemm_cr_splitk, with both operands as six
// FP16 digit planes per row and 26 exact tensor-core products.
int launch_zgemm_dg(int M, int Nn, int K, double alpha, const double2* A, int lda, const double* B, int ldb,
                    bool b_is_nk, double2* C, long long ldc, bool accumulate, const DgScratch& s, cudaStream_t st);


// Exchange sums and force bias of all walkers from one set of digit products f_g = rot_chol_g G^T (N >= kDgMinK
// orbitals): partial[b][chunk] as launch_exchange but exchange_dg_chunks(G) of them (fewer), fb[b][g] = sum_s mult_s tr f_sg.
int exchange_dg_chunks(int G);
size_t exchange_dg_bytes(const Spins& sp, size_t W, size_t N, size_t G);
int launch_exchange_dg(const Spins& sp, int W, int N, int G, const double2* green, double2* partial, double2* fb,
                       const DgScratch& s, cudaStream_t st);

// The same fb, bit for bit, without the exchange sums.  With parts, where all f_gii are there at once, they are handed
// over in it instead (inside the scratch; parts->nspin stays 0 otherwise).
size_t fb_dg_bytes(const Spins& sp, size_t W, size_t N, size_t G);
int launch_fb_dg(const Spins& sp, int W, int N, int G, const double2* green, double2* fb, FbParts* parts,
                 const DgScratch& s, cudaStream_t st);

// C[g][m][j] = (row 2 m, row 2 m + 1) of L_g L_g for `count` real N x N matrices, m < ceil(N / 2) (N even or odd: the
// odd last row's partner is zero).  square_dg_count: matrices a call takes with a scratch of square_dg_bytes.
int square_dg_count(size_t N, size_t G);
size_t square_dg_bytes(size_t N, size_t count);
int launch_square_dg(int N, int count, const double* L, const DgScratch& s, double2** C, cudaStream_t st);

// Trotter propagation (with overlaps and weights in step mode) by digit products; same results as launch_trotter.
size_t trotter_dg_bytes(const Spins& sp, size_t W, size_t N);
int launch_trotter_dg(const Spins& sp, const TrotterArgs& a, const DgScratch& s, cudaStream_t st);

// Batched products of the step adjoint on arrays (walker, column j, orbital p) of nc columns: V (complex N x N per
// walker), E (real N x N) or E^T against every column.
struct DgAdjoint {
  int W, N, nc, K2;                    // K2: terms (l, j) of the cotangent of V
  uint16_t *vimg, *uimg, *eimg, *etimg;
  int16_t *vex, *uex, *eex, *etex;
  int16_t* cexp;                       // (W, K2): exponents of the chain's columns u_l[j], k = (l, j)
  int* status;
};
enum DgOperand { kDgE, kDgET, kDgV };
size_t adjoint_dg_bytes(size_t W, size_t N, size_t nc, size_t K2);
void adjoint_dg_carve(DgAdjoint& d, int W, int N, int nc, int K2, const DgScratch& s);
// digits of E and E^T; of V, or of V^T (transposed)
int adjoint_dg_e(const DgAdjoint& d, const double* E, cudaStream_t st);
int adjoint_dg_v(const DgAdjoint& d, const double2* V, bool transposed, cudaStream_t st);
// walkers with act[b] == 0: a row of V that is not finite counts as zero
int adjoint_dg_v_active(const DgAdjoint& d, const int* act, cudaStream_t st);
// out[b][j][p] (walkers ostride apart) = op . columns of wa (W, N, na) and wb (W, N, nb), conjugated if conj
int adjoint_dg_from_walkers(const DgAdjoint& d, DgOperand op, const double2* wa, int na, const double2* wb, int nb,
                            bool conj, double2* out, long long ostride, cudaStream_t st);
// the same from an array (walker, j, p), walkers sstride apart; term l >= 0: src is u_l, whose exponents gv wants
int adjoint_dg_from_rows(const DgAdjoint& d, DgOperand op, const double2* src, long long sstride, double2* out,
                         long long ostride, cudaStream_t st, int term = -1);
// gv[b][p][q] = sum_{k < K2} S[b][k][p] U[b][k][q], U[b][k] the u_l noted above (the digits of V are overwritten)
int adjoint_dg_gv(const DgAdjoint& d, const double2* S, long long sstride, const double2* U, long long ustride,
                  double2* gv, cudaStream_t st);

// The CISD energy's per-vector terms (cisd_gamma_kernel's) with every contraction over orbitals as a digit product:
// xg[b][g][p][t] = glgp, gpart[b][chunk][4] the four sums (cisd_gamma_dg_chunks(G) chunks per walker).
struct CisdGammaArgs {
  int W, N, n, v, G;
  const double2* green;   // (W, n, N)
  const double* chol;     // (G, N, N)
  const double* lci1;     // (G, N, n)
  const double2* p2;      // (W, N, n)
  const double2* ci1g1;   // (W, n, n)
  double2* xg;
  double2* gpart;
};
// lg1 and B alone, for all walkers: F1[(b, q)][(g, p)] = lg1[p][q], F2[(b, p)][(g, q)] = (G lci1_g)[p][q] (complex,
// W n x G n), both inside the scratch
size_t cisd_lg_dg_bytes(size_t W, size_t N, size_t n, size_t G);
int launch_cisd_lg_dg(const CisdGammaArgs& c, const DgScratch& s, double2** F1, double2** F2, cudaStream_t st);

int cisd_gamma_dg_chunks(int G);
size_t cisd_gamma_dg_bytes(size_t W, size_t N, size_t n, size_t G);
int launch_cisd_gamma_dg(const CisdGammaArgs& c, const DgScratch& s, cudaStream_t st);

}  // namespace trot
