// Non-GEMM device kernels of the GW / HF path (gathers, symmetry unfolding, the batched
// FP64 Dyson solvers and small reductions).  Host launchers; all run on `stream`.
#pragma once

#include "common.cuh"

namespace gg {

// V(k, k1) gather: out[p][Q][i][j] = op_p(S[pos_p][Q])[i][j], op bit0 = conj, bit1 = transpose.
void launch_gather_pairs(const double2* S, const int64_t* pos_d, const int* op_d, int npairs, int NQ, int n,
                         double2* out, cudaStream_t st);

// Gather full-BZ G from the IBZ input (layout [t][s][ink][i][j]):
// out[k][s][t][i][j] = G[t][s][f2r[k]][i][j] (optionally conjugated later).
void launch_gather_g(const double2* G_tskij, const int* k_f2r_d, int nk, int ns, int nts, int ink, int n,
                     double2* out, cudaStream_t st);

// out[k][...][i][j] = conj(...) for every k with tr[k] != 0; per_k elements per k.
void launch_conj_where(double2* X, const int* tr_d, int nk, long per_k, cudaStream_t st);

// gather blocks: out[p][e] = src[idx[p] * src_stride + e] for e < elems
void launch_gather_blocks(const double2* src, const int* idx_d, int nblocks, long elems, long src_stride,
                          double2* out, cudaStream_t st);
// err[0..2] <- (1, base + i, info[i]) for the first failing system i (info != 0), if none is recorded yet
void launch_info_collect(const int* info, int count, int base, int* err, cudaStream_t st);

// Two-component (X2C) spin blocks.  A spinor matrix of order 2n holds the blocks aa (0,0),
// bb (n,n), ab (0,n) and ba (n,0).  Block ss of the pseudo-spin order is (row, col) =
// (ss % 2, ss == 0 ? 0 : ss == 1 ? 1 : ss == 2 ? 1 : 0), i.e. aa, bb, ab, ba (the order of the
// reference's copy_Gk_2c with minus_t = false and copy_Sigma_2c, gw_gpu_kernel.cpp:523-551,
// cugw_qkpt.cu:382-403).
// split: in [nouter][ninner][2n][2n] -> out [nouter][nblk][ninner][n][n] (nblk = 3 or 4)
void launch_x2c_split(const double2* in, long nouter, long ninner, int n, int nblk, double2* out, cudaStream_t st);
// merge: in [nouter][nblk][ninner][n][n] -> out [nouter][ninner][2n][2n]; with nblk = 3 the ba
// block is the adjoint of ab (cuda_common.cu:176-201)
void launch_x2c_merge(const double2* in, long nouter, long ninner, int n, int nblk, double2* out, cudaStream_t st);

// out[b][i][j] = in[b][j][i] for nblocks n x n matrices (32 x 32 tiles through shared memory)
void launch_transpose_blocks(const double2* in, long nblocks, int n, double2* out, cudaStream_t st);

// *flag (device) = nonzero when every G[t][s][k] (layout [nts][ns][ink][n][n]) is Hermitian within tol of its largest element,
// else 0; swap: blocks 2 and 3 are each other's adjoints (X2C)
void launch_hermitian_check(const double2* G, int nts, int ns, int ink, int n, int swap, double tol, int* flag,
                            cudaStream_t st);
// H = the Hermitian parts of G (layout [nk][ns][nts][n][n]) where *flag (device), else a copy
void launch_hermitian_part(const double2* G, int nk, int ns, int nts, int n, int swap, const int* flag, double2* H,
                           cudaStream_t st);
// where *flag (device): the upper triangles of nmat n x n matrices from their lower ones
void launch_mirror_lower(double2* X, int nmat, int n, const int* flag, cudaStream_t st);

// Batched Dyson solve for `nsys` systems of size N x N stored contiguously in P (in place):
// P <- Hermitian-symmetrise(P); A = I - P; Cholesky: P <- (A^{-1} P)^H, LU: P <- sym(A^{-1} P).
// `A` is a workspace of the same size, `info` receives per-system status (0 ok; Cholesky:
// index+1 of the first non-positive pivot; LU: index+1 of the first zero pivot).  LU only: li
// [nsys][ceil(N / b) b][b] with b = dyson_lu_block(N), piv [nsys][N].  Returns the launches.
int dyson_lu_block(int N);
int launch_dyson(double2* P, double2* A, double2* li, int* info, int nsys, int N, int solver, int* piv, cudaStream_t st);

// Hermitian symmetrisation only (cuda_common.cu:249-281), nsys matrices in place.
void launch_hermitian_symmetrize(double2* P, int nsys, int N, cudaStream_t st);

// Hartree term on the stored integrals (pos / op of the diagonal pairs (k, k)):
// c[Q] = scale sum_k sum_{s < nsj} Tr(V^Q(k,k) D[k][s]) (c holds (nk + 1) NQ elements, the partial sums of
// every k after the result), F[s][kr] += sum_Q c[Q] V^Q(k,k) for s < nsj, k = k_r2f[kr].
void launch_hartree_coeff(const double2* S, const int64_t* pos_d, const int* op_d, const double2* D, int nk, int NQ, int n,
                          int ns, int nsj, double scale, double2* c, cudaStream_t st);
void launch_hartree_apply(const double2* S, const int64_t* pos_d, const int* op_d, const int* k_r2f_d, const double2* c,
                          int ink, int NQ, int n, int nsj, double2* F, cudaStream_t st);

}  // namespace gg
