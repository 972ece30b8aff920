// Batched FP64 Dyson solve W = (I - P)^{-1} P over all (q, Omega) systems at once.
//
// The factorisation and the triangular solves are blocked and advance through every system together:
// the O(N^3) work of each block step is one batched product on the FP64 GEMM engine, and only the
// small diagonal blocks (Cholesky) or panels (LU) run in kernels of their own, one CTA per system.
// Diagonal blocks are kept as inverses, so that a triangular solve with one is a product too.
// With one CTA per system doing everything from shared-memory tiles on the FP64 FMA units, 276
// systems of N = 400 took 31.4 ms and 138 LU systems of N = 251 17.7 ms: too few warps in flight, a
// barrier every few hundred FMAs, and in the LU one dependent global load per step.
#include <algorithm>

#include "dmma.cuh"
#include "kernels.cuh"
#include "zgemm.cuh"

namespace gg {
namespace {

constexpr int TPB = 256;
constexpr int CB = 64;      // Cholesky block
constexpr int LU_SMEM = 220 * 1024;

// Hermitian symmetrisation in place, M = (M + M^H) / 2 with a real diagonal
// (cuda_common.cu:249-281); with A != NULL also A = I - M (cu_compute_Pq.cu:44-63), its lower
// triangle only when `lower`.  One 32 x 32 tile pair per CTA: both tiles pass through shared memory,
// so that every access to global memory is a run of 32 elements.
__global__ void __launch_bounds__(TPB) hermitize_kernel(double2* Pall, double2* Aall, int* info, int N, int lower) {
  __shared__ double2 lo[32][33], up[32][33];
  int ti = 0, p = blockIdx.y;
  while (p > ti) p -= ++ti;  // pair (ti, p), p <= ti
  const int tj = p;  // tj <= ti
  const long NN = (long)N * N;
  double2* P = Pall + blockIdx.x * NN;
  double2* A = Aall ? Aall + blockIdx.x * NN : nullptr;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  if (info && blockIdx.y == 0 && threadIdx.x == 0) info[blockIdx.x] = 0;
  for (int r = ty; r < 32; r += 8) {
    const int i = ti * 32 + r, j = tj * 32 + tx;
    if (i < N && j < N) lo[r][tx] = P[(long)i * N + j];
    const int k = tj * 32 + r, l = ti * 32 + tx;
    if (k < N && l < N) up[r][tx] = P[(long)k * N + l];
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int i = ti * 32 + r, j = tj * 32 + tx;
    if (i < N && j < N) {
      const double2 a = lo[r][tx], b = up[tx][r];  // (i, j), (j, i)
      const double2 v = i == j ? make_double2(a.x, 0.0) : make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
      P[(long)i * N + j] = v;
      if (A) A[(long)i * N + j] = i == j ? make_double2(1.0 - v.x, 0.0) : make_double2(-v.x, -v.y);
    }
    const int k = tj * 32 + r, l = ti * 32 + tx;
    if (ti != tj && k < N && l < N) {  // the mirror tile: (k, l) = conj of (l, k)
      const double2 a = lo[tx][r], b = up[r][tx];
      const double2 v = make_double2(0.5 * (a.x + b.x), -0.5 * (a.y - b.y));
      P[(long)k * N + l] = v;
      if (A && !lower) A[(long)k * N + l] = make_double2(-v.x, -v.y);
    }
  }
}

// Cholesky factor L of the jb x jb diagonal block at j0 (its lower triangle is read), replaced by L^{-1}
// (zeros above the diagonal).  Thread (k, ty) keeps elements (ty + 4 i, k) in registers; at step c
// the rank-1 update covers the trailing block (columns k > c) and, for k <= c, the rows of the inverse
// that build up in place of the finished columns.  One barrier per step; bound by the FP64 FMAs
// (16 x 64 per thread) and that barrier: about 12 us per block.
__global__ void __launch_bounds__(TPB) chol_block_kernel(double2* Aall, int* info, int N, int j0, int jb) {
  __shared__ double2 col[2][CB], row[2][CB];
  double2* A = Aall + blockIdx.x * (long)N * N + (long)j0 * N + j0;
  const int k = threadIdx.x & (CB - 1), ty = threadIdx.x / CB;
  double2 a[CB / 4];
#pragma unroll
  for (int i = 0; i < CB / 4; ++i) {
    const int r = ty + 4 * i;
    a[i] = r < jb && k <= r ? A[(long)r * N + k] : make_double2(0.0, 0.0);
  }
  int fail = 0;
  for (int c = 0; c < jb; ++c) {
    double2* const cs = col[c & 1];
    double2* const rs = row[c & 1];
    // column c (raw) and row c of the inverse so far
    if (k == c) {
#pragma unroll
      for (int i = 0; i < CB / 4; ++i) cs[ty + 4 * i] = a[i];
    }
    if ((c & 3) == ty) {
#pragma unroll
      for (int i = 0; i < CB / 4; ++i)
        if (ty + 4 * i == c) rs[k] = a[i];
    }
    __syncthreads();
    double d = cs[c].x;
    if (!(d > 0.0)) {
      if (!fail) fail = j0 + c + 1;
      d = 1.0;
    }
    const double inv = 1.0 / sqrt(d);
    // multiplier of column k: the inverse's row c (k < c), 1 / L_cc (k = c), conj L_kc (k > c)
    const double2 v = k < c ? cscale(rs[k], inv) : k == c ? make_double2(inv, 0.0) : cconj(cscale(cs[k], inv));
#pragma unroll
    for (int i = 0; i < CB / 4; ++i) {
      const int r = ty + 4 * i;
      if (r > c) {
        const double2 l = cscale(cs[r], inv);
        a[i] = csub(k == c ? make_double2(0.0, 0.0) : a[i], cmul(l, v));
      } else if (r == c && k <= c) {
        a[i] = v;
      }
    }
  }
#pragma unroll
  for (int i = 0; i < CB / 4; ++i) {
    const int r = ty + 4 * i;
    if (r < jb && k < jb) A[(long)r * N + k] = k <= r ? a[i] : make_double2(0.0, 0.0);
  }
  if (threadIdx.x == 0 && fail && info[blockIdx.x] == 0) info[blockIdx.x] = fail;
}

// LU panel: columns j0 .. j0 + nb - 1, rows j0 .. N - 1 of one system, with partial pivoting (largest |re| + |im|,
// the lowest row on ties), element (row r, column c) of the panel at pan[c * cs + r * rs]: in shared
// memory by columns when it fits, else in place.  Leaves L below the diagonal block, the
// block's U^{-1} in its place (zeros below), L^{-1} of the block in li (unit diagonal, zeros above),
// and the row interchanges (absolute rows) in piv.
__global__ void __launch_bounds__(TPB) lu_panel_kernel(double2* Aall, double2* li_all, long li_sys, int* piv_all, int* info,
                                                       int N, int j0, int nb, int in_smem) {
  extern __shared__ __align__(16) double2 dsm[];
  __shared__ double red_v[TPB / 32];
  __shared__ int red_i[TPB / 32];
  const int tid = threadIdx.x, lane = tid & 31;
  double2* A = Aall + blockIdx.x * (long)N * N + (long)j0 * N + j0;
  int* piv = piv_all + (long)blockIdx.x * N + j0;
  const int R = N - j0;
  const long cs = in_smem ? (R | 1) : 1, rs = in_smem ? 1 : N;
  double2* pan = in_smem ? dsm : A;
  if (in_smem) {
    for (int e = tid; e < R * nb; e += TPB) pan[(e % nb) * cs + e / nb] = A[(long)(e / nb) * N + e % nb];
    __syncthreads();
  }
  double best = -1.0;
  int bi = 0;
  for (int r = tid; r < R; r += TPB) {
    const double2 x = pan[r * rs];
    const double m = fabs(x.x) + fabs(x.y);
    if (m > best) {
      best = m;
      bi = r;
    }
  }
  int fail = 0;
  for (int c = 0; c < nb; ++c) {
    // largest entry of column c at or below the diagonal
    for (int o = 16; o > 0; o >>= 1) {
      const double ov = __shfl_xor_sync(0xffffffffu, best, o);
      const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
      if (ov > best || (ov == best && oi < bi)) {
        best = ov;
        bi = oi;
      }
    }
    if (lane == 0) {
      red_v[tid >> 5] = best;
      red_i[tid >> 5] = bi;
    }
    __syncthreads();
    best = red_v[0];
    bi = red_i[0];
    for (int w = 1; w < TPB / 32; ++w)
      if (red_v[w] > best || (red_v[w] == best && red_i[w] < bi)) {
        best = red_v[w];
        bi = red_i[w];
      }
    const int p = best < 0.0 ? c : bi;  // no comparable entry (NaN): keep the row
    if (!(best > 0.0) && !fail) fail = j0 + c + 1;
    if (tid == 0) piv[c] = j0 + p;
    if (tid < nb && p != c) {
      const double2 x = pan[tid * cs + c * rs];
      pan[tid * cs + c * rs] = pan[tid * cs + p * rs];
      pan[tid * cs + p * rs] = x;
    }
    __syncthreads();
    const double2 d = pan[c * cs + c * rs];
    const double dn = d.x * d.x + d.y * d.y;
    const double2 inv = dn > 0.0 ? make_double2(d.x / dn, -d.y / dn) : make_double2(0.0, 0.0);
    best = -1.0;
    bi = c + 1;
    for (int r = tid; r < R; r += TPB) {
      if (r <= c) continue;
      const double2 l = cmul(pan[c * cs + r * rs], inv);
      pan[c * cs + r * rs] = l;
      for (int k = c + 1; k < nb; ++k) {
        const double2 x = csub(pan[k * cs + r * rs], cmul(l, pan[k * cs + c * rs]));
        pan[k * cs + r * rs] = x;
        if (k == c + 1) {
          const double m = fabs(x.x) + fabs(x.y);
          if (m > best) {
            best = m;
            bi = r;
          }
        }
      }
    }
  }
  __syncthreads();
  if (in_smem)
    for (int e = tid; e < R * nb; e += TPB)
      if (e / nb >= nb) A[(long)(e / nb) * N + e % nb] = pan[(e % nb) * cs + e / nb];
  // the block's inverses: T = the block, X = L^{-1}, Y = U^{-1}, built by row operations on the identity
  double2 t[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int e = tid + i * TPB, r = e / 32, c = e % 32;
    t[i] = r < nb && c < nb ? pan[c * cs + r * rs] : make_double2(r == c ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  double2 (*T)[33] = reinterpret_cast<double2 (*)[33]>(dsm);
  double2 (*X)[33] = T + 32, (*Y)[33] = T + 64;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int e = tid + i * TPB, r = e / 32, c = e % 32;
    T[r][c] = t[i];
    X[r][c] = make_double2(r == c ? 1.0 : 0.0, 0.0);
    Y[r][c] = make_double2(r == c ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  for (int c = 0; c < nb; ++c) {
    const int b = nb - 1 - c;  // pivot row of the upper solve
    const double2 d = T[b][b];
    const double dn = d.x * d.x + d.y * d.y;
    const double2 inv = dn > 0.0 ? make_double2(d.x / dn, -d.y / dn) : make_double2(0.0, 0.0);
    if (tid < 32) Y[b][tid] = cmul(Y[b][tid], inv);
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int e = tid + i * TPB, r = e / 32, k = e % 32;
      if (r > c && k <= c) X[r][k] = csub(X[r][k], cmul(T[r][c], X[c][k]));
      if (r < b && k >= b) Y[r][k] = csub(Y[r][k], cmul(T[r][b], Y[b][k]));
    }
    __syncthreads();
  }
  double2* li = li_all + blockIdx.x * li_sys;
  for (int e = tid; e < nb * nb; e += TPB) {
    const int r = e / nb, c = e % nb;
    li[e] = X[r][c];
    A[(long)r * N + c] = Y[r][c];
  }
  if (tid == 0 && fail && info[blockIdx.x] == 0) info[blockIdx.x] = fail;
}

// Row interchanges of a panel on the columns outside it (y = 0: A) and on the right-hand side (y = 1: P):
// one thread per column, coalesced across columns.
__global__ void __launch_bounds__(64) lu_swap_kernel(double2* Aall, double2* Pall, const int* piv_all, int N, int j0, int nb) {
  const int c = blockIdx.x * 64 + threadIdx.x;
  const bool rhs = blockIdx.z != 0;
  if (c >= N || (!rhs && c >= j0 && c < j0 + nb)) return;
  double2* M = (rhs ? Pall : Aall) + blockIdx.y * (long)N * N + c;
  const int* piv = piv_all + (long)blockIdx.y * N + j0;
  for (int i = 0; i < nb; ++i) {
    const int p = piv[i];
    if (p != j0 + i) {
      const double2 x = M[(long)(j0 + i) * N];
      M[(long)(j0 + i) * N] = M[(long)p * N];
      M[(long)p * N] = x;
    }
  }
}

// C (M x N) = beta C + alpha A B over `nsys` systems of N x N row-major matrices (leading dimension ld)
struct Product {
  int nsys, ld;
  cudaStream_t st;
  int launches = 0;
  void operator()(int M, int N, int K, const double2* A, bool a_trans, const double2* B, bool b_trans, double2* C,
                  double alpha, double beta, int inplace = 0, long a_sys = -1, int a_ld = 0) {
    if (M <= 0 || N <= 0 || K <= 0) return;
    ZgemmDesc d;
    d.M = M; d.N = N; d.K = K;
    d.A = A; d.a_m.lo = a_trans ? 1 : (a_ld ? a_ld : ld); d.a_k = a_trans ? ld : 1;
    d.B = B; d.b_n.lo = b_trans ? ld : 1; d.b_k = b_trans ? 1 : ld; d.conjB = b_trans ? 1 : 0;
    d.C = C; d.c_m.lo = ld; d.c_n.lo = 1;
    d.nb0 = nsys;
    d.a_b0 = a_sys >= 0 ? a_sys : (long)ld * ld;
    d.b_b0 = d.c_b0 = (long)ld * ld;
    d.alpha = make_double2(alpha, 0.0);
    d.beta = make_double2(beta, 0.0);
    d.inplace = inplace;
    launches += zgemm(d, st);
  }
};

// X = P A^{-1} from the right (P Hermitian, so X = (A^{-1} P)^H, which is what the reference's
// column-major solve leaves in row-major terms): A = L L^H, Y L^H = P, X L = Y, by column blocks.
int cholesky(double2* P, double2* A, int* info, int nsys, int N, cudaStream_t st) {
  Product mul{nsys, N, st};
  int launches = 0;
  for (int j0 = 0; j0 < N; j0 += CB) {
    const int jb = std::min(CB, N - j0), j1 = j0 + jb;
    const double2* Lj = A + (long)j0 * N;         // rows of the block: L_j,0..j
    double2* D = A + (long)j0 * N + j0;           // diagonal block, then its inverse
    mul(N - j0, jb, j0, Lj, false, Lj, true, D, -1.0, 1.0);
    chol_block_kernel<<<nsys, TPB, 0, st>>>(A, info, N, j0, jb);
    GG_CHECK_LAUNCH();
    ++launches;
    double2* below = A + (long)j1 * N + j0;
    mul(N - j1, jb, jb, below, false, D, true, below, 1.0, 0.0, 1);
    mul(N, jb, j0, P, false, Lj, true, P + j0, -1.0, 1.0);
    mul(N, jb, jb, P + j0, false, D, true, P + j0, 1.0, 0.0, 1);
  }
  for (int j0 = (N - 1) / CB * CB; j0 >= 0; j0 -= CB) {
    const int jb = std::min(CB, N - j0), j1 = j0 + jb;
    mul(N, jb, N - j1, P + j1, false, A + (long)j1 * N + j0, false, P + j0, -1.0, 1.0);
    mul(N, jb, jb, P + j0, false, A + (long)j0 * N + j0, false, P + j0, 1.0, 0.0, 1);
  }
  return launches + mul.launches;
}

// P A = L U by panels (right-looking), then the forward and backward solves by row blocks
int lu(double2* P, double2* A, double2* li, int* info, int* piv, int nsys, int N, cudaStream_t st) {
  static_assert(3 * 32 * 33 * 16 <= LU_SMEM, "block inverses");
  Product mul{nsys, N, st};
  int launches = 0;
  const int nb = dyson_lu_block(N);
  const int in_smem = (long)(N | 1) * nb * 16 <= LU_SMEM;
  const size_t smem = std::max<size_t>(in_smem ? (size_t)(N | 1) * nb * 16 : 0, 3 * 32 * 33 * 16);
  GG_CUDA(cudaFuncSetAttribute(lu_panel_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LU_SMEM));
  auto li_of = [&](int j0) { return li + (long)j0 * nb; };
  const long li_sys = (long)ceil_div(N, nb) * nb * nb;
  for (int j0 = 0; j0 < N; j0 += nb) {
    const int jb = std::min(nb, N - j0), j1 = j0 + jb;
    lu_panel_kernel<<<nsys, TPB, smem, st>>>(A, li_of(j0), li_sys, piv, info, N, j0, jb, in_smem);
    GG_CHECK_LAUNCH();
    lu_swap_kernel<<<dim3(ceil_div(N, 64), nsys, 2), 64, 0, st>>>(A, P, piv, N, j0, jb);
    GG_CHECK_LAUNCH();
    launches += 2;
    double2* U = A + (long)j0 * N + j1;
    mul(jb, N - j1, jb, li_of(j0), false, U, false, U, 1.0, 0.0, 2, li_sys, jb);
    mul(N - j1, N - j1, jb, A + (long)j1 * N + j0, false, U, false, A + (long)j1 * N + j1, -1.0, 1.0);
  }
  for (int j0 = 0; j0 < N; j0 += nb) {
    const int jb = std::min(nb, N - j0);
    double2* row = P + (long)j0 * N;
    mul(jb, N, j0, A + (long)j0 * N, false, P, false, row, -1.0, 1.0);
    mul(jb, N, jb, li_of(j0), false, row, false, row, 1.0, 0.0, 2, li_sys, jb);
  }
  for (int j0 = (N - 1) / nb * nb; j0 >= 0; j0 -= nb) {
    const int jb = std::min(nb, N - j0), j1 = j0 + jb;
    double2* row = P + (long)j0 * N;
    mul(jb, N, N - j1, A + (long)j0 * N + j1, false, P + (long)j1 * N, false, row, -1.0, 1.0);
    mul(jb, N, jb, A + (long)j0 * N + j0, false, row, false, row, 1.0, 0.0, 2);
  }
  return launches + mul.launches;
}

void hermitize(double2* P, double2* A, int* info, int nsys, int N, int lower, cudaStream_t st) {
  const int t = ceil_div(N, 32);
  hermitize_kernel<<<dim3(nsys, t * (t + 1) / 2), TPB, 0, st>>>(P, A, info, N, lower);
  GG_CHECK_LAUNCH();
}

}  // namespace

// LU block: 32 columns, or 16 where a panel of 32 does not fit shared memory
int dyson_lu_block(int N) { return (long)(N | 1) * 32 * 16 <= LU_SMEM ? 32 : 16; }

int launch_dyson(double2* P, double2* A, double2* li, int* info, int nsys, int N, int solver, int* piv, cudaStream_t st) {
  if (nsys <= 0) return 0;
  const bool chol = solver == GG_SOLVER_CHOLESKY;
  hermitize(P, A, info, nsys, N, chol ? 1 : 0, st);
  if (chol) return 1 + cholesky(P, A, info, nsys, N, st);
  const int n = lu(P, A, li, info, piv, nsys, N, st);
  hermitize(P, nullptr, nullptr, nsys, N, 0, st);  // cugw_qpt.cu:314-316
  return 2 + n;
}

void launch_hermitian_symmetrize(double2* P, int nsys, int N, cudaStream_t st) {
  if (nsys > 0) hermitize(P, nullptr, nullptr, nsys, N, 0, st);
}

}  // namespace gg
