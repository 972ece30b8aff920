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
#include <type_traits>

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
// triangle only when `lower`.  One CTA per system (fastest) and pair of 32 x 32 tiles, in one grid dimension since
// N > 11552 has more pairs than the second one takes: both tiles pass through shared memory,
// so that every access to global memory is a run of 32 elements.
__global__ void __launch_bounds__(TPB) hermitize_kernel(double2* Pall, double2* Aall, int* info, int nsys, int N, int lower) {
  __shared__ double2 lo[32][33], up[32][33];
  const int sys = blockIdx.x % nsys;
  int ti = 0, p = blockIdx.x / nsys;
  if (info && p == 0 && threadIdx.x == 0) info[sys] = 0;
  while (p > ti) p -= ++ti;  // pair (ti, p), p <= ti
  const int tj = p;  // tj <= ti
  const long NN = (long)N * N;
  double2* P = Pall + sys * NN;
  double2* A = Aall ? Aall + sys * NN : nullptr;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
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
// (16 x 64 per thread) and the chain pivot - reciprocal root - update: 552 blocks of 64 in 154 us.
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
    const double inv = rsqrt(d);  // L_cc itself is not needed
    // multiplier of column k: the inverse's row c (k < c), 1 / L_cc (k = c), conj L_kc (k > c)
    const double2 v = k < c ? cscale(rs[k], inv) : k == c ? make_double2(inv, 0.0) : cconj(cscale(cs[k], inv));
    const double2 m = cscale(v, -inv);  // rows below take L_rc v = cs[r] inv v off
#pragma unroll
    for (int i = 0; i < CB / 4; ++i) {
      const int r = ty + 4 * i;
      if (r > c) {
        const double2 l = cs[r];
        const double2 x = k == c ? make_double2(0.0, 0.0) : a[i];
        a[i].x = fma(l.x, m.x, fma(-l.y, m.y, x.x));
        a[i].y = fma(l.x, m.y, fma(l.y, m.x, x.y));
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

// LU panel: columns j0 .. j0 + nb - 1 (nb <= 32), rows j0 .. N - 1 of one system, with partial pivoting (largest
// |re| + |im|, the lowest row on ties), element (row r, column c) of the panel at pan[c * cs + r * rs]: in
// shared memory by columns when it fits, else in place.  Leaves L below the diagonal block, the
// block's U^{-1} in its place (zeros below), L^{-1} of the block in li (unit diagonal, zeros above),
// and the row interchanges (absolute rows) in piv.
// Bound by the chain of columns (FP64 latencies, not throughput).  Warp k % 8 owns column k, lanes go down the
// rows; the owner of column c + 1 updates it first, finds its pivot within the warp and scales it while
// the other warps still apply column c, so that a column costs one barrier.  With all threads on rows, a
// block-wide FP64 search and two barriers per column a panel of 69 systems of N = 140 took 67 us, now 54;
// of 552 systems of N = 120 159 and 129 us.
__device__ __forceinline__ double2 cinv(double2 d) {
  const double dn = d.x * d.x + d.y * d.y;
  if (!(dn > 0.0)) return make_double2(0.0, 0.0);
  // 1 / dn overflows for |d| below 7e-155, where the inverse itself is still finite: quotients there (everywhere they
  // would lengthen the chain of columns: gamma-point build of NQ 140 1.36 -> 1.39 ms)
  if (dn < 0x1p-1000) return make_double2(d.x / dn, -d.y / dn);
  const double f = 1.0 / dn;
  return make_double2(d.x * f, -d.y * f);
}

__global__ void __launch_bounds__(TPB, 2) lu_panel_kernel(double2* Aall, double2* li_all, long li_sys, int* piv_all, int* info,
                                                       int N, int j0, int nb, int in_smem) {
  extern __shared__ __align__(16) double2 dsm[];
  __shared__ int s_piv[32];
  __shared__ int s_fail;
  constexpr int W = TPB / 32;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double2* A = Aall + blockIdx.x * (long)N * N + (long)j0 * N + j0;
  const int R = N - j0;
  const long cs = in_smem ? (R | 1) : 1, rs = in_smem ? 1 : N;
  double2* pan = in_smem ? dsm : A;
  if (tid == 0) s_fail = 0;
  if (in_smem && lane < nb)
    for (int r = warp; r < R; r += W) pan[lane * cs + r] = A[(long)r * N + lane];
  __syncthreads();
  // pivot of column c (owner warp only): search rows >= c, interchange inside the column, scale
  auto pivot = [&](int c) {
    double2* col = pan + c * cs;
    // magnitudes compared as the bits of non-negative doubles: three warp reductions (high word, low
    // word, lowest row) instead of five rounds of FP64 comparisons; a NaN counts as zero
    unsigned hi = 0, lo = 0;
    int bi = c;
    for (int r = lane; r < R; r += 32) {
      const double2 x = col[r * rs];
      const double m = fabs(x.x) + fabs(x.y);
      const unsigned long long bits = r >= c && m == m ? __double_as_longlong(m) : 0;
      const unsigned h = (unsigned)(bits >> 32), w = (unsigned)bits;
      if (h > hi || (h == hi && w > lo)) {
        hi = h;
        lo = w;
        bi = r;
      }
    }
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    const bool some = mh != 0 || ml != 0;
    const int p = some ? (int)__reduce_min_sync(0xffffffffu, hi == mh && lo == ml ? (unsigned)bi : 0xffffffffu) : c;
    const double2 d = col[p * rs];
    const double2 top = col[c * rs];
    __syncwarp();
    if (lane == 0) {
      col[p * rs] = top;
      col[c * rs] = d;
      s_piv[c] = p;
      if (!some && s_fail == 0) s_fail = j0 + c + 1;
    }
    __syncwarp();
    const double2 inv = cinv(d);
    for (int r0 = lane; r0 < R; r0 += 128) {
      double2 x[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = r0 + 32 * i < R ? col[(r0 + 32 * i) * rs] : make_double2(0.0, 0.0);
#pragma unroll
      for (int i = 0; i < 4; ++i) x[i] = cmul(x[i], inv);
#pragma unroll
      for (int i = 0; i < 4; ++i)
        if (r0 + 32 * i > c && r0 + 32 * i < R) col[(r0 + 32 * i) * rs] = x[i];
    }
  };
  // column c applied to Q of this warp's columns, k0, k0 + W, ...: all loads of a step before its stores,
  // so that the FP64 latencies overlap
  auto update = [&](int c, int k0, auto count) {
    constexpr int Q = decltype(count)::value;
    const double2* l = pan + c * cs;
    double2 u[Q];
    double2* col[Q];
    bool ok[Q];
#pragma unroll
    for (int q = 0; q < Q; ++q) {
      ok[q] = k0 + W * q < nb;
      col[q] = pan + (ok[q] ? k0 + W * q : c) * cs;
      u[q] = col[q][c * rs];
    }
    for (int r0 = lane; r0 < R; r0 += 64) {
      double2 lv[2], x[2][Q];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = r0 + 32 * i < R ? r0 + 32 * i : R - 1;
        lv[i] = l[r * rs];
#pragma unroll
        for (int q = 0; q < Q; ++q) x[i][q] = col[q][r * rs];
      }
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int r = r0 + 32 * i;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
          x[i][q] = csub(x[i][q], cmul(lv[i], u[q]));
          if (ok[q] && r > c && r < R) col[q][r * rs] = x[i][q];
        }
      }
    }
  };
  if (warp == 0) pivot(0);
  __syncthreads();
  for (int c = 0; c < nb; ++c) {
    const int p = s_piv[c];
    const int k = warp + W * lane;  // the warp's columns: one lane interchanges each
    if (k < nb && k != c && p != c) {
      const double2 x = pan[k * cs + c * rs];
      pan[k * cs + c * rs] = pan[k * cs + p * rs];
      pan[k * cs + p * rs] = x;
    }
    __syncwarp();
    const bool next = c + 1 < nb && (c + 1) % W == warp;
    if (next) {
      update(c, c + 1, std::integral_constant<int, 1>());
      __syncwarp();
      pivot(c + 1);
    }
    // the warp's columns beyond c (and beyond c + 1 where that one is done), from the first such k
    const int first = c + (next ? 2 : 1);
    const int k0 = first + (warp - first % W + W) % W, left = (nb - k0 + W - 1) / W;
    if (left > 2) update(c, k0, std::integral_constant<int, 4>());
    else if (left == 2) update(c, k0, std::integral_constant<int, 2>());
    else if (left == 1) update(c, k0, std::integral_constant<int, 1>());
    __syncthreads();
  }
  int* piv = piv_all + (long)blockIdx.x * N + j0;
  if (tid < nb) piv[tid] = j0 + s_piv[tid];
  if (in_smem && lane < nb)
    for (int r = nb + warp; r < R; r += W) A[(long)r * N + lane] = pan[lane * cs + r];
  // the block's inverses X = L^{-1} and Y = U^{-1}, built by row operations on the identity: T holds L below the
  // diagonal and U D^{-1} above it (D the diagonal of U), Y's rows are scaled at the end
  double2 t[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = warp + W * i, c = lane;
    t[i] = r < nb && c < nb ? pan[c * cs + r * rs] : make_double2(r == c ? 1.0 : 0.0, 0.0);
    if (r < c && c < nb) t[i] = cmul(t[i], cinv(pan[c * cs + c * rs]));
  }
  __syncthreads();
  double2 (*T)[33] = reinterpret_cast<double2 (*)[33]>(dsm);
  double2 (*X)[33] = T + 32, (*Y)[33] = T + 64;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = warp + W * i, c = lane;
    T[r][c] = t[i];
    X[r][c] = Y[r][c] = make_double2(r == c ? 1.0 : 0.0, 0.0);
  }
  __syncthreads();
  for (int c = 0; c < nb; ++c) {
    const int b = nb - 1 - c;  // pivot row of the upper solve
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = warp + W * i, k = lane;
      if (r > c && k <= c) X[r][k] = csub(X[r][k], cmul(T[r][c], X[c][k]));
      if (r < b && k >= b) Y[r][k] = csub(Y[r][k], cmul(T[r][b], Y[b][k]));
    }
    __syncthreads();
  }
  double2* li = li_all + blockIdx.x * li_sys;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = warp + W * i, c = lane;
    if (r < nb && c < nb) {
      li[r * nb + c] = X[r][c];
      A[(long)r * N + c] = cmul(cinv(T[r][r]), Y[r][c]);
    }
  }
  if (tid == 0 && s_fail && info[blockIdx.x] == 0) info[blockIdx.x] = s_fail;
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
  hermitize_kernel<<<(unsigned)((long)nsys * t * (t + 1) / 2), TPB, 0, st>>>(P, A, info, nsys, N, lower);
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
