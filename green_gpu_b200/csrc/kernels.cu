// Non-GEMM device kernels: gathers, symmetry helpers, spin blocks, Hartree term (Dyson solvers: dyson.cu).
#include "kernels.cuh"

#include <algorithm>

namespace gg {
namespace {

constexpr int TPB = 256;

__global__ void gather_pairs_kernel(const double2* __restrict__ S, const int64_t* __restrict__ pos,
                                    const int* __restrict__ op, int NQ, int n, double2* __restrict__ out) {
  // one block per (pair, Q); 32x32 tiles through shared memory for the transposed case
  __shared__ double2 tile[32][33];
  const int pq = blockIdx.x;
  const int p = pq / NQ, Q = pq % NQ;
  const double2* src = S + (pos[p] * NQ + Q) * (long)n * n;
  double2* dst = out + ((long)p * NQ + Q) * n * n;
  const int o = op[p];
  const bool cj = o & 1, tr = (o >> 1) & 1;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;  // 32 x 8
  for (int i0 = 0; i0 < n; i0 += 32)
    for (int j0 = 0; j0 < n; j0 += 32) {
      if (!tr) {
        for (int r = ty; r < 32; r += 8) {
          int i = i0 + r, j = j0 + tx;
          if (i < n && j < n) {
            double2 v = src[(long)i * n + j];
            dst[(long)i * n + j] = cj ? cconj(v) : v;
          }
        }
      } else {
        // dst[i][j] = src[j][i]: read rows of src (i index = j0..), write rows of dst
        for (int r = ty; r < 32; r += 8) {
          int si = j0 + r, sj = i0 + tx;  // src element (si, sj) -> dst (sj, si)
          tile[r][tx] = (si < n && sj < n) ? src[(long)si * n + sj] : make_double2(0, 0);
        }
        __syncthreads();
        for (int r = ty; r < 32; r += 8) {
          int i = i0 + r, j = j0 + tx;
          if (i < n && j < n) {
            double2 v = tile[tx][r];
            dst[(long)i * n + j] = cj ? cconj(v) : v;
          }
        }
        __syncthreads();
      }
    }
}

__global__ void gather_g_kernel(const double2* __restrict__ G, const int* __restrict__ f2r, int nk, int ns, int nts,
                                int ink, int n, double2* __restrict__ out) {
  const long nn = (long)n * n;
  const long total = (long)nk * ns * nts * nn;
  for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total; idx += (long)gridDim.x * blockDim.x) {
    long e = idx % nn;
    long r = idx / nn;
    int t = (int)(r % nts);
    r /= nts;
    int s = (int)(r % ns);
    int k = (int)(r / ns);
    out[idx] = G[(((long)t * ns + s) * ink + f2r[k]) * nn + e];
  }
}

__global__ void conj_where_kernel(double2* X, const int* tr, int nk, long per_k) {
  const long total = (long)nk * per_k;
  for (long idx = blockIdx.x * (long)blockDim.x + threadIdx.x; idx < total; idx += (long)gridDim.x * blockDim.x) {
    if (tr[idx / per_k]) X[idx].y = -X[idx].y;
  }
}

__global__ void gather_blocks_kernel(const double2* __restrict__ src, const int* __restrict__ idx, long elems,
                                     long stride, int nblocks, double2* __restrict__ out) {
  const long total = (long)nblocks * elems;
  for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < total; i += (long)gridDim.x * blockDim.x) {
    long b = i / elems, e = i % elems;
    out[i] = src[(long)idx[b] * stride + e];
  }
}

__global__ void transpose_blocks_kernel(const double2* __restrict__ in, int n, int tiles, double2* __restrict__ out) {
  __shared__ double2 t[32][33];
  const long b = blockIdx.y;
  const int ti = blockIdx.x / tiles, tj = blockIdx.x % tiles;
  const double2* src = in + b * (long)n * n;
  double2* dst = out + b * (long)n * n;
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int i = ti * 32 + r, j = tj * 32 + threadIdx.x;
    if (i < n && j < n) t[r][threadIdx.x] = src[(long)i * n + j];
  }
  __syncthreads();
  for (int r = threadIdx.y; r < 32; r += 8) {
    const int j = tj * 32 + r, i = ti * 32 + threadIdx.x;
    if (i < n && j < n) dst[(long)j * n + i] = t[threadIdx.x][r];
  }
}

// One CTA per matrix (blockIdx.x = (t * ns + s) * ink + k): clears *flag unless G[t][s][k] and G[t][s'][k]^H agree
// within tol of the largest element of either, s' = s or, with `swap` (X2C spin blocks), 0, 1, 3, 2
__global__ void __launch_bounds__(128) hermitian_check_kernel(const double2* __restrict__ G, int ns, int ink, int n, int swap,
                                                              double tol, int* flag) {
  __shared__ double red[2][4];
  const long nn = (long)n * n;
  const long b = blockIdx.x;
  const int s = (int)((b / ink) % ns), p = swap && s >= 2 ? 5 - s : s;
  const double2* X = G + b * nn;
  const double2* Y = X + (long)(p - s) * ink * nn;
  double big = 0.0, off = 0.0;
  bool bad = false;
  for (int e = threadIdx.x; e < nn; e += 128) {
    const int i = e / n, j = e - i * n;
    const double2 x = X[e], y = Y[(long)j * n + i];
    const double m = fmax(fmax(fabs(x.x), fabs(x.y)), fmax(fabs(y.x), fabs(y.y)));
    const double dr = fabs(x.x - y.x), di = fabs(x.y + y.y);
    bad = bad || !(dr <= 1e300) || !(di <= 1e300);  // NaN and infinities, each by itself: fmax drops a NaN
    big = fmax(big, m);
    off = fmax(off, fmax(dr, di));
  }
  for (int o = 16; o > 0; o >>= 1) {
    big = fmax(big, __shfl_xor_sync(0xffffffffu, big, o));
    off = fmax(off, __shfl_xor_sync(0xffffffffu, off, o));
  }
  if ((threadIdx.x & 31) == 0) {
    red[0][threadIdx.x >> 5] = big;
    red[1][threadIdx.x >> 5] = off;
  }
  const int any_bad = __syncthreads_or(bad);
  if (threadIdx.x == 0) {
    for (int w = 1; w < 4; ++w) {
      big = fmax(big, red[0][w]);
      off = fmax(off, red[1][w]);
    }
    if (any_bad || off > tol * big) *flag = 0;
  }
}

// One CTA per matrix b = (k * ns + s) * nts + t, b < nmat (fastest), and 32 x 32 tile: H = (G + G'^H) / 2 where *flag, else G, with
// G'(s) as in the check.  Reads every tile and its mirror once each, through shared memory (HBM-bound).
__global__ void __launch_bounds__(TPB) hermitian_part_kernel(const double2* __restrict__ G, int nmat, int ns, int nts, int n,
                                                             int swap, const int* flag, double2* __restrict__ H) {
  __shared__ double2 m[32][33];
  const int tiles = (n + 31) / 32, tile = blockIdx.x / nmat, ti = tile / tiles, tj = tile % tiles;
  const long b = blockIdx.x % nmat, nn = (long)n * n;
  const int s = (int)((b / nts) % ns), p = swap && s >= 2 ? 5 - s : s;
  const double2* X = G + b * nn;
  const double2* Y = X + (long)(p - s) * nts * nn;
  const bool half = *flag != 0;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  if (half)
    for (int r = ty; r < 32; r += 8) {
      const int i = tj * 32 + r, j = ti * 32 + tx;
      if (i < n && j < n) m[r][tx] = Y[(long)i * n + j];
    }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int i = ti * 32 + r, j = tj * 32 + tx;
    if (i >= n || j >= n) continue;
    double2 x = X[(long)i * n + j];
    if (half) {
      const double2 y = m[tx][r];
      x = make_double2(0.5 * (x.x + y.x), 0.5 * (x.y - y.y));
    }
    H[b * nn + (long)i * n + j] = x;
  }
}

// where *flag: X[b][i][j] = conj(X[b][j][i]) above the diagonal and a real diagonal; one CTA per matrix
// (fastest) and 32 x 32 tile pair
__global__ void __launch_bounds__(TPB) mirror_lower_kernel(double2* X, int nmat, int n, const int* flag) {
  __shared__ double2 s[32][33];
  if (!*flag) return;
  int ti = 0, tj = blockIdx.x / nmat;
  while (tj > ti) tj -= ++ti;  // tile row ti >= tile column tj
  double2* M = X + blockIdx.x % nmat * (long)n * n;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (int r = ty; r < 32; r += 8) {
    const int i = ti * 32 + r, j = tj * 32 + tx;
    if (i < n && j < n) s[r][tx] = M[(long)i * n + j];
  }
  __syncthreads();
  for (int r = ty; r < 32; r += 8) {
    const int i = tj * 32 + r, j = ti * 32 + tx;
    if (i < n && j < n && j >= i) M[(long)i * n + j] = i == j ? make_double2(s[r][r].x, 0.0) : cconj(s[tx][r]);
  }
}

inline unsigned grid_for(long n, int tpb = TPB) {
  long b = (n + tpb - 1) / tpb;
  return (unsigned)std::max(1L, std::min(b, 148L * 32));
}

// One CTA per (Q, k): cp[k][Q] = sum_{s < nsj} Tr(V^Q(k,k) D_s(k)), V(k,k) = op(stored).  The stored
// matrix is read in its own order, so that the pass streams the integrals once (HBM-bound); the
// element of D that meets S[r][c] is D[c][r], or D[r][c] under a transpose.
__global__ void __launch_bounds__(128) hartree_coeff_kernel(const double2* __restrict__ S, const int64_t* __restrict__ pos,
                                                            const int* __restrict__ op, const double2* __restrict__ D, int NQ,
                                                            int n, int ns, int nsj, double2* __restrict__ cp) {
  __shared__ double2 red[4];
  const int Q = blockIdx.x, k = blockIdx.y;
  const int nn = n * n;
  const double2* v = S + (pos[k] * NQ + Q) * (long)nn;
  const double2* d = D + (long)k * ns * nn;
  const bool cj = op[k] & 1, tr = (op[k] >> 1) & 1;
  double2 acc = make_double2(0, 0);
  for (int e = threadIdx.x; e < nn; e += 128) {
    const int r = e / n, c = e - r * n;
    double2 x = v[e];
    if (cj) x.y = -x.y;
    for (int s = 0; s < nsj; ++s) acc = cadd(acc, cmul(x, d[(long)s * nn + (tr ? e : c * n + r)]));
  }
  for (int o = 16; o > 0; o >>= 1) {
    acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
    acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
  }
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) cp[(long)k * NQ + Q] = cadd(cadd(red[0], red[1]), cadd(red[2], red[3]));
}

// c[Q] = scale sum_k cp[k][Q], in the order of k
__global__ void hartree_sum_kernel(const double2* __restrict__ cp, int nk, int NQ, double scale, double2* __restrict__ c) {
  const int Q = blockIdx.x * blockDim.x + threadIdx.x;
  if (Q >= NQ) return;
  double2 acc = make_double2(0, 0);
  for (int k = 0; k < nk; ++k) acc = cadd(acc, cp[(long)k * NQ + Q]);
  c[Q] = cscale(acc, scale);
}

// F[s][kr] += op(sum_Q c[Q] S[Q]) for s < nsj: one CTA per (32 elements, kr), eight warps sharing the Q
__global__ void __launch_bounds__(256) hartree_apply_kernel(const double2* __restrict__ S, const int64_t* __restrict__ pos,
                                                            const int* __restrict__ op, const int* __restrict__ k_r2f,
                                                            const double2* __restrict__ c, int ink, int NQ, int n, int nsj,
                                                            double2* __restrict__ F) {
  __shared__ double2 red[8][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int kr = blockIdx.y, k = k_r2f[kr], nn = n * n, e = blockIdx.x * 32 + lane;
  const bool cj = op[k] & 1, tr = (op[k] >> 1) & 1;
  const double2* v = S + pos[k] * NQ * (long)nn;
  double2 acc = make_double2(0, 0);
  if (e < nn)
    for (int Q = w; Q < NQ; Q += 8) {
      double2 x = v[(long)Q * nn + e];
      if (cj) x.y = -x.y;
      acc = cadd(acc, cmul(c[Q], x));
    }
  red[w][lane] = acc;
  __syncthreads();
  if (w != 0 || e >= nn) return;
  for (int i = 1; i < 8; ++i) acc = cadd(acc, red[i][lane]);
  const int r = e / n, q = e - r * n, o = tr ? q * n + r : e;
  for (int s = 0; s < nsj; ++s) {
    double2* f = F + ((long)s * ink + kr) * nn + o;
    *f = cadd(*f, acc);
  }
}

}  // namespace

void launch_gather_pairs(const double2* S, const int64_t* pos_d, const int* op_d, int npairs, int NQ, int n,
                         double2* out, cudaStream_t st) {
  if (npairs <= 0) return;
  gather_pairs_kernel<<<npairs * NQ, 256, 0, st>>>(S, pos_d, op_d, NQ, n, out);
  GG_CHECK_LAUNCH();
}

void launch_gather_g(const double2* G, const int* f2r, int nk, int ns, int nts, int ink, int n, double2* out,
                     cudaStream_t st) {
  long total = (long)nk * ns * nts * n * n;
  gather_g_kernel<<<grid_for(total), TPB, 0, st>>>(G, f2r, nk, ns, nts, ink, n, out);
  GG_CHECK_LAUNCH();
}

void launch_conj_where(double2* X, const int* tr, int nk, long per_k, cudaStream_t st) {
  conj_where_kernel<<<grid_for((long)nk * per_k), TPB, 0, st>>>(X, tr, nk, per_k);
  GG_CHECK_LAUNCH();
}

void launch_gather_blocks(const double2* src, const int* idx, int nblocks, long elems, long stride, double2* out,
                          cudaStream_t st) {
  if (nblocks <= 0) return;
  gather_blocks_kernel<<<grid_for((long)nblocks * elems), TPB, 0, st>>>(src, idx, elems, stride, nblocks, out);
  GG_CHECK_LAUNCH();
}

namespace {
__device__ __forceinline__ void x2c_block(int ss, int& a, int& b) {
  a = ss & 1;
  b = (ss == 1 || ss == 2) ? 1 : 0;
}

__global__ void x2c_split_kernel(const double2* in, long nouter, long ninner, int n, int nblk, double2* out) {
  const long nn = (long)n * n, total = nouter * nblk * ninner * nn;
  const int n2 = 2 * n;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const long ij = e % nn;
    long r = e / nn;
    const long kin = r % ninner;
    r /= ninner;
    const int ss = (int)(r % nblk);
    const long o = r / nblk;
    int a, b;
    x2c_block(ss, a, b);
    const int i = (int)(ij / n), j = (int)(ij % n);
    out[e] = in[((o * ninner + kin) * n2 + a * n + i) * n2 + b * n + j];
  }
}

__global__ void x2c_merge_kernel(const double2* in, long nouter, long ninner, int n, int nblk, double2* out) {
  const int n2 = 2 * n;
  const long nn = (long)n * n, mm = (long)n2 * n2, total = nouter * ninner * mm;
  for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < total; e += (long)gridDim.x * blockDim.x) {
    const int J = (int)(e % n2), I = (int)((e / n2) % n2);
    const long r = e / mm, kin = r % ninner, o = r / ninner;
    const int a = I >= n, b = J >= n, i = I - a * n, j = J - b * n;
    // block index of (a, b): aa 0, bb 1, ab 2, ba 3
    const int ss = (a == b) ? a : (a == 0 ? 2 : 3);
    double2 v;
    if (ss == 3 && nblk == 3) {
      const double2 u = in[((o * nblk + 2) * ninner + kin) * nn + (long)j * n + i];
      v = make_double2(u.x, -u.y);
    } else {
      v = in[((o * nblk + ss) * ninner + kin) * nn + (long)i * n + j];
    }
    out[e] = v;
  }
}
}  // namespace

void launch_x2c_split(const double2* in, long nouter, long ninner, int n, int nblk, double2* out, cudaStream_t st) {
  x2c_split_kernel<<<grid_for(nouter * nblk * ninner * (long)n * n), TPB, 0, st>>>(in, nouter, ninner, n, nblk, out);
  GG_CHECK_LAUNCH();
}

void launch_x2c_merge(const double2* in, long nouter, long ninner, int n, int nblk, double2* out, cudaStream_t st) {
  x2c_merge_kernel<<<grid_for(nouter * ninner * 4L * n * n), TPB, 0, st>>>(in, nouter, ninner, n, nblk, out);
  GG_CHECK_LAUNCH();
}

namespace {
__global__ void __launch_bounds__(TPB) info_collect_kernel(const int* info, int count, int base, int* err) {
  __shared__ int first;
  if (threadIdx.x == 0) first = count;
  __syncthreads();
  for (int i = threadIdx.x; i < count; i += TPB)
    if (info[i] != 0) atomicMin(&first, i);
  __syncthreads();
  if (threadIdx.x == 0 && first < count && err[0] == 0) {
    err[0] = 1;
    err[1] = base + first;
    err[2] = info[first];
  }
}
}  // namespace

void launch_info_collect(const int* info, int count, int base, int* err, cudaStream_t st) {
  info_collect_kernel<<<1, TPB, 0, st>>>(info, count, base, err);
  GG_CHECK_LAUNCH();
}

void launch_transpose_blocks(const double2* in, long nblocks, int n, double2* out, cudaStream_t st) {
  if (nblocks <= 0 || n <= 0) return;
  if (nblocks > 65535) throw Error(GG_ERR_ARG, "transpose: too many blocks for one launch");
  const int tiles = (n + 31) / 32;
  transpose_blocks_kernel<<<dim3((unsigned)(tiles * tiles), (unsigned)nblocks), dim3(32, 8), 0, st>>>(in, n, tiles, out);
  GG_CHECK_LAUNCH();
}

void launch_hermitian_check(const double2* G, int nts, int ns, int ink, int n, int swap, double tol, int* flag,
                            cudaStream_t st) {
  GG_CUDA(cudaMemsetAsync(flag, 1, sizeof(int), st));
  hermitian_check_kernel<<<nts * ns * ink, 128, 0, st>>>(G, ns, ink, n, swap, tol, flag);
  GG_CHECK_LAUNCH();
}

void launch_hermitian_part(const double2* G, int nk, int ns, int nts, int n, int swap, const int* flag, double2* H,
                           cudaStream_t st) {
  const int t = ceil_div(n, 32);
  const int nmat = nk * ns * nts;
  hermitian_part_kernel<<<(unsigned)((long)nmat * t * t), TPB, 0, st>>>(G, nmat, ns, nts, n, swap, flag, H);
  GG_CHECK_LAUNCH();
}

void launch_mirror_lower(double2* X, int nmat, int n, const int* flag, cudaStream_t st) {
  const int t = ceil_div(n, 32);
  mirror_lower_kernel<<<(unsigned)((long)nmat * t * (t + 1) / 2), TPB, 0, st>>>(X, nmat, n, flag);
  GG_CHECK_LAUNCH();
}

void launch_hartree_coeff(const double2* S, const int64_t* pos_d, const int* op_d, const double2* D, int nk, int NQ, int n,
                          int ns, int nsj, double scale, double2* c, cudaStream_t st) {
  hartree_coeff_kernel<<<dim3(NQ, nk), 128, 0, st>>>(S, pos_d, op_d, D, NQ, n, ns, nsj, c + NQ);
  GG_CHECK_LAUNCH();
  hartree_sum_kernel<<<ceil_div(NQ, 64), 64, 0, st>>>(c + NQ, nk, NQ, scale, c);
  GG_CHECK_LAUNCH();
}

void launch_hartree_apply(const double2* S, const int64_t* pos_d, const int* op_d, const int* k_r2f_d, const double2* c,
                          int ink, int NQ, int n, int nsj, double2* F, cudaStream_t st) {
  hartree_apply_kernel<<<dim3(ceil_div((long)n * n, 32), ink), 256, 0, st>>>(S, pos_d, op_d, k_r2f_d, c, ink, NQ, n, nsj, F);
  GG_CHECK_LAUNCH();
}

}  // namespace gg
