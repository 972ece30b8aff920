// FP64 complex GEMM for products too small to fill the GPU (see zgemm.cuh).
//
// One CTA of four warps per 8 x 8 tile; the warps share the reduction and add their partial tiles in order
// through shared memory.  Fragments go from global memory straight to registers, CH groups of 4 at a
// time: nothing is reused inside a CTA that would pay for staging, and what bounds such a product is
// latency - the launch, a round of loads, a few DMMAs - which a staged pipeline lengthens.  Against the best staged
// tile: 52^3 6.9 -> 5.2 us, 64 x 64 x 200 11.3 -> 6.8, 100^3 9.2 -> 5.8, eight of 20 x 20 x 120 9.3 -> 5.1.
#include <atomic>

#include "dmma.cuh"
#include "zgemm_kernel.cuh"

namespace gg {
namespace {

__global__ void __launch_bounds__(128) zgemm_small_kernel(const __grid_constant__ ZgemmDesc d, ZGrid g) {
  constexpr int CH = 8;
  __shared__ double2 part[3][8][8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int fr = lane >> 2, fk = lane & 3;
  const ZItem w = zitem(d, g.tiles_m * g.tiles_n, blockIdx.x);
  const int tn = (int)((unsigned)w.tile / (unsigned)g.tiles_m), tm = w.tile - tn * g.tiles_m;
  const int ma = tm * 8 + fr, nb = tn * 8 + fr;  // this lane's row of A and column of B
  const bool oka = ma < d.M, okb = nb < d.N;
  const double2* A = d.A + w.b0 * d.a_b0 + w.b1 * d.a_b1 + w.b2 * d.a_b2 + fk * d.a_k + (oka ? zmap(d.a_m, ma) : 0);
  const double2* B = d.B + w.b0 * d.b_b0 + w.b1 * d.b_b1 + w.b2 * d.b_b2 + fk * d.b_k + (okb ? zmap(d.b_n, nb) : 0);
  const int sa = d.conjA ? (int)0x80000000 : 0, sb = d.conjB ? (int)0x80000000 : 0;
  double cr[2] = {0.0, 0.0}, ci[2] = {0.0, 0.0};
  const int g1 = (int)((long)g.groups * (warp + 1) / 4);
  int grp = (int)((long)g.groups * warp / 4);
  int kb = grp / g.gpb, kin = grp - kb * g.gpb;
  for (; grp < g1; grp += CH) {
    double2 a[CH], b[CH];
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      const bool v = grp + c < g1 && 4 * kin + fk < d.K;
      a[c] = v && oka ? A[kb * d.a_kb + 4L * kin * d.a_k] : make_double2(0.0, 0.0);
      b[c] = v && okb ? B[kb * d.b_kb + 4L * kin * d.b_k] : make_double2(0.0, 0.0);
      if (++kin == g.gpb) {
        kin = 0;
        ++kb;
      }
    }
#pragma unroll
    for (int c = 0; c < CH; ++c) {
      if (grp + c >= g1) break;
      const double ai = zflip(a[c].y, sa), bi = zflip(b[c].y, sb);
      dmma(cr[0], cr[1], a[c].x, b[c].x);
      dmma(ci[0], ci[1], a[c].x, bi);
      dmma(cr[0], cr[1], -ai, bi);
      dmma(ci[0], ci[1], ai, b[c].x);
    }
  }
  if (warp > 0) {
#pragma unroll
    for (int e = 0; e < 2; ++e) part[warp - 1][fr][2 * fk + e] = make_double2(cr[e], ci[e]);
  }
  __syncthreads();
  if (warp > 0 || !oka) return;
  const bool use_beta = d.beta.x != 0.0 || d.beta.y != 0.0;
  double2* const row = d.C + w.b0 * d.c_b0 + w.b1 * d.c_b1 + w.b2 * d.c_b2 + zmap(d.c_m, ma);
#pragma unroll
  for (int e = 0; e < 2; ++e) {
    const int n = tn * 8 + 2 * fk + e;
    if (n >= d.N) continue;
    double2 v = make_double2(cr[e], ci[e]);
#pragma unroll
    for (int p = 0; p < 3; ++p) v = cadd(v, part[p][fr][2 * fk + e]);
    v = cmul(d.alpha, v);
    double2* c = row + zmap(d.c_n, n);
    if (use_beta) v = cadd(v, cmul(d.beta, *c));
    *c = v;
  }
}

}  // namespace

void zgemm_launch_small(const ZgemmDesc& d, const ZGrid& g, cudaStream_t st) {
  zgemm_small_kernel<<<(unsigned)g.items, 128, 0, st>>>(d, g);
  GG_CHECK_LAUNCH();
}

}  // namespace gg
