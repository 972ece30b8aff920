// Batched complex FP64 GEMM engine: choice of the tile shape and split-K factor, launch and the
// ordered split-K reduction (kernels: zgemm_kernel.cuh).
#include <algorithm>
#include <atomic>
#include <cmath>

#include "zgemm_kernel.cuh"

namespace gg {
namespace {

// C = alpha sum_s work[s] + beta C.  SL threads share the partial sums of an element (consecutive runs,
// then combined in order), eight loads in flight each, so that hundreds of partial sums of a small
// output are not one chain of loads.
template <int SL>
__global__ void __launch_bounds__(256) zgemm_reduce(ZgemmDesc d) {
  __shared__ double2 part[SL > 1 ? SL : 1][SL > 1 ? 256 / SL : 1];
  const long mn = (long)d.M * d.N, total = (long)d.nb0 * d.nb1 * d.nb2 * mn;
  const int lane = threadIdx.x % (256 / SL), sl = threadIdx.x / (256 / SL);
  const long i = blockIdx.x * (long)(256 / SL) + lane;
  double2 acc = make_double2(0.0, 0.0);
  if (i < total) {
    const double2* w = d.work + i;
    int s = d.splits * sl / SL;
    const int end = d.splits * (sl + 1) / SL;
    for (; s + 8 <= end; s += 8) {
      double2 p[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) p[j] = w[(s + j) * total];
#pragma unroll
      for (int j = 0; j < 8; ++j) acc = cadd(acc, p[j]);
    }
    for (; s < end; ++s) acc = cadd(acc, w[s * total]);
  }
  if constexpr (SL > 1) {
    part[sl][lane] = acc;
    __syncthreads();
    if (sl != 0) return;
    for (int j = 1; j < SL; ++j) acc = cadd(acc, part[j][lane]);
  }
  if (i >= total) return;
  const long batch = i / mn, e = i % mn;
  const int m = (int)(e / d.N), n = (int)(e % d.N);
  if (d.tri && *d.tri && n > m) return;
  const int b0 = (int)(batch % d.nb0), b1 = (int)((batch / d.nb0) % d.nb1), b2 = (int)(batch / ((long)d.nb0 * d.nb1));
  double2* c = d.C + b0 * d.c_b0 + b1 * d.c_b1 + b2 * d.c_b2 + d.c_m(m) + d.c_n(n);
  double2 v = cmul(d.alpha, acc);
  if (d.beta.x != 0.0 || d.beta.y != 0.0) v = cadd(v, cmul(d.beta, *c));
  *c = v;
}

// tiles on and below the diagonal of a square product
int tri_tiles(int tiles_m, int tiles_n, int bm, int bn) {
  int count = 0;
  for (int tn = 0; tn < tiles_n; ++tn) count += std::max(0, tiles_m - zfirst_row(tn, bm, bn));
  return count;
}

// Least split-K factor.  The rounding error of a sum grows with its length (120 x 120 x 5408: 2.7e-15 as one sum, 6.7e-16
// as four), so a four-product sum is cut until an accumulator adds up at most 128 groups, as far as the parts leave at
// most four 64 x 64 tiles per SM, 256 parts and room for them: beyond that the pass over the parts
// costs more (exchange of the Fock build 5.3 -> 5.5 ms with 547 parts instead of 296).  By time alone small tiles, which fill
// the GPU with few parts, have long sums: Sigma of nao 26, NQ 120 (P0 in 4 parts, now 11) was off by 5.3 to 8.4e-15 and is by
// 2.2 to 2.9e-15, of nao 36, NQ 250 (1 part, now 4) 3.3e-15 and 9.5e-16.  It costs 0 to 2 % of a build (spinors of
// 2 x 26 10.82 -> 10.92 ms; nao 26, NQ 120 33.9 -> 33.7).
long least_splits(const ZgemmDesc& d, long batch, long groups, int sms) {
  if (d.gauss || d.inplace || !d.work) return 1;
  const double out = (double)d.M * d.N * batch;
  const long tiles64 = (long)ceil_div(d.M, 64) * ceil_div(d.N, 64) * batch;
  const long parts = std::min(std::min((groups + 127) / 128, (4L * sms + tiles64 - 1) / tiles64), 256L);
  return std::max(1L, std::min(parts, std::min(groups / 8, (long)((double)d.work_elems / out))));
}

}  // namespace

// The choice minimises a cycle estimate fitted to timings of every shape and split on 33 of the
// library's products (outputs of 20..400 columns, reductions of 20..280000, batches of 1..72; the chosen
// one is within 2 % of the best measured one on average, 20 % at worst):
//   pipe   the SM with the most tiles issues tiles x warps/4 x groups x MT NT P DMMAs (P = 4 or 3
//          products) of 16 cycles on each sub-partition.  The pipe is busy 0.89 - 0.5 / (MT NT) of the
//          time (V^T W of NQ 400, nao 52, 72 tau: 7.54 ms on 64 x 80 tiles, 8.93 ms on 64 x 16), a fifth
//          less with three products, which add FP64 sums, and 10 % less on squares of one
//          warp per row of 8 x 8 tiles; a tile's output costs 100 cycles per 8 x 8 tile;
//   chain  groups of one tile follow one another: its DMMAs, or the copy warp's work, per group, and
//          about 6000 cycles from the first copy to the last store (a 52^3 product: 7.2 us on 16 tiles
//          of 16 x 16, 17.3 us on one of 64 x 64);
//   l2     operand tiles arrive at about 40 bytes per cycle and SM.
// Splitting the reduction multiplies the tiles and adds a launch and the pass over the partial sums.
ZChoice zgemm_choose(const ZgemmDesc& d, long batch, long groups, int sms) {
  static const int kSplits[] = {1, 2, 3, 4, 5, 6, 8, 10, 12, 16, 20, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512};
  const ZShape* const table = d.gauss ? kZShape3 : kZShape;
  const int count = d.gauss ? kZShapes3 : kZShapes;
  const double prods = d.gauss ? 3.0 : 4.0;
  const double out = (double)d.M * d.N * batch;
  const int least = (int)least_splits(d, batch, groups, sms);
  ZChoice best;
  double best_cost = 0.0;
  bool have = false;
  for (int i = 0; i < count; ++i) {
    const ZShape& s = table[i];
    const int tm = ceil_div(d.M, s.bm), tn = ceil_div(d.N, s.bn);
    if ((d.inplace == 1 && tn > 1) || (d.inplace == 2 && tm > 1)) continue;
    const double tiles = (double)(d.tri ? tri_tiles(tm, tn, s.bm, s.bn) : tm * tn) * batch;
    const int t88 = s.mt * s.nt;
    const double mma = t88 * prods * 16.0, busy =
        (0.89 - 0.5 / t88) * (d.gauss ? 0.8 : 1.0) * (s.square() ? 0.9 : 1.0);
    const double group = std::max(1.15 * mma + 100.0, 150.0 + 7.0 * (s.bm + s.bn));
    auto consider = [&](int sp) {
      if (sp < least) return;
      if (sp > 1 && (d.inplace || !d.work || groups / sp < 8 || out * sp > (double)d.work_elems)) return;
      const double g = (double)((groups + sp - 1) / sp), items = tiles * sp;
      const double per_sm = std::ceil(items / sms), waves = std::ceil(items / ((double)sms * s.teams));
      const double pipe = per_sm * s.warps / 4.0 * (g * mma / busy + 100.0 * t88);
      const double chain = waves * (g * group + 100.0 * t88 + 6000.0);
      const double l2 = per_sm * (s.bm + s.bn) * g * 64.0 / 40.0;
      double cost = std::max(std::max(pipe, chain), l2);
      if (sp > 1) cost += 7000.0 + 100.0 * std::min(sp, 64) + out * (sp + 1) * 16.0 / 3000.0;
      if (!have || cost < best_cost) {
        have = true;
        best_cost = cost;
        best.shape = i;
        best.splits = sp;
      }
    };
    for (int sp : kSplits) consider(sp);
    consider(least);
    // splits that fill whole rounds of SMs: with 256 of them over 148 SMs, 40 SMs have one CTA and the others two
    // (36 x 36 x 279936: 194 us, 171 us with 296; Z V^+ of nao 37, three products: 0.252 -> 0.229 ms)
    for (int r = 1; r <= 4; ++r) {
      const int sp = (int)(r * sms / tiles);
      if (sp > 1 && sp <= 512) consider(sp);
    }
  }
  if (!have) throw Error(GG_ERR_INTERNAL, "zgemm: no tile shape for an in-place product of this size");
  return best;
}

int current_device() {
  int dev = 0;
  GG_CUDA(cudaGetDevice(&dev));
  if (dev < 0 || dev >= kMaxDevices) throw Error(GG_ERR_ARG, "device index " + std::to_string(dev) + " out of range");
  return dev;
}

int device_sm_count() {
  static std::atomic<int> counts[kMaxDevices];
  const int dev = current_device();
  int n = counts[dev].load(std::memory_order_relaxed);
  if (!n) {
    GG_CUDA(cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev));
    counts[dev].store(n, std::memory_order_relaxed);
  }
  return n;
}

int zgemm(const ZgemmDesc& d0, cudaStream_t stream) {
  ZgemmDesc d = d0;
  if (d.M <= 0 || d.N <= 0 || d.nb0 <= 0 || d.nb1 <= 0 || d.nb2 <= 0) return 0;
  if (d.K < 0 || d.KB < 1) throw Error(GG_ERR_ARG, "zgemm: bad K");
  if (d.tri && d.M != d.N) throw Error(GG_ERR_INTERNAL, "zgemm: the lower triangle of a product that is not square");
  const long batch = (long)d.nb0 * d.nb1 * d.nb2;
  const int gpb = std::max(1, ceil_div(d.K, 4));
  const long groups = (long)d.KB * gpb;
  const int sms = device_sm_count();
  // one round of 8 x 8 tiles (four CTAs per SM) with at most 24 groups per warp: the latency-bound kernel (beyond
  // it the staged tiles win: eight of 100^3 10.6 against 13.3 us)
  const long tiles8 = (long)ceil_div(d.M, 8) * ceil_div(d.N, 8) * batch;
  if (tiles8 <= 4L * sms && groups <= 96 && !d.tri && !d.inplace) {
    ZGrid g = {};
    g.gpb = gpb;
    g.tiles_m = ceil_div(d.M, 8);
    g.tiles_n = ceil_div(d.N, 8);
    g.items = (int)tiles8;
    g.groups = (int)groups;
    d.splits = 1;
    zgemm_launch_small(d, g, stream);
    return 1;
  }
  if (d.a_k != 1) d.gauss = 0;  // the three-product kernels exist where split builds use them (k-contiguous A)
  const ZChoice ch = zgemm_choose(d, batch, groups, sms);
  d.splits = ch.splits;
  return zgemm_shape(d, ch.shape, stream);
}

int zgemm_shape(const ZgemmDesc& d, int shape, cudaStream_t stream) {
  const bool ak = (d.a_k == 1), bk = (d.b_k == 1);
  const ZShape& s = d.gauss ? kZShape3[shape] : kZShape[shape];
  const long batch = (long)d.nb0 * d.nb1 * d.nb2;
  const int sms = device_sm_count();
  ZGrid g = {};
  g.gpb = std::max(1, ceil_div(d.K, 4));
  const long groups = (long)d.KB * g.gpb;
  g.tiles_m = ceil_div(d.M, s.bm);
  g.tiles_n = ceil_div(d.N, s.bn);
  g.tri_tiles = tri_tiles(g.tiles_m, g.tiles_n, s.bm, s.bn);
  const long items = (long)g.tiles_m * g.tiles_n * d.splits * batch;
  if (items > 0x7fffffffL - 4096 || groups > 0x7fffffffL) throw Error(GG_ERR_ARG, "zgemm: grid too large");
  g.items = (int)items;
  g.groups = (int)groups;
  g.wrap_a = d.a_kb - 4L * (g.gpb - 1) * d.a_k;
  g.wrap_b = d.b_kb - 4L * (g.gpb - 1) * d.b_k;
  const long teams = std::min<long>(items, (long)sms * s.teams);
  // start the teams of a paired CTA a tile's DMMA time apart where they walk several short tiles (B-build of P0,
  // nao 52, NQ 400: 0.96 -> 0.86 ms on 64 x 56 tiles, X G 1.56 -> 1.47 ms on 64 x 64; long tiles hide the output
  // anyway, and CTAs of one team drift apart by themselves)
  const double tile_ns = (double)groups / d.splits * s.mt * s.nt * (d.gauss ? 3 : 4) * 16.0 * s.warps / 4 / 1.9;
  g.stagger = items >= 4 * teams && tile_ns < 200e3 ? (int)tile_ns : 0;
  if (ak && bk) zgemm_launch_kk(shape, d.gauss != 0, d, g, stream);
  else if (ak) zgemm_launch_kn(shape, d.gauss != 0, d, g, stream);
  else if (bk) zgemm_launch_nk(shape, d, g, stream);
  else zgemm_launch_nn(shape, d, g, stream);
  int launches = 1;
  if (d.splits > 1) {
    const long total = (long)d.M * d.N * batch;
    if (d.splits > 32)
      zgemm_reduce<8><<<(unsigned)((total + 31) / 32), 256, 0, stream>>>(d);
    else
      zgemm_reduce<1><<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(d);
    GG_CHECK_LAUNCH();
    ++launches;
  }
  return launches;
}

}  // namespace gg
