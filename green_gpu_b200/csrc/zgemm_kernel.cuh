// The FP64 complex GEMM kernel (see zgemm.cuh) and its tile shapes.
//
// One CTA computes tiles of 8 MT WM x 8 NT WN complex elements with WM x WN DMMA warps, each owning
// MT x NT DMMA tiles of 8 x 8, and one copy warp.  The reduction runs in groups of 4 (the DMMA's
// k), two groups per pipeline stage; a group never crosses a K-batch boundary, so a reduction block
// of K = nao pads to a multiple of 4 only.  The copy warp stages the operands by 16-byte cp.async
// into a ring of STAGES stages whose layout follows the operand's contiguous direction ([row][k] or
// [k][row]) with an XOR swizzle, so that copies and 16-byte fragment loads are free of bank
// conflicts.  CTAs are persistent: the copies of the next tile start while the current one is finished.
// The two sides meet on hardware named barriers, a full and an empty one per stage.
//
// What bounds it: the FP64 pipe (one DMMA per 16 cycles and sub-partition, 37 TFLOP/s measured; FP64
// FMAs share that pipe).  A warp that computes addresses issues no DMMA, and with two DMMA warps per
// sub-partition nothing else fills the gap: with the copies issued by the DMMA warps themselves
// the short reductions (K = 52) spent 40 % of their time on fixed-latency integer work.
#pragma once

#include "dmma.cuh"
#include "zgemm.cuh"

namespace gg {

// Tile shape of one kernel.  DB = 2 loads the next group's fragments before the current group's DMMAs issue,
// which pays only for tiles of one or two DMMA tiles per warp (6 to 20 % there; 4 to 8 % lost on larger
// ones, whose two warps per sub-partition cover the loads).  PAIR: one CTA per SM
// holds two independent teams (four DMMA warps, two copy warps and a ring each), and the copy
// warps hand registers to the DMMA warps (56 and 224 per thread of the 168 that the 384
// threads are launched with; two CTAs of five warps get 168).
template <int MT_, int NT_, int WM_, int WN_, int MINB_, int STAGES_, int DB_, bool PAIR_ = false>
struct ZTile {
  static constexpr int MT = MT_, NT = NT_, WM = WM_, WN = WN_, MINB = MINB_, STAGES = STAGES_, DB = DB_;
  static constexpr bool PAIR = PAIR_;
  static constexpr int BM = 8 * MT * WM, BN = 8 * NT * WN, WARPS = WM * WN;
  static constexpr int TEAMS = PAIR ? 2 : 1, CW = PAIR ? 2 : 1;  // teams, copy warps of each
  static constexpr int THREADS = 32 * TEAMS * (WARPS + CW), TEAM_THREADS = 32 * (WARPS + CW);
  static constexpr int SMEM = TEAMS * STAGES * (BM + BN) * 8 * 16;
  static_assert(!PAIR || (WARPS == 4 && MINB == 1), "whole warpgroups exchange registers");
  static_assert(TEAMS * 2 * STAGES <= 15, "named barriers");
};

constexpr int kZBK = 8;  // reduction elements per stage: two groups of 4

struct ZGrid {
  int tiles_m, tiles_n;
  int items;            // tiles_m * tiles_n * splits * batch
  int tri_tiles;        // tiles on and below the diagonal
  int stagger;          // nanoseconds by which the second team of a CTA starts later
  int gpb;              // groups of 4 per K-batch
  int groups;           // KB * gpb
  long wrap_a, wrap_b;  // from the last group of a K-batch to the first of the next
};

__device__ __forceinline__ long zmap(const IdxMap& f, int i) {
  return f.split > 0 ? (long)(i / f.split) * f.hi + (long)(i % f.split) * f.lo : (long)i * f.lo;
}

// x with its sign bit XORed with the sign bit of `s` (s = 0 or 0x80000000)
__device__ __forceinline__ double zflip(double x, int s) {
  return __hiloint2double(__double2hiint(x) ^ s, __double2loint(x));
}

// swizzled position of tile element (row r, k) in a stage of R rows
template <bool KMAJ, int R>
__device__ __forceinline__ int zsidx(int r, int k) {
  return KMAJ ? r * kZBK + (k ^ ((r & 1) << 2)) : k * R + (r ^ ((k & 3) << 1));
}

// named barriers (hardware; id 0 is __syncthreads): `threads` threads meet, arrive does not wait
__device__ __forceinline__ void zbar_sync(int id, int threads) {
  asm volatile("barrier.cta.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void zbar_arrive(int id, int threads) {
  asm volatile("barrier.cta.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// two neighbouring elements as one 32-byte store
__device__ __forceinline__ void zstore2(double2* p, double2 v0, double2 v1) {
  asm volatile("st.global.v4.f64 [%0], {%1, %2, %3, %4};" ::"l"(p), "d"(v0.x), "d"(v0.y), "d"(v1.x), "d"(v1.y) : "memory");
}

// tile row that holds the diagonal of tile column tn: the first one of a lower-triangle product
__host__ __device__ __forceinline__ int zfirst_row(int tn, int bm, int bn) { return (int)((long)tn * bn / bm); }

// first row and column of a tile (tile rows vary fastest)
template <int BM, int BN>
__device__ __forceinline__ void ztile_origin(const ZGrid& g, bool tri, int tile, int& m0, int& n0) {
  int tn = (int)((unsigned)tile / (unsigned)g.tiles_m), tm = tile - tn * g.tiles_m;
  if (tri) {
    for (tn = 0;; ++tn) {
      const int first = zfirst_row(tn, BM, BN), count = g.tiles_m - first;
      if (tile < count) {
        tm = first + tile;
        break;
      }
      tile -= count;
    }
  }
  m0 = tm * BM;
  n0 = tn * BN;
}

// tile, split and batch indices of item `it`
struct ZItem {
  int tile, split, batch, b0, b1, b2;
};
__device__ __forceinline__ ZItem zitem(const ZgemmDesc& d, int ntile, int it) {
  ZItem w;
  unsigned rest = (unsigned)it / (unsigned)ntile;
  w.tile = it - (int)rest * ntile;
  w.split = 0;
  if (d.splits > 1) {
    w.split = (int)(rest % (unsigned)d.splits);
    rest /= (unsigned)d.splits;
  }
  w.batch = (int)rest;
  w.b0 = w.batch;
  w.b1 = w.b2 = 0;
  if (d.nb1 > 1 || d.nb2 > 1) {
    w.b0 = (int)(rest % (unsigned)d.nb0);
    rest /= (unsigned)d.nb0;
    w.b1 = (int)(rest % (unsigned)d.nb1);
    w.b2 = (int)(rest / (unsigned)d.nb1);
  }
  return w;
}

// group range of item `it` (split-K)
__device__ __forceinline__ void zrange(const ZgemmDesc& d, const ZGrid& g, int ntile, int it, int& g0, int& g1) {
  g0 = 0;
  g1 = g.groups;
  if (d.splits > 1) {
    const int split = (it / ntile) % d.splits;
    g0 = (int)((long)g.groups * split / d.splits);
    g1 = (int)((long)g.groups * (split + 1) / d.splits);
  }
}

// Rows of one operand that a lane of CW copy warps fetches, R rows x 8 k per stage (`lane` counts through
// the warps).  [row][k]: lane (r = lane / 8, kk = lane % 8) takes rows r + 4 CW i; [k][row]: rows
// r = lane % 32 + 32 i, the warps sharing the kk.
template <bool KMAJ, int R, int CW>
struct ZRows {
  static constexpr int N = KMAJ ? (R + 4 * CW - 1) / (4 * CW) : (R + 31) / 32;
  const double2* p[N];
  unsigned ok;
  __device__ __forceinline__ void begin(const double2* base, const IdxMap& map, long ks, int row0, int rows, int lane) {
    ok = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
      const int r = KMAJ ? lane / 8 + 4 * CW * i : lane % 32 + 32 * i;
      const bool v = r < R && row0 + r < rows;
      ok |= v ? 1u << i : 0u;
      p[i] = base + (v ? zmap(map, row0 + r) : 0) + (KMAJ ? (lane & 3) * ks : 0);
    }
  }
  // one stage: group offsets o0 / o1 and their valid counts
  __device__ __forceinline__ void copy(double2* dst, long ks, long o0, long o1, int cnt0, int cnt1, int lane,
                                       const double2* any) const {
    if constexpr (KMAJ) {
      const int kk = lane & 7;
      const bool kv = (kk & 3) < (kk < 4 ? cnt0 : cnt1);
      const long o = kk < 4 ? o0 : o1;
      double2* s = dst + zsidx<true, R>(lane / 8, kk);  // rows step by an even number: the swizzle term stays
#pragma unroll
      for (int i = 0; i < N; ++i) {
        if (R % (4 * CW) != 0 && lane / 8 + 4 * CW * i >= R) continue;
        const bool v = kv && (ok >> i & 1);
        cp_async16(s + i * 4 * CW * kZBK, v ? p[i] + o : any, v);
      }
    } else {
#pragma unroll
      for (int k = 0; k < kZBK; k += CW) {
        const int kk = k + (CW > 1 ? lane / 32 : 0);
        const bool kv = (kk & 3) < (kk < 4 ? cnt0 : cnt1);
        const long o = (kk < 4 ? o0 : o1) + (kk & 3) * ks;
#pragma unroll
        for (int i = 0; i < N; ++i) {
          if (R % 32 != 0 && lane % 32 + 32 * i >= R) continue;
          const bool v = kv && (ok >> i & 1);
          cp_async16(dst + zsidx<false, R>(lane % 32 + 32 * i, kk), v ? p[i] + o : any, v);
        }
      }
    }
  }
};

// G3: three real products per complex product (ZgemmDesc::gauss)
template <class T, bool A_K, bool B_K, bool G3>
__global__ void __launch_bounds__(T::THREADS, T::MINB) zgemm_kernel(const __grid_constant__ ZgemmDesc d, ZGrid g) {
  extern __shared__ __align__(16) double2 zsm[];
  constexpr int MT = T::MT, NT = T::NT, BM = T::BM, BN = T::BN, S = T::STAGES, NTHR = T::TEAM_THREADS;
  constexpr int ASZ = BM * kZBK, BSZ = BN * kZBK;
  const bool copier = threadIdx.x >= 32 * T::TEAMS * T::WARPS;
  const int wid = (copier ? threadIdx.x - 32 * T::TEAMS * T::WARPS : threadIdx.x) >> 5;
  const int team = T::PAIR ? wid / (copier ? T::CW : T::WARPS) : 0;
  const int FULL = 1 + team * 2 * S, EMPTY = FULL + S;
  double2* const As = zsm + team * S * (ASZ + BSZ);
  double2* const Bs = As + S * ASZ;
  const int lane = threadIdx.x & 31;
  const bool tri = d.tri && *d.tri;
  const int ntile = tri ? g.tri_tiles : g.tiles_m * g.tiles_n;
  const int items = tri ? g.items / (g.tiles_m * g.tiles_n) * g.tri_tiles : g.items;
  // the second round of items starts on other SMs before any SM's second team gets one
  const int it0 = blockIdx.x + team * gridDim.x, stride = gridDim.x * T::TEAMS;

  if (copier) {
    if (T::PAIR) asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    // teams that start together also write their tiles at the same time, with the DMMA pipe idle
    if (T::PAIR && team && g.stagger) __nanosleep(g.stagger);
    const int cl = lane + 32 * (T::PAIR ? wid % T::CW : 0);  // lane of the team's copy warps
    // ---------------- copy warp.  Stage t is announced once it has landed and stage t + S - 2 has been
    // issued: the copies of S - 2 stages are in flight, and one landed stage waits for its turn
    constexpr int LAG = S - 2;
    ZRows<A_K, BM, T::CW> ra;
    ZRows<B_K, BN, T::CW> rb;
    int t = 0, st = 0;  // steps issued, stage of the next one
    int sa = 0;         // stage of the next announcement
    for (int it = it0; it < items; it += stride) {
      {
        const ZItem w = zitem(d, ntile, it);
        int m0, n0;
        ztile_origin<BM, BN>(g, tri, w.tile, m0, n0);
        ra.begin(d.A + w.b0 * d.a_b0 + w.b1 * d.a_b1 + w.b2 * d.a_b2, d.a_m, d.a_k, m0, d.M, cl);
        rb.begin(d.B + w.b0 * d.b_b0 + w.b1 * d.b_b1 + w.b2 * d.b_b2, d.b_n, d.b_k, n0, d.N, cl);
      }
      int g0, g1;
      zrange(d, g, ntile, it, g0, g1);
      int left = g1 - g0;
      const int kb = g0 / g.gpb;
      int kin = g0 - kb * g.gpb;
      long goff_a = kb * d.a_kb + 4L * kin * d.a_k, goff_b = kb * d.b_kb + 4L * kin * d.b_k;
      // valid element count of the next group (0 past the end of the item) and step past it
      auto next_group = [&](long& oa, long& ob, int& cnt) {
        oa = goff_a;
        ob = goff_b;
        cnt = left > 0 ? d.K - 4 * kin : 0;
        --left;
        if (++kin == g.gpb) {
          kin = 0;
          goff_a += g.wrap_a;
          goff_b += g.wrap_b;
        } else {
          goff_a += 4L * d.a_k;
          goff_b += 4L * d.b_k;
        }
      };
      while (left > 0) {
        if (t >= S) zbar_sync(EMPTY + st, NTHR);
        long oa0, ob0, oa1, ob1;
        int cnt0, cnt1;
        next_group(oa0, ob0, cnt0);
        next_group(oa1, ob1, cnt1);
        ra.copy(As + st * ASZ, d.a_k, oa0, oa1, cnt0, cnt1, cl, d.A);
        rb.copy(Bs + st * BSZ, d.b_k, ob0, ob1, cnt0, cnt1, cl, d.B);
        cp_commit();
        if (t >= LAG) {
          cp_wait<LAG>();
          zbar_arrive(FULL + sa, NTHR);
          sa = sa + 1 == S ? 0 : sa + 1;
        }
        ++t;
        st = st + 1 == S ? 0 : st + 1;
      }
    }
    cp_wait<0>();
    for (int i = 0; i < min(t, LAG); ++i) {
      zbar_arrive(FULL + sa, NTHR);
      sa = sa + 1 == S ? 0 : sa + 1;
    }
    // the last stages' releases: every barrier is complete when the CTA ends
    for (int i = t > S ? t - S : 0; i < t; ++i) zbar_sync(EMPTY + i % S, NTHR);
    return;
  }

  // ---------------- DMMA warps
  if (T::PAIR) asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
  const int warp = T::PAIR ? wid % T::WARPS : wid;
  const int wm = warp % T::WM, wn = warp / T::WM;
  const int fr = lane >> 2, fk = lane & 3;
  // accumulators: c0 / c1 = re / im (four products) or c0 / c1 / c2 = rr, ii, (r+i)(r+i)
  double c0[MT][NT][2], c1[MT][NT][2], c2[G3 ? MT : 1][G3 ? NT : 1][2];
  auto zero_acc = [&]() {
#pragma unroll
    for (int a = 0; a < MT; ++a)
#pragma unroll
      for (int b = 0; b < NT; ++b)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          c0[a][b][j] = 0.0;
          c1[a][b][j] = 0.0;
          if constexpr (G3) c2[a][b][j] = 0.0;
        }
  };
  zero_acc();
  // conjugation flips the sign bit of the imaginary part (an integer XOR, no FP64 multiply)
  const int sa = d.conjA ? (int)0x80000000 : 0;
  const int sb = d.conjB ? (int)0x80000000 : 0;
  double2 fa[T::DB][MT], fb[T::DB][NT];
  auto load = [&](int buf, int st, int grp) {
    const double2* as = As + st * ASZ;
    const double2* bs = Bs + st * BSZ;
#pragma unroll
    for (int i = 0; i < MT; ++i) fa[buf][i] = as[zsidx<A_K, BM>(wm * 8 * MT + i * 8 + fr, grp * 4 + fk)];
#pragma unroll
    for (int i = 0; i < NT; ++i) fb[buf][i] = bs[zsidx<B_K, BN>(wn * 8 * NT + i * 8 + fr, grp * 4 + fk)];
  };
  // passes over all accumulator tiles: consecutive DMMAs never share an accumulator
  auto mma = [&](int buf) {
    double ai[MT], ax[MT], bi[NT];
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      ai[i] = zflip(fa[buf][i].y, sa);
      ax[i] = G3 ? fa[buf][i].x + ai[i] : -ai[i];
    }
#pragma unroll
    for (int i = 0; i < NT; ++i) bi[i] = zflip(fb[buf][i].y, sb);
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
      for (int j = 0; j < NT; ++j) dmma(c0[i][j][0], c0[i][j][1], fa[buf][i].x, fb[buf][j].x);
    if constexpr (G3) {
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) dmma(c1[i][j][0], c1[i][j][1], ai[i], bi[j]);
#pragma unroll
      for (int j = 0; j < NT; ++j) bi[j] += fb[buf][j].x;
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) dmma(c2[i][j][0], c2[i][j][1], ax[i], bi[j]);
    } else {
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) dmma(c1[i][j][0], c1[i][j][1], fa[buf][i].x, bi[j]);
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) dmma(c0[i][j][0], c0[i][j][1], ax[i], bi[j]);
#pragma unroll
      for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j) dmma(c1[i][j][0], c1[i][j][1], ai[i], fb[buf][j].x);
    }
  };
  // Output of a tile.  No DMMA issues from this warp meanwhile, so the addresses are kept to one
  // pointer per row and one column offset that steps by 8 (a division per tile, not per element), and the
  // usual case - no scaling, no accumulation - has a loop of its own.
  auto epilogue = [&](int it) {
    const ZItem w = zitem(d, ntile, it);
    int m0, n0;
    ztile_origin<BM, BN>(g, tri, w.tile, m0, n0);
    m0 += wm * 8 * MT + fr;
    n0 += wn * 8 * NT + 2 * fk;
    const bool part = d.splits > 1;
    const bool plain = part || (d.alpha.x == 1.0 && d.alpha.y == 0.0 && d.beta.x == 0.0 && d.beta.y == 0.0);
    const bool use_beta = d.beta.x != 0.0 || d.beta.y != 0.0;
    double2* const cb = part ? d.work + ((long)w.split * (d.nb0 * d.nb1 * d.nb2) + w.batch) * d.M * d.N
                             : d.C + w.b0 * d.c_b0 + w.b1 * d.c_b1 + w.b2 * d.c_b2;
    double2* row[MT];
    bool rok[MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) {
      rok[i] = m0 + i * 8 < d.M;
      row[i] = cb + (!rok[i] ? 0 : part ? (long)(m0 + i * 8) * d.N : zmap(d.c_m, m0 + i * 8));
    }
    auto value = [&](int i, int j, int e) {
      if constexpr (G3)
        return make_double2(c0[i][j][e] - c1[i][j][e], c2[i][j][e] - c0[i][j][e] - c1[i][j][e]);
      else
        return make_double2(c0[i][j][e], c1[i][j][e]);
    };
    const int split = part ? 0 : d.c_n.split;
    const long lo = part ? 1 : d.c_n.lo;
    // short reductions into contiguous rows (X G): a row's pointer and immediate offsets.  They spend a third of a
    // tile's instructions on its output (X G of nao 52 1.24 -> 1.22 ms, with three products 1.07 -> 1.03, nao 37
    // 0.31 -> 0.29, nao 20 49.9 -> 45.9 us); the other layouts have long reductions, where the second loop
    // only costs registers (Z V^+ of nao 52 0.84 -> 0.90 ms)
    if (A_K && !B_K && plain && split == 0 && lo == 1) {
      const int left = d.N - n0;
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        if (!rok[i]) continue;
        double2* const p = row[i] + n0;
        const bool wide = ((size_t)p & 31) == 0;  // columns step by 8: the same for the whole row
#pragma unroll
        for (int j = 0; j < NT; ++j) {
          const double2 v0 = value(i, j, 0), v1 = value(i, j, 1);
          if (wide && j * 8 + 1 < left) {
            zstore2(p + j * 8, v0, v1);
          } else {
            if (j * 8 < left) p[j * 8] = v0;
            if (j * 8 + 1 < left) p[j * 8 + 1] = v1;
          }
        }
      }
      return;
    }
    const long wrap = split > 0 ? d.c_n.hi - split * lo : 0;
    int r[2];
    long off[2];
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      r[e] = n0 + e;
      off[e] = (long)r[e] * lo;
      if (split > 0) {
        const int q = r[e] / split;
        r[e] -= q * split;
        off[e] = q * d.c_n.hi + r[e] * lo;
      }
    }
    // a lane's two columns are neighbours in memory where C is contiguous along n: one 32-byte store (a full
    // sector) where the address allows it, else one after the other, since they share sectors
#pragma unroll
    for (int j = 0; j < NT; ++j) {
      const bool ok0 = n0 + j * 8 < d.N, ok1 = n0 + j * 8 + 1 < d.N;
#pragma unroll
      for (int i = 0; i < MT; ++i) {
        if (!rok[i]) continue;
        double2* const p0 = row[i] + off[0];
        double2* const p1 = row[i] + off[1];
        double2 v0 = value(i, j, 0), v1 = value(i, j, 1);
        if (!plain) {
          v0 = cmul(d.alpha, v0);
          v1 = cmul(d.alpha, v1);
          if (use_beta) {
            if (ok0) v0 = cadd(v0, cmul(d.beta, *p0));
            if (ok1) v1 = cadd(v1, cmul(d.beta, *p1));
          }
        }
        if (ok1 && p1 == p0 + 1 && ((size_t)p0 & 31) == 0) {
          zstore2(p0, v0, v1);
        } else {
          if (ok0) *p0 = v0;
          if (ok1) *p1 = v1;
        }
      }
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        off[e] += 8 * lo;
        if (split > 0) {
          r[e] += 8;
          while (r[e] >= split) {
            r[e] -= split;
            off[e] += wrap;
          }
        }
      }
    }
  };

  // the barrier in the middle of a step makes the next stage visible; the current one is released
  // as soon as its last fragments are in registers
  constexpr int D = T::DB - 1;  // fragment buffer of the second group
  int st = 0;
  if (it0 < items) zbar_sync(FULL, NTHR);
  if (D) load(0, 0, 0);
  for (int it = it0; it < items; it += stride) {
    int g0, g1;
    zrange(d, g, ntile, it, g0, g1);
    const bool more = it + stride < items;
    for (int n = g1 - g0; n > 0; n -= 2) {
      if (!D) {
        load(0, st, 0);
        mma(0);
      }
      load(D, st, 1);
      zbar_arrive(EMPTY + st, NTHR);
      if (D) mma(0);
      st = st + 1 == S ? 0 : st + 1;
      if (n > 2 || more) {
        zbar_sync(FULL + st, NTHR);
        if (D) load(0, st, 0);
      }
      if (n > 1) mma(D);
    }
    epilogue(it);
    zero_acc();
  }
}

// The launch tables: one translation unit per operand layout (zgemm_kk.cu, ...), each holding every
// tile shape.  64 x 64 and 64 x 80 serve wide outputs (80 divides NQ = 400, 64 pads it to 448);
// 64 x 8 NT and 32 x 8 NT serve outputs of at most 56 columns (N = nao), where one tile spans the
// width; squares of 24, 32, 40, 48 and 56 serve nao x nao outputs of long reductions (exchange), 16 x 16
// products whose few tiles would leave most SMs idle.  The three-product
// kernels hold three accumulators per element, so their tiles are smaller.  Each shape has as many
// CTAs per SM as its registers allow (64 x 32: two -> three, operand build of nao 26 95 -> 87 us, Z V^+ of nao 20
// 64 -> 50 us; a fourth CTA of 64 x 24 lost 3 % on V^T W and exchange products).
struct ZShape {
  int bm, bn, mt, nt, warps, teams;  // teams resident per SM
  constexpr bool square() const { return mt == 1 && warps == nt; }
};
constexpr ZShape kZShape[] = {
    {64, 64, 4, 4, 4, 2}, {64, 80, 4, 5, 4, 2}, {64, 56, 2, 7, 4, 2}, {64, 48, 2, 6, 4, 2}, {64, 40, 2, 5, 4, 2},
    {64, 32, 2, 4, 4, 3}, {64, 24, 2, 3, 4, 3}, {64, 16, 2, 2, 4, 4}, {64, 8, 2, 1, 4, 4}, {32, 56, 1, 7, 4, 3},
    {56, 56, 1, 7, 7, 2}, {48, 48, 1, 6, 6, 2}, {40, 40, 1, 5, 5, 3}, {24, 24, 1, 3, 3, 4}, {32, 32, 2, 2, 4, 3},
    {16, 16, 1, 1, 4, 4}};
constexpr ZShape kZShape3[] = {
    {64, 48, 4, 3, 4, 2}, {64, 56, 2, 7, 4, 2}, {64, 40, 2, 5, 4, 2}, {64, 32, 2, 4, 4, 2}, {64, 24, 2, 3, 4, 3},
    {64, 16, 2, 2, 4, 3}, {64, 8, 2, 1, 4, 4},  {32, 56, 1, 7, 4, 3}, {32, 32, 2, 2, 4, 3}, {16, 16, 1, 1, 4, 4}};
constexpr int kZShapes = sizeof(kZShape) / sizeof(ZShape), kZShapes3 = sizeof(kZShape3) / sizeof(ZShape);

template <int I, bool G3>
struct ZTileOf;
template <> struct ZTileOf<0, false> { using T = ZTile<4, 4, 2, 2, 1, 3, 1, true>; };
template <> struct ZTileOf<1, false> { using T = ZTile<4, 5, 2, 2, 1, 3, 1, true>; };
template <> struct ZTileOf<2, false> { using T = ZTile<2, 7, 4, 1, 1, 3, 1, true>; };
template <> struct ZTileOf<3, false> { using T = ZTile<2, 6, 4, 1, 1, 3, 1, true>; };
template <> struct ZTileOf<4, false> { using T = ZTile<2, 5, 4, 1, 2, 4, 1>; };
template <> struct ZTileOf<5, false> { using T = ZTile<2, 4, 4, 1, 3, 4, 1>; };
template <> struct ZTileOf<6, false> { using T = ZTile<2, 3, 4, 1, 3, 4, 1>; };
template <> struct ZTileOf<7, false> { using T = ZTile<2, 2, 4, 1, 4, 4, 1>; };
template <> struct ZTileOf<8, false> { using T = ZTile<2, 1, 4, 1, 4, 5, 2>; };
template <> struct ZTileOf<9, false> { using T = ZTile<1, 7, 4, 1, 3, 4, 1>; };
template <> struct ZTileOf<10, false> { using T = ZTile<1, 7, 7, 1, 2, 7, 1>; };
template <> struct ZTileOf<11, false> { using T = ZTile<1, 6, 6, 1, 2, 7, 1>; };
template <> struct ZTileOf<12, false> { using T = ZTile<1, 5, 5, 1, 3, 6, 1>; };
template <> struct ZTileOf<13, false> { using T = ZTile<1, 3, 3, 1, 4, 7, 2>; };
template <> struct ZTileOf<14, false> { using T = ZTile<2, 2, 2, 2, 3, 5, 1>; };
template <> struct ZTileOf<15, false> { using T = ZTile<1, 1, 2, 2, 4, 7, 2>; };
template <> struct ZTileOf<0, true> { using T = ZTile<4, 3, 2, 2, 1, 3, 1, true>; };
template <> struct ZTileOf<1, true> { using T = ZTile<2, 7, 4, 1, 1, 3, 1, true>; };
template <> struct ZTileOf<2, true> { using T = ZTile<2, 5, 4, 1, 1, 3, 1, true>; };
template <> struct ZTileOf<3, true> { using T = ZTile<2, 4, 4, 1, 1, 3, 1, true>; };
template <> struct ZTileOf<4, true> { using T = ZTile<2, 3, 4, 1, 3, 4, 1>; };
template <> struct ZTileOf<5, true> { using T = ZTile<2, 2, 4, 1, 3, 4, 1>; };
template <> struct ZTileOf<6, true> { using T = ZTile<2, 1, 4, 1, 4, 5, 2>; };
template <> struct ZTileOf<7, true> { using T = ZTile<1, 7, 4, 1, 3, 4, 1>; };
template <> struct ZTileOf<8, true> { using T = ZTile<2, 2, 2, 2, 3, 5, 1>; };
template <> struct ZTileOf<9, true> { using T = ZTile<1, 1, 2, 2, 4, 7, 2>; };

// tile shape and split-K factor of a descriptor on a GPU of `sms` SMs (zgemm.cu)
struct ZChoice {
  int shape = 0, splits = 1;
};
ZChoice zgemm_choose(const ZgemmDesc& d, long batch, long groups, int sms);
// the product with shape `shape` of the table (three products: of kZShape3) and d.splits partial sums, the pass over
// which follows; returns the launches (zgemm.cu)
int zgemm_shape(const ZgemmDesc& d, int shape, cudaStream_t stream);
// launch shape `shape` of one layout (G3 where the layout has it)
void zgemm_launch_kk(int shape, bool g3, const ZgemmDesc& d, const ZGrid& g, cudaStream_t st);
void zgemm_launch_kn(int shape, bool g3, const ZgemmDesc& d, const ZGrid& g, cudaStream_t st);
void zgemm_launch_nk(int shape, const ZgemmDesc& d, const ZGrid& g, cudaStream_t st);
void zgemm_launch_nn(int shape, const ZgemmDesc& d, const ZGrid& g, cudaStream_t st);
// products that do not fill the GPU, any layout: one CTA per 8 x 8 tile (zgemm_small.cu)
void zgemm_launch_small(const ZgemmDesc& d, const ZGrid& g, cudaStream_t st);

// CTAs for `items` tiles with `resident` teams per SM.  Paired: one CTA per SM as long as there are items, so that no SM's
// second team gets one before every SM has its first.  Unpaired: up to four rounds of items go out as a CTA each, which
// the hardware deals to SMs as they become free (a fixed assignment gives SMs whose CTAs all have one
// item more than others: 160 x 160 x 3200, batch 12: 0.33 against 0.27 ms), more as persistent CTAs.
inline long zgemm_ctas(long items, long sms, int resident, bool pair) {
  if (pair) return items < sms ? items : sms;
  const long teams = sms * resident;
  return items <= 4 * teams ? items : teams;
}

template <class T, bool A_K, bool B_K, bool G3>
void zlaunch(const ZgemmDesc& d, const ZGrid& g, cudaStream_t st) {
  // the shared-memory attribute is per device: set once on each
  static std::atomic<bool> cfg[kMaxDevices];
  const int dev = current_device();
  if (!cfg[dev].load(std::memory_order_acquire)) {
    GG_CUDA(cudaFuncSetAttribute(zgemm_kernel<T, A_K, B_K, G3>, cudaFuncAttributeMaxDynamicSharedMemorySize, T::SMEM));
    cfg[dev].store(true, std::memory_order_release);
  }
  const unsigned ctas = (unsigned)zgemm_ctas(g.items, device_sm_count(), T::TEAMS * T::MINB, T::PAIR);
  zgemm_kernel<T, A_K, B_K, G3><<<ctas, T::THREADS, T::SMEM, st>>>(d, g);
  GG_CHECK_LAUNCH();
}

template <bool A_K, bool B_K, bool G3, int I = 0>
void zlaunch_shape(int shape, const ZgemmDesc& d, const ZGrid& g, cudaStream_t st) {
  if constexpr (I < (G3 ? kZShapes3 : kZShapes)) {
    using T = typename ZTileOf<I, G3>::T;
    constexpr ZShape s = G3 ? kZShape3[I < kZShapes3 ? I : 0] : kZShape[I];
    static_assert(T::BM == s.bm && T::BN == s.bn && T::MT == s.mt && T::NT == s.nt && T::WARPS == s.warps &&
                      T::TEAMS * T::MINB == s.teams,
                  "shape table");
    if (shape == I) zlaunch<T, A_K, B_K, G3>(d, g, st);
    else zlaunch_shape<A_K, B_K, G3, I + 1>(shape, d, g, st);
  }
}

}  // namespace gg
