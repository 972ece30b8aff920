// Internal functions of libgreen_b200.so behind plain C calls, for the tests that look at them directly.
#include <atomic>

#include "engine.cuh"
#include "zgemm_kernel.cuh"

// out: q points, k points, tau points, Dyson systems per chunk, bytes; returns the error code of a refused shape
extern "C" int plan_work(const gg_shape* s, int nspin, int slices, int solver, int64_t budget, int64_t* out) {
  try {
    const gg::Plan p = gg::plan_work(*s, nspin, slices, solver, (size_t)budget);
    out[0] = p.qc;
    out[1] = p.kc;
    out[2] = p.tb;
    out[3] = p.dyson_batch;
    out[4] = (int64_t)p.bytes;
    return GG_OK;
  } catch (const gg::Error& e) {
    return e.code;
  }
}

extern "C" int64_t zgemm_ctas(int64_t items, int64_t sms, int resident, int pair) {
  return gg::zgemm_ctas(items, sms, resident, pair != 0);
}

// split factor chosen for `batch` products of M x N x (KB K) with room for `room` partial sums
extern "C" int zgemm_splits(int M, int N, int K, int KB, int batch, int tri, int gauss, int64_t room, int sms) {
  static int flag;
  gg::ZgemmDesc d;
  d.M = M; d.N = N; d.K = K; d.KB = KB; d.nb0 = batch; d.gauss = gauss; d.a_k = 1;
  d.tri = tri ? &flag : nullptr;
  d.work = room ? reinterpret_cast<double2*>(16) : nullptr;
  d.work_elems = room;
  return gg::zgemm_choose(d, batch, (long)KB * ((K + 3) / 4), sms).splits;
}

// number of tile shapes; rows and columns of one and its teams per SM
extern "C" int zgemm_shapes(int gauss) { return gauss ? gg::kZShapes3 : gg::kZShapes; }
extern "C" void zgemm_tile(int gauss, int shape, int64_t* out) {
  const gg::ZShape& s = gauss ? gg::kZShape3[shape] : gg::kZShape[shape];
  out[0] = s.bm;
  out[1] = s.bn;
  out[2] = s.teams;
}

// One product from a flat descriptor (see tests/test_gpu_zgemm_shapes.py): shape < 0 lets the library choose.  Returns
// the launches or minus the error code; synchronises.
extern "C" int zgemm_desc(const int64_t* v, const double* ab, const void* A, const void* B, void* C, void* work,
                          const void* tri, int shape, int splits) {
  gg::ZgemmDesc d;
  auto map = [&](gg::IdxMap& m) {
    m.split = (int)*v++;
    m.hi = *v++;
    m.lo = *v++;
  };
  d.M = (int)*v++; d.N = (int)*v++; d.K = (int)*v++; d.KB = (int)*v++;
  d.A = (const double2*)A; map(d.a_m); d.a_k = *v++; d.a_kb = *v++;
  d.B = (const double2*)B; map(d.b_n); d.b_k = *v++; d.b_kb = *v++;
  d.C = (double2*)C; map(d.c_m); map(d.c_n);
  d.nb0 = (int)*v++; d.nb1 = (int)*v++; d.nb2 = (int)*v++;
  d.a_b0 = *v++; d.a_b1 = *v++; d.a_b2 = *v++;
  d.b_b0 = *v++; d.b_b1 = *v++; d.b_b2 = *v++;
  d.c_b0 = *v++; d.c_b1 = *v++; d.c_b2 = *v++;
  d.conjA = (int)*v++; d.conjB = (int)*v++; d.gauss = (int)*v++; d.inplace = (int)*v++;
  d.work = (double2*)work; d.work_elems = *v++;
  d.alpha = make_double2(ab[0], ab[1]);
  d.beta = make_double2(ab[2], ab[3]);
  d.tri = (const int*)tri;
  d.splits = splits;
  try {
    const int n = shape < 0 ? gg::zgemm(d, nullptr) : gg::zgemm_shape(d, shape, nullptr);
    GG_CUDA(cudaStreamSynchronize(nullptr));
    return n;
  } catch (const gg::Error& e) {
    return -e.code;
  }
}
