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
