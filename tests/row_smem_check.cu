// Host check: the shared-memory limit that a row-tile launch sets on its kernel
// covers every lattice that launches the same kernel, whatever ran before.  Runs
// on the CPU: the launches themselves fail for want of a device.
#include <cuda_runtime.h>

#include <cstdio>
#include <map>

static std::map<const void*, int> g_limit;
template <class F>
static cudaError_t record_limit(F* fn, cudaFuncAttribute, int bytes) {
  g_limit[reinterpret_cast<const void*>(fn)] = bytes;
  return cudaSuccess;
}
#define cudaFuncSetAttribute record_limit
#include "../gpu-sims_b200/csrc/phys_rows.cuh"

using namespace lbm;

static Ctx box(int n) {
  Ctx c{};
  PhysGeom& g = c.pp.g;
  g.nx = g.ny = g.nz = n;
  g.n = (size_t)n * n * n;
  g.gy = g.gz = 1;
  g.px = (n + 1 + 7) / 8 * 8;
  g.py = g.pz = n + 2;
  g.pxy = (uint32_t)(g.px * g.py);
  g.slot_stride = (size_t)g.pxy * g.pz;
  return c;
}

int main() {
  int devices = 0;
  if (cudaGetDeviceCount(&devices) == cudaSuccess && devices > 0) {
    std::printf("a device is visible: nothing is launched\n");
    return 2;
  }
  // one kernel, five stages (store above ROWS_DEEP_BYTES) and two
  const Ctx deep = box(160), shallow = box(96);
  auto* fn = &k_phys_rows<LBM_PREC_F32, LBM_COLL_BGK, 0, false, false, false>;
  const int need = ROWS_MAXST * rows_stage<LBM_PREC_F32>();
  int bad = 0;
  for (const Ctx* c : {&deep, &shallow, &deep}) {
    launch_row_tiles<LBM_PREC_F32, LBM_COLL_BGK, 0, false, false, false>(*c, 0, nullptr);
    bad += g_limit[reinterpret_cast<const void*>(fn)] < need;
  }
  std::printf("limit %d bytes, need %d, %d errors\n", g_limit[reinterpret_cast<const void*>(fn)], need, bad);
  return bad != 0;
}
