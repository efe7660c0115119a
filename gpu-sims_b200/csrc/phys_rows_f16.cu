// Row-tile step kernels with f16 population storage.
#include "phys_rows.cuh"

LBM_DEFINE_PHYS_ROWS(phys_rows_f16, LBM_PREC_F16S)

namespace lbm {
uint32_t phys_rows_tiles(const PhysGeom& g) {
  const RowTiles rt = row_tiles(g);
  return rt.R ? rt.ntiles : 0;
}
bool phys_rows_pay(const PhysParams& p, const lbm_desc& d) { return row_tiles_pay(p, d); }
}  // namespace lbm
