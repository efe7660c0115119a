// Row-tile step kernels with f32 population storage.
#include "phys_rows.cuh"

LBM_DEFINE_PHYS_ROWS(phys_rows_f32, LBM_PREC_F32)
