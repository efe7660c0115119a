// Row-tile step kernels with f16 population storage.
#include "phys_rows.cuh"

LBM_DEFINE_PHYS_ROWS(phys_rows_f16, LBM_PREC_F16S)
