// Row-tile step kernels with bf16 population storage.
#include "phys_rows.cuh"

LBM_DEFINE_PHYS_ROWS(phys_rows_bf16, LBM_PREC_BF16S)
