// ntt_cols_inv_trunc5.cu -- inverse columns of transforms truncated to 5 eighths.
#define PREC_TRUNC_E 5
#define PREC_TRUNC_FWD 0
#include "ntt_cols_trunc.inc"
