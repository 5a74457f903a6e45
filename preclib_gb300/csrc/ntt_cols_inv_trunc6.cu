// ntt_cols_inv_trunc6.cu -- inverse columns of transforms truncated to 6 eighths.
#define PREC_TRUNC_E 6
#define PREC_TRUNC_FWD 0
#include "ntt_cols_trunc.inc"
