// ntt_cols_inv_trunc7.cu -- inverse columns of transforms truncated to 7 eighths.
#define PREC_TRUNC_E 7
#define PREC_TRUNC_FWD 0
#include "ntt_cols_trunc.inc"
