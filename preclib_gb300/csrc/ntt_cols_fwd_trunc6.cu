// ntt_cols_fwd_trunc6.cu -- forward columns of transforms truncated to 6 eighths.
#define PREC_TRUNC_E 6
#define PREC_TRUNC_FWD 1
#include "ntt_cols_trunc.inc"
