// ntt_cols_fwd_trunc7.cu -- forward columns of transforms truncated to 7 eighths.
#define PREC_TRUNC_E 7
#define PREC_TRUNC_FWD 1
#include "ntt_cols_trunc.inc"
