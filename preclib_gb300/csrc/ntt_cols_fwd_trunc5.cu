// ntt_cols_fwd_trunc5.cu -- forward columns of transforms truncated to 5 eighths.
#define PREC_TRUNC_E 5
#define PREC_TRUNC_FWD 1
#include "ntt_cols_trunc.inc"
