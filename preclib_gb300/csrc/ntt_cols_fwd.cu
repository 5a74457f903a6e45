// ntt_cols_fwd.cu -- instantiations and launcher of the forward column
// kernel (k_fwd_cols, ntt_cols.cuh).
#include "ntt_cols.cuh"

namespace precgpu {

void launch_fwd_cols(int set, const ProdArgs& a, cudaStream_t st, const ProdPtrs* batch, int count, int nprimes) {
    if (nprimes <= 0) nprimes = kSetPrimes[set];
    int cg, mr;
    col_config(set_base(set), a.k1, a.cg, a.cmr, cg, mr);
    const dim3 grid((1u << a.k2) / cg, (a.square || a.operand_only ? 1 : 2) * nprimes, count);
    const size_t smem = col_smem(a.k1, cg);
    if (a.keep < 8) {  // (the plan checked that the kernel exists)
        if (a.keep == 5) launch_fwd_cols_trunc5(set, a, cg, mr, grid, smem, st, batch);
        else if (a.keep == 6) launch_fwd_cols_trunc6(set, a, cg, mr, grid, smem, st, batch);
        else launch_fwd_cols_trunc7(set, a, cg, mr, grid, smem, st, batch);
        count_launches(1);
        return;
    }
    if (launch_fwd_cols_k2(set, a, cg, mr, grid, smem, st, batch)) {
        count_launches(1);
        return;
    }
#define X(S, MM, CC, RR)                                                     \
    if (set == S && a.k1 == MM && cg == CC && mr == RR) {                     \
        launch_pdl(a.chain != 0, k_fwd_cols<S, MM, CC, RR>, grid, col_threads(CC, MM), smem, st, a, batch); \
        count_launches(1);                                                  \
        return;                                                             \
    }
    PREC_COLS_CONFIGS(X)
    PREC_COLS_WIDE_CONFIGS(X)
#undef X
}

bool cols_trunc_supported(int set, int k1, int k2, int cg, int mr, int keep) {
    col_config(set_base(set), k1, cg, mr, cg, mr);
#define X(S, MM, CC, RR, KK) \
    if (set == S && k1 == MM && cg == CC && mr == RR && k2 == KK) return true;
    if (keep == 6) {
        PREC_COLS_FWD_TRUNC6_CONFIGS(X)
    }
    PREC_COLS_FWD_TRUNC_CONFIGS(X)
#undef X
    return false;
}

int configure_fwd_cols() {
    cudaError_t e = (cudaError_t)configure_fwd_cols_k2();
    if (!e) e = (cudaError_t)configure_fwd_cols_trunc5();
    if (!e) e = (cudaError_t)configure_fwd_cols_trunc6();
    if (!e) e = (cudaError_t)configure_fwd_cols_trunc7();
#define X(S, MM, CC, RR)                                                                                   \
    if (!e) e = cudaFuncSetAttribute(k_fwd_cols<S, MM, CC, RR>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                     (int)col_smem(MM, CC));
    PREC_COLS_CONFIGS(X)
    PREC_COLS_WIDE_CONFIGS(X)
#undef X
    return (int)e;
}

}  // namespace precgpu
