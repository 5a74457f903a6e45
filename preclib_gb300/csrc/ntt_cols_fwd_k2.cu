// ntt_cols_fwd_k2.cu -- the forward column kernels of the default
// configurations compiled for their constant row length
// (PREC_COLS_FWD_K2_CONFIGS, ntt_cols.cuh).
#include "ntt_cols.cuh"

namespace precgpu {

bool launch_fwd_cols_k2(int set, const ProdArgs& a, int cg, int mr, dim3 grid, size_t smem, cudaStream_t st,
                        const ProdPtrs* batch) {
#define X(S, MM, CC, RR, KK)                                                                   \
    if (set == S && a.k1 == MM && cg == CC && mr == RR && a.k2 == KK) {                         \
        launch_pdl(a.chain != 0, k_fwd_cols<S, MM, CC, RR, KK>, grid, col_threads(CC, MM), smem, st, a, batch);        \
        return true;                                                                            \
    }
    PREC_COLS_FWD_K2_CONFIGS(X)
    PREC_COLS_FWD_BATCH_CONFIGS(X)
    PREC_COLS_FWD_BATCH_SHORT_CONFIGS(X)
    PREC_COLS_BATCH_SHORTEST_CONFIGS(X)
#undef X
    return false;
}

int configure_fwd_cols_k2() {
    cudaError_t e = cudaSuccess;
#define X(S, MM, CC, RR, KK)                                                                             \
    if (!e) e = cudaFuncSetAttribute(k_fwd_cols<S, MM, CC, RR, KK>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                     (int)col_smem(MM, CC));
    PREC_COLS_FWD_K2_CONFIGS(X)
    PREC_COLS_FWD_BATCH_CONFIGS(X)
    PREC_COLS_FWD_BATCH_SHORT_CONFIGS(X)
    PREC_COLS_BATCH_SHORTEST_CONFIGS(X)
#undef X
    return (int)e;
}

}  // namespace precgpu
