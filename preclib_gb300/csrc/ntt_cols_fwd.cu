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

struct TableArgs {
    FieldArgs f;
    uint32_t fold[kMaxPrimes];
};

__global__ void __launch_bounds__(256) k_fourstep_table(uint2* t4, TableArgs a, int k1, int k2) {
    const int prime = blockIdx.y, np = gridDim.y, k = k1 + k2;
    const PrimeC pc = a.f.pc[prime];
    const uint32_t N = 1u << k;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < N; i += gridDim.x * blockDim.x) {
        const uint32_t e = (i & ((1u << k2) - 1)) * brev_bits(i >> k2, k1);
#pragma unroll
        for (int dir = 0; dir < 2; ++dir) {
            uint32_t w = fourstep_twiddle<0>(a.f, prime, dir ? (0u - e) & (N - 1) : e, k);
            if (dir) w = mont_lazy(w, a.fold[prime], pc);
            w = red1(mont_lazy(w, 1u, pc), pc.p);
            t4[((size_t)(dir * np + prime) << k) + i] = make_uint2(w, (uint32_t)(((uint64_t)w << 32) / pc.p));
        }
    }
}

void launch_fourstep_table(uint2* t4, const FieldArgs& f, const uint32_t* fold, int nprimes, int k1, int k2,
                           cudaStream_t st) {
    TableArgs a;
    a.f = f;
    for (int j = 0; j < nprimes; ++j) a.fold[j] = fold[j];
    k_fourstep_table<<<dim3((1u << (k1 + k2)) / 256 > 1024 ? 1024 : (1u << (k1 + k2)) / 256, nprimes), 256, 0, st>>>(
        t4, a, k1, k2);
    count_launches(1);
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
    cudaError_t e = load_kernel(k_fourstep_table);
    if (!e) e = (cudaError_t)configure_fwd_cols_k2();
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
