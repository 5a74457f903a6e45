// ntt_cols.cuh -- column passes of the four-step NTT (index i = i1*N2 + i2).
//
// k_fwd_cols: for C adjacent columns i2 of one operand and one prime, the
//   limbs are read as 32-bit digits (sets 2 and 3: whole 64-bit limbs) (the
//   reference's ntt_digits and mont_in, src/mul_ntt.cpp:331-342, 357-360,
//   fused into the load), reduced, run through a DIF transform over i1 (the
//   first log2(N1) stages of ntt_forward, mul_ntt.cpp:193-255) and
//   multiplied by the four-step twiddle w_N^(i2*k1).  Output row slot s
//   holds frequency k1 = bitrev(s).
// k_inv_cols: the inverse four-step twiddle w_N^-(i2*k1) times the prime's
//   CRT scale (CrtConst/Crt5Const::fold: the Garner constant that would
//   otherwise cost the CRT one product per prime and coefficient), then the
//   DIT transform over the row slots (the last stages of ntt_inverse,
//   mul_ntt.cpp:257-329) back to natural coefficient order.
// Both generate their twiddles as running powers over a thread's 32 slots of one
// column (sets 0 and 2: a chain of Shoup products, twiddle32_shoup; sets 1 and 3:
// Montgomery products, twiddle32), or read them from a table (col_table).
// Columns are interleaved in shared memory (element i of column c at
// P(i)*C + c); a warp covers C columns x 32/C items, so every global access
// moves whole 32-byte sectors.
// Template parameters: SET prime set, M = log2 N1 (column length), C
// columns per CTA (launched with col_threads(C, M) threads), MR the pass radix cap (MR = 6: a 2^11-point column runs
// as a radix-64 and a radix-32 pass; MR = 4: radix-8, -8, -32), K2 =
// log2 N2 (the row length, the stride between a column's elements) as a
// constant, or 0: from the arguments.  The instantiated (SET, M, C, MR)
// configurations are PREC_COLS_CONFIGS, with K2 = 0; the autotuner picks C
// and MR per transform length.  The default configuration of every
// transform length also has a K2 instantiation (PREC_COLS_*_K2_CONFIGS,
// ntt_cols_fwd_k2.cu, ntt_cols_inv_k2.cu).  Its global addresses are a
// constant offset from one base per item.  At 2^21 points on the 64-bit plan
// the forward columns measured 71.5 -> 63.1 us, and the inverse columns
// 34.8 -> 32.8 us.
#pragma once
#include "ntt_engine.cuh"

namespace precgpu {

// the batch classes' configurations (more than 8 columns per CTA) read their
// four-step twiddles from a table, one Shoup product per value instead of a
// Montgomery product and a chain step (a third of the forward pass's
// multiplier time).  4096 products of 200 .. 65536 limbs 8.52 -> 8.23 ms.  Past
// 2^19 points the tables no longer stay in L2 beside the residues: 2^20
// points 86 -> 109 us, 2^21 157 -> 197.
__host__ __device__ constexpr bool col_table(int cg) { return cg > 8; }

// Top DIF pass of a digit tile whose upper half (rows 2^(M-1) and up) is
// zero -- every operand of at most N/2 digits, i.e. both operands of a
// balanced product: only the lower half is staged and reduced, and the
// first stage (x, 0) -> (x, x*w) needs one twiddle product per pair.
// Set 2 stages 64-bit limbs as two words per element (stage_limbs): the
// element's digit is read from its row and the row 2^(M-1) above it.
// E: the transform is truncated to E eighths (ntt_engine.cuh).
template <int SET, int M, int C, int MR, int E = 8>
__device__ __forceinline__ void col_top_upper_zero(uint32_t* sm, const uint2* __restrict__ tw, const PrimeC& c) {
    using G = Geom<M, 0, MR>;
    static_assert(G::LO >= 5, "the top pass of a multi-pass transform");
    constexpr int H = G::R / 2;
    for (int w = threadIdx.x; w < (C << G::LGI); w += blockDim.x) {
        const int col = w & (C - 1);
        const uint32_t u = w / C;
        const uint32_t ulo = u & G::LOMASK;
        uint32_t* s = sm + G::pbase(u) * C + col;
        uint32_t x[1][G::R];
#pragma unroll
        for (int q = 0; q < H; ++q) {
            uint32_t d;
            if constexpr (set_wide(SET)) d = Ar<SET>::digit64(s[q * G::QS * C], s[(q + H) * G::QS * C], c);
            else d = Ar<SET>::digit(s[q * G::QS * C], c);
            const uint2 wq = __ldg(&tw[(1u << (G::LO + G::RB - 1)) + (ulo | ((uint32_t)q << G::LO))]);
            x[0][q] = d;
            x[0][q + H] = Ar<SET>::twiddle(d, wq, c);
        }
        constexpr int LIM = E * G::R / 8;
        dif_regs<SET, G::LO, G::RB, 1, G::RB - 2, LIM>(x, ulo, tw, c);
#pragma unroll
        for (int q = 0; q < LIM; ++q) s[q * G::QS * C] = x[0][q];
    }
}

// The forward column pass: column group x (C columns) and y = prime*2 +
// operand (or just the prime for a square or a launch of one operand) of
// product z; nx = column groups per (prime, operand).
template <int SET, int M, int C, int MR, int K2 = 0, int E = 8>
__global__ void __launch_bounds__(col_threads(C, M), cols_minb(M, MR, C)) k_fwd_cols(ProdArgs args, const ProdPtrs* __restrict__ batch) {
    extern __shared__ uint32_t sm[];
    pdl_enter();
#define PREC_K2 K2
#define PREC_E E
#define PREC_TILE_X blockIdx.x
#define PREC_TILE_Y blockIdx.y
#define PREC_TILE_NX gridDim.x
#define PREC_TILE_PRODUCT select_product(args, batch)
#include "ntt_cols_fwd_body.inc"
#undef PREC_K2
#undef PREC_E
#undef PREC_TILE_X
#undef PREC_TILE_Y
#undef PREC_TILE_NX
#undef PREC_TILE_PRODUCT
}

// One tile of the forward column pass at the indices ix (a persistent kernel's).
template <int SET, int M, int C, int MR>
__device__ __forceinline__ void fwd_cols_tile(const ProdArgs& args, const ProdPtrs* __restrict__ batch,
                                              const TileIdx& ix, uint32_t* sm) {
#define PREC_K2 0
#define PREC_E 8
#define PREC_TILE_X ix.bx
#define PREC_TILE_Y ix.by
#define PREC_TILE_NX ix.nbx
#define PREC_TILE_PRODUCT select_product_at(args, batch, ix.bz)
#include "ntt_cols_fwd_body.inc"
#undef PREC_K2
#undef PREC_E
#undef PREC_TILE_X
#undef PREC_TILE_Y
#undef PREC_TILE_NX
#undef PREC_TILE_PRODUCT
}

// The inverse column pass: column group x, prime args.prime0 + y of
// product z.
template <int SET, int M, int C, int MR, int K2 = 0, int E = 8>
__global__ void __launch_bounds__(col_threads(C, M), cols_minb(M, MR, C)) k_inv_cols(ProdArgs args, const ProdPtrs* __restrict__ batch) {
    extern __shared__ uint32_t sm[];
    pdl_enter();
#define PREC_K2 K2
#define PREC_E E
#define PREC_TILE_X blockIdx.x
#define PREC_TILE_Y blockIdx.y
#define PREC_TILE_PRODUCT select_product(args, batch)
#include "ntt_cols_inv_body.inc"
#undef PREC_K2
#undef PREC_E
#undef PREC_TILE_X
#undef PREC_TILE_Y
#undef PREC_TILE_PRODUCT
}

// One tile of the inverse column pass at the indices ix.
template <int SET, int M, int C, int MR>
__device__ __forceinline__ void inv_cols_tile(const ProdArgs& args, const ProdPtrs* __restrict__ batch,
                                              const TileIdx& ix, uint32_t* sm) {
#define PREC_K2 0
#define PREC_E 8
#define PREC_TILE_X ix.bx
#define PREC_TILE_Y ix.by
#define PREC_TILE_PRODUCT select_product_at(args, batch, ix.bz)
#include "ntt_cols_inv_body.inc"
#undef PREC_K2
#undef PREC_E
#undef PREC_TILE_X
#undef PREC_TILE_Y
#undef PREC_TILE_PRODUCT
}

// ---------------------------------------------------------------------------

#define PREC_COLS_CONFIGS(X)                                                                            \
    X(0, 6, 4, 6) X(0, 6, 8, 6) X(0, 7, 4, 6) X(0, 7, 8, 6) X(0, 8, 4, 6) X(0, 8, 8, 6) X(0, 9, 4, 6)     \
    X(0, 9, 8, 6) X(0, 10, 4, 4) X(0, 10, 8, 4) X(0, 10, 4, 6) X(0, 10, 8, 6) X(0, 11, 4, 4)              \
    X(0, 11, 8, 4) X(0, 11, 4, 6) X(0, 11, 8, 6) X(1, 11, 4, 4) X(1, 11, 8, 4) X(1, 11, 4, 6)             \
    X(1, 11, 8, 6) X(1, 12, 4, 6) X(1, 13, 4, 6) X(1, 10, 4, 6) X(1, 10, 8, 6)

// the forward column kernels of sets 2 and 3 (64-bit digits) in the
// (M, C, MR) configurations of sets 0 and 1; their other kernels are set 0's
// and set 1's
#define PREC_COLS_WIDE_CONFIGS(X)                                                                       \
    X(2, 6, 4, 6) X(2, 6, 8, 6) X(2, 7, 4, 6) X(2, 7, 8, 6) X(2, 8, 4, 6) X(2, 8, 8, 6) X(2, 9, 4, 6)     \
    X(2, 9, 8, 6) X(2, 10, 4, 4) X(2, 10, 8, 4) X(2, 10, 4, 6) X(2, 10, 8, 6) X(2, 11, 4, 4)              \
    X(2, 11, 8, 4) X(2, 11, 4, 6) X(2, 11, 8, 6) X(3, 10, 4, 6) X(3, 10, 8, 6) X(3, 11, 4, 4)             \
    X(3, 11, 8, 4) X(3, 11, 4, 6) X(3, 11, 8, 6) X(3, 12, 4, 6)

// (SET, M, C, MR, K2) of the default configurations (set 0: N1 =
// 2^floor(k/2), set 2 also wide_column_log2's; sets 1 and 3: N2 = 2^13), compiled
// with a constant row length.  The inverse columns of sets 2 and 3 are set 0's and set 1's.
#define PREC_COLS_FWD_K2_CONFIGS(X)                                                                        \
    X(0, 6, 8, 6, 7) X(0, 7, 8, 6, 7) X(0, 7, 8, 6, 8) X(0, 8, 8, 6, 8) X(0, 8, 8, 6, 9) X(0, 9, 8, 6, 9)   \
    X(0, 9, 8, 6, 10) X(0, 10, 8, 6, 10) X(0, 10, 8, 6, 11) X(0, 11, 8, 6, 11) X(0, 11, 8, 6, 12)           \
    X(2, 9, 8, 6, 9) X(2, 9, 8, 6, 10) X(2, 10, 8, 6, 10) X(2, 10, 8, 6, 11) X(2, 11, 8, 6, 11)             \
    X(2, 10, 8, 6, 12)                                                                                     \
    X(1, 11, 8, 6, 13) X(1, 12, 4, 6, 13) X(1, 13, 4, 6, 13) X(3, 10, 8, 6, 13) X(3, 11, 8, 6, 13)         \
    X(3, 12, 4, 6, 13)
#define PREC_COLS_INV_K2_CONFIGS(X)                                                                        \
    X(0, 6, 8, 6, 7) X(0, 7, 8, 6, 7) X(0, 7, 8, 6, 8) X(0, 8, 8, 6, 8) X(0, 8, 8, 6, 9) X(0, 9, 8, 6, 9)   \
    X(0, 9, 8, 6, 10) X(0, 10, 8, 6, 10) X(0, 10, 8, 6, 11) X(0, 11, 8, 6, 11) X(0, 11, 8, 6, 12)           \
    X(0, 10, 8, 6, 12)                                                                                     \
    X(1, 10, 8, 6, 13) X(1, 11, 8, 6, 13) X(1, 12, 4, 6, 13) X(1, 13, 4, 6, 13)

// Batch classes with enough products take more short columns per CTA, 8192
// points as the 2^10-point columns have (col_batch_group): the bottom pass
// has 32 points per thread, so a tile of 8 columns of 2^8 points keeps 2 of its 8
// warps busy there and the other six at the barrier.
#define PREC_COLS_FWD_BATCH_CONFIGS(X) X(0, 8, 32, 6, 8) X(0, 8, 32, 6, 9) X(0, 9, 16, 6, 9) X(2, 9, 16, 6, 9) X(2, 9, 16, 6, 10)
#define PREC_COLS_INV_BATCH_CONFIGS(X) X(0, 8, 32, 6, 8) X(0, 8, 32, 6, 9) X(0, 9, 16, 6, 9) X(0, 9, 16, 6, 10)
#define PREC_COLS_FWD_BATCH_SHORT_CONFIGS(X) X(0, 7, 64, 6, 7) X(0, 7, 64, 6, 8)
#define PREC_COLS_INV_BATCH_SHORT_CONFIGS(X) X(0, 7, 64, 6, 7) X(0, 7, 64, 6, 8)
// (2^6-point columns: whole transforms only)
#define PREC_COLS_BATCH_SHORTEST_CONFIGS(X) X(0, 6, 64, 6, 7)

// The same configurations with columns of at least 2^7 points for transforms
// truncated to E eighths (E = 5, 7: 2^8 points and up; ntt_cols_trunc.inc).
#define PREC_COLS_FWD_TRUNC6_CONFIGS(X) X(0, 7, 8, 6, 7) X(0, 7, 8, 6, 8) PREC_COLS_FWD_BATCH_SHORT_CONFIGS(X)
#define PREC_COLS_INV_TRUNC6_CONFIGS(X) X(0, 7, 8, 6, 7) X(0, 7, 8, 6, 8) PREC_COLS_INV_BATCH_SHORT_CONFIGS(X)
#define PREC_COLS_FWD_TRUNC_CONFIGS(X)                                                                      \
    X(0, 8, 8, 6, 8) X(0, 8, 8, 6, 9) X(0, 9, 8, 6, 9) X(0, 9, 8, 6, 10) X(0, 10, 8, 6, 10)                 \
    X(0, 10, 8, 6, 11) X(0, 11, 8, 6, 11) X(0, 11, 8, 6, 12) X(2, 9, 8, 6, 9) X(2, 9, 8, 6, 10)             \
    PREC_COLS_FWD_BATCH_CONFIGS(X) X(2, 10, 8, 6, 10) X(2, 10, 8, 6, 11) X(2, 10, 8, 6, 12) X(1, 11, 8, 6, 13) X(1, 12, 4, 6, 13)          \
    X(1, 13, 4, 6, 13) X(3, 10, 8, 6, 13) X(3, 11, 8, 6, 13) X(3, 12, 4, 6, 13)
#define PREC_COLS_INV_TRUNC_CONFIGS(X)                                                                      \
    X(0, 8, 8, 6, 8) X(0, 8, 8, 6, 9) X(0, 9, 8, 6, 9) X(0, 9, 8, 6, 10) X(0, 10, 8, 6, 10)                 \
    X(0, 10, 8, 6, 11) X(0, 11, 8, 6, 11) X(0, 11, 8, 6, 12) X(1, 10, 8, 6, 13) X(1, 11, 8, 6, 13)          \
    X(0, 10, 8, 6, 12) PREC_COLS_INV_BATCH_CONFIGS(X) X(1, 12, 4, 6, 13) X(1, 13, 4, 6, 13)

inline size_t col_smem(int m, int cg) { return (size_t)cg * astride_for(m) * sizeof(uint32_t); }

// the K2 instantiations (ntt_cols_fwd_k2.cu, ntt_cols_inv_k2.cu): launch the
// one matching (set, a.k1, cg, mr, a.k2) and return true, or return false.
bool launch_fwd_cols_k2(int set, const ProdArgs& a, int cg, int mr, dim3 grid, size_t smem, cudaStream_t st,
                        const ProdPtrs* batch);
bool launch_inv_cols_k2(int set, const ProdArgs& a, int cg, int mr, dim3 grid, size_t smem, cudaStream_t st,
                        const ProdPtrs* batch);
int configure_fwd_cols_k2();
int configure_inv_cols_k2();
// the truncated instantiations of E eighths (a.keep = E), one translation
// unit per direction and E
#define PREC_TRUNC_DECL(E)                                                                                     \
    bool launch_fwd_cols_trunc##E(int set, const ProdArgs& a, int cg, int mr, dim3 grid, size_t smem, cudaStream_t st, \
                                  const ProdPtrs* batch);                                                     \
    bool launch_inv_cols_trunc##E(int set, const ProdArgs& a, int cg, int mr, dim3 grid, size_t smem, cudaStream_t st, \
                                  const ProdPtrs* batch);                                                     \
    int configure_fwd_cols_trunc##E();                                                                        \
    int configure_inv_cols_trunc##E();
PREC_TRUNC_DECL(5)
PREC_TRUNC_DECL(6)
PREC_TRUNC_DECL(7)
#undef PREC_TRUNC_DECL

}  // namespace precgpu
