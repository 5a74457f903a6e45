// ntt_lat.cu -- the transform passes of one mid-size product (2^13 .. 2^18
// points), built for latency.
//
// Such a product leaves the GPU mostly idle: its passes are chains of a
// load, a few register passes and a store, and what counts is how long one
// thread's share is.  The throughput kernels (ntt_cols.cuh, ntt_rows.cuh)
// give a thread 32 points of the last pass, two operands' in the rows, 1200 -
// 3200 instructions in a row from two or three warps per SM.  Here a thread
// holds 8 points (two operands' in the rows): columns and rows of 2^M points
// run as a radix-2^(M-6), a radix-8 and a radix-8 pass, with four to eight
// times the threads; the first pass reads global memory directly.
// Shared memory has one spare word per eight (element i at P(i) = i + i/8):
// conflict-free for both radix-8 passes.
// Whole products, throughput kernels -> these: 2^14 points 18.4 -> 11.4 us, 2^15
// 18.2 -> 12.5, 2^16 18.9 -> 13.8, 2^17 19.6 -> 14.9, 2^18 (64-bit digits) 31.6 ->
// 28.1.  From 2^19 points, and in batches, the GPU is full
// and the fewer passes of the throughput kernels count.
#include <cooperative_groups.h>

#include "ntt_engine.cuh"

namespace precgpu {

namespace {

__device__ __forceinline__ constexpr int p8(int i) { return i + (i >> 3); }
constexpr int lat_words(int m) { return (1 << m) + (1 << (m - 3)); }  // padded words of one array
constexpr int kLatC = 8;          // columns per column CTA
constexpr int kLatRowThreads = 64;  // threads of a row CTA

__device__ __forceinline__ constexpr int brev3(int q) { return ((q & 1) << 2) | (q & 2) | (q >> 2); }

// x[brev3(j)] *= t * g^j
template <int SET>
__device__ __forceinline__ void twiddle8(uint32_t (&x)[8], uint32_t t, uint32_t g, const PrimeC& pc) {
    // (two chains by g^2: half as long)
    uint32_t s = Ar<SET>::mul(t, g, pc);
    const uint32_t g2 = Ar<SET>::mul(g, g, pc);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
        x[brev3(j)] = Ar<SET>::mul(x[brev3(j)], t, pc);
        x[brev3(j + 1)] = Ar<SET>::mul(x[brev3(j + 1)], s, pc);
        if (j < 6) {
            t = Ar<SET>::mul(t, g2, pc);
            s = Ar<SET>::mul(s, g2, pc);
        }
    }
}

}  // namespace

// Forward columns: grid (N2 / 8, primes * operands), 2^M threads.  E: the
// transform is truncated to E eighths (ntt_engine.cuh; both operands in the
// lower half).
template <int SET, int M, int K2, int E>
__global__ void __launch_bounds__(1 << M) k_fwd_cols_lat(ProdArgs args) {
    constexpr int C = kLatC, R = 1 << (M - 6), KK = M + K2, KEPT = E == 8 ? R : E * R / 8;
    static_assert(E == 8 || E * R % 8 == 0, "whole blocks of the first pass");
    constexpr uint32_t N2 = 1u << K2;
    __shared__ uint32_t sm[lat_words(M) * C];  // element i of column c at P(i) * C + c
    pdl_enter();
    const bool one = args.square != 0;
    const int prime = one ? blockIdx.y : blockIdx.y >> 1;
    const int operand = one ? 0 : blockIdx.y & 1;
    const PrimeC pc = args.f.pc[prime];
    const uint2* __restrict__ tw = args.f.tf[prime];
    const uint32_t c0 = blockIdx.x * C;
    const uint64_t* __restrict__ src = after_entry(operand ? args.b : args.a);
    const uint64_t nl = operand ? args.lb : args.la;
    // the carry kernel's look-back words start at zero
    if (blockIdx.y == 0)
        for (int i = blockIdx.x * blockDim.x + threadIdx.x; i <= args.nblk; i += gridDim.x * blockDim.x) args.scratch[i] = 0;
    // digit of row i1 of a column, zero past the operand
    auto digit = [&](int i1, int col) -> uint32_t {
        const uint64_t i = (uint64_t)i1 * N2 + c0 + col;
        if constexpr (set_wide(SET)) {
            const uint64_t v = i < nl ? src[i] : 0;
            return Ar<SET>::digit64((uint32_t)v, (uint32_t)(v >> 32), pc);
        } else {
            return i < 2 * nl ? Ar<SET>::digit(reinterpret_cast<const uint32_t*>(src)[i], pc) : 0u;
        }
    };
    const bool half = (set_wide(SET) ? nl : 2 * nl) <= (1ull << (KK - 1));  // the upper half is zero
#pragma unroll
    for (int w = threadIdx.x; w < 64 * C; w += 1 << M) {
        const int col = w % C, u = w / C;
        uint32_t x[1][R];
        if constexpr (R == 1) {
            x[0][0] = digit(u, col);
        } else if (half) {
#pragma unroll
            for (int q = 0; q < R / 2; ++q) {
                x[0][q] = digit(q * 64 + u, col);
                x[0][q + R / 2] = Ar<SET>::twiddle(x[0][q], __ldg(&tw[(1u << (M - 1)) + q * 64 + u]), pc);
            }
            if constexpr (R > 2) dif_regs<SET, 6, M - 6, 1, M - 8, E * R / 8>(x, u, tw, pc);
        } else if constexpr (E == 8) {
#pragma unroll
            for (int q = 0; q < R; ++q) x[0][q] = digit(q * 64 + u, col);
            dif_regs<SET, 6, M - 6, 1>(x, u, tw, pc);
        } else {  // a truncated plan has both operands in the lower half
            if (threadIdx.x == 0) atomicOr(args.err, kDevErrPlan);
            return;
        }
#pragma unroll
        for (int q = 0; q < KEPT; ++q) sm[p8(q * 64 + u) * C + col] = x[0][q];
    }
    __syncthreads();
    const int col = threadIdx.x % C, u = threadIdx.x / C;
    const bool on = E == 8 || threadIdx.x < (E << M) / 8;  // items of the kept eighths
    uint32_t x[1][8];
    if (on) {
        uint32_t* s = sm + p8((u >> 3) * 64 + (u & 7)) * C + col;
#pragma unroll
        for (int q = 0; q < 8; ++q) x[0][q] = s[q * 9 * C];
        dif_regs<SET, 3, 3, 1>(x, u & 7, tw, pc);
#pragma unroll
        for (int q = 0; q < 8; ++q) s[q * 9 * C] = x[0][q];
    }
    // slot 8u + q holds k1 = brev3(q) << (M-3) | brev(u): twiddle t * g^brev3(q)
    const uint32_t i2 = c0 + col;
    const uint32_t t = fourstep_twiddle<SET>(args.f, prime, i2 * brev_bits(u, M - 3), KK);
    const uint32_t g = fourstep_twiddle<SET>(args.f, prime, i2 << (M - 3), KK);
    __syncthreads();
    if (!on) return;
    const uint32_t* s = sm + 9 * u * C + col;
#pragma unroll
    for (int q = 0; q < 8; ++q) x[0][q] = s[q * C];
    dif_regs<SET, 0, 3, 1>(x, 0, tw, pc);
    twiddle8<SET>(x[0], t, g, pc);
    uint32_t* __restrict__ dst = args.work + ((uint64_t)(prime * 2 + operand) << KK) + (uint64_t)(8 * u) * N2 + i2;
#pragma unroll
    for (int q = 0; q < 8; ++q) dst[q * N2] = x[0][q];
}

// Rows: 2^(M-3) threads per row, both operands; grid (N1 / rows per CTA, primes).
template <int SET, int M, bool SQ>
__global__ void __launch_bounds__(kLatRowThreads) k_rows_lat(ProdArgs args) {
    constexpr int TPR = 1 << (M - 3), RPC = kLatRowThreads / TPR, R = 1 << (M - 6);
    constexpr int AS = lat_words(M), NA = SQ ? 1 : 2;
    __shared__ uint32_t sm[RPC * NA * AS];
    pdl_enter();
    const int prime = blockIdx.y;
    const PrimeC pc = args.f.pc[prime];
    const uint2* __restrict__ twf = args.f.tf[prime];
    const uint2* __restrict__ twi = args.f.ti[prime];
    const int r = threadIdx.x / TPR, v = threadIdx.x % TPR;
    uint32_t* __restrict__ A = after_entry(args.work) + ((uint64_t)(prime * 2) << args.k) +
                               ((uint64_t)(blockIdx.x * RPC + r) << M);
    const uint32_t* B = A + (1ull << args.k);
    uint32_t* srow = sm + r * NA * AS;
#pragma unroll
    for (int u = v; u < 64; u += TPR) {
        uint32_t x[NA][R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            x[0][q] = A[q * 64 + u];
            if constexpr (!SQ) x[NA - 1][q] = B[q * 64 + u];
        }
        dif_regs<SET, 6, M - 6, NA>(x, u, twf, pc);
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
            for (int q = 0; q < R; ++q) srow[a * AS + p8(q * 64 + u)] = x[a][q];
    }
    __syncthreads();
    uint32_t* smid = srow + p8((v >> 3) * 64 + (v & 7));
    uint32_t x[NA][8];
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int q = 0; q < 8; ++q) x[a][q] = smid[a * AS + q * 9];
    dif_regs<SET, 3, 3, NA>(x, v & 7, twf, pc);
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int q = 0; q < 8; ++q) smid[a * AS + q * 9] = x[a][q];
    __syncthreads();
    uint32_t* sbot = srow + 9 * v;
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
        for (int q = 0; q < 8; ++q) x[a][q] = sbot[a * AS + q];
    dif_regs<SET, 0, 3, NA>(x, 0, twf, pc);
    uint32_t y[1][8];
#pragma unroll
    for (int q = 0; q < 8; ++q) y[0][q] = Ar<SET>::mul(x[0][q], x[NA - 1][q], pc);
    dit_regs<SET, 0, 3, 1>(y, 0, twi, pc);
#pragma unroll
    for (int q = 0; q < 8; ++q) sbot[q] = y[0][q];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) y[0][q] = smid[q * 9];
    dit_regs<SET, 3, 3, 1>(y, v & 7, twi, pc);
#pragma unroll
    for (int q = 0; q < 8; ++q) smid[q * 9] = y[0][q];
    __syncthreads();
#pragma unroll
    for (int u = v; u < 64; u += TPR) {
        uint32_t z[1][R];
#pragma unroll
        for (int q = 0; q < R; ++q) z[0][q] = srow[p8(q * 64 + u)];
        dit_regs<SET, 6, M - 6, 1>(z, u, twi, pc);
#pragma unroll
        for (int q = 0; q < R; ++q) A[q * 64 + u] = Ar<SET>::half(z[0][q], pc);
    }
}

// Inverse columns: grid (N2 / 8, primes), 2^M threads.
template <int SET, int M, int K2, int E>
__global__ void __launch_bounds__(1 << M) k_inv_cols_lat(ProdArgs args) {
    constexpr int C = kLatC, R = 1 << (M - 6), KK = M + K2, KEPT = E == 8 ? R : E * R / 8;
    constexpr uint32_t N2 = 1u << K2;
    __shared__ uint32_t sm[lat_words(M) * C];
    const int prime = blockIdx.y;
    const PrimeC pc = args.f.pc[prime];
    const uint2* __restrict__ tw = args.f.ti[prime];
    const int col = threadIdx.x % C, u = threadIdx.x / C;
    const uint32_t c0 = blockIdx.x * C, i2 = c0 + col;
    constexpr uint32_t nmask = (1u << KK) - 1;
    const uint32_t fold = args.f.nprimes == kMaxPrimes ? args.crt5.fold[prime] : args.crt.fold[prime];
    const uint32_t t = Ar<SET>::mul(fourstep_twiddle<SET>(args.f, prime, (0u - i2 * brev_bits(u, M - 3)) & nmask, KK),
                                    fold, pc);
    const uint32_t g = fourstep_twiddle<SET>(args.f, prime, (0u - (i2 << (M - 3))) & nmask, KK);
    pdl_enter();
    uint32_t* __restrict__ wk = after_entry(args.work) + ((uint64_t)(prime * 2) << KK);
    const bool on = E == 8 || threadIdx.x < (E << M) / 8;  // items of the kept eighths
    uint32_t x[1][8];
    if (on) {
        const uint32_t* src = wk + (uint64_t)(8 * u) * N2 + i2;
#pragma unroll
        for (int q = 0; q < 8; ++q) x[0][q] = src[q * N2];
        twiddle8<SET>(x[0], t, g, pc);
        dit_regs<SET, 0, 3, 1>(x, 0, tw, pc);
        uint32_t* s0 = sm + 9 * u * C + col;
#pragma unroll
        for (int q = 0; q < 8; ++q) s0[q * C] = x[0][q];
    }
    __syncthreads();
    uint32_t* s = sm + p8((u >> 3) * 64 + (u & 7)) * C + col;
    if (on) {
#pragma unroll
        for (int q = 0; q < 8; ++q) x[0][q] = s[q * 9 * C];
        dit_regs<SET, 3, 3, 1>(x, u & 7, tw, pc);
    }
    if constexpr (R == 1) {
#pragma unroll
        for (int q = 0; q < 8; ++q) wk[(uint64_t)((u >> 3) * 64 + (u & 7) + 8 * q) * N2 + i2] = x[0][q];
    } else {
        if (on) {
#pragma unroll
            for (int q = 0; q < 8; ++q) s[q * 9 * C] = x[0][q];
        }
        __syncthreads();
#pragma unroll
        for (int w = threadIdx.x; w < 64 * C; w += 1 << M) {
            const int cl = w % C, uu = w / C;
            uint32_t z[1][R];
#pragma unroll
            for (int q = 0; q < KEPT; ++q) z[0][q] = sm[p8(q * 64 + uu) * C + cl];
            if constexpr (E == 8) dit_regs<SET, 6, M - 6, 1>(z, uu, tw, pc);
            else dit_top_trunc<SET, 6, M - 6, E>(z, uu, args.f.tf[prime], tw, pc);
#pragma unroll
            for (int q = 0; q < KEPT; ++q) wk[(uint64_t)(q * 64 + uu) * N2 + c0 + cl] = z[0][q];
        }
    }
}

// CRT and carries of up to 8 * 1024 * L limbs (32-bit digits) as one cluster:
// L limbs per thread; each CTA puts its carry aggregate into every CTA's shared
// memory, one cluster barrier, and every limb is written once, final.  (The
// general kernel's join by the last block -- fence, counter, aggregates
// read back -- is a third of its time at these sizes.)  Products of 2^14
// points 12.9 -> 11.4 us, 2^15 13.3 -> 12.5; with 4 limbs per thread 2^16 would
// go 13.8 -> 17.2, eight SMs are too few.
constexpr int kClThreads = 1024;
constexpr int kClCtas = 8;

template <int L>
__global__ void __launch_bounds__(kClThreads) k_crt_cluster(ProdArgs args) {
    namespace cg = cooperative_groups;
    __shared__ uint32_t s_wg[32], s_wp[32], s_blk[kClCtas];
    __shared__ uint64_t s_hi[32];
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = blockIdx.x, ranks = gridDim.x;
    cluster.barrier_arrive();  // (the other CTAs' shared memory exists once all arrived)
    pdl_enter();
    const uint64_t N = 1ull << args.k;
    const uint64_t nc = (uint64_t)args.keep << args.k >> 3;  // coefficients there are
    const uint32_t* __restrict__ r0 = after_entry(args.work);
    const uint32_t* __restrict__ r1 = r0 + 2 * N;
    const uint32_t* __restrict__ r2 = r0 + 4 * N;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t m0 = ((int64_t)rank * kClThreads + threadIdx.x) * L;
    u128 T[L];
    {
        uint2 y[3][L];
#pragma unroll
        for (int k = 0; k < L; ++k) {
            const uint64_t i = 2 * (uint64_t)(m0 + k);  // even, as nc
            const bool in = i < nc;
            y[0][k] = in ? *reinterpret_cast<const uint2*>(r0 + i) : make_uint2(0, 0);
            y[1][k] = in ? *reinterpret_cast<const uint2*>(r1 + i) : make_uint2(0, 0);
            y[2][k] = in ? *reinterpret_cast<const uint2*>(r2 + i) : make_uint2(0, 0);
        }
#pragma unroll
        for (int k = 0; k < L; ++k)
            T[k] = crt3_folded<0>(y[0][k].x, y[1][k].x, y[2][k].x, args.crt, args.f) +
                   (crt3_folded<0>(y[0][k].y, y[1][k].y, y[2][k].y, args.crt, args.f) << 32);
    }
    const uint64_t hi_last = (uint64_t)(T[L - 1] >> 64);
    uint64_t prev_hi = __shfl_up_sync(0xffffffffu, hi_last, 1);
    if (lane == 31) s_hi[warp] = hi_last;
    if (threadIdx.x == 0) {  // the limb below the CTA's first
        prev_hi = 0;
        const uint64_t i = 2 * (uint64_t)(m0 - 1);
        if (m0 > 0 && i < nc) {
            const uint2 a = *reinterpret_cast<const uint2*>(r0 + i), b = *reinterpret_cast<const uint2*>(r1 + i),
                        c = *reinterpret_cast<const uint2*>(r2 + i);
            prev_hi = (uint64_t)((crt3_folded<0>(a.x, b.x, c.x, args.crt, args.f) +
                                  (crt3_folded<0>(a.y, b.y, c.y, args.crt, args.f) << 32)) >> 64);
        }
    }
    __syncthreads();
    if (lane == 0 && warp > 0) prev_hi = s_hi[warp - 1];
    uint64_t v[L];
    uint32_t gbits;
    bool G, P;
    limbs_from_sums<L>(T, prev_hi, v, gbits, G, P);
    const uint32_t gm = __ballot_sync(0xffffffffu, G), pm = __ballot_sync(0xffffffffu, P);
    if (lane == 0) {
        s_wg[warp] = (uint32_t)(carry_chain(gm, pm, false) >> 32) & 1;
        s_wp[warp] = pm == 0xffffffffu;
    }
    __syncthreads();
    const uint32_t bg = __ballot_sync(0xffffffffu, s_wg[lane] != 0), bp = __ballot_sync(0xffffffffu, s_wp[lane] != 0);
    const uint64_t c0 = carry_chain(bg, bp, false);
    cluster.barrier_wait();
    if (ranks > 1) {
        if (warp == 0 && lane < (int)ranks)
            *cluster.map_shared_rank(&s_blk[rank], lane) = ((uint32_t)(c0 >> 32) & 1) | (bp == 0xffffffffu ? 2u : 0u);
        cluster.sync();
    }
    bool cin = false;
    for (uint32_t r = 0; r < rank; ++r) cin = (s_blk[r] & 1) || ((s_blk[r] & 2) && cin);
    const uint64_t cw = carry_chain(bg, bp, cin);
    limbs_finish<L>(m0, args.lout, v, gbits, (carry_chain(gm, pm, (cw >> warp) & 1) >> lane) & 1, args.out);
    if (rank == ranks - 1 && threadIdx.x == 0 && (cw >> 32) & 1)
        atomicOr(args.err, kDevErrCarry);  // a product fits La+Lb limbs
}

template <int L>
static void launch_cluster(const ProdArgs& a, cudaStream_t st) {
    const unsigned n = (unsigned)((a.lout + kClThreads * L - 1) / (kClThreads * L));
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = n;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = n;
    cfg.blockDim = kClThreads;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, k_crt_cluster<L>, a);
    count_launches(1);
}

// (k1, k2) of the default configurations (set 2's fit from 2^18 points) and
// the eighths they are instantiated for
#define PREC_LAT(X) \
    X(0, 6, 7, 8) X(0, 7, 7, 8) X(0, 7, 8, 8) X(0, 8, 8, 8) X(0, 8, 8, 6) X(0, 8, 9, 8) X(0, 8, 9, 6) X(0, 9, 9, 8) \
    X(0, 9, 9, 7) X(0, 9, 9, 6) X(0, 9, 9, 5) X(2, 9, 9, 8) X(2, 9, 9, 7) X(2, 9, 9, 6) X(2, 9, 9, 5)

int lat_keep(int set, int k1, int k2, int keep) {
    for (; keep <= 8; ++keep) {
#define X(S, A, B, E) \
    if (set == S && k1 == A && k2 == B && keep == E) return E;
        PREC_LAT(X)
#undef X
    }
    return 0;
}

template <int M>
static void launch_rows_lat(const ProdArgs& a, int nprimes, cudaStream_t st) {
    const dim3 grid(((unsigned)a.keep << a.k1) / 8 / (kLatRowThreads >> (M - 3)), nprimes);
    if (a.square) launch_pdl(false, k_rows_lat<0, M, true>, grid, kLatRowThreads, 0, st, a);
    else launch_pdl(false, k_rows_lat<0, M, false>, grid, kLatRowThreads, 0, st, a);
}

void ntt_launch_lat(int set, const ProdArgs& a, cudaStream_t st, cudaEvent_t* ev) {
    const int np = kSetPrimes[set];
    if (ev) cudaEventRecord(ev[0], st);
#define X(S, A, B, E)                                                                                          \
    if (set == S && a.k1 == A && a.k2 == B && a.keep == E)                                                     \
        launch_pdl(false, k_fwd_cols_lat<S, A, B, E>, dim3((1u << B) / kLatC, (a.square ? 1 : 2) * np), 1 << A, 0, st, a);
    PREC_LAT(X)
#undef X
    if (ev) cudaEventRecord(ev[1], st);
    if (a.k2 == 7) launch_rows_lat<7>(a, np, st);
    else if (a.k2 == 8) launch_rows_lat<8>(a, np, st);
    else launch_rows_lat<9>(a, np, st);
    if (ev) cudaEventRecord(ev[2], st);
#define X(S, A, B, E)                                                                       \
    if (S == 0 && a.k1 == A && a.k2 == B && a.keep == E)                                    \
        launch_pdl(false, k_inv_cols_lat<0, A, B, E>, dim3((1u << B) / kLatC, np), 1 << A, 0, st, a);
    PREC_LAT(X)
#undef X
    if (ev) cudaEventRecord(ev[3], st);
    count_launches(3);
    constexpr uint64_t one = (uint64_t)kClThreads * kClCtas;
    if (set == 0 && a.lout <= one) launch_cluster<1>(a, st);
    else if (set == 0 && a.lout <= 2 * one) launch_cluster<2>(a, st);
    else launch_crt_carry(set, a, st);
    if (ev) cudaEventRecord(ev[4], st);
}

int configure_lat() {
    cudaError_t e = cudaSuccess;
#define X(S, A, B, E)                                      \
    if (!e) e = load_kernel(k_fwd_cols_lat<S, A, B, E>);   \
    if (!e && S == 0) e = load_kernel(k_inv_cols_lat<0, A, B, E>);
    PREC_LAT(X)
#undef X
#define X(M)                                        \
    if (!e) e = load_kernel(k_rows_lat<0, M, true>); \
    if (!e) e = load_kernel(k_rows_lat<0, M, false>);
    X(7) X(8) X(9)
#undef X
    if (!e) e = load_kernel(k_crt_cluster<1>);
    if (!e) e = load_kernel(k_crt_cluster<2>);
    return (int)e;
}

}  // namespace precgpu
