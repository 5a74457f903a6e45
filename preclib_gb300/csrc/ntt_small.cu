// ntt_small.cu -- single-CTA products (transforms of 2^5 .. 2^12 points).
//
// One CTA runs the whole of the reference's mul_ntt (src/mul_ntt.cpp:494-518)
// for one product in shared memory: digits of both operands, forward DIF,
// pointwise product and inverse DIT for each of the three primes, then CRT
// and the carry chain (block-wide scan).  With a descriptor array the same
// kernel runs one product per CTA for a whole batch of a length class.
//
// Bound by the integer multiply pipe.  A third of the threads to each prime: the
// bottom pass, half of the work, has an item for every thread and the barriers
// are those of one prime's transform.  (The primes in turn, with eight
// points per thread: three quarters of the threads had no bottom item.  ns per
// product of a large batch, before -> now: 256 x 256 limbs 29.1 -> 20.2, 512 x 512
// 70 -> 39, 1024 x 1024 111 -> 91; 200 products of 256 limbs 22.6 -> 14.7 us; one of
// 128 limbs between host arrays 41 -> 30.)
#include "ntt_engine.cuh"

namespace precgpu {

// Threads per prime: one for each of the bottom pass's items (32 points), a warp
// at least.  The three primes run side by side.
constexpr int small_tp(int m) { return m <= 10 ? 32 : 1 << (m - 5); }
constexpr int small_threads(int m) { return kPrimes * small_tp(m); }
constexpr int kSmallRadix = 5;  // register passes of up to 5 stages
// Resident CTAs the registers are limited for: what shared memory holds
// (six arrays of 2^m words); short lengths run alone and are not limited.
constexpr int small_minb(int m) { return m < 9 ? 1 : 768 / small_threads(m); }

// pass T over NA arrays of one prime by its TP threads
template <int M, int T, bool DIT, int NA>
__device__ __forceinline__ void small_pass(uint32_t* s0, int t, const uint2* __restrict__ tw, const PrimeC& pc) {
    using G = Geom<M, T, kSmallRadix>;
    constexpr int AS = astride_for(M);
    for (uint32_t u = t; u < (1u << G::LGI); u += small_tp(M)) {
        uint32_t* s = s0 + G::pbase(u);
        uint32_t x[NA][G::R];
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
            for (int q = 0; q < G::R; ++q) x[a][q] = s[a * AS + q * G::QS];
        regs_pass<0, M, T, DIT, NA, kSmallRadix>(x, u, tw, pc);
#pragma unroll
        for (int a = 0; a < NA; ++a)
#pragma unroll
            for (int q = 0; q < G::R; ++q) s[a * AS + q * G::QS] = x[a][q];
    }
}

template <int M>
__global__ void __launch_bounds__(small_threads(M), small_minb(M))
    k_small(const SmallDesc* __restrict__ descs, SmallDesc single, FieldArgs f, CrtConst crt) {
    extern __shared__ uint32_t sm[];
    __shared__ BlockCarryShared sh;
    __shared__ uint64_t s_hi[small_threads(M) / 32];
    constexpr int MR = kSmallRadix;
    constexpr int NP = sch_np(M, MR);
    constexpr int AS = astride_for(M);
    constexpr int TP = small_tp(M);
    const int prime = threadIdx.x / TP, t = threadIdx.x % TP;
    const PrimeC pc = f.pc[prime];
    const uint2* __restrict__ twf = f.tf[prime];
    const uint2* __restrict__ twi = f.ti[prime];
    uint32_t* const s0 = sm + prime * 2 * AS;  // this prime's arrays: a (then the product), b
    pdl_enter();
    SmallDesc d = descs ? descs[blockIdx.x] : single;
    d.a = after_entry(d.a);
    d.b = after_entry(d.b);
    const uint32_t* __restrict__ da = reinterpret_cast<const uint32_t*>(d.a);
    const uint32_t* __restrict__ db = reinterpret_cast<const uint32_t*>(d.b);
    const uint32_t nda = 2 * (uint32_t)d.la, ndb = 2 * (uint32_t)d.lb;

    {   // top DIF pass from the limbs
        using G = Geom<M, 0, MR>;
        for (uint32_t u = t; u < (1u << G::LGI); u += TP) {
            const uint32_t base = G::base(u);
            uint32_t x[2][G::R];
#pragma unroll
            for (int q = 0; q < G::R; ++q) {
                const uint32_t i = base + ((uint32_t)q << G::LO);
                x[0][q] = i < nda ? Ar<0>::digit(__ldg(&da[i]), pc) : 0u;
                x[1][q] = i < ndb ? Ar<0>::digit(__ldg(&db[i]), pc) : 0u;
            }
            regs_pass<0, M, 0, false, 2, MR>(x, u, twf, pc);
            if constexpr (NP == 1) {  // 32 points: one register pass does everything
                uint32_t y[1][G::R];
#pragma unroll
                for (int q = 0; q < G::R; ++q) y[0][q] = Ar<0>::mul(x[0][q], x[1][q], pc);
                regs_pass<0, M, 0, true, 1, MR>(y, 0, twi, pc);
#pragma unroll
                for (int q = 0; q < G::R; ++q) s0[padded(q)] = y[0][q];
            } else {
                uint32_t* s = s0 + G::pbase(u);
#pragma unroll
                for (int q = 0; q < G::R; ++q) {
                    s[q * G::QS] = x[0][q];
                    s[AS + q * G::QS] = x[1][q];
                }
            }
        }
        __syncthreads();
    }
    if constexpr (NP > 1) {
        if constexpr (NP > 2) {
            static_assert(NP == 3);
            small_pass<M, 1, false, 2>(s0, t, twf, pc);
            __syncthreads();
        }
        if (t < (1 << (M - 5))) {  // bottom: last DIF stages, product, first DIT stages
            uint32_t* s = s0 + 33 * t;
            uint32_t x[2][32];
#pragma unroll
            for (int q = 0; q < 32; ++q) {
                x[0][q] = s[q];
                x[1][q] = s[AS + q];
            }
            regs_pass<0, M, NP - 1, false, 2, MR>(x, t, twf, pc);
            uint32_t y[1][32];
#pragma unroll
            for (int q = 0; q < 32; ++q) y[0][q] = Ar<0>::mul(x[0][q], x[1][q], pc);
            regs_pass<0, M, NP - 1, true, 1, MR>(y, t, twi, pc);
#pragma unroll
            for (int q = 0; q < 32; ++q) s[q] = y[0][q];
        }
        __syncthreads();
        if constexpr (NP > 2) {
            small_pass<M, 1, true, 1>(s0, t, twi, pc);
            __syncthreads();
        }
        small_pass<M, 0, true, 1>(s0, t, twi, pc);
        __syncthreads();
    }

    // CRT + carries over the block, L limbs per thread
    constexpr int L = 6;
    static_assert(small_threads(M) * L >= (1 << M) / 2, "every limb in one round");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int m0 = (int)threadIdx.x * L;
    u128 T[L];
#pragma unroll
    for (int k = 0; k < L; ++k) {
        u128 c[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int i = 2 * (m0 + k) + e, pi = padded(i);
            c[e] = i < (1 << M) ? crt3(sm[pi], sm[2 * AS + pi], sm[4 * AS + pi], crt, f) : (u128)0;
        }
        T[k] = c[0] + (c[1] << 32);
    }
    const uint64_t hi = (uint64_t)(T[L - 1] >> 64);
    uint64_t prev_hi = __shfl_up_sync(0xffffffffu, hi, 1);
    if (lane == 31) s_hi[warp] = hi;
    __syncthreads();
    if (lane == 0) prev_hi = warp ? s_hi[warp - 1] : 0;
    uint64_t v[L];
    uint32_t gbits;
    bool G, P;
    limbs_from_sums<L>(T, prev_hi, v, gbits, G, P);
    const bool cin = block_carry_in0(G, P, sh, [](bool, bool) {});  // (no carry out: the product fits)
    limbs_finish<L>(m0, d.lout, v, gbits, cin, d.out);
}

// ---------------------------------------------------------------------------

size_t ntt_small_smem_bytes(int k) { return (size_t)2 * kPrimes * astride_for(k) * sizeof(uint32_t); }

#define PREC_SMALL(X) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12)

void ntt_launch_small(const SmallDesc* d_descs, const SmallDesc* single, int count, int k, const FieldArgs& f,
                      const CrtConst& crt, cudaStream_t st, cudaEvent_t* ev) {
    SmallDesc one{};
    if (single) one = *single;
    if (ev) cudaEventRecord(ev[0], st);
    const int threads = small_threads(k);
    const size_t smem = ntt_small_smem_bytes(k);
#define X(MM) \
    if (k == MM) {                                                     \
        launch_pdl(false, k_small<MM>, count, threads, smem, st, d_descs, one, f, crt); \
        count_launches(1);                                             \
    }
    PREC_SMALL(X)
#undef X
    if (ev) cudaEventRecord(ev[1], st);
}

int configure_small() {
    cudaError_t e = cudaSuccess;
#define X(MM)                                                                                    \
    if (!e) e = cudaFuncSetAttribute(k_small<MM>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                     (int)ntt_small_smem_bytes(MM));
    PREC_SMALL(X)
#undef X
    return (int)e;
}

}  // namespace precgpu
