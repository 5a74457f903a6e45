// fft_kernels.cuh -- FP64 FFT band: arguments and launchers.
#pragma once
#include <cstddef>
#include <cstdint>

#include <cuda_runtime.h>

#include "ntt_kernels.cuh"

namespace precgpu {

constexpr int kFftMaxLog2 = 16;     // largest FP64 transform (6144 x 6144 limbs fits)
constexpr int kDevErrFftRound = 4;  // device error bit: max distance above 0.25

struct FftArgs {
    const uint64_t* a;    // operands and result: device or page-locked host memory
    const uint64_t* bp;
    uint64_t* out;
    double2* work;        // N complex values
    long long* coef;      // N rounded coefficients
    double* maxdist;      // max |x - round(x)| of this product
    double* host_dist;    // page-locked copy of it for the host, or nullptr
    int* err;
    const double2* tw;    // e^(2 pi i e / 2^16), e < 2^15
    const double2* twr;   // e^(-pi i 0.b0b1..), q = ..b1b0 < 2^15
    uint64_t la, lb, lout;
    uint64_t da, db;      // balanced digit counts
    uint64_t ncoef;       // N
    int b;                // digit width in bits
    int k, k1, k2;        // log2 N = k1 + k2 (column length 2^k1, row length 2^k2)
};

// ---- the carry (k_fft_carry), in functions that the host can call
//
// c_i + 2^62 - 2^(62-b) (for i = 0: c_i + 2^62) is positive, and over all N
// coefficients these add up to the product plus 2^(bN + 62 - b), past every limb
// of the product, so the carries are 0 or 1: S_m, the sum of the coefficients
// that start in limb m, gives limb lo64(S_m) + hi64(S_m-1) + carry, as in the NTT band.
// coef(i): coefficient i, called for i < ncoef.
template <class Coef>
__host__ __device__ __forceinline__ unsigned __int128 fft_limb_sum(Coef coef, uint64_t ncoef, int b, int64_t m) {
    if (m < 0) return 0;
    const uint32_t bit = (uint32_t)m * 64;
    const uint32_t i0 = (bit + b - 1) / b;
    const uint32_t off = i0 * b - bit;
    long long c[8];  // b >= 8: at most 8 coefficients start in a limb
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) c[u] = off + u * b < 64 && i0 + u < ncoef ? coef(i0 + u) : 0;
    unsigned __int128 s = 0;
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) {
        if (off + u * b < 64 && i0 + u < ncoef) {
            const uint64_t v = (uint64_t)c[u] + (1ull << 62) - (i0 + u ? 1ull << (62 - b) : 0);
            s += (unsigned __int128)v << (off + u * b);
        }
    }
    return s;
}

// A product of la x lb limbs must fit la + lb limbs.  Its coefficients from
// da + db - 1 on are zero (k_fft_inv_cols checks that), so what the others add up
// to is below 2^(64 lout + 2b + 50) either way (|c_i| < 2^51, b (da + db - 2) <= 64
// lout + 2b - 2): with b <= 30, if the two limbs past the product hold the
// offset's bit and nothing else, every limb past it does.
constexpr int kFftPastLimbs = 2;
__host__ __device__ inline uint64_t fft_past_value(int b, uint64_t ncoef, int64_t m) {
    const uint64_t bit = (uint64_t)b * ncoef + 62 - b;
    return (int64_t)(bit >> 6) == m ? 1ull << (bit & 63) : 0;
}

// One cluster of up to 8 CTAs, 16 warps each and 1 to 3 limbs per thread.  4096, 8192
// and 12288 limbs fill that cluster: with the limbs past them they take 17 warps.
// (One more limb per thread there instead: 2048 x 2048 limbs 39.4 -> 40.4 us, 6144 x
// 6144 54.0 -> 55.2.  17 warps for every length: 0.3 us more per call.)
constexpr int kFftCarryCluster = 8;
__host__ __device__ constexpr int fft_carry_limbs(uint64_t lout) {
    constexpr uint64_t one = (uint64_t)16 * 32 * kFftCarryCluster;
    return (int)((lout + one - 1) / one);
}
__host__ __device__ constexpr int fft_carry_warps(uint64_t lout) {
    return lout + kFftPastLimbs <= (uint64_t)16 * 32 * kFftCarryCluster * fft_carry_limbs(lout) ? 16 : 17;
}
__host__ __device__ constexpr unsigned fft_carry_ctas(uint64_t lout) {
    const uint64_t per = (uint64_t)32 * fft_carry_warps(lout) * fft_carry_limbs(lout);
    return (unsigned)((lout + kFftPastLimbs + per - 1) / per);
}

// both twiddle tables: tw, then twr at tw + 2^15
size_t fft_table_bytes();
void fft_build_table(double2* tw, cudaStream_t st);
// The product's 5 kernels on `st`.  Returns a cudaError_t.
int fft_launch(const FftArgs& f, cudaStream_t st);
int configure_fft();

}  // namespace precgpu
