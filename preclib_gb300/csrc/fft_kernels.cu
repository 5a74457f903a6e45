// fft_kernels.cu -- FP64 FFT band (193 .. 6144 limbs) of the multiply.
//
// Replaces preclib's mul_fft (src/mul_fft.cpp:340-394) with the same method
// -- both operands packed as the real and imaginary parts of one complex
// FP64 FFT (fft_load_digits, 234-246), the two spectra separated and
// multiplied (fft_pair_convolution, 248-305), the inverse FFT, rounding to
// the nearest integer (307-309, 364-376) and a carry back to limbs
// (fft_from_digits, 311-338) -- laid out for many SMs:
//
//  digits   balanced b-bit digits (|d| <= 2^(b-1)), b chosen per transform
//           length from a worst-case error bound (host side); every digit
//           is computed on its own: d_i = raw_i - 2^b t_i + t_{i-1} with
//           t_j = [raw_j >= 2^(b-1)], so no carry chain is needed.
//  twiddles two tables from sincospi() (the reference builds per-stage tables
//           by a recurrence, mul_fft.cpp:57-76): e^(2 pi i e / 2^16) in
//           natural order for the inverse, e^(-pi i 0.b0b1b2..) by the bits
//           of the block index for the forward transform.
//  four-step N = N1 * N2:
//    k_fft_digits    limbs (device or page-locked host memory) -> digits
//    k_fft_fwd_cols  columns: the top log2 N1 levels of the transform
//    k_fft_rows      rows k1 and N1-k1 together: the other levels, product
//                    (P_-k = conj P_k), fold to half length, inverse levels
//    k_fft_inv_cols  columns of the inverse -> x scale -> nearest integer,
//                    max distance
//    k_fft_carry     limbs from the signed coefficients; writes nothing when
//                    the max distance exceeds 0.25.
//
// What bounds it: FP64 issue.  GB300 takes one FP64 warp instruction per 64
// cycles on each SM quarter (measured; 19 cycles per SM with all four
// busy), whatever the kind and at no extra latency.  So the transform is
// arranged for few FP64 instructions and for four warps per SM, and integer
// work, shared memory and barriers come free beside it:
//   * a butterfly (x + wy, x - wy) is 8 fused operations, two chained fma per
//     part (x - wy = 2x - (x + wy) would make it 6, 1.5 us less at 3000 x 3000
//     limbs, but its mean rounding distance came out 7% above the earlier
//     kernels'; this form's is 2% below);
//   * forward: block q of a level splits x^2m - r^2 into x^m -+ r, one twiddle
//     per block, natural to bit-reversed order: the four-step twiddles are
//     part of the rows' own twiddles and cost nothing;
//   * inverse: stage b pairs i and i + 2^b with w^(i mod 2^b), over the whole
//     index: again no separate twiddles;
//   * product: 4 i P_k = F_k^2 - conj(F_-k)^2, 7 operations;
//   * the inverse output is real: P is folded to Z_k = E_k + i O_k of half
//     length, whose inverse has the even coefficients as real and the odd
//     ones as imaginary parts.
// Per C call from host memory (the Python binding adds about 8 us): 256 x 193 limbs
// 45.5 -> 32.0 us, 3000 x 3000 59.5 -> 42.1, 6144 x 6144 80.4 -> 54.5 (kernels alone
// 34 -> 20, 46 -> 28, 63 -> 37).
#include <cuda_runtime.h>

#include <cooperative_groups.h>

#include "fft_kernels.cuh"
#include "ntt_engine.cuh"

namespace precgpu {

// raw b-bit digit starting at bit `bit` of the limbs s (one past them readable)
__device__ __forceinline__ uint32_t raw_digit(const uint64_t* s, uint32_t bit, int b) {
    const uint32_t l = bit >> 6, sh = bit & 63;
    uint64_t v = s[l] >> sh;
    if (sh + b > 64) v |= s[l + 1] << (64 - sh);
    return (uint32_t)(v & ((1ull << b) - 1));
}

// an exact double from an integer |d| < 2^31
__device__ __forceinline__ double small_double(int d) {
    return __hiloint2double(0x43300000, d ^ (int)0x80000000) - __hiloint2double(0x43300000, (int)0x80000000);
}

constexpr int kDigitThreads = 256;
constexpr int kDigitLimbs = kDigitThreads * 30 / 64 + 4;  // limbs 257 digits of up to 30 bits touch, and one more

// digits of both operands: element i = (a_i, b_i); starts the distance at 0
__global__ void __launch_bounds__(kDigitThreads) k_fft_digits(FftArgs f) {
    __shared__ uint64_t s[2][kDigitLimbs];
    pdl_enter();
    const uint64_t i0 = (uint64_t)blockIdx.x * kDigitThreads;
    // from digit i0 - 1 (its top bit decides digit i0's carry)
    const uint64_t first = i0 ? i0 - 1 : 0;
    const uint64_t l0 = first * f.b >> 6;
    const uint64_t* __restrict__ pa = after_entry(f.a);
    const uint64_t* __restrict__ pb = after_entry(f.bp);
    const int nl = (int)(((i0 + kDigitThreads) * f.b + 63) / 64 - l0) + 1;
    for (int t = threadIdx.x; t < nl; t += kDigitThreads) {
        s[0][t] = l0 + t < f.la ? __ldg(&pa[l0 + t]) : 0;
        s[1][t] = l0 + t < f.lb ? __ldg(&pb[l0 + t]) : 0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *f.maxdist = 0.0;
    __syncthreads();
    const uint64_t i = i0 + threadIdx.x;
    const uint32_t half = 1u << (f.b - 1);
    const uint32_t bit = (uint32_t)(i * f.b - (l0 << 6));
    double v[2];
#pragma unroll
    for (int o = 0; o < 2; ++o) {
        const uint32_t r = raw_digit(s[o], bit, f.b);
        const int t_in = i > 0 && raw_digit(s[o], bit - f.b, f.b) >= half ? 1 : 0;
        const int d = (int)r - (r >= half ? 1 << f.b : 0) + t_in;
        v[o] = small_double(i < (o ? f.db : f.da) ? d : 0);
    }
    if (i < f.ncoef) f.work[i] = make_double2(v[0], v[1]);
}

// (x, y) -> (x + wy, x - wy)
__device__ __forceinline__ void butterfly(double2& x, double2& y, double2 w) {
    const double re = fma(w.x, y.x, fma(-w.y, y.y, x.x));
    const double im = fma(w.x, y.y, fma(w.y, y.x, x.y));
    y = make_double2(fma(-w.x, y.x, fma(w.y, y.y, x.x)), fma(-w.x, y.y, fma(-w.y, y.x, x.y)));
    x = make_double2(re, im);
}
// w = 1, and w = -i
__device__ __forceinline__ void butterfly1(double2& x, double2& y) {
    const double2 t = x;
    x = make_double2(t.x + y.x, t.y + y.y);
    y = make_double2(t.x - y.x, t.y - y.y);
}
__device__ __forceinline__ void butterfly_mi(double2& x, double2& y) {
    const double2 t = x;
    x = make_double2(t.x + y.y, t.y - y.x);
    y = make_double2(t.x - y.y, t.y + y.x);
}

// One column of 2^M points: N1/2 threads, one butterfly each per level; C
// columns per CTA (one, once a column fills a warp).
template <int M>
struct ColGeom {
    static constexpr int HALF = 1 << (M - 1);
    static constexpr int THREADS = HALF < 32 ? 32 : HALF;
    static constexpr int C = THREADS / HALF;
};

// forward columns: levels 0 .. M-1; grid N2 / C
template <int M>
__global__ void __launch_bounds__(ColGeom<M>::THREADS) k_fft_fwd_cols(FftArgs f) {
    using G = ColGeom<M>;
    constexpr int H = G::HALF, N1 = 2 * H;
    __shared__ double2 s[G::C][N1];
    const int col = threadIdx.x / H, j = threadIdx.x % H;
    const uint32_t N2 = 1u << f.k2;
    const uint32_t c = blockIdx.x * G::C + col;
    double2 w[M];
#pragma unroll
    for (int l = 2; l < M; ++l) w[l] = __ldg(&f.twr[j >> (M - 1 - l)]);
    pdl_enter();
    const double2* __restrict__ src = after_entry(f.work);
    const uint64_t nd = f.da > f.db ? f.da : f.db;
    const bool upper = nd > f.ncoef / 2;  // else the upper half is zero: level 0 copies
    const uint64_t i = (uint64_t)j * N2 + c;
    double2 x = make_double2(0.0, 0.0), y = x;
    if (i < nd) x = src[i];
    if (upper && i + f.ncoef / 2 < nd) y = src[i + f.ncoef / 2];
    if (upper) butterfly1(x, y);
    else y = x;
    int pos = j;
#pragma unroll
    for (int l = 1; l < M; ++l) {
        s[col][pos] = x;
        s[col][pos + (H >> (l - 1))] = y;
        __syncthreads();
        const int h = H >> l;
        const int q = j / h;
        pos = q * 2 * h + j % h;
        x = s[col][pos];
        y = s[col][pos + h];
        if (l == 1) {
            if (q) butterfly_mi(x, y);
            else butterfly1(x, y);
        } else {
            butterfly(x, y, w[l]);
        }
        if (l + 1 < M) __syncthreads();
    }
    f.work[(uint64_t)pos * N2 + c] = x;
    f.work[(uint64_t)(pos + 1) * N2 + c] = y;
}

__device__ __forceinline__ uint32_t bitrev(uint32_t x, int bits) { return bits ? __brev(x) >> (32 - bits) : 0u; }

// row pass: CTA r handles frequency rows k1 = r and N1 - r (one row when
// they coincide); grid N1/2 + 1, N2 threads (2^M = N2)
template <int M>
__global__ void __launch_bounds__(M < 5 ? 32 : 1 << M) k_fft_rows(FftArgs f) {
    constexpr int N2 = 1 << M, H = N2 / 2, Q = N2 / 4;
    __shared__ double2 s[2][N2];
    const int N1 = 1 << f.k1;
    const uint32_t ka = blockIdx.x, kb = (N1 - blockIdx.x) & (N1 - 1);
    const bool one = ka == kb;
    const uint32_t sl[2] = {bitrev(ka, f.k1), bitrev(kb, f.k1)};
    const int r = threadIdx.x / H & 1, j = threadIdx.x % H;
    const bool on = threadIdx.x < N2 && !(one && r);
    const uint32_t slot = r ? sl[1] : sl[0];
    double2 w[M];
#pragma unroll
    for (int l = 0; l < M; ++l) w[l] = __ldg(&f.twr[(slot << l) + (j >> (M - 1 - l))]);
    const uint32_t k1 = r ? kb : ka;
    // fold twiddle i e^(2 pi i k / N) of this thread's frequency pair k, k + N/2
    const double2 e = __ldg(&f.tw[(k1 + ((uint32_t)bitrev(j, M - 1) << f.k1)) << (kFftMaxLog2 - f.k)]);
    pdl_enter();
    const double2* __restrict__ src = after_entry(f.work) + (uint64_t)slot * N2;
    double2 x, y;
    if (on) {
        x = src[j];
        y = src[j + H];
    }
    int pos = j;
#pragma unroll
    for (int l = 0; l < M; ++l) {
        const int h = H >> l;
        if (l) {
            __syncthreads();
            pos = (j / h) * 2 * h + j % h;
            if (on) {
                x = s[r][pos];
                y = s[r][pos + h];
            }
            __syncthreads();
        }
        if (on) {
            butterfly(x, y, w[l]);
            s[r][pos] = x;
            s[r][pos + h] = y;
        }
    }
    __syncthreads();
    // product and fold: slots 2j, 2j + 1 hold k and k + N/2; the partner of
    // slot t (frequency -k) is slot N2-1-t of the other row, in row 0 the
    // slot of the negated index
    double2 z;
    if (on) {
        const int pr = one ? 0 : 1 - r;
        int p0 = N2 - 1 - 2 * j, p1 = p0 - 1;
        if (k1 == 0) {
            p0 = bitrev((N2 - bitrev(2 * j, M)) & (N2 - 1), M);
            p1 = bitrev((N2 - bitrev(2 * j + 1, M)) & (N2 - 1), M);
        }
        const double2 F0 = s[r][2 * j], F1 = s[r][2 * j + 1], G0 = s[pr][p0], G1 = s[pr][p1];
        // 4 P = (2 m, t)
        const double m0 = fma(F0.x, F0.y, G0.x * G0.y);
        const double t0 = fma(F0.y, F0.y, fma(-F0.x, F0.x, fma(-G0.y, G0.y, G0.x * G0.x)));
        const double m1 = fma(F1.x, F1.y, G1.x * G1.y);
        const double t1 = fma(F1.y, F1.y, fma(-F1.x, F1.x, fma(-G1.y, G1.y, G1.x * G1.x)));
        const double a1 = m0 + m1, a2 = m0 - m1, b1 = t0 + t1, b2 = t0 - t1;
        // 8 Z = (2 a1 + i b1) + u (2 a2 + i b2), u = i e
        const double ur = -e.y, ui = e.x;
        z = make_double2(fma(2.0, a1, fma(2.0 * ur, a2, -ui * b2)), fma(ur, b2, fma(2.0 * ui, a2, b1)));
    }
    __syncthreads();
    // inverse levels over N2/2 points in bit-reversed order; real and
    // imaginary parts by different threads (four busy warps at N2 = 128)
    double* sd = reinterpret_cast<double*>(&s[0][0]);
    auto at = [&](int row, int part, int i) -> double& { return sd[(row * 2 + part) * H + i]; };
    if (on) {
        at(r, 0, j) = z.x;
        at(r, 1, j) = z.y;
    }
    const int part = threadIdx.x / H & 1;
    const int ir = (threadIdx.x % H) / Q, ij = threadIdx.x % Q;
    const bool ion = threadIdx.x < N2 && !(one && ir);
#pragma unroll
    for (int b = 0; b < M - 1; ++b) {
        const int h = 1 << b;
        const int p = (ij >> b) * 2 * h + (ij & (h - 1));
        double2 wt = make_double2(1.0, 0.0);
        if (b) wt = __ldg(&f.tw[(uint32_t)(ij & (h - 1)) << (kFftMaxLog2 - 1 - b)]);
        __syncthreads();
        double o0 = 0.0, o1 = 0.0;
        if (ion) {
            const double xs = at(ir, part, p), ys = at(ir, part, p + h);
            if (b == 0) {
                o0 = xs + ys;
                o1 = xs - ys;
            } else {
                const double yo = at(ir, 1 - part, p + h);
                o0 = fma(wt.x, ys, fma(part ? wt.y : -wt.y, yo, xs));
                o1 = fma(-wt.x, ys, fma(part ? -wt.y : wt.y, yo, xs));
            }
        }
        __syncthreads();
        if (ion) {
            at(ir, part, p) = o0;
            at(ir, part, p + h) = o1;
        }
    }
    __syncthreads();
    if (on) f.work[(uint64_t)slot * N2 + j] = make_double2(at(r, 0, j), at(r, 1, j));
}

// 1.5 * 2^52: adding it rounds |v| < 2^51 to the nearest integer (ties to
// even, as rint) and leaves that integer in the low bits
__device__ __forceinline__ double round_magic() { return 6755399441055744.0; }

// inverse columns (half length: N2/2 columns of N1 points), scaling,
// rounding; grid N2 / 2 / C
template <int M>
__global__ void __launch_bounds__(ColGeom<M>::THREADS) k_fft_inv_cols(FftArgs f) {
    using G = ColGeom<M>;
    constexpr int H = G::HALF, N1 = 2 * H;
    __shared__ double2 s[G::C][N1];
    __shared__ unsigned long long s_max[G::THREADS / 32];
    const int col = threadIdx.x / H, j = threadIdx.x % H;
    const uint32_t N2 = 1u << f.k2, N2h = N2 / 2;
    const uint32_t c = blockIdx.x * G::C + col;
    const bool on = c < N2h;  // (N = 64 has fewer columns than one CTA takes)
    double2 w[M];
#pragma unroll
    for (int b = 0; b < M; ++b)
        w[b] = __ldg(&f.tw[((uint32_t)(j & ((1 << b) - 1)) * N2h + (on ? c : 0)) << (kFftMaxLog2 - f.k2 - b)]);
    pdl_enter();
    const double2* __restrict__ src = after_entry(f.work);
    double2 x = make_double2(0.0, 0.0), y = x;
    if (on) {
        x = src[(uint64_t)(2 * j) * N2 + c];
        y = src[(uint64_t)(2 * j + 1) * N2 + c];
    }
    int pos = 2 * j;
#pragma unroll
    for (int b = 0; b < M; ++b) {
        const int h = 1 << b;
        if (b) {
            s[col][pos] = x;
            s[col][pos + (h >> 1)] = y;
            __syncthreads();
            pos = (j >> b) * 2 * h + (j & (h - 1));
            x = s[col][pos];
            y = s[col][pos + h];
            if (b + 1 < M) __syncthreads();
        }
        butterfly(x, y, w[b]);
    }
    // element i1 = pos, pos + H of column c: coefficients 2n, 2n + 1 of n = i1 N2/2 + c
    const double scale = __hiloint2double((1023 - f.k - 2) << 20, 0);  // 2^-(k+2)
    const double magic = round_magic();
    unsigned long long dmax = 0;
    auto round1 = [&](double v) -> long long {
        const double m = fma(v, scale, magic);
        const double r = m - magic;
        const double d = fma(v, scale, -r);
        // |d| by its bits (non-negative doubles order like them; NaN above
        // all); a value past 2^51 cannot be rounded this way: refused
        unsigned long long bits = (unsigned long long)__double_as_longlong(d) & 0x7fffffffffffffffull;
        const unsigned long long big = (unsigned long long)__double_as_longlong(r) & 0x7fffffffffffffffull;
        if (big >= 0x4320000000000000ull) bits = 0x7ff0000000000000ull;
        dmax = bits > dmax ? bits : dmax;
        return __double_as_longlong(m) - __double_as_longlong(magic);
    };
    longlong2* coef = reinterpret_cast<longlong2*>(f.coef);
    const long long x0 = round1(x.x), x1 = round1(x.y), y0 = round1(y.x), y1 = round1(y.y);
    if (on) {
        coef[(uint64_t)pos * N2h + c] = make_longlong2(x0, x1);
        coef[(uint64_t)(pos + H) * N2h + c] = make_longlong2(y0, y1);
    }
    {   // no coefficient past the last digits' product
        const uint64_t end = f.da + f.db - 1, i = 2 * ((uint64_t)pos * N2h + c), j = i + 2 * (uint64_t)H * N2h;
        const bool past = on && ((i >= end && x0) || (i + 1 >= end && x1) || (j >= end && y0) || (j + 1 >= end && y1));
        if (__any_sync(0xffffffffu, past) && (threadIdx.x & 31) == 0) atomicOr(f.err, kDevErrCarry);
    }
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long v = __shfl_xor_sync(0xffffffffu, dmax, o);
        dmax = v > dmax ? v : dmax;
    }
    if (G::THREADS > 32) {
        if ((threadIdx.x & 31) == 0) s_max[threadIdx.x >> 5] = dmax;
        __syncthreads();
        if (threadIdx.x == 0)
            for (int i = 1; i < G::THREADS / 32; ++i) dmax = s_max[i] > dmax ? s_max[i] : dmax;
    }
    if (threadIdx.x == 0) atomicMax(reinterpret_cast<unsigned long long*>(f.maxdist), dmax);
}

// Carry: limbs of the product sum c_i 2^(bi) from the signed coefficients
// (fft_limb_sum).  The product runs as one cluster of up to 8 CTAs: each puts its carry aggregate
// into every CTA's shared memory, one cluster barrier, and every limb is
// written once, final.  (As separate CTAs joined by the last one over the
// carry maps of signed limbs this kernel took 9 - 11 us.)
template <int L, int NW>
__global__ void __launch_bounds__(32 * NW) k_fft_carry(FftArgs f) {
    namespace cg = cooperative_groups;
    __shared__ uint32_t s_wg[NW], s_wp[NW];
    __shared__ uint32_t s_blk[kFftCarryCluster];
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = blockIdx.x, ranks = gridDim.x;
    cluster.barrier_arrive();  // (the other CTAs' shared memory exists once all arrived)
    pdl_enter();
    const long long* __restrict__ coef = after_entry(f.coef);
    const double dist = *f.maxdist;
    if (f.host_dist && rank == 0 && threadIdx.x == 0) *f.host_dist = dist;
    if (!(dist <= 0.25)) {  // also NaN / inf: nothing is written
        if (rank == 0 && threadIdx.x == 0) atomicOr(f.err, kDevErrFftRound);
        cluster.barrier_wait();
        return;
    }
    const int b = f.b;
    const int64_t m0 = ((int64_t)rank * 32 * NW + threadIdx.x) * L;
    const int64_t lim = (int64_t)f.lout + kFftPastLimbs;
    u128 T[L + 1];  // S of limbs m0 - 1 .. m0 + L - 1
#pragma unroll
    for (int k = 0; k <= L; ++k) {
        const int64_t m = m0 + k - 1;
        T[k] = m < lim ? fft_limb_sum([&](uint32_t i) { return coef[i]; }, f.ncoef, b, m) : (u128)0;
    }
    u128 S[L];
#pragma unroll
    for (int k = 0; k < L; ++k) S[k] = T[k + 1];
    uint64_t v[L];
    uint32_t gbits;
    bool G, P;
    limbs_from_sums<L>(S, (uint64_t)(T[0] >> 64), v, gbits, G, P);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t gm = __ballot_sync(0xffffffffu, G), pm = __ballot_sync(0xffffffffu, P);
    if (lane == 0) {
        s_wg[warp] = (uint32_t)(carry_chain(gm, pm, false) >> 32) & 1;
        s_wp[warp] = pm == 0xffffffffu;
    }
    __syncthreads();
    // warp aggregates as bits; the CTA's own aggregate to every CTA of the cluster
    const uint32_t bg = __ballot_sync(0xffffffffu, lane < NW && s_wg[lane] != 0);
    const uint32_t bp = __ballot_sync(0xffffffffu, lane < NW && s_wp[lane] != 0);
    cluster.barrier_wait();
    if (ranks > 1) {
        if (warp == 0 && lane < (int)ranks) {
            const uint32_t agg = ((uint32_t)(carry_chain(bg, bp, false) >> NW) & 1) | (bp == (1u << NW) - 1 ? 2u : 0u);
            *cluster.map_shared_rank(&s_blk[rank], lane) = agg;
        }
        cluster.sync();
    }
    bool cin = false;
    for (uint32_t r = 0; r < rank; ++r) cin = (s_blk[r] & 1) || ((s_blk[r] & 2) && cin);
    const bool wcin = (carry_chain(bg, bp, cin) >> warp) & 1;
    bool c = (carry_chain(gm, pm, wcin) >> lane) & 1;
#pragma unroll
    for (int k = 0; k < L; ++k) {
        const uint64_t x = v[k] + (c ? 1u : 0u);
        c = ((gbits >> k) & 1) || (v[k] == ~0ull && c);
        const int64_t m = m0 + k;
        if (m < (int64_t)f.lout) f.out[m] = x;
        else if (m < lim && x != fft_past_value(b, f.ncoef, m)) atomicOr(f.err, kDevErrCarry);  // a product fits La+Lb limbs
    }
}

// e^(2 pi i e / 2^16) for e < 2^15, then e^(-pi i 0.b0b1..) for q = ..b1b0 < 2^15
__global__ void k_fft_table(double2* tw) {
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < (1 << (kFftMaxLog2 - 1))) {
        double s, c;
        sincospi((double)e / (double)(1 << (kFftMaxLog2 - 1)), &s, &c);
        tw[e] = make_double2(c, s);
        const int q = (int)bitrev((uint32_t)e, kFftMaxLog2 - 1);
        sincospi((double)e / (double)(1 << (kFftMaxLog2 - 1)), &s, &c);
        tw[(1 << (kFftMaxLog2 - 1)) + q] = make_double2(c, -s);
    }
}

// ---------------------------------------------------------------------------

size_t fft_table_bytes() { return (size_t)sizeof(double2) << kFftMaxLog2; }

void fft_build_table(double2* tw, cudaStream_t st) {
    k_fft_table<<<(1 << (kFftMaxLog2 - 1)) / 256, 256, 0, st>>>(tw);
    count_launches(1);
}

template <int L, int NW>
static void launch_carry(const FftArgs& f, cudaStream_t st) {
    const unsigned n = fft_carry_ctas(f.lout);
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = n;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = n;
    cfg.blockDim = 32 * NW;
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    cudaLaunchKernelEx(&cfg, k_fft_carry<L, NW>, f);
}

#define PREC_FFT_LOG2(X) X(3) X(4) X(5) X(6) X(7) X(8)

// (limbs per thread, warps)
#define PREC_FFT_CARRY(X) X(1, 16) X(1, 17) X(2, 16) X(2, 17) X(3, 16) X(3, 17)

int configure_fft() {
    cudaError_t e = load_kernel(k_fft_digits);
#define X(M)                                        \
    if (!e) e = load_kernel(k_fft_fwd_cols<M>);     \
    if (!e) e = load_kernel(k_fft_rows<M>);         \
    if (!e) e = load_kernel(k_fft_inv_cols<M>);
    PREC_FFT_LOG2(X)
#undef X
#define X(L, W) \
    if (!e) e = load_kernel(k_fft_carry<L, W>);
    PREC_FFT_CARRY(X)
#undef X
    return (int)e;
}

int fft_launch(const FftArgs& f, cudaStream_t st) {
    const uint64_t nd = f.da > f.db ? f.da : f.db;
    launch_pdl(false, k_fft_digits, (unsigned)((nd + kDigitThreads - 1) / kDigitThreads), kDigitThreads, 0, st, f);
#define X(M) \
    if (f.k1 == M) launch_pdl(false, k_fft_fwd_cols<M>, (1u << f.k2) / ColGeom<M>::C, ColGeom<M>::THREADS, 0, st, f);
    PREC_FFT_LOG2(X)
#undef X
#define X(M) \
    if (f.k2 == M) launch_pdl(false, k_fft_rows<M>, (1u << f.k1) / 2 + 1, M < 5 ? 32 : 1 << M, 0, st, f);
    PREC_FFT_LOG2(X)
#undef X
#define X(M) \
    if (f.k1 == M) launch_pdl(false, k_fft_inv_cols<M>, ((1u << f.k2) / 2 + ColGeom<M>::C - 1) / ColGeom<M>::C, ColGeom<M>::THREADS, 0, st, f);
    PREC_FFT_LOG2(X)
#undef X
    static_assert(fft_carry_limbs(2 * 6144) == 3, "the band's longest product");
    const int L = fft_carry_limbs(f.lout), NW = fft_carry_warps(f.lout);
#define X(LL, W) \
    if (L == LL && NW == W) launch_carry<LL, W>(f, st);
    PREC_FFT_CARRY(X)
#undef X
    count_launches(5);
    return (int)cudaGetLastError();
}

}  // namespace precgpu
