// ntt_carry.cuh -- CRT recombination and carry propagation of the four-step
// path (crt_carry_tile): the reference's ntt_crt2/ntt_crt3 and serial
// ntt_from_residues carry loop (src/mul_ntt.cpp:405-487) as one pass over
// the natural-order residues.  Shared by the carry kernel (ntt_carry.cu)
// and the batch form's persistent class kernel (ntt_class.cu).
//
// Phase 1 (every block): each thread turns 8 coefficients into 4 limbs
// (set 2: 4 coefficients of up to 150 bits, one per limb, into 4 limbs),
// the limb carry chain is resolved per warp (ballot) and per block (one
// barrier), and the limbs are written.  The block finds its own carry-in: it
// recombines the limbs just below its first one too, and the carry out of
// that limb is known unless the limb is all ones (its own carry-in then decides).
// A block that does not know its carry-in takes 0 and says so in the aggregate that it
// publishes (G = carry out, P = a carry-in would pass through).
// Phase 2, only if some block did not know: the last block to finish (found with a
// fence and an atomic counter) scans the aggregates into per-block carry-ins
// and adds the carry into those blocks that took 0 instead of 1.  No block
// ever waits on another.  (Every block with carry-in 0 and the scan on every
// product: 65536 x 65536 limbs 22.5 us, now 20.9; 20011 x 13001 15.5, now 14.9;
// 1M x 1M 156.0, now 154.2; 4096 products of 200 .. 65536 limbs 8.15 ms, now 8.13.  Counting
// before the limbs are stored, which only needs to wait in a block that does not
// know: the batch 8.09, but 20011 x 13001 15.7.)
#pragma once
#include "ntt_engine.cuh"

namespace precgpu {

// residue loads: COH reads through L2 only (data written earlier in the
// same launch); otherwise as before (read-only path for the vector loads)
template <bool COH>
__device__ __forceinline__ uint4 ld_work4(const uint32_t* p) {
    if constexpr (COH) return __ldcg(reinterpret_cast<const uint4*>(p));
    else return __ldg(reinterpret_cast<const uint4*>(p));
}
template <bool COH>
__device__ __forceinline__ uint32_t ld_work(const uint32_t* p) {
    if constexpr (COH) return __ldcg(p);
    else return *p;
}

// ---- set 2: one coefficient per 64-bit limb

// a coefficient c < p1..p5 < 2^150 as three words (w2 < 2^22)
struct Coef3 {
    uint64_t w0, w1;
    uint32_t w2;
};

// Garner over the five primes (the constants of Crt5Const) from the
// inverse-transform outputs y_j = (value) * a_j (times 2^32 for j > 0), a_j
// applied by the inverse column pass: v_j = y_j - sum_{i<j} v_i b_ij mod p_j as
// one 64-bit sum of products and one Montgomery reduction, then
// c = v0 + p0 (v1 + p1 (v2 + p2 (v3 + p3 v4))) in 32-bit words.  LAZY (set 2,
// p < 2^30): y_j in [0, 4p), the sum below 2^32 p_j; otherwise (set 3, p <
// 2^31) y_j in [0, p), the sum below 1.8 * 2^32 p_j and 2^63.2 (and with the
// reduction's multiple of p_j below 2^64).
// (Each product reduced by itself, ten Shoup products and their corrections,
// and 128-bit arithmetic for c took 194 instructions per coefficient instead
// of 149; 1M x 1M limbs 163.1 -> 160.6 us.)
template <bool LAZY>
__device__ __forceinline__ Coef3 crt5(const uint32_t (&y)[5], const Crt5Const& cc, const FieldArgs& f) {
    uint32_t v[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) {
        const uint32_t p = f.pc[j].p, p2 = f.pc[j].p2;
        uint32_t r = y[j];
        if (j) {
            uint64_t t = r;
#pragma unroll
            for (int i = 0; i < j; ++i) t += (uint64_t)v[i] * cc.n[j * (j - 1) / 2 + i];
            const uint32_t m = (uint32_t)t * f.pc[j].pinv;
            r = (uint32_t)((t + (uint64_t)m * p) >> 32);  // LAZY: below 2p; else below 2.8 p < 2^32
        }
        if (LAZY ? j == 0 : j > 1) r = red1(r, p2);
        v[j] = (LAZY || j) ? red1(r, p) : r;
    }
    // words of c, one multiply-add per word and prime
    uint32_t w[5] = {v[4], 0, 0, 0, 0};
#pragma unroll
    for (int j = 3; j >= 0; --j) {
        uint32_t carry = v[j];
#pragma unroll
        for (int i = 0; i < 4 - j; ++i) {
            const uint64_t t = (uint64_t)w[i] * f.pc[j].p + carry;
            w[i] = (uint32_t)t;
            carry = (uint32_t)(t >> 32);
        }
        w[4 - j] = carry;
    }
    Coef3 c;
    c.w0 = (uint64_t)w[1] << 32 | w[0];
    c.w1 = (uint64_t)w[3] << 32 | w[2];
    c.w2 = w[4];
    return c;
}

template <bool LAZY>
__device__ __forceinline__ Coef3 coef5(const uint32_t* __restrict__ work, uint64_t N, int64_t i,
                                       const ProdArgs& args) {
    if (i < 0 || (uint64_t)i >= N) return Coef3{0, 0, 0};
    uint32_t y[5];
#pragma unroll
    for (int j = 0; j < 5; ++j) y[j] = work[(uint64_t)(2 * j) * N + i];
    return crt5<LAZY>(y, args.crt5, args.f);
}

// sum of limb m: S_m = w0(c_m) + w1(c_(m-1)) + w2(c_(m-2)) < 2^66
__device__ __forceinline__ u128 limb_sum(const Coef3& c0, uint64_t w1_prev, uint32_t w2_prev2) {
    return (u128)c0.w0 + w1_prev + w2_prev2;
}

struct WideEdge {
    uint64_t w1;  // w1 of the warp's last coefficient
    uint32_t w2a, w2b;  // w2 of its last two coefficients
    uint32_t hi;  // S >> 64 of its last limb
};

// T[k] = S_(m0+k) for this thread's limbs and hi(S_(m0-1)); the words the
// first limbs need from below come from the lane below or, for a warp's
// lane 0, from the warp below (shared memory).  The block's thread 0 holds
// the four coefficients just below the block's first limb and outputs
// nothing, so every thread recombines exactly four coefficients (three lanes
// of warp 0 recomputing the block's edge after their own four kept the
// other warps waiting at the barrier: 3.9 stalled warps per issue).
template <bool LAZY>
__device__ __forceinline__ void wide_sums(const uint32_t* __restrict__ work, const ProdArgs& args, int64_t m0, u128 (&T)[kCarryLimbs],
                                          uint64_t& prev_hi, WideEdge* s_edge) {
    static_assert(kCarryLimbs >= 4 && kCarryLimbs % 4 == 0, "limbs per thread: whole 16-byte loads");
    constexpr int L = kCarryLimbs;
    const uint64_t N = 1ull << args.k;
    const uint64_t nc = (uint64_t)args.keep << args.k >> 3;  // coefficients there are
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Coef3 c[L];
    if (m0 >= 0 && (uint64_t)m0 + L <= nc) {  // (block 0's thread 0 starts at -4)
#pragma unroll
        for (int h = 0; h < L / 4; ++h) {
            uint4 r[5];
#pragma unroll
            for (int j = 0; j < 5; ++j)
                r[j] = __ldg(reinterpret_cast<const uint4*>(work + (uint64_t)(2 * j) * N + m0) + h);
            uint32_t y[5];
#pragma unroll
            for (int j = 0; j < 5; ++j) y[j] = r[j].x;
            c[4 * h] = crt5<LAZY>(y, args.crt5, args.f);
#pragma unroll
            for (int j = 0; j < 5; ++j) y[j] = r[j].y;
            c[4 * h + 1] = crt5<LAZY>(y, args.crt5, args.f);
#pragma unroll
            for (int j = 0; j < 5; ++j) y[j] = r[j].z;
            c[4 * h + 2] = crt5<LAZY>(y, args.crt5, args.f);
#pragma unroll
            for (int j = 0; j < 5; ++j) y[j] = r[j].w;
            c[4 * h + 3] = crt5<LAZY>(y, args.crt5, args.f);
        }
    } else {
#pragma unroll
        for (int k = 0; k < L; ++k) c[k] = (uint64_t)(m0 + k) < nc ? coef5<LAZY>(work, N, m0 + k, args) : Coef3{0, 0, 0};
    }
    const u128 s_last = limb_sum(c[L - 1], c[L - 2].w1, c[L - 3].w2);
    const uint32_t hi_last = (uint32_t)(s_last >> 64);
    // words from the thread below: w1(c_-1), w2(c_-1), w2(c_-2), hi(S_-1)
    uint64_t w1m1 = __shfl_up_sync(0xffffffffu, c[L - 1].w1, 1);
    uint32_t w2m1 = __shfl_up_sync(0xffffffffu, c[L - 1].w2, 1);
    uint32_t w2m2 = __shfl_up_sync(0xffffffffu, c[L - 2].w2, 1);
    uint32_t him1 = __shfl_up_sync(0xffffffffu, hi_last, 1);
    if (lane == 31) s_edge[warp] = WideEdge{c[L - 1].w1, c[L - 1].w2, c[L - 2].w2, hi_last};
    __syncthreads();
    if (lane == 0 && warp > 0) {
        const WideEdge e = s_edge[warp - 1];
        w1m1 = e.w1;
        w2m1 = e.w2a;
        w2m2 = e.w2b;
        him1 = e.hi;
    }
    T[0] = limb_sum(c[0], w1m1, w2m2);
    T[1] = limb_sum(c[1], c[0].w1, w2m1);
#pragma unroll
    for (int k = 2; k < L; ++k) T[k] = limb_sum(c[k], c[k - 1].w1, c[k - 2].w2);
    prev_hi = him1;
}

// One carry block (x, from args.crt_blk0 in a chunked CRT) of product z;
// nx: blocks of this launch (the chunk's, or every block of the product).
// scratch layout: [0] finished-block counter, [1 .. nblk] aggregates
// (bit0 G, bit1 P).  COH: the residues were written earlier in the same
// launch (the batch form's persistent class kernel) and are read through L2
// (ld.global.cg), never a non-coherent cache.
template <int SET, bool COH = false, class I>
__device__ __forceinline__ void crt_carry_tile(const ProdArgs& args, const ProdPtrs* __restrict__ batch, const I& ix) {
    __shared__ BlockCarryShared sh;
    __shared__ uint32_t s_last;
    __shared__ WideEdge s_edge[kCarryThreads / 32];
    const ProdPtrs PP = select_product_at(args, batch, ix.z());
    const uint32_t* __restrict__ work = after_entry(PP.work);
    const uint32_t bid = args.crt_blk0 + ix.x();  // chunked CRT: blocks from crt_blk0
    if ((int)bid >= PP.nblk) return;  // batch: a shorter product of the class
    const uint64_t N = 1ull << args.k;
    const int lane = threadIdx.x & 31;
    constexpr int BL = crt_block_limbs(SET);  // limbs the block outputs
    // 64-bit digits: thread 0 takes the four coefficients below the block
    const int64_t m0 = (int64_t)bid * BL + ((int)threadIdx.x - (set_wide(SET) ? 1 : 0)) * kCarryLimbs;
    const bool edge_only = set_wide(SET) && threadIdx.x == 0;

    u128 T[kCarryLimbs];
    uint64_t prev_hi = 0;
    u128 below = 0;  // thread 0: value and carry of the limb below the block
    if constexpr (set_wide(SET)) {
        wide_sums<SET == kWideSet>(work, args, m0, T, prev_hi, s_edge);
    } else {
        const uint32_t* __restrict__ r0 = work;
        const uint32_t* __restrict__ r1 = work + 2 * N;
        const uint32_t* __restrict__ r2 = work + 4 * N;
        const uint64_t i0 = 2 * (uint64_t)m0;
        const uint64_t nc = (uint64_t)args.keep << args.k >> 3;  // coefficients there are
        if (i0 + 2 * kCarryLimbs <= nc) {
            uint32_t y[3][2 * kCarryLimbs];
#pragma unroll
            for (int h = 0; h < 2 * kCarryLimbs / 4; ++h) {
                const uint4 a = ld_work4<COH>(r0 + i0 + 4 * h);
                const uint4 b = ld_work4<COH>(r1 + i0 + 4 * h);
                const uint4 c = ld_work4<COH>(r2 + i0 + 4 * h);
                y[0][4 * h] = a.x; y[0][4 * h + 1] = a.y; y[0][4 * h + 2] = a.z; y[0][4 * h + 3] = a.w;
                y[1][4 * h] = b.x; y[1][4 * h + 1] = b.y; y[1][4 * h + 2] = b.z; y[1][4 * h + 3] = b.w;
                y[2][4 * h] = c.x; y[2][4 * h + 1] = c.y; y[2][4 * h + 2] = c.z; y[2][4 * h + 3] = c.w;
            }
#pragma unroll
            for (int k = 0; k < kCarryLimbs; ++k) {
                const u128 c0 = crt3_folded<SET>(y[0][2 * k], y[1][2 * k], y[2][2 * k], args.crt, args.f);
                const u128 c1 =
                    crt3_folded<SET>(y[0][2 * k + 1], y[1][2 * k + 1], y[2][2 * k + 1], args.crt, args.f);
                T[k] = c0 + (c1 << 32);
            }
        } else {
#pragma unroll
            for (int k = 0; k < kCarryLimbs; ++k) {
                u128 c[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const uint64_t i = i0 + 2 * k + e;
                    c[e] = i < nc ? crt3_folded<SET>(ld_work<COH>(r0 + i), ld_work<COH>(r1 + i), ld_work<COH>(r2 + i),
                                                    args.crt, args.f)
                                 : (u128)0;
                }
                T[k] = c[0] + (c[1] << 32);
            }
        }
        // hi(T) of the limb just below this thread's first limb; lanes 0 and 1
        // recombine the two limbs below the warp's first
        prev_hi = __shfl_up_sync(0xffffffffu, (uint64_t)(T[kCarryLimbs - 1] >> 64), 1);
        u128 E = 0;
        const int64_t e0 = 2 * (m0 - (int64_t)lane * kCarryLimbs - 1 - lane);  // its first coefficient
        if (lane < 2 && e0 >= 0 && (uint64_t)e0 + 1 < nc) {
            const u128 c0 = crt3_folded<SET>(ld_work<COH>(r0 + e0), ld_work<COH>(r1 + e0), ld_work<COH>(r2 + e0), args.crt,
                                             args.f);
            const u128 c1 = crt3_folded<SET>(ld_work<COH>(r0 + e0 + 1), ld_work<COH>(r1 + e0 + 1),
                                             ld_work<COH>(r2 + e0 + 1), args.crt, args.f);
            E = c0 + (c1 << 32);
        }
        const uint64_t hi2 = __shfl_down_sync(0xffffffffu, (uint64_t)(E >> 64), 1);
        if (lane == 0) {
            prev_hi = (uint64_t)(E >> 64);
            below = (u128)(uint64_t)E + hi2;
        }
    }
    uint64_t v[kCarryLimbs];
    uint32_t gbits;
    bool G, P;
    limbs_from_sums<kCarryLimbs>(T, prev_hi, v, gbits, G, P);
    if (edge_only) {  // its last limb is the one below the block, and it outputs nothing
        below = (u128)v[kCarryLimbs - 1] | (u128)(gbits >> (kCarryLimbs - 1) & 1) << 64;
        G = false;
        P = true;
    }
    // thread 0 puts the carry into the block (0 if it is not known) into its own (G, P)
    const bool known = (uint64_t)below != ~0ull;
    const bool c_in = known && (uint64_t)(below >> 64) != 0;
    if (threadIdx.x == 0 && known) {
        G = G || (P && c_in);
        P = false;
    }

    const bool chunked = args.chunk_words != nullptr;
    uint32_t* counter = chunked ? &args.chunk_words[2 * args.crt_chunk] : &PP.scratch[0];
    const int blo = chunked ? args.crt_blk0 : 0;
    const int bhi = chunked ? args.crt_blk0 + (int)ix.nx() : PP.nblk;
    // the carry out of the run of blocks
    auto run_out = [&](bool cout) {
        if (chunked && !args.crt_last) args.chunk_words[2 * args.crt_chunk + 3] = cout ? 1u : 0u;
        else if (cout) atomicOr(args.err, kDevErrCarry);  // a product fits La+Lb limbs
    };
    uint32_t* agg = PP.scratch + 1;
    auto publish = [&](bool Gb, bool Pb) {
        agg[bid] = (Gb ? 1u : 0u) | (Pb ? 2u : 0u) | (known ? 0u : 4u);
        if (known && (int)bid == bhi - 1) run_out(Gb);
    };
    bool cin = block_carry_in0(G, P, sh, publish);
    if (threadIdx.x == 0) cin = c_in;
    if (!edge_only) limbs_finish<kCarryLimbs>(m0, PP.lout, v, gbits, cin, PP.out);

    // ---- phase 2: the last block resolves the carries not known.
    // The barrier orders every thread's limb and aggregate stores before
    // thread 0's device-scope fence, which orders them before the counter.
    // A chunked CRT (one launch per run of blocks, in order on one stream)
    // joins each chunk on its own: the carry into the chunk comes from the
    // previous chunk's join, and its carry out goes to the next.
    constexpr uint32_t kUnknown = 1u << 31;  // counter bit: some block did not know
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        if (!known) atomicOr(counter, kUnknown);
        const uint32_t done = atomicAdd(counter, 1u);
        s_last = done == (kUnknown | ((uint32_t)(bhi - blo) - 1)) ? 1u : 0u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    const bool cin_chunk = chunked && __ldcg(&args.chunk_words[2 * args.crt_chunk + 1]) != 0;
    const int nb = bhi - blo;
    const int per = (nb + blockDim.x - 1) / blockDim.x;  // aggregates per thread
    const int b0 = blo + threadIdx.x * per, b1 = min(b0 + per, bhi);
    const int n = b1 > b0 ? b1 - b0 : 0;  // this thread's run of blocks
    auto chunk_in = [&](bool, bool) -> bool { return cin_chunk; };
    // the carry enters block b: +1 ripples through its all-ones limbs
    auto ripple = [&](int b) {
        const uint64_t lim_end = min((uint64_t)(b + 1) * BL, PP.lout);
        for (uint64_t m = (uint64_t)b * BL; m < lim_end; ++m) {
            const uint64_t x = __ldcg(&PP.out[m]) + 1;
            PP.out[m] = x;
            if (x != 0) break;
        }
    };
    // The aggregates are loaded kAggBatch at a time in one unrolled group
    // (independent loads in flight together, not one L2 round trip each).
    constexpr int kAggBatch = 16;
    bool cout;  // the carry out of this thread's last block
    if (per <= 64) {
        // the run as bit masks (bit i: block b0 + i; G and P, with G = 0,
        // P = 1 past the run): the run's own aggregate and, once the carry
        // into it is known, the carry into each of its blocks come from one
        // carry-chain addition each (a product up to 2^24 limbs)
        uint64_t gm = 0, pm = 0, um = 0;  // um: blocks that took 0
        for (int base = 0; base < per; base += kAggBatch) {
            uint32_t h[kAggBatch];
#pragma unroll
            for (int i = 0; i < kAggBatch; ++i) h[i] = base + i < n ? __ldcg(&agg[b0 + base + i]) : 2u;
#pragma unroll
            for (int i = 0; i < kAggBatch; ++i) {
                gm |= (uint64_t)(h[i] & 1u) << (base + i);
                pm |= (uint64_t)((h[i] >> 1) & 1u) << (base + i);
                um |= (uint64_t)((h[i] >> 2) & 1u) << (base + i);
            }
        }
        const u128 A = (u128)(gm | pm), B = (u128)gm;
        const uint64_t nmask = n >= 64 ? ~0ull : ((1ull << n) - 1);
        const bool tG = (uint64_t)(((A + B) ^ A ^ B) >> n) & 1;  // carry out of the run, carry-in 0
        const bool tP = (pm & nmask) == nmask;
        const bool c = block_carry(tG, tP, sh, chunk_in);  // carry into this thread's first block
        const u128 cc = (A + B + (c ? 1u : 0u)) ^ A ^ B;   // bit i: carry into block b0 + i
        for (uint64_t enter = (uint64_t)cc & nmask & um; enter; enter &= enter - 1) ripple(b0 + __ffsll((long long)enter) - 1);
        cout = (uint64_t)(cc >> n) & 1;
    } else {
        // longer runs: two passes over the aggregates
        bool tG = false, tP = true;
        for (int base = b0; base < b1; base += kAggBatch) {
            uint32_t h[kAggBatch];
#pragma unroll
            for (int i = 0; i < kAggBatch; ++i) h[i] = base + i < b1 ? __ldcg(&agg[base + i]) : 2u;
#pragma unroll
            for (int i = 0; i < kAggBatch; ++i) {
                tG = (h[i] & 1u) || (tG && (h[i] & 2u));
                tP = tP && (h[i] & 2u);
            }
        }
        bool c = block_carry(tG, tP, sh, chunk_in);  // carry into this thread's first block
        for (int b = b0; b < b1; ++b) {
            const uint32_t a = __ldcg(&agg[b]);
            if (c && (a & 4u)) ripple(b);
            c = (a & 1u) || (c && (a & 2u));
        }
        cout = c;
    }
    if (b0 < bhi && b1 == bhi) run_out(cout);  // the thread holding the last block
}

}  // namespace precgpu
