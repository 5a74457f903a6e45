// mul_direct.cu -- direct (schoolbook) products of short operands.
//
// preclib forms products below its FFT band by schoolbook and Karatsuba
// (src/mul_basic.cpp:206-269); here the direct form takes the short products
// of the device-pointer calls: 32-bit digits, every column sum
// S_c = sum_{i+j=c} a_i b_j exact in 96 bits, then the carry chain over the
// limbs T_m = S_2m + 2^32 S_2m+1.
//
// Work split.  Columns are taken R at a time, and column block c together
// with block c + na (na, nb: digit blocks of the longer and the shorter
// operand): with j running over the nb digit blocks of b, column block c
// meets a-blocks c-j for j <= c and column block c + na meets a-blocks
// c-j+na for j >= c, so every pair costs exactly nb + 1 block steps of R x R
// multiply-adds and no thread waits for a longer neighbour.  One block step
// takes 2R - 1 digits of a (a window that slides by one block) and R of b.
//
// What bounds it: the 32x32->64-bit multiply-add, one per digit pair; 8192
// products of 512 x 96 limbs reach 6.2 T multiply-adds/s, 40000 of 64 x 64
// limbs 5.1 T/s (there the flushes and the carry stage show).  44643 products of
// 58 .. 66 limbs: kernels 0.98 -> 0.18 ms against the single-CTA transform.
// A single product is bound by latency instead: launch, two trips to L2 and
// the carries of the last CTA; 1024 x 1000 limbs 28.7 -> 8.1 us.
#include "mul_direct.cuh"

#include "ntt_engine.cuh"

namespace precgpu {

// (lo, mid, hi) += x * y
__device__ __forceinline__ void mac96(uint32_t& lo, uint32_t& mid, uint32_t& hi, uint32_t x, uint32_t y) {
    asm("mad.lo.cc.u32 %0, %3, %4, %0;\n\t"
        "madc.hi.cc.u32 %1, %3, %4, %1;\n\t"
        "addc.u32 %2, %2, 0;"
        : "+r"(lo), "+r"(mid), "+r"(hi)
        : "r"(x), "r"(y));
}

// digit blocks in shared memory: R words at a stride that keeps 16-byte
// loads of consecutive blocks by consecutive lanes free of bank conflicts
template <int R>
struct Blk {
    static constexpr int S = R == 8 ? 12 : R;  // (12 words: 8 lanes cover the 32 banks once)
    static_assert(S == 12, "bank-conflict-free strides");
    static __device__ __forceinline__ void load(uint32_t (&x)[R], const uint32_t* p) {
#pragma unroll
        for (int h = 0; h < R / 4; ++h) {
            const uint4 v = *reinterpret_cast<const uint4*>(p + 4 * h);
            x[4 * h] = v.x;
            x[4 * h + 1] = v.y;
            x[4 * h + 2] = v.z;
            x[4 * h + 3] = v.w;
        }
    }
    // limb l of an operand: digits 2l, 2l + 1
    static __device__ __forceinline__ void put(uint32_t* s, int l, uint64_t v) {
        const int d = 2 * l;
        *reinterpret_cast<uint64_t*>(s + (d / R) * S + d % R) = v;
    }
};

// R column sums
template <int R>
struct Acc {
    uint32_t w[3][R];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int k = 0; k < 3; ++k)
#pragma unroll
            for (int r = 0; r < R; ++r) w[k][r] = 0;
    }
    // one block step: a-blocks `lower` and `upper` (the next block up), b-block y
    __device__ __forceinline__ void step(const uint32_t (&lower)[R], const uint32_t (&upper)[R],
                                         const uint32_t (&y)[R]) {
#pragma unroll
        for (int s = 0; s < R; ++s)
#pragma unroll
            for (int r = 0; r < R; ++r)
                mac96(w[0][r], w[1][r], w[2][r], r >= s ? upper[r - s] : lower[R + r - s], y[s]);
    }
};

// ---------------------------------------------------------------------------
// batch form
// ---------------------------------------------------------------------------

// G threads per product (G <= 32: 32 / G products per warp)
template <int R, int G>
struct DirectGeom {
    static constexpr int A_BLKS = G + 2;             // zero block, up to G blocks, zero block
    static constexpr int B_BLKS = G + 1;             // up to G blocks, zero block
    static constexpr int COLS = 2 * R * G;
    static constexpr int PCOLS = COLS + COLS / R;    // padded: column c at c + c / R
    static constexpr int WORDS = (A_BLKS + B_BLKS) * Blk<R>::S + 3 * PCOLS;
    static constexpr int THREADS = G <= 32 ? 128 : G;
    static constexpr int PER_CTA = THREADS / G;
    static constexpr size_t SMEM = (size_t)WORDS * PER_CTA * sizeof(uint32_t);
};

template <int G>
__device__ __forceinline__ void group_sync() {
    if constexpr (G <= 32) __syncwarp();
    else __syncthreads();
}

constexpr int kListThreads = 256;

// Classes by list: a warp's lanes of one class take their places together.
// (With every class's launch going over all items, mostly empty groups kept
// the shared memory of half-empty CTAs: 44643 products of 58 .. 66 limbs,
// two classes, 299 us of kernels; with lists 175.)
__global__ void __launch_bounds__(kListThreads) k_direct_lists(const DirectItem* __restrict__ items, int count, uint32_t* lists,
                                                      uint32_t* n) {
    pdl_enter();
    const int64_t i = direct_first(blockIdx.x, kListThreads) + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const int cls = i < count ? direct_class(items[i].la, items[i].lb) : -1;
    const uint32_t same = __match_any_sync(0xffffffffu, cls);
    const int leader = __ffs(same) - 1;
    uint32_t at = 0;
    if (cls >= 0 && lane == leader) at = atomicAdd(&n[cls], (uint32_t)__popc(same));
    at = __shfl_sync(0xffffffffu, at, leader) + __popc(same & ((1u << lane) - 1));
    if (cls >= 0) lists[(size_t)cls * count + at] = (uint32_t)i;
}

template <int R, int G>
__global__ void __launch_bounds__(DirectGeom<R, G>::THREADS) k_direct(const DirectItem* __restrict__ items, int count,
                                                                   const uint32_t* __restrict__ list,
                                                                   const uint32_t* n) {
    using D = DirectGeom<R, G>;
    constexpr int S = Blk<R>::S;
    extern __shared__ __align__(16) uint32_t dsm[];
    __shared__ BlockCarryShared sh;
    pdl_enter();
    pdl_next();
    if (n) count = (int)*after_entry(n);
    list = after_entry(list);
    const int sub = threadIdx.x / G;
    const int g = threadIdx.x & (G - 1);
    uint32_t* sa = dsm + sub * D::WORDS;  // block i of a at (i + 1) * S
    uint32_t* sb = sa + D::A_BLKS * S;
    uint32_t* cols = sb + D::B_BLKS * S;
    const int64_t stride = direct_first(gridDim.x, D::PER_CTA);
    for (int64_t base = direct_first(blockIdx.x, D::PER_CTA); base < count; base += stride) {
        const bool live = base + sub < count;  // a group past the end runs an empty product
        const int64_t at = live ? base + sub : count - 1;
        const DirectItem d = items[list ? list[at] : at];
        const bool swap = d.la < d.lb;
        const uint64_t* __restrict__ pa = swap ? d.b : d.a;
        const uint64_t* __restrict__ pb = swap ? d.a : d.b;
        const int la = live ? (int)(swap ? d.lb : d.la) : 0, lb = live ? (int)(swap ? d.la : d.lb) : 0;
        const int na = (2 * la + R - 1) / R, nb = (2 * lb + R - 1) / R;  // digit blocks
        for (int i = g; i < na * (R / 2); i += G) Blk<R>::put(sa + S, i, i < la ? __ldg(&pa[i]) : 0ull);
        for (int i = g; i < (nb + 1) * (R / 2); i += G) Blk<R>::put(sb, i, i < lb ? __ldg(&pb[i]) : 0ull);
        if (g < R) {
            sa[g] = 0;
            sa[(na + 1) * S + g] = 0;
        }
        group_sync<G>();

        const bool active = g < na;
        const int c = g;  // column block
        if (active) {
            Acc<R> acc;
            acc.zero();
            auto flush = [&](int blk) {
                uint32_t* p = cols + blk * (R + 1);
#pragma unroll
                for (int k = 0; k < 3; ++k)
#pragma unroll
                    for (int r = 0; r < R; ++r) p[k * D::PCOLS + r] = acc.w[k][r];
            };
            uint32_t upper[R];
            Blk<R>::load(upper, sa + (c + 1) * S);
            int jb = 0, ab = c;
            bool high = false;
            for (int t = 0; t <= nb; ++t) {
                if (t == c + 1) {  // from column block c to block c + na
                    flush(c);
                    acc.zero();
                    high = true;
                    jb = c;
                    ab = na;
#pragma unroll
                    for (int r = 0; r < R; ++r) upper[r] = 0;
                }
                uint32_t lower[R], y[R];
                Blk<R>::load(lower, sa + ab * S);  // block ab - 1
                Blk<R>::load(y, sb + jb * S);
                acc.step(lower, upper, y);
#pragma unroll
                for (int r = 0; r < R; ++r) upper[r] = lower[r];
                ++jb;
                --ab;
            }
            flush(high ? na + c : c);
        }
        group_sync<G>();

        // limbs g*R .. g*R + R - 1
        const int lout = la + lb;
        const int m0 = g * R;
        auto col = [&](int i) -> u128 {
            const uint32_t* p = cols + i + i / R;
            return ((u128)p[2 * D::PCOLS] << 64) | ((uint64_t)p[D::PCOLS] << 32) | p[0];
        };
        u128 T[R];
#pragma unroll
        for (int k = 0; k < R; ++k) T[k] = m0 + k < lout ? col(2 * (m0 + k)) + (col(2 * (m0 + k) + 1) << 32) : (u128)0;
        uint64_t prev_hi = 0;
        if (g > 0 && m0 - 1 < lout) prev_hi = (uint64_t)((col(2 * m0 - 2) + (col(2 * m0 - 1) << 32)) >> 64);
        uint64_t v[R];
        uint32_t gbits;
        bool cg, cp;
        limbs_from_sums<R>(T, prev_hi, v, gbits, cg, cp);
        bool cin;
        if constexpr (G <= 32) {
            constexpr uint32_t mask = G == 32 ? 0xffffffffu : (1u << G) - 1;
            const int sh0 = (threadIdx.x & 31) & ~(G - 1);  // the group's first lane
            const uint32_t gm = (__ballot_sync(0xffffffffu, cg) >> sh0) & mask;
            const uint32_t pm = (__ballot_sync(0xffffffffu, cp) >> sh0) & mask;
            cin = (carry_chain(gm, pm, false) >> g) & 1;
            __syncwarp();
        } else {
            cin = block_carry(cg, cp, sh, [](bool, bool) { return false; });
        }
        // the limbs through shared memory (limb m at m + m / R) to whole-line stores
        uint64_t* st = reinterpret_cast<uint64_t*>(cols);
        limbs_finish<R>(m0, (uint64_t)lout, v, gbits, cin, st + g);
        group_sync<G>();
        for (int m = g; m < lout; m += G) d.out[m] = st[m + m / R];
        group_sync<G>();  // the next product's operands
    }
}

// (class, R, G): the longer operand up to R G / 2 limbs
#define PREC_DIRECT(X) X(0, 8, 16) X(1, 12, 16) X(2, 8, 32) X(3, 8, 64) X(4, 8, 128)

void launch_direct_lists(const DirectItem* d_items, int count, uint32_t* lists, uint32_t* n, cudaStream_t st) {
    launch_pdl(false, k_direct_lists, direct_ctas(count, kListThreads, 0x7fffffff), kListThreads, 0, st, d_items, count, lists, n);
    count_launches(1);
}

void launch_direct_batch(const DirectItem* d_items, int count, int cls, cudaStream_t st, const uint32_t* list,
                         const uint32_t* n) {
    // with a list of unknown length: as many CTAs as stay resident, a few times over
    const int cap = n ? device_sm_count() * 64 : 0x7fffffff;
#define X(C, R, G)                                                                                          \
    if (cls == C) {                                                                                         \
        using D = DirectGeom<R, G>;                                                                         \
        launch_pdl(false, k_direct<R, G>, direct_ctas(count, D::PER_CTA, cap), D::THREADS, D::SMEM, st,     \
                   d_items, count, list, n);                                                                \
        count_launches(1);                                                                                  \
    }
    PREC_DIRECT(X)
#undef X
}

// ---------------------------------------------------------------------------
// single product over the whole GPU
// ---------------------------------------------------------------------------

constexpr int kGridR = 8;
constexpr int kGridThreads = 512;

struct DirectArgs {
    const uint64_t* a;  // the longer operand
    const uint64_t* b;
    uint64_t* out;
    uint64_t* sums;     // per limb m: T_m = S_2m + 2^32 S_2m+1, two words
    uint32_t* counter;
    int* err;
    int la, lb, na, nb; // limbs and digit blocks
};

// CB column blocks (with their partners na blocks up) per CTA, their nb + 1
// block steps split over kGridThreads / CB threads each; the partial sums
// are added in shared memory, the column sums go to scratch, and the last
// CTA to finish (fence and counter) resolves the carries.
template <int CB>
__global__ void __launch_bounds__(kGridThreads) k_direct_grid(DirectArgs f) {
    constexpr int R = kGridR, S = Blk<R>::S;
    constexpr int SL = kGridThreads / CB;  // slices per column block
    extern __shared__ __align__(16) uint32_t dsm[];
    __shared__ BlockCarryShared sh;
    __shared__ uint32_t s_last;
    uint32_t* sa = dsm;
    uint32_t* sb = sa + (f.na + 2) * S;
    // partial sums: slot s < SL of a column block holds slice s's sums, slot
    // SL the low part of the slice that crosses from block c to block c + na
    uint32_t* part = sb + (f.nb + 1) * S;
    pdl_enter();
    pdl_next();
    f.a = after_entry(f.a);
    f.b = after_entry(f.b);
    constexpr int PS = 3 * R + 1;  // words per slot (odd: no bank conflicts across slots)
#pragma unroll 4
    for (int i = threadIdx.x; i < f.na * (R / 2); i += kGridThreads) Blk<R>::put(sa + S, i, i < f.la ? __ldg(&f.a[i]) : 0ull);
#pragma unroll 4
    for (int i = threadIdx.x; i < (f.nb + 1) * (R / 2); i += kGridThreads) Blk<R>::put(sb, i, i < f.lb ? __ldg(&f.b[i]) : 0ull);
    if (threadIdx.x < R) {
        sa[threadIdx.x] = 0;
        sa[(f.na + 1) * S + threadIdx.x] = 0;
    }
    __syncthreads();
    const int c0 = blockIdx.x * CB;
    const int steps = f.nb + 1;
    {
        const int cl = threadIdx.x / SL, s = threadIdx.x % SL;
        const int c = c0 + cl;
        const int t0 = (int)((long long)steps * s / SL), t1 = (int)((long long)steps * (s + 1) / SL);
        uint32_t* slots = part + cl * (SL + 1) * PS;
        Acc<R> acc;
        acc.zero();
        auto put = [&](int slot) {
#pragma unroll
            for (int k = 0; k < 3; ++k)
#pragma unroll
                for (int r = 0; r < R; ++r) slots[slot * PS + k * R + r] = acc.w[k][r];
        };
        if (c < f.na) {
            for (int t = t0; t < t1; ++t) {
                if (t == c + 1 && t > t0) {
                    put(SL);
                    acc.zero();
                }
                const bool high = t > c;
                const int jb = high ? t - 1 : t;             // t = c + 1: j = c
                const int ab = c - jb + (high ? f.na : 0);   // -1 <= ab - 1, ab <= na
                uint32_t lower[R], upper[R], y[R];
                Blk<R>::load(lower, sa + ab * S);
                Blk<R>::load(upper, sa + (ab + 1) * S);
                Blk<R>::load(y, sb + jb * S);
                acc.step(lower, upper, y);
            }
        }
        put(s);
    }
    __syncthreads();
    {   // add the slices: P threads per column
        constexpr int OUT = CB * 2 * R;  // columns of this CTA
        // (at most 16: two neighbouring columns share a warp)
        constexpr int P = kGridThreads / OUT < 16 ? kGridThreads / OUT : 16;
        const int o = threadIdx.x / P, p = threadIdx.x % P;
        const int cl = o / (2 * R), half = (o / R) & 1, r = o % R;
        const int c = c0 + cl;
        const uint32_t* slots = part + cl * (SL + 1) * PS;
        // first slice that ends past the low steps 0 .. c
        int x = SL, cross = 0;
        if (c + 1 < steps) {
            // slice s covers [steps*s/SL, steps*(s+1)/SL): the one holding step c + 1
            x = (int)(((long long)(c + 1) * SL + SL) / steps);
            if (x > SL) x = SL;
            while (x > 0 && (int)((long long)steps * x / SL) > c + 1) --x;
            while ((int)((long long)steps * (x + 1) / SL) <= c + 1) ++x;
            cross = (int)((long long)steps * x / SL) < c + 1;  // it also holds low steps
        }
        uint64_t lo = 0, hi = 0;  // 96-bit sums as lo + 2^32 * hi (both below 2^64)
        auto add = [&](int slot) {
            const uint32_t* q = slots + slot * PS + r;
            lo += q[0];
            hi += (uint64_t)q[R] + ((uint64_t)q[2 * R] << 32);
        };
        if (o < OUT) {
            const int s0 = half ? x : 0, s1 = half ? SL : x;
            for (int s = s0 + p; s < s1; s += P) add(s);
            if (!half && cross && p == 0) add(SL);
        }
#pragma unroll
        for (int k = P / 2; k > 0; k >>= 1) {
            lo += __shfl_down_sync(0xffffffffu, lo, k, P);
            hi += __shfl_down_sync(0xffffffffu, hi, k, P);
        }
        // T = S_2m + 2^32 S_2m+1: the odd column's sum from the next output
        const uint64_t lo1 = __shfl_down_sync(0xffffffffu, lo, P);
        const uint64_t hi1 = __shfl_down_sync(0xffffffffu, hi, P);
        if (o < OUT && p == 0 && !(r & 1) && c < f.na && (!half || c < f.nb)) {
            const u128 T = (u128)lo + ((u128)hi << 32) + ((u128)lo1 << 32) + ((u128)hi1 << 64);
            const int m = ((c + (half ? f.na : 0)) * R + r) / 2;
            *reinterpret_cast<ulonglong2*>(f.sums + 2 * m) = make_ulonglong2((uint64_t)T, (uint64_t)(T >> 64));
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        s_last = atomicAdd(f.counter, 1u) == gridDim.x - 1 ? 1u : 0u;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x == 0) *f.counter = 0;
    // carries over the block, L limbs per thread per round
    constexpr int L = 8;
    const int lout = f.la + f.lb;
    bool carry = false;
    for (int r0 = 0; r0 < lout; r0 += kGridThreads * L) {
        const int m0 = r0 + threadIdx.x * L;
        u128 T[L];
#pragma unroll
        for (int k = 0; k < L; ++k) {
            ulonglong2 w = make_ulonglong2(0, 0);
            if (m0 + k < lout) w = __ldcg(reinterpret_cast<const ulonglong2*>(f.sums) + m0 + k);
            T[k] = ((u128)w.y << 64) | w.x;
        }
        const uint64_t prev_hi = m0 > 0 && m0 - 1 < lout ? __ldcg(&f.sums[2 * (m0 - 1) + 1]) : 0;
        uint64_t v[L];
        uint32_t gbits;
        bool G, P;
        limbs_from_sums<L>(T, prev_hi, v, gbits, G, P);
        auto cin_fn = [&](bool Gb, bool Pb) -> bool {
            sh.block_cin = (Gb || (Pb && carry)) ? 1u : 0u;
            return carry;
        };
        const bool cin = block_carry(G, P, sh, cin_fn);
        limbs_finish<L>(m0, (uint64_t)lout, v, gbits, cin, f.out);
        const int last = lout - 1 - m0;  // a product fits La+Lb limbs
        if (last >= 0 && last < L && limbs_overflow<L>(last, T, v, gbits, cin)) atomicOr(f.err, kDevErrCarry);
        __syncthreads();
        carry = sh.block_cin != 0;
        __syncthreads();
    }
}

static int grid_blocks(uint64_t limbs) { return (int)((2 * limbs + kGridR - 1) / kGridR); }

static size_t grid_smem(int cb, int na, int nb) {
    return ((size_t)(na + 2 + nb + 1) * Blk<kGridR>::S + (size_t)cb * (kGridThreads / cb + 1) * (3 * kGridR + 1)) *
           sizeof(uint32_t);
}

// Direct up to 2^22 limb pairs: measured 5.9 us at 64 x 64 limbs (transform
// 12.6), 8.1 at 1024 x 1000 (28.7), 14.9 at 2048 x 2048 and 16.4 at
// 4096 x 1000 (19.2).  4096 limbs are what one CTA's shared memory takes.
bool direct_single(uint64_t la, uint64_t lb) {
    const uint64_t hi = la > lb ? la : lb;
    return hi <= kDirectGridMax && la * lb <= 1ull << 22;
}

size_t direct_scratch_bytes(uint64_t la, uint64_t lb) {
    return (size_t)(grid_blocks(la) + grid_blocks(lb)) * kGridR * sizeof(uint64_t);
}

#define PREC_DIRECT_GRID(X) X(1) X(2) X(4) X(8)

void launch_direct_single(const uint64_t* a, uint64_t la, const uint64_t* b, uint64_t lb, uint64_t* out,
                          uint8_t* scratch, uint32_t* counter, int* err, cudaStream_t st) {
    const bool swap = la < lb;
    DirectArgs f;
    f.a = swap ? b : a;
    f.b = swap ? a : b;
    f.la = (int)(swap ? lb : la);
    f.lb = (int)(swap ? la : lb);
    f.na = grid_blocks(f.la);
    f.nb = grid_blocks(f.lb);
    f.out = out;
    f.sums = reinterpret_cast<uint64_t*>(scratch);
    f.counter = counter;
    f.err = err;
    int cb = 1;
    while (cb < 8 && (f.na + cb - 1) / cb > device_sm_count()) cb *= 2;
#define X(C)                                                                                           \
    if (cb == C) {                                                                                     \
        launch_pdl(false, k_direct_grid<C>, (f.na + C - 1) / C, kGridThreads, grid_smem(C, f.na, f.nb), st, f); \
        count_launches(1);                                                                             \
    }
    PREC_DIRECT_GRID(X)
#undef X
}

int configure_direct() {
    cudaError_t e = load_kernel(k_direct_lists);
#define X(C, R, G) \
    if (!e) e = cudaFuncSetAttribute(k_direct<R, G>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)DirectGeom<R, G>::SMEM);
    PREC_DIRECT(X)
#undef X
    const int nmax = grid_blocks(kDirectGridMax);
#define X(C) \
    if (!e) e = cudaFuncSetAttribute(k_direct_grid<C>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)grid_smem(C, nmax, nmax));
    PREC_DIRECT_GRID(X)
#undef X
    return (int)e;
}

}  // namespace precgpu
