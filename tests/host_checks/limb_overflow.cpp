// The check that a product ends with its last limb, on the host with the
// kernels' own functions: limb sums of a number of 1 .. L limbs pass, and the
// same sums with 2^64n more or with a larger last limb do not.
#include <cstdio>

#include "ntt_engine.cuh"

using namespace precgpu;

static uint64_t state = 99;
static uint64_t rnd() {
    state = state * 6364136223846793005ull + 1442695040888963407ull;
    return (state ^ (state >> 29)) * 0xBF58476D1CE4E5B9ull ^ state >> 17;
}

int main() {
    constexpr int L = 8;
    int over = 0;
    for (int t = 0; t < 20000; ++t) {
        const int n = 1 + t % L;  // limbs of the product among this thread's
        u128 T[L] = {};
        const bool ones = t % 3 == 0, cin = rnd() & 1;
        uint64_t prev = t % 5 == 0 ? rnd() >> 40 : 0;
        for (int k = 0; k < n; ++k) T[k] = (u128)(ones ? ~0ull : rnd()) | (u128)(k + 1 < n || t % 2 ? rnd() >> 40 : 0) << 64;
        if (t % 7 == 0) T[n - 1] = ~0ull;
        uint64_t v[L];
        uint32_t gbits;
        bool G, P;
        limbs_from_sums<L>(T, prev, v, gbits, G, P);
        // the sum of T_k 2^64k + prev + cin, carried by hand
        u128 c = (u128)prev + (cin ? 1 : 0);
        for (int k = 0; k < n; ++k) {
            const u128 s = (u128)(uint64_t)T[k] + (uint64_t)c;
            c = (c >> 64) + (T[k] >> 64) + (s >> 64);
        }
        const bool want = c != 0;
        over += want;
        if (limbs_overflow<L>(n - 1, T, v, gbits, cin) != want) {
            std::printf("case %d, %d limbs: expected %d\n", t, n, (int)want);
            return 1;
        }
    }
    return over > 2000 && over < 18000 ? 0 : 1;
}
