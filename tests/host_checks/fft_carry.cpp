// The FP64 band's carry on the host, with the kernel's own limb sums: exact
// products of short operands come out whole and pass the check of the limbs past
// the product, and a coefficient off by any amount that takes the number out of
// the product's limbs (or below zero) fails it, as the full signed carry over
// every limb that a coefficient reaches would.  Also: the cluster covers the
// product and the checked limbs for every length of the band.
#include <cstdio>
#include <cstdlib>
#include <vector>

#include "fft_kernels.cuh"

using namespace precgpu;
typedef __int128 i128;
typedef unsigned __int128 u128;

static uint64_t rng_state = 12345;
static uint64_t rnd() {
    uint64_t z = rng_state += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

static std::vector<long long> digits(const std::vector<uint64_t>& a, int b, size_t n) {
    std::vector<long long> d(n);
    auto raw = [&](size_t i) -> uint32_t {
        uint32_t r = 0;
        for (int k = 0; k < b; ++k) {
            const size_t bit = i * b + k;
            if (bit / 64 < a.size()) r |= (uint32_t)(a[bit / 64] >> (bit % 64) & 1) << k;
        }
        return r;
    };
    const uint32_t half = 1u << (b - 1);
    for (size_t i = 0; i < n; ++i)
        d[i] = (long long)raw(i) - (raw(i) >= half ? 1 << b : 0) + (i > 0 && raw(i - 1) >= half ? 1 : 0);
    return d;
}

// limbs [0, n) of sum c_i 2^(bi) as a signed number, and the carry out of them
static std::vector<uint64_t> signed_limbs(const std::vector<long long>& c, int b, size_t n, i128& out) {
    std::vector<uint64_t> r(n);
    i128 carry = 0;
    size_t i = 0;
    for (size_t m = 0; m < n; ++m) {
        u128 lo = (u128)carry & 0xffffffffffffffffull;
        i128 hi = carry >> 64;
        for (; i < c.size() && i * b < 64 * (m + 1); ++i) {
            const int s = (int)(i * b - 64 * m);
            const i128 v = (i128)c[i] * ((i128)1 << s);
            lo += (u128)v & 0xffffffffffffffffull;
            hi += v >> 64;
        }
        r[m] = (uint64_t)lo;
        carry = hi + (i128)(lo >> 64);
    }
    out = carry;
    return r;
}

// the kernel's way: limbs and whether the check passes
static bool kernel_limbs(const std::vector<long long>& c, int b, size_t lout, std::vector<uint64_t>& r) {
    bool ok = true;
    uint64_t carry = 0;
    r.assign(lout, 0);
    auto coef = [&](uint32_t i) { return c[i]; };
    for (size_t m = 0; m < lout + kFftPastLimbs; ++m) {
        const u128 s = (u128)(uint64_t)fft_limb_sum(coef, c.size(), b, (int64_t)m) +
                       (uint64_t)(fft_limb_sum(coef, c.size(), b, (int64_t)m - 1) >> 64) + carry;
        carry = (uint64_t)(s >> 64);
        if (m < lout) r[m] = (uint64_t)s;
        else if ((uint64_t)s != fft_past_value(b, c.size(), (int64_t)m)) ok = false;
    }
    return ok;
}

int main() {
    for (uint64_t lout = 2; lout <= 12288; ++lout) {
        const int L = fft_carry_limbs(lout);
        const int warps = fft_carry_warps(lout);
        const uint64_t ctas = fft_carry_ctas(lout);
        if (L < 1 || L > 3 || warps < 16 || warps > 17 || ctas < 1 || ctas > kFftCarryCluster ||
            ctas * 32 * warps * L < lout + kFftPastLimbs) {
            std::printf("%llu limbs: %d per thread do not cover them\n", (unsigned long long)lout, L);
            return 1;
        }
    }
    int caught = 0, inside = 0;
    for (int t = 0; t < 4000; ++t) {
        const int b = t % 5 == 4 ? 30 - t % 13 : 8 + (int)(rnd() % 9);
        const size_t la = 1 + rnd() % 9, lb = 1 + rnd() % 9, lout = la + lb;
        std::vector<uint64_t> x(la), y(lb);
        const int kind = (int)(rnd() % 3);
        for (auto& v : x) v = kind == 0 ? ~0ull : rnd();
        for (auto& v : y) v = kind == 0 ? ~0ull : rnd();
        if (kind == 2) x[la - 1] = y[lb - 1] = 0;  // far below the top
        const size_t da = (64 * la + b - 1) / b + 1, db = (64 * lb + b - 1) / b + 1;
        size_t N = 64;
        while (N < da + db - 1) N *= 2;
        const auto dx = digits(x, b, da), dy = digits(y, b, db);
        std::vector<long long> c(N, 0);
        for (size_t i = 0; i < da; ++i)
            for (size_t j = 0; j < db; ++j) c[i + j] += dx[i] * dy[j];
        std::vector<uint64_t> r;
        i128 out;
        const size_t all = (b * N + 63) / 64 + 3;  // every limb that a coefficient reaches
        auto ref = signed_limbs(c, b, all, out);
        if (!kernel_limbs(c, b, lout, r)) {
            std::printf("refused an exact product: b %d, %zu x %zu\n", b, la, lb);
            return 1;
        }
        for (size_t m = 0; m < lout; ++m)
            if (r[m] != ref[m]) {
                std::printf("limb %zu: b %d, %zu x %zu\n", m, b, la, lb);
                return 1;
            }
        // one coefficient off
        for (int e = 0; e < 8; ++e) {
            auto w = c;
            const size_t i = e < 4 ? da + db - 2 - rnd() % 5 : rnd() % (da + db - 1);
            w[i] += (rnd() & 1 ? 1ll : -1ll) * (1ll << rnd() % 40);
            ref = signed_limbs(w, b, all, out);
            bool fits = out == 0;
            for (size_t m = lout; m < all; ++m) fits = fits && ref[m] == 0;
            if (kernel_limbs(w, b, lout, r) != fits) {
                std::printf("b %d, %zu x %zu, N %zu, coefficient %zu off: expected %d\n", b, la, lb, N, i, (int)fits);
                return 1;
            }
            ++(fits ? inside : caught);
        }
    }
    if (caught < 1000 || inside < 1000) {
        std::printf("caught %d, inside %d\n", caught, inside);
        return 1;
    }
    return 0;
}
