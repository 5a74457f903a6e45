// Walks the item ranges of the direct batch kernels on the host, with the
// kernels' own index functions: every CTA's rounds for the given item counts.
// Exits 1 at the first index out of range, or if the items are not covered once.
#include <cstdio>
#include <cstdlib>

#include "mul_direct.cuh"

using namespace precgpu;

static int walk(int count, int per, int cap) {
    const int ctas = direct_ctas(count, per, cap);
    if (ctas < 1 || ctas > cap || (ctas < cap && (int64_t)ctas * per < count)) return 1;
    const int64_t stride = direct_first((uint32_t)ctas, per);
    int64_t covered = 0;
    for (int c = 0; c < ctas; c += ctas > 4096 && c >= 8 && c < ctas - 64 ? ctas - 64 - c : 1) {
        int64_t last = -1;
        for (int64_t base = direct_first((uint32_t)c, per); base < count; base += stride) {
            if (base < 0 || base <= last) return 1;
            last = base;
            covered += base + per < count ? per : count - base;
        }
    }
    return ctas <= 4096 && covered != count ? 1 : 0;
}

int main() {
    const int counts[] = {1, 7, 8, 9, 44643, (1 << 30) - 1, 1 << 30, (1 << 30) + 1, 0x7fffff00, 0x7fffffff};
    const int pers[] = {1, 4, 8, 256};
    const int caps[] = {1, 1024, 152 * 64, 0x7fffffff};
    for (int n : counts)
        for (int p : pers)
            for (int c : caps)
                if (!(c == 1 && n > 1 << 20) && walk(n, p, c)) {
                    std::printf("count %d, %d at a time, at most %d CTAs\n", n, p, c);
                    return 1;
                }
    return 0;
}
