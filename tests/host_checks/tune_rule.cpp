// The autotuner's acceptance rule: faster whole transforms do not buy slower
// truncated ones.  (First case: 2^22 points as 2^10 x 2^12 instead of 2^11 x 2^11
// on 32-bit digits, measured.)
#include "prec_gpu_internal.h"

using precgpu::tune_better;

int main() {
    const float dflt[4] = {185.9f, 169.5f, 145.0f, 125.8f};
    const float whole_only[4] = {180.9f, 179.7f, 176.7f, 175.7f};
    const float all[4] = {180.9f, 165.0f, 141.0f, 122.0f};
    const float truncated_only[4] = {185.8f, 160.0f, 135.0f, 115.0f};
    const float failed[4] = {180.9f, 165.0f, -1.0f, 122.0f};
    const float mixed[4] = {170.0f, 165.0f, 144.0f, 127.0f};
    if (tune_better(whole_only, dflt) || tune_better(truncated_only, dflt) || tune_better(failed, dflt)) return 1;
    if (tune_better(dflt, dflt)) return 1;
    return tune_better(all, dflt) && tune_better(mixed, dflt) ? 0 : 1;
}
