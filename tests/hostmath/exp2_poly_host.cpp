// Host build of the polynomial with which attention_tc05.cu evaluates some of its exponentials.
#include <math.h>
#include <stdint.h>
#include "../../pointtransformerv3_b200/csrc/exp2_poly.cuh"

using namespace ptv3;

extern "C" void host_exp2_poly(const float* r, int64_t n, float* out)
{
    for (int64_t i = 0; i < n; ++i) {
        float p = fmaf(r[i], EXP2_C5, EXP2_C4);
        p = fmaf(p, r[i], EXP2_C3);
        p = fmaf(p, r[i], EXP2_C2);
        p = fmaf(p, r[i], EXP2_C1);
        out[i] = fmaf(p, r[i], EXP2_C0);
    }
}
