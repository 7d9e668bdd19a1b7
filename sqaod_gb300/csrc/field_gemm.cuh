// field_gemm.cuh -- compensated fp32 summation of the local fields and energy row sums.
//
// GB300 runs FP64 at 1/64 of the fp32 rate, so sums of exact fp32 products (spins
// times couplings) are kept as (sum, compensation) pairs.
#pragma once

#include <cstdint>

namespace sq103 {

__device__ __forceinline__ void two_sum_acc(float &s, float &c, float x) {
    const float t = __fadd_rn(s, x);
    const float bp = __fsub_rn(t, s);
    const float err = __fadd_rn(__fsub_rn(s, __fsub_rn(t, bp)), __fsub_rn(x, bp));
    s = t;
    c = __fadd_rn(c, err);
}

}  // namespace sq103
