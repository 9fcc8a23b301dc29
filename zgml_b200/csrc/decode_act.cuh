// The activation chain of a gated feed-forward, element by element (the two fused decode kernels).
#pragma once
#include "zg_internal.cuh"

namespace {

// the general activation chain of one element (fused_elementwise steps, src/backend/reference.zig:262-300); out of line
__device__ __noinline__ float act_chain(const ZgDecStep* steps, uint32_t n_steps, float gt, float up, float sec0, int first_ext, uint32_t k) {
    float v = gt;
    for (uint32_t s = 0; s < n_steps; s++) {
        const ZgDecStep st = steps[s];
        if (st.op == ZG_EW_ADD || st.op == ZG_EW_MUL) {
            const float o2 = st.sec_kind == 1 ? gt : (st.sec_kind == 2 ? up : ((int)s == first_ext ? sec0 : __ldg(st.sec + k)));
            if (st.op == ZG_EW_ADD) v = st.is_swapped ? __fadd_rn(o2, v) : __fadd_rn(v, o2);
            else v = st.is_swapped ? __fmul_rn(o2, v) : __fmul_rn(v, o2);
        } else v = apply_unary(st.op, v);
    }
    return v;
}

} // namespace
