// The Adagrad step of one element, shared by the kernels that update node rows.
#pragma once
#include "common.cuh"

namespace ge2 {

constexpr float kAdagradEps = 1e-10f;  // literal in cpp/src/data/batch.cpp:266 of the reference project

// state += g*g ; delta = -lr * g / (sqrt(state) + eps), one IEEE operation at a time
__device__ __forceinline__ void adagrad_elem(float g, float& state, float& delta, float& upd, float neg_lr) {
    upd = __fmul_rn(g, g);
    state = __fadd_rn(state, upd);
    const float den = __fadd_rn(__fsqrt_rn(state), kAdagradEps);
    delta = __fmul_rn(neg_lr, __fdiv_rn(g, den));
}

}  // namespace ge2
