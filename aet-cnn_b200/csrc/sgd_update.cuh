// The SGD-momentum update of one parameter (mtcs/MtcsConvLayer.c:618-631 with its two NaN scrubs, :586-587), shared by the
// update kernels and by the weight gradient that applies it in its epilogue: the same operations in the same order, so that
// a parameter's value does not depend on which of them moved it.
#pragma once

namespace {

// u = U + G; scrub; u += decay * w; w += rate * u; u *= momentum.  A frozen parameter (a layer that is not updated now) only
// adds the gradient to its pending update.  `index` is the element's position in its segment.
struct SgdStep {
    float rate, momentum, decay;
    int scrub;
    bool frozen;
};
// seg: {learning-rate multiplier (negative: frozen), decay flag, scrub kind, ...}; hyper: {rate / B, momentum, -decay * B, ...}
__device__ __forceinline__ SgdStep sgd_step(const float *seg, const float *hyper) {
    SgdStep s;
    s.frozen = seg[0] < 0.f;
    s.rate = hyper[0] * seg[0];
    s.momentum = hyper[1];
    s.decay = seg[1] != 0.f ? hyper[2] : 0.f;
    s.scrub = (int)seg[2];
    return s;
}
// Non-finite scrub of the reference's GPU update.  kind 1 = a weight segment: a NaN/Inf pending update becomes 0
// (resetNanAndInf) and a NaN/Inf weight becomes 1 / (index + 1) (fixNanAndInf), mtcs/MtcsConvLayer.c:586-587,
// mtcs/MtcsTool.c:77-107.  kind 2 = a bias / scale segment of a batch-norm layer with try_fix_nan: the pending
// update becomes 1 / (index + 1), dnn/NLayer.c:318-323.  `index` is the element's position in its segment.
// Returns true when something was replaced.
__device__ __forceinline__ bool scrub1(float &w, float &u, int kind, size_t index) {
    bool hit = false;
    if (kind == 1) {
        if (isnan(u) || isinf(u)) { u = 0.f; hit = true; }
        if (isnan(w) || isinf(w)) { w = 1.0f / ((float)index + 1.f); hit = true; }
    } else if (kind == 2) {
        if (isnan(u) || isinf(u)) { u = 1.0f / ((float)index + 1.f); hit = true; }
    }
    return hit;
}
__device__ __forceinline__ void sgd_move(float &w, float &u, float rate, float momentum, float decay) {
    u = __fmaf_rn(decay, w, u);
    w = __fmaf_rn(rate, u, w);
    u = __fmul_rn(u, momentum);
}

}  // namespace
