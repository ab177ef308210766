// Elementwise pieces of the surrogate network shared by its kernels.
#pragma once

namespace mlpmath {

__device__ __forceinline__ float gelu(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

__device__ __forceinline__ float gelu_grad(float x)
{
    return 0.5f * (1.0f + erff(x * 0.70710678118654752f)) +
           x * 0.39894228040143268f * expf(-0.5f * x * x);
}

struct AdamW {
    float lr, b1, b2, eps, wd, c1, c2;
};

// One AdamW update of a master parameter w with moments m, v and gradient gi.
// Explicit operations: the compiler contracts the sums of two products one way
// or the other depending on what is around them, and every kernel that updates
// parameters has to give the same bits.
__device__ __forceinline__ void adamw(float &w, float &m, float &v, float gi, const AdamW &p,
                                      float wd)
{
    const float mi = __fmaf_rn(1.f - p.b1, gi, __fmul_rn(p.b1, m));
    const float vi = __fmaf_rn(__fmul_rn(1.f - p.b2, gi), gi, __fmul_rn(p.b2, v));
    m = mi;
    v = vi;
    const float mh = mi / p.c1, vh = vi / p.c2;
    const float u = mh / (sqrtf(vh) + p.eps);
    w = __fmaf_rn(-p.lr, __fmaf_rn(wd, w, u), w);
}

}  // namespace mlpmath
