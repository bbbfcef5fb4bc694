// soft_cap.cuh — tanh for soft-capped scores.  Plain arithmetic (compiled by the host compiler in tests/test_soft_cap_host.py).
#pragma once
#include <cmath>

#if defined(__CUDACC__)
#define SOFT_CAP_FN __host__ __device__ __forceinline__
#else
#define SOFT_CAP_FN inline
#endif

// tanh(x), |x| < SOFT_CAP_SMALL: x times a polynomial in x^2, the interpolant of tanh(x) / x at the Chebyshev nodes of [0, SOFT_CAP_SMALL^2] (1e-9 off), 1e-7 in f32
// with its roundings.  Through an exponential, 1 - 2 / (e^2x + 1), the same is off by 1e-7 of 1, not of itself: 1e-5 of a score of 5 under a cap of 50.
constexpr float SOFT_CAP_SMALL = 0.55f;
SOFT_CAP_FN float tanh_small(float x) {
    const float u = x * x;
    float p = fmaf(-0.006238845642656088f, u, 0.021042168140411377f);
    p = fmaf(p, u, -0.05384336784482002f);
    p = fmaf(p, u, 0.13332468271255493f);
    p = fmaf(p, u, -0.3333331048488617f);
    p = fmaf(p, u, 1.0f);
    return x * p;
}
