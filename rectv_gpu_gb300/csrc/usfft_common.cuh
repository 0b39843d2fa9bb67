// Device helpers shared by the USFFT gather/scatter kernels.
#pragma once

#include <cuda_runtime.h>

#include "rectv_internal.cuh"

namespace rectv {

__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// (a.x b.x + c.x, a.y b.y + c.y) as one packed FP32x2 FMA (each lane an IEEE
// fma.rn, so results equal two fmaf calls).
__device__ __forceinline__ float2 ffma2(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(d)
        : "l"(*reinterpret_cast<const unsigned long long *>(&a)), "l"(*reinterpret_cast<const unsigned long long *>(&b)),
          "l"(*reinterpret_cast<const unsigned long long *>(&c)));
    return *reinterpret_cast<const float2 *>(&d);
}

// Position of polar sample (theta, k): identical float operation sequence to
// the host plan (plan.cpp) and to takexy (kernels_radonusfft.cuh:73-78).
__device__ __forceinline__ void sample_pos(int k, float2 sc, const UsGeo &g, float &x0, float &y0, int &fx,
                                           int &fy) {
    const float q = __fdiv_rn((float)(k - g.n / 2), (float)g.n);
    x0 = __fmul_rn(q, sc.x);
    y0 = __fmul_rn(q, sc.y);
    if (x0 >= 0.5f) x0 = 0.5f - 1e-5f;
    if (y0 >= 0.5f) y0 = 0.5f - 1e-5f;
    fx = (int)floorf(__fmul_rn(g.tn, x0));
    fy = (int)floorf(__fmul_rn(g.tn, y0));
}

// Gaussian weight exp(-pi^2/mu d^2) of tap i of the 9 taps per axis
// (gather, kernels_radonusfft.cuh:116-118; pi/mu and 1/n are applied once).
__device__ __forceinline__ float tap_weight(int f, int i, float p0, const UsGeo &g) {
    const float d = (float)(f - kR + i) * g.inv2n - p0;
    return __expf(-g.wexp * d * d);
}

__device__ __forceinline__ void tap_weights(int f, float p0, const UsGeo &g, float (&e)[kTaps]) {
#pragma unroll
    for (int i = 0; i < kTaps; ++i) e[i] = tap_weight(f, i, p0, g);
}

// Adds samples (j, j + 1) of cell (KX, KY)'s sum X(k) to the zeroed Hermitian half
// planes of the C2R inverse (base: the slice's entry of its plane): the adjoint
// only needs Re IFFT2(X), the C2R of H(k) = (X(k) + conj X(-k)) / 2 on kx <= n,
// so X(k)/2 goes to H(k) and conj(X(k))/2 to H(-k) where they lie in the half
// plane (at most two adds per value, onto zeros: the sum does not depend on
// their order).  v is X / 2 with the pre-IFFT fftshift sign.  ONE: sample j alone.
// PLANAR: the half planes are the planar images cuFFT transforms (base: the
// first of the group's time samples; sample j + 1 is added where there is one).
template <bool ONE, bool PLANAR>
__device__ __forceinline__ void add_hermitian(float2 *__restrict__ base, const UsGeo &g, int KX, int KY, int j,
                                              const float4 &v, bool two) {
    const int P = g.P, half = P / 2;
    if (KY >= P || KX >= P) return;
    auto add = [&](int X, int Y, const float4 &a) {
        if constexpr (PLANAR) {
            const int pitch = planar_pitch(g.n);
            float2 *d = base + (long long)j * P * pitch + (long long)Y * pitch + X;
            atomicAdd(d, make_float2(a.x, a.y));
            if (!ONE && two) atomicAdd(d + (long long)P * pitch, make_float2(a.z, a.w));
            return;
        }
        float2 *d = base + ((long long)(Y + kVH) * g.vp + X + kVH) * 16 + j;
        if constexpr (ONE) atomicAdd(d, make_float2(a.x, a.y));
        else atomicAdd(reinterpret_cast<float4 *>(d), a);
    };
    if (KX <= half) add(KX, KY, v);
    if (KX >= half || KX == 0) add(KX ? P - KX : 0, KY ? P - KY : 0, make_float4(v.x, -v.y, v.z, -v.w));
}

// where the samples of slice z, group jgrp are added: its entries of its plane, or
// its first planar image
template <bool PLANAR>
__device__ __forceinline__ float2 *adj_base(float2 *spec, const UsGeo &g, int z, int jgrp) {
    if constexpr (PLANAR) return spec + ((long long)z * g.m + 16 * jgrp) * g.P * planar_pitch(g.n);
    else return spec + vec_plane_of(g, z, jgrp) * g.vplane + vec_entry(g, z);
}

}  // namespace rectv
