// Mixed-radix FFT passes in shared memory for transform lengths that are no
// power of two (fft_general_fwd.cu, fft_general_inv.cu): Stockham passes of
// radix 2 .. 16, 17 and 19, at most four for the lengths in use, C transforms interleaved
// (element i of transform c at i C + c).
#pragma once

#include <cuda_runtime.h>

#include "rectv_internal.cuh"

namespace rectv {
namespace gen {

__device__ __forceinline__ float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 mul(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// cos and sin of 2 pi e / n at compile time: the angle reduced to the first
// octant, then the Taylor series (to 1e-17 below pi/4)
constexpr double kPi = 3.14159265358979323846;
constexpr double taylor_cos(double x) {
    double t = 1.0, s = 1.0;
    for (int i = 1; i < 14; ++i) {
        t *= -x * x / ((2 * i - 1) * (2 * i));
        s += t;
    }
    return s;
}
constexpr double taylor_sin(double x) {
    double t = x, s = x;
    for (int i = 1; i < 14; ++i) {
        t *= -x * x / ((2 * i) * (2 * i + 1));
        s += t;
    }
    return s;
}
constexpr double cosq(int e, int n);
constexpr double sinq(int e, int n) {  // sin(2 pi e / n)
    e %= n;
    if (2 * e > n) return -sinq(n - e, n);
    if (4 * e > n) return 2 * e == n ? 0.0 : (4 * (n - 2 * e) == 2 * n ? 1.0 : sinq(n - 2 * e, 2 * n));
    if (8 * e > n) return taylor_cos(2 * kPi * (n - 4 * e) / (4.0 * n));
    return taylor_sin(2 * kPi * e / n);
}
constexpr double cosq(int e, int n) { return sinq(4 * (e % n) + n, 4 * n); }  // sin(x + pi/2)

// a exp(DIR 2 pi i E / N) for compile-time E, N
template <int E, int N, int DIR>
__device__ __forceinline__ float2 rot(float2 a) {
    constexpr int e = E % N;
    if constexpr (e == 0) {
        return a;
    } else if constexpr (2 * e == N) {
        return make_float2(-a.x, -a.y);
    } else if constexpr (4 * e == N) {
        return DIR < 0 ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
    } else if constexpr (4 * e == 3 * N) {
        return DIR < 0 ? make_float2(-a.y, a.x) : make_float2(a.y, -a.x);
    } else {
        constexpr float c = (float)cosq(e, N), s = (float)(DIR * sinq(e, N));
        return make_float2(a.x * c - a.y * s, a.x * s + a.y * c);
    }
}

template <int R, int DIR>
struct Dft;

// odd primes: pairs x_k +- x_(R-k), then X_m = x_0 + sum cos t_k +- i sum sin s_k
template <int R, int DIR>
struct DftPrime {
    template <int M, int K>
    __device__ static __forceinline__ void term(const float2 *t, const float2 *s, float2 &a, float2 &b) {
        if constexpr (K <= R / 2) {
            constexpr float c = (float)cosq(M * K, R), sn = (float)(DIR * sinq(M * K, R));
            a.x = fmaf(c, t[K].x, a.x);
            a.y = fmaf(c, t[K].y, a.y);
            b.x = fmaf(-sn, s[K].y, b.x);  // i sn s
            b.y = fmaf(sn, s[K].x, b.y);
            term<M, K + 1>(t, s, a, b);
        }
    }
    template <int M>
    __device__ static __forceinline__ void out(const float2 *t, const float2 *s, float2 x0, float2 *v) {
        if constexpr (M <= R / 2) {
            float2 a = x0, b = make_float2(0.f, 0.f);
            term<M, 1>(t, s, a, b);
            v[M] = add(a, b);
            v[R - M] = sub(a, b);
            out<M + 1>(t, s, x0, v);
        }
    }
    __device__ static __forceinline__ void run(float2 *v) {
        float2 t[R / 2 + 1], s[R / 2 + 1], x0 = v[0], sum = v[0];
#pragma unroll
        for (int k = 1; k <= R / 2; ++k) {
            t[k] = add(v[k], v[R - k]);
            s[k] = sub(v[k], v[R - k]);
            sum = add(sum, t[k]);
        }
        out<1>(t, s, x0, v);
        v[0] = sum;
    }
};

// R = A B: DFT_A over n1 of x[B n1 + n2], twiddle, DFT_B over n2; X[k1 + A k2]
template <int A, int B, int DIR>
struct DftComposite {
    template <int N2, int K1>
    __device__ static __forceinline__ void twiddle(float2 (*y)[A]) {
        if constexpr (N2 < B) {
            if constexpr (K1 < A) {
                y[N2][K1] = rot<N2 * K1, A * B, DIR>(y[N2][K1]);
                twiddle<N2, K1 + 1>(y);
            } else {
                twiddle<N2 + 1, 1>(y);
            }
        }
    }
    __device__ static __forceinline__ void run(float2 *v) {
        float2 y[B][A];
#pragma unroll
        for (int n2 = 0; n2 < B; ++n2) {
#pragma unroll
            for (int n1 = 0; n1 < A; ++n1) y[n2][n1] = v[B * n1 + n2];
            Dft<A, DIR>::run(y[n2]);
        }
        twiddle<1, 1>(y);
#pragma unroll
        for (int k1 = 0; k1 < A; ++k1) {
            float2 z[B];
#pragma unroll
            for (int n2 = 0; n2 < B; ++n2) z[n2] = y[n2][k1];
            Dft<B, DIR>::run(z);
#pragma unroll
            for (int k2 = 0; k2 < B; ++k2) v[k1 + A * k2] = z[k2];
        }
    }
};

template <int R, int DIR>
struct Dft : DftPrime<R, DIR> {};
template <int DIR>
struct Dft<2, DIR> {
    __device__ static __forceinline__ void run(float2 *v) {
        const float2 s = add(v[0], v[1]), d = sub(v[0], v[1]);
        v[0] = s;
        v[1] = d;
    }
};
template <int DIR>
struct Dft<4, DIR> {
    __device__ static __forceinline__ void run(float2 *v) {
        const float2 s0 = add(v[0], v[2]), d0 = sub(v[0], v[2]), s1 = add(v[1], v[3]), d1 = rot<1, 4, DIR>(sub(v[1], v[3]));
        v[0] = add(s0, s1);
        v[1] = add(d0, d1);
        v[2] = sub(s0, s1);
        v[3] = sub(d0, d1);
    }
};
template <int DIR>
struct Dft<6, DIR> : DftComposite<2, 3, DIR> {};
template <int DIR>
struct Dft<8, DIR> : DftComposite<2, 4, DIR> {};
template <int DIR>
struct Dft<9, DIR> : DftComposite<3, 3, DIR> {};
template <int DIR>
struct Dft<10, DIR> : DftComposite<2, 5, DIR> {};
template <int DIR>
struct Dft<12, DIR> : DftComposite<3, 4, DIR> {};
template <int DIR>
struct Dft<15, DIR> : DftComposite<3, 5, DIR> {};
template <int DIR>
struct Dft<16, DIR> : DftComposite<4, 4, DIR> {};

// The transforms' values; all passes address it by element offsets, so that
// every access is a shared-memory one.
extern __shared__ __align__(16) float2 gen_sh[];

// One Stockham pass from offset so to offset d0: items (c, j), j < P / R, read
// x[j + (P/R) r], twiddle by exp(DIR 2 pi i r (j mod Ns) / (Ns R)), DFT, write
// to (j / Ns) Ns R + j mod Ns + r Ns.  PART: only elements [off, off + cnt) of
// the source exist (stored from so on), the others are zero.
template <int R, int DIR, int C, bool PART>
__device__ __forceinline__ void pass(int so, int d0, const GenPlan &g, int p, const float2 *__restrict__ tw, int c,
                                     int j0, int jstep, int off, int cnt) {
    const int M = g.P / R, Ns = g.Ns[p], MC = M * C;
    const uint32_t magic = g.magic[p];
    for (int j = j0; j < M; j += jstep) {
        float2 v[R];
        int si = so + (PART ? j - off : j) * C + c, row = j - off;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            v[r] = !PART || (unsigned)row < (unsigned)cnt ? gen_sh[si] : make_float2(0.f, 0.f);
            si += MC;
            if (PART) row += M;
        }
        const int jq = Ns > 1 ? (int)__umulhi((uint32_t)j, magic) : j, k = j - jq * Ns;
        if (Ns > 1) {
            int ti = g.toff[p] + k;  // lanes: consecutive k
#pragma unroll
            for (int r = 1; r < R; ++r) {
                float2 w = __ldg(tw + ti);
                ti += Ns;
                if (DIR > 0) w.y = -w.y;
                v[r] = mul(v[r], w);
            }
        }
        Dft<R, DIR>::run(v);
        int di = d0 + (jq * Ns * R + k) * C + c;
#pragma unroll
        for (int r = 0; r < R; ++r) {
            gen_sh[di] = v[r];
            di += Ns * C;
        }
    }
}

template <int DIR, int C, bool PART>
__device__ __forceinline__ void any_pass(int so, int d0, const GenPlan &g, int p, const float2 *__restrict__ tw, int c,
                                         int j0, int jstep, int off, int cnt) {
    switch (g.R[p]) {
#define RECTV_PASS(R) \
    case R: pass<R, DIR, C, PART>(so, d0, g, p, tw, c, j0, jstep, off, cnt); break;
        RECTV_PASS(2)
        RECTV_PASS(3)
        RECTV_PASS(4)
        RECTV_PASS(5)
        RECTV_PASS(6)
        RECTV_PASS(7)
        RECTV_PASS(8)
        RECTV_PASS(9)
        RECTV_PASS(10)
        RECTV_PASS(11)
        RECTV_PASS(12)
        RECTV_PASS(13)
        RECTV_PASS(15)
        RECTV_PASS(16)
        RECTV_PASS(17)
        RECTV_PASS(19)
#undef RECTV_PASS
    }
}

// Passes first .. of the plan between the buffers at offsets a and b; the
// result's offset.  All threads of the block.
template <int DIR, int C>
__device__ __forceinline__ int passes(int a, int b, int first, const GenPlan &g, const float2 *__restrict__ tw, int c,
                                      int j0, int jstep) {
    for (int i = first; i < g.np; ++i) {
        any_pass<DIR, C, false>(a, b, g, i, tw, c, j0, jstep, 0, 0);
        __syncthreads();
        const int t = a;
        a = b;
        b = t;
    }
    return a;
}

// Column pass over the vector layout: persistent blocks take tiles of C
// values of one column's cells, copied (cp.async) into the second exchange
// buffer.  Forward: rows [n/2, 3n/2) in (the others are zero), all P rows out;
// inverse: P rows in, rows [n/2, 3n/2) out, in place.
template <int C, int DIR>
__device__ __forceinline__ void cols(float2 *__restrict__ spec, const GenPlan &p, const float2 *__restrict__ tw,
                                     const UsGeo &g, int nlv, int ntiles) {
    const int n = g.n, P = g.P, lrows = DIR < 0 ? n : P;
    const int in0 = DIR < 0 ? n / 2 : 0, out0 = DIR < 0 ? 0 : n / 2, orows = DIR < 0 ? P : n;
    const int X = 0, Y = P * C;  // two exchange buffers; the tile's rows land in the second
    const int tid = threadIdx.x, nthr = blockDim.x, c = tid % C, j0 = tid / C, js = nthr / C;
    constexpr int H = C / 2;  // 16-byte pieces of a row
    const int per_pl = (n + 1) * nlv;
    auto base = [&](int tile) {  // value 0 of row 0 of the tile's column
        const int pl = tile / per_pl, r = tile - pl * per_pl, kx = r / nlv, q = r - kx * nlv;
        return spec + pl * g.vplane + ((long long)kVH * g.vp + kVH + kx) * 16 + q * C;
    };
    const long long pitch = (long long)g.vp * 16;
    auto fetch = [&](int tile) {
        const float2 *b = base(tile) + in0 * pitch;
        for (int i = tid; i < lrows * H; i += nthr) {
            const int y = i / H, h = i % H;
            const unsigned sa = (unsigned)__cvta_generic_to_shared(gen_sh + Y + y * C + 2 * h);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(b + y * pitch + 2 * h) : "memory");
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        __syncthreads();  // the previous tile has left X and Y
        fetch(tile);
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        any_pass<DIR, C, (DIR < 0)>(Y, X, p, 0, tw, c, j0, js, in0, lrows);
        __syncthreads();
        const int a = passes<DIR, C>(X, Y, 1, p, tw, c, j0, js);
        float2 *o = base(tile) + out0 * pitch;
        for (int i = tid; i < orows * H; i += nthr) {
            const int y = i / H, h = i % H;
            *reinterpret_cast<float4 *>(o + y * pitch + 2 * h) = *reinterpret_cast<const float4 *>(gen_sh + a + (out0 + y) * C + 2 * h);
        }
    }
}

}  // namespace gen
}  // namespace rectv
