// Two-dimensional FFTs of the USFFT operators for P = 2n a power of two
// (256 <= P <= 2048), written for the zero padding of the reference's grids.
//
// The reference pads the deapodised n x n image into the centre of a P x P
// grid, modulates it by (-1)^(X+Y) and runs a P x P FFT (divphi, fftshift and
// the cuFFT 2D plan, radonusfft.cu:85-90, kernels_radonusfft.cuh:4-38); the
// adjoint runs the inverse FFT and crops the centre (radonusfft.cu:127-132).
// Three quarters of the forward input and of the adjoint output are padding,
// so the passes here touch only what is not:
//
//  forward  rows    the n rows of two images at a time: their deapodised real
//                   rows are one complex P-point FFT (a + i b, split after the
//                   transform), input read straight from the volume; writes
//                   the n+1 half-plane columns of rows [n/2, 3n/2)
//           columns n+1 columns of P points whose input rows outside
//                   [n/2, 3n/2) are zero (not read); writes all P rows
//  adjoint  columns n+1 inverse P-point FFTs of the Hermitian half planes;
//                   writes only rows [n/2, 3n/2) (in place)
//           rows    two images at a time: the Hermitian extension of their half
//                   rows as one complex inverse FFT (Re -> first, Im -> second),
//                   only the n centre outputs, deapodised and added into u
//
// The spectra are in the vector layout (UsGeo): the two images of a transform
// are neighbouring values of a cell.
//
// The same transform core also runs the n-point row transforms between the
// gather and the scatter (k_resid_rows: inverse row FFT, residual, fftshift
// and the adjoint's row R2C in one pass, n a power of two in [256, 1024]).
//
// Every transform is P = 16 x 16 x R3 points (R3 = P/256) computed by P/16
// threads holding 16 values each: a 16-point DFT in registers, twiddles,
// exchange through shared memory, a 16-point DFT, twiddles, exchange, and
// R3-point DFTs.  Twiddles come from a table evaluated in double precision on
// the host, laid out so that the lanes of a warp read consecutive entries:
// [k2][n1] = exp(-2 pi i n1 k2 / P) for stage 1, then [j2][m1] =
// exp(-2 pi i 16 m1 j2 / P) for stage 2.  Results equal cuFFT's to FP32
// rounding.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <string>
#include <vector>

#include "rectv_internal.cuh"
#include "tcgen05.cuh"

namespace rectv {

namespace {

__device__ __forceinline__ float2 operator+(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 operator-(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
__device__ __forceinline__ float2 cmul_(float2 a, float2 b) {
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// a * exp(DIR * i pi / 2): DIR = -1 (forward) multiplies by -i, DIR = +1 by +i
template <int DIR>
__device__ __forceinline__ float2 rot4(float2 a) {
    return DIR < 0 ? make_float2(a.y, -a.x) : make_float2(-a.y, a.x);
}

// a * exp(DIR * 2 pi i e / 16) for a compile-time e in [0, 16)
template <int E, int DIR>
__device__ __forceinline__ float2 tw16(float2 a) {
    constexpr int e = E & 15;
    constexpr float C1 = 0.92387953251128674f;  // cos(pi/8)
    constexpr float S1 = 0.38268343236508977f;  // sin(pi/8)
    constexpr float R2 = 0.70710678118654752f;  // cos(pi/4)
    constexpr float cs[16] = {1.f, C1, R2, S1, 0.f, -S1, -R2, -C1, -1.f, -C1, -R2, -S1, 0.f, S1, R2, C1};
    constexpr float sn[16] = {0.f, S1, R2, C1, 1.f, C1, R2, S1, 0.f, -S1, -R2, -C1, -1.f, -C1, -R2, -S1};
    if constexpr (e == 0) {
        return a;
    } else if constexpr (e == 4) {
        return rot4<DIR>(a);
    } else if constexpr (e == 8) {
        return make_float2(-a.x, -a.y);
    } else if constexpr (e == 12) {
        return rot4<-DIR>(a);
    } else {
        constexpr float c = cs[e], s = DIR * sn[e];
        return make_float2(a.x * c - a.y * s, a.x * s + a.y * c);
    }
}

template <int DIR>
__device__ __forceinline__ void dft2(float2 &x0, float2 &x1) {
    const float2 s = x0 + x1, d = x0 - x1;
    x0 = s;
    x1 = d;
}

template <int DIR>
__device__ __forceinline__ void dft4(float2 &x0, float2 &x1, float2 &x2, float2 &x3) {
    const float2 s02 = x0 + x2, d02 = x0 - x2, s13 = x1 + x3, d13 = rot4<DIR>(x1 - x3);
    x0 = s02 + s13;
    x2 = s02 - s13;
    x1 = d02 + d13;
    x3 = d02 - d13;
}

// in place, natural order in and out: v[k] = sum_r v[r] exp(DIR 2 pi i r k / 8)
template <int DIR>
__device__ __forceinline__ void dft8(float2 *v) {
    // r = 2a + b, k = c + 4d
    dft4<DIR>(v[0], v[2], v[4], v[6]);  // b = 0 -> y0[c] at v[0], v[2], v[4], v[6]
    dft4<DIR>(v[1], v[3], v[5], v[7]);  // b = 1
    v[3] = tw16<2, DIR>(v[3]);          // omega8^c = omega16^(2c)
    v[5] = tw16<4, DIR>(v[5]);
    v[7] = tw16<6, DIR>(v[7]);
    float2 o[8];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        o[c] = v[2 * c] + v[2 * c + 1];
        o[c + 4] = v[2 * c] - v[2 * c + 1];
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = o[i];
}

// in place, natural order in and out: v[k] = sum_r v[r] exp(DIR 2 pi i r k / 16)
template <int DIR>
__device__ __forceinline__ void dft16(float2 *v) {
    // r = 4a + b, k = c + 4d: DFT4 over a for each b, twiddle omega16^(bc), DFT4 over b
#pragma unroll
    for (int b = 0; b < 4; ++b) dft4<DIR>(v[b], v[4 + b], v[8 + b], v[12 + b]);  // y[b][c] at v[4c + b]
    v[4 * 1 + 1] = tw16<1, DIR>(v[5]);
    v[4 * 1 + 2] = tw16<2, DIR>(v[6]);
    v[4 * 1 + 3] = tw16<3, DIR>(v[7]);
    v[4 * 2 + 1] = tw16<2, DIR>(v[9]);
    v[4 * 2 + 2] = tw16<4, DIR>(v[10]);
    v[4 * 2 + 3] = tw16<6, DIR>(v[11]);
    v[4 * 3 + 1] = tw16<3, DIR>(v[13]);
    v[4 * 3 + 2] = tw16<6, DIR>(v[14]);
    v[4 * 3 + 3] = tw16<9, DIR>(v[15]);
#pragma unroll
    for (int c = 0; c < 4; ++c) dft4<DIR>(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);  // over b
    // V[c + 4d] sits at v[4c + d]: transpose the 4x4 index
    float2 o[16];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int d = 0; d < 4; ++d) o[c + 4 * d] = v[4 * c + d];
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = o[i];
}

template <int R, int DIR>
__device__ __forceinline__ void dftR(float2 *v) {
    if constexpr (R == 2) dft2<DIR>(v[0], v[1]);
    if constexpr (R == 4) dft4<DIR>(v[0], v[1], v[2], v[3]);
    if constexpr (R == 8) dft8<DIR>(v);
    if constexpr (R == 16) dft16<DIR>(v);
}

__device__ __forceinline__ float2 twiddle(const float2 *__restrict__ tw, int e, int dir) {
    const float2 w = __ldg(tw + e);
    return dir < 0 ? w : make_float2(w.x, -w.y);
}

// Shared-memory layouts of one transform's values at the two exchanges.
//  INTERLEAVED (column kernels, thread = c + C t): element i of transform c
//    at i*C + c; stage-2 output of pair p, m1 at p*Q + m1 (Q = R3+1 odd).
//  regions (row kernels, thread = t + (P/16) c): element i of transform c at
//    c*S + i; stage-2 output at p*R3 + ((m1 + p/(16/R3)) mod R3).
// Both make the exchanges free of bank conflicts for P >= 1024 (at P = 512
// one exchange of the column kernels keeps a two-way conflict).
template <int N, bool INTERLEAVED, int C>
struct FftLayout {
    static constexpr int N1 = N / 16;
    static constexpr int R3 = N / 256;
    static constexpr int P1 = N1 + R3;
    static constexpr int Q = INTERLEAVED ? (R3 == 1 ? 1 : R3 + 1) : R3;
    static constexpr int S1 = 16 * P1;
    static constexpr int S2 = 256 * Q;
    static constexpr int S = (S1 > S2 ? S1 : S2) > N ? (S1 > S2 ? S1 : S2) : N;  // elements per transform
    __device__ static __forceinline__ int a1(int c, int i) { return INTERLEAVED ? i * C + c : c * S + i; }
    __device__ static __forceinline__ int a2(int c, int p, int m1) {
        if constexpr (INTERLEAVED) {
            return (p * Q + m1) * C + c;
        } else {
            constexpr int G = (R3 >= 16) ? 1 : 16 / R3;
            return c * S + p * R3 + ((R3 == 1) ? 0 : ((m1 + p / G) & (R3 - 1)));
        }
    }
};

// One P-point FFT per transform c; thread t of the transform enters with
// v[r] = x[t + N1 r] (r < 16) and leaves with v[q R3 + j1] = X[t + N1 q +
// 256 j1] (q < 16/R3, j1 < R3).  All threads of the block must call it.
template <int N, int DIR, class L>
__device__ __forceinline__ void fft_core(float2 *v, float2 *sh, int c, int t, const float2 *__restrict__ tw) {
    constexpr int N1 = L::N1, R3 = L::R3;
    // stage 1: 16-point DFT over n2 of x[n1 + N1 n2], twiddle omega_N^(n1 k2)
    dft16<DIR>(v);
#pragma unroll
    for (int k2 = 1; k2 < 16; ++k2) v[k2] = cmul_(v[k2], twiddle(tw, k2 * N1 + t, DIR));
#pragma unroll
    for (int k2 = 0; k2 < 16; ++k2) sh[L::a1(c, k2 * L::P1 + t)] = v[k2];
    __syncthreads();
    // stage 2: thread (k2, m1), 16-point DFT over m2 of y[k2][m1 + R3 m2]
    const int k2 = t / R3, m1 = t - k2 * R3;
#pragma unroll
    for (int m2 = 0; m2 < 16; ++m2) v[m2] = sh[L::a1(c, k2 * L::P1 + m1 + R3 * m2)];
    __syncthreads();
    dft16<DIR>(v);
#pragma unroll
    for (int j2 = 1; j2 < 16; ++j2) v[j2] = cmul_(v[j2], twiddle(tw, N + j2 * R3 + m1, DIR));
#pragma unroll
    for (int j2 = 0; j2 < 16; ++j2) sh[L::a2(c, k2 + 16 * j2, m1)] = v[j2];
    __syncthreads();
    // stage 3: R3-point DFTs over m1 for the pairs p = t + N1 q
#pragma unroll
    for (int q = 0; q < 16 / R3; ++q)
#pragma unroll
        for (int i = 0; i < R3; ++i) v[q * R3 + i] = sh[L::a2(c, t + N1 * q, i)];
    if constexpr (R3 > 1) {
#pragma unroll
        for (int q = 0; q < 16 / R3; ++q) dftR<R3, DIR>(v + q * R3);
    }
}

constexpr int kRowThreads = 512;  // threads per block of the row kernels
// values per tile of the column passes (32- to 128-byte runs; 512 threads but for P = 256)
constexpr int vec_col_c(int N) { return N >= 2048 ? 4 : (N == 1024 ? 8 : 16); }

// ---------------------------------------------------------------------------
// Forward rows into the vector layout (UsGeo): one row y of the images of one
// plane.  The two images of a value pair (2p, 2p+1) are the real and imaginary
// part of one complex FFT, so that the split half spectra leave as 16-byte
// stores and the C pairs of a block as C x 16 contiguous bytes per cell
// (64-128 bytes).  Thread = (pair c, point t) with c fastest: C transforms
// interleaved in shared memory as in the column kernels, R rows per block.
// With one time sample per slice the two values would be two slices, and a NaN
// or the rounding of a bright slice would reach its neighbour: there (YP) a
// transform takes the rows y and y + 1 of one image, a block C images.
// ---------------------------------------------------------------------------
template <int N>
struct VecRows {
    static constexpr int N1 = N / 16;
    static constexpr int C = N1 * 8 <= kRowThreads ? 8 : 4;  // pairs per block
    static constexpr int R = kRowThreads / (N1 * C);         // rows per block
    using L = FftLayout<N, true, C>;
    static constexpr size_t SMEM = sizeof(float2) * (size_t)L::S * C * R;
    // real rows of the block's 2C images in shared memory, image c of the
    // pairs' first values, C + c of their second ones: 16-byte rows whose
    // pitch spreads the lanes (c, t) over the banks
    static constexpr int n = N / 2;
    static constexpr int RP = n + (C == 8 ? 4 : 8);
    static_assert(2 * C * RP <= 2 * L::S * C, "real rows fit the exchange buffer");
    static constexpr int PER = 2 * C * (n / 4) / (C * N1);  // float4 of the rows per thread (4)
    // the 16-byte piece i of this row's thread tr: image j, column x (a multiple of 4)
    __device__ static __forceinline__ void piece(int i, int tr, int &j, int &x) {
        const int e = i * (C * N1) + tr;
        j = e / (n / 4);
        x = 4 * (e - j * (n / 4));
    }
};

template <int N, bool YP>
__global__ void __launch_bounds__(kRowThreads, 2)
    k_fft_rows_fwd(const float *__restrict__ u, float2 *__restrict__ spec, const float *__restrict__ dp,
                       const float2 *__restrict__ tw, UsGeo g, int zb, float inv4n2) {
    using V = VecRows<N>;
    using L = typename V::L;
    constexpr int N1 = V::N1, C = V::C, R = V::R;
    extern __shared__ float2 fft_sh[];
    const int n = N / 2;
    const int c = threadIdx.x % C, t = (threadIdx.x / C) % N1, rr = threadIdx.x / (C * N1);
    constexpr int G = YP ? 16 / C : 8 / C;  // blocks per row (pair)
    const int ry = (blockIdx.x / G) * R + rr, pl = blockIdx.y;
    const int y = YP ? 2 * ry : ry, y1 = YP ? y + 1 : y;
    // the pair's values v0, v0 + 1 of the plane (YP: value v0, rows y and y + 1)
    const int v0 = (YP ? 1 : 2) * ((blockIdx.x % G) * C + c), v1 = YP ? v0 : v0 + 1;
    if (!vec_live(g, zb, pl, v0 - (YP ? 1 : 2) * c)) return;  // the block's values hold no data
    float2 *sh = fft_sh + rr * (L::S * C);
    const int za = vec_slice(g, pl, v0), ta = vec_time(g, pl, v0);
    const int zc = vec_slice(g, pl, v1), tb = vec_time(g, pl, v1);
    const bool oka = za < zb && ta < g.m, okb = zc < zb && tb < g.m;
    float2 v[16];
    {
        const float *ua = u + (((long long)(oka ? za : 0) * g.m + (oka ? ta : 0)) * n + y) * n;
        const float *ub = u + (((long long)(okb ? zc : 0) * g.m + (okb ? tb : 0)) * n + y1) * n;
        const float sy = (((y + n / 2) & 1) ? -dp[y] : dp[y]) * inv4n2;
        const float sy1 = YP ? (((y1 + n / 2) & 1) ? -dp[y1] : dp[y1]) * inv4n2 : sy;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            v[r] = make_float2(0.f, 0.f);
            if (r >= 4 && r < 12) {  // X = t + N1 r in [n/2, 3n/2)
                const int x = t + N1 * (r - 4), X = x + n / 2;
                const float d = (X & 1) ? -__ldg(dp + x) : __ldg(dp + x), w = d * sy;
                if (oka) v[r].x = __ldg(ua + x) * w;
                if (okb) v[r].y = __ldg(ub + x) * (YP ? d * sy1 : w);
            }
        }
    }
    fft_core<N, -1, L>(v, sh, c, t, tw);
    // Z in natural order, then A(k) = (Z(k) + conj Z(-k))/2, B(k) = (Z(k) - conj Z(-k))/(2i)
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16 / L::R3; ++q)
#pragma unroll
        for (int j1 = 0; j1 < L::R3; ++j1) sh[(t + N1 * q + 256 * j1) * C + c] = v[q * L::R3 + j1];
    __syncthreads();
    if (!oka && !okb) return;
    float2 *row = spec + pl * g.vplane + ((long long)(y + n / 2 + kVH) * g.vp + kVH) * 16 + v0;
    for (int k = t; k <= n; k += N1) {
        const float2 zk = sh[k * C + c], zm = sh[((N - k) & (N - 1)) * C + c];
        const float4 o = make_float4(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y), 0.5f * (zk.y + zm.y),
                                     0.5f * (zm.x - zk.x));
        if constexpr (YP) {
            row[(long long)k * 16] = make_float2(o.x, o.y);
            row[((long long)g.vp + k) * 16] = make_float2(o.z, o.w);
        } else {
            reinterpret_cast<float4 *>(row)[(long long)k * 8] = o;
        }
    }
}

// TMA tile copies of the column kernels: boxes of 4 columns (8 floats) x BR
// rows of one image, landing in shared memory as [row][column].
__device__ __forceinline__ void tma_load3(void *dst, const CUtensorMap *map, int x, int y, int z, void *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
        "[%5];\n" ::"r"(tc::smem_addr(dst)),
        "l"((unsigned long long)map), "r"(x), "r"(y), "r"(z), "r"(tc::smem_addr(bar))
        : "memory");
}
__device__ __forceinline__ void tma_store3(const CUtensorMap *map, int x, int y, int z, const void *src) {
    asm volatile("cp.async.bulk.tensor.3d.global.shared::cta.tile.bulk_group [%0, {%1, %2, %3}], [%4];\n" ::"l"(
                     (unsigned long long)map),
                 "r"(x), "r"(y), "r"(z), "r"(tc::smem_addr(src))
                 : "memory");
}
__device__ __forceinline__ void tma_store_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read 0;\n" ::: "memory");
}
__device__ __forceinline__ void mbar_expect(void *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(tc::smem_addr(bar)), "r"(bytes)
                 : "memory");
}


// ---------------------------------------------------------------------------
// Column passes.  Persistent blocks take tiles of C values of one column's
// cells (C x 8 contiguous bytes), round-robin, the values of a cell fastest so
// that the blocks in flight share the cells' 128-byte lines; the tile after
// the current one is loaded by TMA into the second landing buffer while the
// current one is transformed, and each output tile leaves by TMA stores from
// the exchange buffer, which the next tile reuses once those stores have read
// it.
//
// Forward: the row pass's output (rows [n/2, 3n/2); the others are zero and
// not read), P-point FFT, all P rows written back in place.
// Inverse: inverse P-point FFT of the columns of the Hermitian half planes;
// only rows [n/2, 3n/2) are written back.
// ---------------------------------------------------------------------------
template <int N, int C, int DIR>
struct ColPass {
    static constexpr int n = N / 2;
    static constexpr int BR = n < 256 ? n : 256;                  // rows per TMA box
    static constexpr int IN_ROWS = DIR < 0 ? n : N;               // rows loaded per tile
    static constexpr int OUT_ROWS = DIR < 0 ? N : n;              // rows stored per tile
    static constexpr int IN_Y0 = DIR < 0 ? kVH + n / 2 : kVH;     // first loaded row (window coordinates)
    static constexpr int OUT_Y0 = DIR < 0 ? kVH : kVH + n / 2;    // first stored row
    // first float of tile group gr of a plane, nlv groups of values per cell
    __device__ static __forceinline__ int x0(int gr, int nlv) {
        const int k = gr / nlv;
        return 32 * (kVH + k) + 2 * C * (gr - k * nlv);
    }
    using L = FftLayout<N, true, C>;
    static constexpr size_t EX = (size_t)L::S * C > (size_t)OUT_ROWS * C ? (size_t)L::S * C : (size_t)OUT_ROWS * C;
    static constexpr size_t LAND = (size_t)IN_ROWS * C;          // float2 per landing buffer
    static constexpr size_t SMEM = sizeof(float2) * (EX + 2 * LAND);
};

template <int N, int C, int DIR>
__global__ void __launch_bounds__(C *(N / 16), 1)
    k_fft_cols(const __grid_constant__ CUtensorMap tmap, const float2 *__restrict__ tw, int ngroups, int nlv,
               int ntiles, int *__restrict__ err) {
    using CP = ColPass<N, C, DIR>;
    using L = typename CP::L;
    constexpr int N1 = N / 16, n = N / 2, BR = CP::BR;
    extern __shared__ __align__(1024) float2 fft_sh[];
    float2 *ex = fft_sh;  // exchange buffer / output tile; landing buffers follow it
    __shared__ uint64_t bar[2];
    const int c = threadIdx.x % C, t = threadIdx.x / C;
    if (threadIdx.x == 0) {
        tc::mbar_init(&bar[0], 1);
        tc::mbar_init(&bar[1], 1);
        tc::fence_mbar_init();
    }
    __syncthreads();
    auto fetch = [&](int tile, int buf) {  // one thread
        const int x = CP::x0(tile % ngroups, nlv), img = tile / ngroups;
        mbar_expect(&bar[buf], (uint32_t)(CP::LAND * sizeof(float2)));
        for (int i = 0; i < CP::IN_ROWS / BR; ++i)
            tma_load3(fft_sh + CP::EX + buf * CP::LAND + i * BR * C, &tmap, x, CP::IN_Y0 + i * BR, img, &bar[buf]);
    };
    if (threadIdx.x == 0 && (int)blockIdx.x < ntiles) fetch(blockIdx.x, 0);
    bool ok = true;
    int it = 0;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, ++it) {
        const int buf = it & 1;
        // the other landing buffer was read in the previous iteration, before
        // at least one block barrier: it takes the next tile
        if (threadIdx.x == 0 && tile + (int)gridDim.x < ntiles) fetch(tile + gridDim.x, buf ^ 1);
        ok = tc::mbar_wait(&bar[buf], (uint32_t)((it >> 1) & 1), ok) && ok;
        float2 v[16];
        const float2 *in = fft_sh + CP::EX + buf * CP::LAND;
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            if constexpr (DIR < 0)
                v[r] = (r >= 4 && r < 12) ? in[(t + N1 * r - n / 2) * C + c] : make_float2(0.f, 0.f);
            else
                v[r] = in[(t + N1 * r) * C + c];
        }
        if (threadIdx.x == 0) tma_store_wait_read();  // the previous output tile has left the exchange buffer
        __syncthreads();
        fft_core<N, DIR, L>(v, ex, c, t, tw);
        __syncthreads();
#pragma unroll
        for (int q = 0; q < 16 / L::R3; ++q)
#pragma unroll
            for (int j1 = 0; j1 < L::R3; ++j1) {
                const int Y = t + N1 * q + 256 * j1;
                if constexpr (DIR < 0) {
                    ex[Y * C + c] = v[q * L::R3 + j1];
                } else {
                    if (Y >= n / 2 && Y < n / 2 + n) ex[(Y - n / 2) * C + c] = v[q * L::R3 + j1];
                }
            }
        tc::fence_proxy_async();
        __syncthreads();
        if (threadIdx.x == 0) {
            const int x = CP::x0(tile % ngroups, nlv), img = tile / ngroups;
            for (int i = 0; i < CP::OUT_ROWS / BR; ++i) tma_store3(&tmap, x, CP::OUT_Y0 + i * BR, img, ex + i * BR * C);
            asm volatile("cp.async.bulk.commit_group;\n" ::: "memory");
        }
    }
    if (threadIdx.x == 0) {
        asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory");  // the last tiles are written
        if (!ok) atomicAdd(err, 1);
    }
}

// ---------------------------------------------------------------------------
// Adjoint rows from the vector layout: the two images of a value pair are the
// real and imaginary part of one inverse FFT (as k_fft_rows_fwd); the
// centre outputs pass through shared memory once more so that the rows of u
// are read and written as whole lines.
// ---------------------------------------------------------------------------
template <int N, bool YP>
__global__ void __launch_bounds__(kRowThreads, 2)
    k_fft_rows_inv(const float2 *__restrict__ spec, float *__restrict__ u, const float *__restrict__ dp,
                       const float2 *__restrict__ tw, UsGeo g, int zb, float cscale) {
    using V = VecRows<N>;
    using L = typename V::L;
    constexpr int N1 = V::N1, C = V::C, R = V::R, n = N / 2;
    extern __shared__ float2 fft_sh[];
    const int c = threadIdx.x % C, t = (threadIdx.x / C) % N1, rr = threadIdx.x / (C * N1);
    constexpr int G = YP ? 16 / C : 8 / C;
    const int ry = (blockIdx.x / G) * R + rr, pl = blockIdx.y, y = YP ? 2 * ry : ry;
    const int vb = (YP ? 1 : 2) * (blockIdx.x % G) * C;  // the block's first value
    if (!vec_live(g, zb, pl, vb)) return;  // the block's values hold no data
    float2 *sh = fft_sh + rr * (L::S * C);
    const float2 *row = spec + pl * g.vplane + ((long long)(y + n / 2 + kVH) * g.vp + kVH) * 16 + vb + (YP ? 1 : 2) * c;
    auto load = [&](int k) {  // column k of the pair's two half rows
        if constexpr (YP) {
            const float2 a = row[(long long)k * 16], b = row[((long long)g.vp + k) * 16];
            return make_float4(a.x, a.y, b.x, b.y);
        } else {
            return *reinterpret_cast<const float4 *>(row + (long long)k * 16);
        }
    };
    // A + i B at k = t + N1 r: the stored half k <= n is read once; its mirror
    // image at N - k belongs to thread N1 - t and goes there through shared memory
    float2 v[16];
    {
        float4 f[9];
#pragma unroll
        for (int r = 0; r < 8; ++r) f[r] = load(t + N1 * r);
        f[8] = t == 0 ? load(n) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (t == 0) f[0].y = f[0].w = f[8].y = f[8].w = 0.f;  // columns 0 and n of a real image's spectrum
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            v[r] = make_float2(f[r].x - f[r].w, f[r].y + f[r].z);
            const int k = t + N1 * r;
            if (k > 0) sh[(N - k - n) * C + c] = make_float2(f[r].x + f[r].w, f[r].z - f[r].y);
        }
        if (t == 0) sh[c] = make_float2(f[8].x - f[8].w, f[8].y + f[8].z);
    }
    __syncthreads();
#pragma unroll
    for (int r = 8; r < 16; ++r) v[r] = sh[(t + N1 * r - n) * C + c];
    __syncthreads();
    fft_core<N, 1, L>(v, sh, c, t, tw);
    __syncthreads();
    float *rows = reinterpret_cast<float *>(sh);
#pragma unroll
    for (int q = 0; q < 16 / L::R3; ++q)
#pragma unroll
        for (int j1 = 0; j1 < L::R3; ++j1) {
            const int x = t + N1 * q + 256 * j1 - n / 2;
            if (x >= 0 && x < n) {
                rows[c * V::RP + x] = v[q * L::R3 + j1].x;
                rows[(C + c) * V::RP + x] = v[q * L::R3 + j1].y;
            }
        }
    const float sy = (((y + n / 2) & 1) ? -dp[y] : dp[y]) * cscale;
    const float sy1 = YP ? (((y + 1 + n / 2) & 1) ? -dp[y + 1] : dp[y + 1]) * cscale : sy;
    float4 *up[V::PER], f[V::PER];
    const int tr = threadIdx.x % (C * N1);
#pragma unroll
    for (int i = 0; i < V::PER; ++i) {  // the rows of u are on their way during the barrier
        int j, x;
        V::piece(i, tr, j, x);
        const int vj = YP ? vb + j % C : vb + 2 * (j % C) + j / C, yj = YP ? y + j / C : y;
        const int z = vec_slice(g, pl, vj), tt = vec_time(g, pl, vj);
        up[i] = z < zb && tt < g.m ? reinterpret_cast<float4 *>(u + (((long long)z * g.m + tt) * n + yj) * n + x) : nullptr;
        if (up[i]) f[i] = *up[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < V::PER; ++i) {
        if (!up[i]) continue;
        int j, x;
        V::piece(i, tr, j, x);
        const float4 o = *reinterpret_cast<const float4 *>(rows + j * V::RP + x);
        const float4 d = __ldg(reinterpret_cast<const float4 *>(dp + x));
        const float syj = YP && j >= C ? sy1 : sy;
        const float s0 = ((x + n / 2) & 1) ? -syj : syj;  // (-1)^X of column x; the next ones alternate
        f[i].x += o.x * d.x * s0;
        f[i].y -= o.y * d.y * s0;
        f[i].z += o.z * d.z * s0;
        f[i].w -= o.w * d.w * s0;
        *up[i] = f[i];
    }
}

template <int N>
size_t rows_smem() {
    return sizeof(float2) * (size_t)FftLayout<N, false, kRowThreads / (N / 16)>::S * (kRowThreads / (N / 16));
}

// ---------------------------------------------------------------------------
// Residual rows of the inner step, fused: for two gathered rows a, b (rows of
// n complex values, already multiplied by (-1)^(k+1) shift(k) (pi/mu)/n):
//   x = Re IFFT_n(row)                                  (radonusfft.cu:98-102)
//   r(s) = x(s) (-1)^(s+1) / sqrt(n ntheta) - g(s)      (residual, admm.cu:92)
//   w(s) = (-1)^(s+1) r(s)                              (fftshift of adjR, radonusfft.cu:115)
//   R = FFT_n(w), k = 0 .. n/2                          (the adjoint's row transform)
// Re IFFT(a) + i Re IFFT(b) is the inverse FFT of Ha + i Hb (H = Hermitian
// part), and FFT(wa + i wb) splits into the two half spectra, so a row pair
// costs one inverse and one forward n-point FFT; the residual never goes to
// memory.  Rows are the flattened (slice, angle) index, in runs of nrows
// (blockIdx.y); N = n.
// ---------------------------------------------------------------------------
// HALF: the rows hold H(k) itself, k = 0 .. n/2 (direction path).
// FWD: the forward operator of the direction path, fout = tau R u, without the
// residual and the second transform.  (A C2R transform of each row leaves all of
// its rounding in the real output, a pair's is shared by two rows: the operator at
// width 1024, 2880 angles, 16 samples is 2.15e-7 off its 64-bit value, 2.74e-7 with
// C2R, and 917 us instead of 939 at 3 slices.)
template <int N, bool HALF, bool FWD>
__global__ void __launch_bounds__(kRowThreads, 2)
    k_resid_rows(const float2 *__restrict__ rows, const float *__restrict__ gdata, float2 *__restrict__ out,
                 const float2 *__restrict__ tw, long long nrows, float scale, float *__restrict__ fout, float tau) {
    constexpr int N1 = N / 16, RP = kRowThreads / N1;
    using L = FftLayout<N, false, RP>;
    extern __shared__ float2 fft_sh[];
    const int t = threadIdx.x % N1, c = threadIdx.x / N1;
    const long long ra = 2 * ((long long)blockIdx.x * RP + c), rb = ra + 1;
    const bool oka = ra < nrows, okb = rb < nrows;
    constexpr int RN = HALF ? N / 2 + 1 : N;  // values per row
    rows += blockIdx.y * nrows * RN;
    if constexpr (FWD) {
        fout += blockIdx.y * nrows * N;
    } else {
        gdata += blockIdx.y * nrows * N;
        out += blockIdx.y * nrows * (N / 2 + 1);
    }
    const float2 *ga = rows + (oka ? ra : 0) * RN, *gb = rows + (okb ? rb : 0) * RN;
    float2 v[16];
#pragma unroll
    for (int r = 0; r < 16; ++r) {  // Ha + i Hb at k = t + N1 r
        const int k = t + N1 * r, km = (N - k) & (N - 1);
        float2 a = make_float2(0.f, 0.f), b = make_float2(0.f, 0.f);
        if constexpr (HALF) {
            const bool hi = k > N / 2;
            if (oka) a = __ldg(ga + (hi ? km : k));
            if (okb) b = __ldg(gb + (hi ? km : k));
            if (hi) {
                a.y = -a.y;
                b.y = -b.y;
            } else if (k == N / 2) {  // the transform's output is real: its Nyquist bin is too
                a.y = b.y = 0.f;
            }
            v[r] = make_float2(a.x - b.y, a.y + b.x);
            continue;
        }
        if (oka) {
            const float2 p = ga[k], q = ga[km];
            a = make_float2(0.5f * (p.x + q.x), 0.5f * (p.y - q.y));
        }
        if (okb) {
            const float2 p = gb[k], q = gb[km];
            b = make_float2(0.5f * (p.x + q.x), 0.5f * (p.y - q.y));
        }
        v[r] = make_float2(a.x - b.y, a.y + b.x);
    }
    fft_core<N, 1, L>(v, fft_sh, c, t, tw);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16 / L::R3; ++q)
#pragma unroll
        for (int j1 = 0; j1 < L::R3; ++j1) fft_sh[c * L::S + t + N1 * q + 256 * j1] = v[q * L::R3 + j1];
    __syncthreads();
    if constexpr (FWD) {
#pragma unroll
        for (int r = 0; r < 16; ++r) {
            const int sidx = t + N1 * r;
            const float2 x = fft_sh[c * L::S + sidx];
            const float sc = (sidx & 1) ? scale : -scale;
            if (oka) fout[ra * N + sidx] = tau * (x.x * sc);
            if (okb) fout[rb * N + sidx] = tau * (x.y * sc);
        }
        return;
    }
    const float *da = gdata + (oka ? ra : 0) * N, *db = gdata + (okb ? rb : 0) * N;
#pragma unroll
    for (int r = 0; r < 16; ++r) {
        const int sidx = t + N1 * r;
        const float2 x = fft_sh[c * L::S + sidx];
        const float sg = (sidx & 1) ? 1.f : -1.f;
        // as the separate passes: v = x (+-scale), r = v - g, w = (+-) r
        const float wa = oka ? sg * (sg * (x.x * scale) - da[sidx]) : 0.f;
        const float wb = okb ? sg * (sg * (x.y * scale) - db[sidx]) : 0.f;
        v[r] = make_float2(wa, wb);
    }
    __syncthreads();
    fft_core<N, -1, L>(v, fft_sh, c, t, tw);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16 / L::R3; ++q)
#pragma unroll
        for (int j1 = 0; j1 < L::R3; ++j1) fft_sh[c * L::S + t + N1 * q + 256 * j1] = v[q * L::R3 + j1];
    __syncthreads();
    constexpr int HN = N / 2 + 1;
    for (int k = t; k < HN; k += N1) {
        const float2 zk = fft_sh[c * L::S + k], zm = fft_sh[c * L::S + ((N - k) & (N - 1))];
        if (oka) out[ra * HN + k] = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
        if (okb) out[rb * HN + k] = make_float2(0.5f * (zk.y + zm.y), 0.5f * (zm.x - zk.x));
    }
}

template <int N, bool HALF, bool FWD>
void resid_n(const float2 *rows, const float *gdata, float2 *out, const float2 *tw, long long nrows, int runs,
             float scale, float *fout, float tau, cudaStream_t s) {
    constexpr int N1 = N / 16, RP = kRowThreads / N1;
    const long long npairs = (nrows + 1) / 2;
    const long long nblk = (npairs + RP - 1) / RP;
    if (nblk > 2147483647LL) throw Error(1, "residual rows: too many rows");
    for (int y = 0; y < runs; y += 65535) {
        const long long r0 = y * nrows;
        k_resid_rows<N, HALF, FWD><<<dim3((unsigned)nblk, std::min(65535, runs - y)), kRowThreads, rows_smem<N>(), s>>>(
            rows + r0 * (HALF ? N / 2 + 1 : N), FWD ? nullptr : gdata + r0 * N, FWD ? nullptr : out + r0 * (N / 2 + 1), tw,
            nrows, scale, FWD ? fout + r0 * N : nullptr, tau);
        LAUNCH_CHECK("k_resid_rows");
    }
}

template <int N>
void set_attrs_n() {
    constexpr auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    constexpr int C = vec_col_c(N);
    CUDA_CHECK(cudaFuncSetAttribute(k_resid_rows<N, false, false>, attr, (int)rows_smem<N>()));
    CUDA_CHECK(cudaFuncSetAttribute(k_resid_rows<N, true, false>, attr, (int)rows_smem<N>()));
    CUDA_CHECK(cudaFuncSetAttribute(k_resid_rows<N, true, true>, attr, (int)rows_smem<N>()));
    CUDA_CHECK(cudaFuncSetAttribute(k_fft_rows_fwd<N, false>, attr, (int)VecRows<N>::SMEM));
    CUDA_CHECK(cudaFuncSetAttribute(k_fft_rows_fwd<N, true>, attr, (int)VecRows<N>::SMEM));
    CUDA_CHECK(cudaFuncSetAttribute(k_fft_rows_inv<N, false>, attr, (int)VecRows<N>::SMEM));
    CUDA_CHECK(cudaFuncSetAttribute(k_fft_rows_inv<N, true>, attr, (int)VecRows<N>::SMEM));
    CUDA_CHECK(cudaFuncSetAttribute(k_fft_cols<N, C, -1>, attr, (int)ColPass<N, C, -1>::SMEM));
    CUDA_CHECK(cudaFuncSetAttribute(k_fft_cols<N, C, 1>, attr, (int)ColPass<N, C, 1>::SMEM));
}

template <int N, int DIR>
void launch_cols(const CUtensorMap &map, const float2 *tw, int zb, int *err, const UsGeo &g, cudaStream_t s) {
    constexpr int C = vec_col_c(N), thr = C * (N / 16);
    constexpr size_t smem = ColPass<N, C, DIR>::SMEM;
    const int nlv = vec_groups(g, zb, C), ngroups = (N / 2 + 1) * nlv;
    const long long ntiles = (long long)ngroups * vec_planes(g, zb);
    if (ntiles > 2147483647LL - 65536) throw Error(1, "pad FFT: too many column tiles");
    // persistent: as many blocks per SM as shared memory and 1024 threads allow
    const int per_sm = std::max(1, std::min((int)((size_t)227 * 1024 / (smem + 1024)), 1024 / thr));
    const int grid = (int)std::min<long long>(ntiles, (long long)per_sm * sm_count());
    k_fft_cols<N, C, DIR><<<grid, thr, smem, s>>>(map, tw, ngroups, nlv, (int)ntiles, err);
    LAUNCH_CHECK(DIR < 0 ? "k_fft_cols (forward)" : "k_fft_cols (inverse)");
}

template <int N>
void fwd_n(const float *u, float2 *spec, int zb, const float *deapod, const float2 *tw, const CUtensorMap &map,
           int *err, const UsGeo &g, cudaStream_t s) {
    using V = VecRows<N>;
    const int n = N / 2;
    const float inv4n2 = (float)(1.0 / (4.0 * n * (double)n));
    const dim3 gr(n / V::R * (8 / V::C), vec_planes(g, zb));
    (g.tg == 1 ? k_fft_rows_fwd<N, true> : k_fft_rows_fwd<N, false>)<<<gr, kRowThreads, V::SMEM, s>>>(u, spec, deapod, tw, g,
                                                                                               zb, inv4n2);
    LAUNCH_CHECK("k_fft_rows_fwd");
    launch_cols<N, -1>(map, tw, zb, err, g, s);
}

template <int N>
void inv_n(float2 *spec, float *u, int zb, float cscale, const float *deapod, const float2 *tw, const CUtensorMap &map,
           int *err, const UsGeo &g, cudaStream_t s) {
    using V = VecRows<N>;
    launch_cols<N, 1>(map, tw, zb, err, g, s);
    const dim3 gr(N / 2 / V::R * (8 / V::C), vec_planes(g, zb));
    (g.tg == 1 ? k_fft_rows_inv<N, true> : k_fft_rows_inv<N, false>)<<<gr, kRowThreads, V::SMEM, s>>>(spec, u, deapod, tw, g,
                                                                                               zb, cscale);
    LAUNCH_CHECK("k_fft_rows_inv");
}

PFN_cuTensorMapEncodeTiled_v12000 tmap_encoder() {
    static const PFN_cuTensorMapEncodeTiled_v12000 encode = [] {
        PFN_cuTensorMapEncodeTiled_v12000 e = nullptr;
        cudaDriverEntryPointQueryResult q;
        CUDA_CHECK(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", (void **)&e, 12000, cudaEnableDefault, &q));
        if (q != cudaDriverEntryPointSuccess || !e) throw Error(1, "cuTensorMapEncodeTiled unavailable");
        return e;
    }();
    return encode;
}

}  // namespace

int sm_count() {
    static const int nsm = [] {
        int dev = 0, v = 0;
        CUDA_CHECK(cudaGetDevice(&dev));
        CUDA_CHECK(cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev));
        return v;
    }();
    return nsm;
}

// P <= 2048: the column passes' two landing tiles and exchange buffer fit in
// shared memory up to that size
bool pad_fft_supported(int P) { return P >= 256 && P <= 2048 && (P & (P - 1)) == 0; }

void pad_fft_prepare() {
    set_attrs_n<256>();
    set_attrs_n<512>();
    set_attrs_n<1024>();
    set_attrs_n<2048>();
}

std::vector<float2> pad_fft_twiddles(int P) {
    const int N1 = P / 16, R3 = P / 256;
    std::vector<float2> w((size_t)P + 16 * R3);
    const double pi = 3.14159265358979323846;
    auto cis = [&](long long e) {
        const double a = -2.0 * pi * (double)(e % P) / (double)P;
        return make_float2((float)std::cos(a), (float)std::sin(a));
    };
    for (int k2 = 0; k2 < 16; ++k2)
        for (int t = 0; t < N1; ++t) w[(size_t)k2 * N1 + t] = cis((long long)t * k2);
    for (int j2 = 0; j2 < 16; ++j2)
        for (int m1 = 0; m1 < R3; ++m1) w[(size_t)P + j2 * R3 + m1] = cis(16LL * m1 * j2);
    return w;
}

// float view [planes][rows][32 cells], boxes of one tile's values x min(n, 256) rows
void make_vec_fft_map(CUtensorMap *map, float2 *spec, int npl, const UsGeo &g) {
    const cuuint64_t dims[3] = {(cuuint64_t)32 * g.vp, (cuuint64_t)g.vrows, (cuuint64_t)npl};
    const cuuint64_t strides[2] = {(cuuint64_t)128 * g.vp, (cuuint64_t)8 * g.vplane};
    const cuuint32_t box[3] = {(cuuint32_t)(2 * vec_col_c(g.P)), (cuuint32_t)(g.n < 256 ? g.n : 256), 1};
    const cuuint32_t es[3] = {1, 1, 1};
    const CUresult r = tmap_encoder()(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3, spec, dims, strides, box, es,
                                      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                                      CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw Error(1, "cuTensorMapEncodeTiled failed for the column FFT");
}

void launch_pad_fft_fwd(const float *u, float2 *spec, int zb, const float *deapod, const float2 *tw,
                        const CUtensorMap &map, int *err, const UsGeo &g, cudaStream_t s) {
    if (vec_planes(g, zb) > 65535) throw Error(1, "pad FFT: too many planes per batch");
    switch (g.P) {
        case 256: fwd_n<256>(u, spec, zb, deapod, tw, map, err, g, s); break;
        case 512: fwd_n<512>(u, spec, zb, deapod, tw, map, err, g, s); break;
        case 1024: fwd_n<1024>(u, spec, zb, deapod, tw, map, err, g, s); break;
        case 2048: fwd_n<2048>(u, spec, zb, deapod, tw, map, err, g, s); break;
        default: throw Error(1, "pad FFT: unsupported grid size");
    }
}

bool resid_rows_supported(int n) { return n >= 256 && n <= 1024 && (n & (n - 1)) == 0; }

// A pair of rows must not lie in two slices (a NaN or the rounding of a bright
// slice would reach the other): one run of all rows where a slice has an even
// number, else one run per slice, whose last row has no partner.
int resid_runs(int zb, int ntheta) { return ntheta % 2 == 0 ? 1 : zb; }

namespace {
template <int N>
void resid_any(const float2 *rows, const float *gdata, float2 *out, const float2 *tw, int zb, bool half, const UsGeo &g,
               float *fout, float tau, cudaStream_t s) {
    const int runs = resid_runs(zb, g.ntheta);
    const long long nrows = (long long)zb * g.ntheta / runs;
    const float scale = (float)(1.0 / std::sqrt((double)g.n * (double)g.ntheta));
    (fout ? resid_n<N, true, true> : half ? resid_n<N, true, false> : resid_n<N, false, false>)(rows, gdata, out, tw, nrows,
                                                                                         runs, scale, fout, tau, s);
}
void resid_switch(const float2 *rows, const float *gdata, float2 *out, const float2 *tw, int zb, bool half, const UsGeo &g,
                  float *fout, float tau, cudaStream_t s) {
    switch (g.n) {
        case 256: resid_any<256>(rows, gdata, out, tw, zb, half, g, fout, tau, s); break;
        case 512: resid_any<512>(rows, gdata, out, tw, zb, half, g, fout, tau, s); break;
        case 1024: resid_any<1024>(rows, gdata, out, tw, zb, half, g, fout, tau, s); break;
        default: throw Error(1, "residual rows: unsupported detector width");
    }
}
}  // namespace

// tw_n: the twiddle table of the n-point transforms, pad_fft_twiddles(n)
void launch_resid_rows(const float2 *rows, const float *gdata, float2 *out, const float2 *tw_n, int zb, bool half,
                       const UsGeo &g, cudaStream_t s) {
    resid_switch(rows, gdata, out, tw_n, zb, half, g, nullptr, 0.f, s);
}

void launch_fwd_rows(const float2 *hrows, float *out, float tau, const float2 *tw_n, int zb, const UsGeo &g,
                     cudaStream_t s) {
    resid_switch(hrows, nullptr, nullptr, tw_n, zb, true, g, out, tau, s);
}

void launch_pad_fft_inv_accum(float2 *spec, float *u, int zb, float tau, const float *deapod, const float2 *tw,
                              const CUtensorMap &map, int *err, const UsGeo &g, cudaStream_t s) {
    if (vec_planes(g, zb) > 65535) throw Error(1, "pad FFT: too many planes per batch");
    const double scale = 1.0 / std::sqrt((double)g.n * (double)g.ntheta);
    const float c = (float)(tau * scale / (4.0 * g.n * (double)g.n));
    switch (g.P) {
        case 256: inv_n<256>(spec, u, zb, c, deapod, tw, map, err, g, s); break;
        case 512: inv_n<512>(spec, u, zb, c, deapod, tw, map, err, g, s); break;
        case 1024: inv_n<1024>(spec, u, zb, c, deapod, tw, map, err, g, s); break;
        case 2048: inv_n<2048>(spec, u, zb, c, deapod, tw, map, err, g, s); break;
        default: throw Error(1, "pad FFT: unsupported grid size");
    }
}

}  // namespace rectv
