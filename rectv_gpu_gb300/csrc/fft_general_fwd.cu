// Forward padded-grid FFT for grid sides 2n that are no
// power of two in [256, 2048] but a product of radices up to 19 (detector
// widths such as 480 and 504), in the vector layout: the passes of
// fft_kernels.cu (rows of value pairs as one complex transform, only the n
// non-zero rows; columns with the padding not read) on the mixed-radix core
// of fft_general.cuh.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "fft_general.cuh"

namespace rectv {

namespace {

// columns: as the inverse's (8 planes of 505 columns of 1008 points 0.327 ms, 0.341
// with 256 threads, 0.400 with 352; 4 planes of 65 x 128 points 5.2 us, 7.4 with 256)
constexpr int kThr = 256, kColThr = 192;

template <int C>
__global__ void __launch_bounds__(kColThr, C == 8 ? 4 : 3)
    k_gen_cols_fwd(float2 *__restrict__ spec, const __grid_constant__ GenPlan p, const float2 *__restrict__ tw, UsGeo g, int nlv, int ntiles) {
    gen::cols<C, -1>(spec, p, tw, g, nlv, ntiles);
}

// One row y of C value pairs of a plane: the pair's two real rows are one
// complex transform, split into the two half spectra (YP, one time sample per
// slice: the rows y and y + 1 of C values, so that slices stay apart).
template <int C, bool YP>
__global__ void __launch_bounds__(kThr, 3)
    k_gen_rows_fwd(const float *__restrict__ u, float2 *__restrict__ spec, const float *__restrict__ dp, const __grid_constant__ GenPlan p,
                   const float2 *__restrict__ tw, UsGeo g, int zb, float inv4n2) {
    using gen::gen_sh;
    const int n = g.n, P = g.P;
    const int X = 0, Y = P * C;
    const int c = threadIdx.x % C, j0 = threadIdx.x / C;
    constexpr int js = kThr / C;
    constexpr int G = YP ? 16 / C : 8 / C;  // blocks per row (pair)
    const int y = (YP ? 2 : 1) * (blockIdx.x / G), y1 = YP ? min(y + 1, n - 1) : y, pl = blockIdx.y;
    const int v0 = (YP ? 1 : 2) * ((blockIdx.x % G) * C + c), v1 = YP ? v0 : v0 + 1;
    if (!vec_live(g, zb, pl, v0 - (YP ? 1 : 2) * c)) return;  // the block's values hold no data
    const int za = vec_slice(g, pl, v0), ta = vec_time(g, pl, v0);
    const int zc = vec_slice(g, pl, v1), tb = vec_time(g, pl, v1);
    const bool oka = za < zb && ta < g.m, okb = zc < zb && tb < g.m && !(YP && y + 1 >= n);
    const float *ua = u + (((long long)(oka ? za : 0) * g.m + (oka ? ta : 0)) * n + y) * n;
    const float *ub = u + (((long long)(okb ? zc : 0) * g.m + (okb ? tb : 0)) * n + y1) * n;
    const float sy = (((y + n / 2) & 1) ? -dp[y] : dp[y]) * inv4n2;
    const float sy1 = YP ? (((y1 + n / 2) & 1) ? -dp[y1] : dp[y1]) * inv4n2 : sy;
    for (int xb = j0; xb < n; xb += 4 * js) {  // deapodised, times (-1)^(X+Y); eight loads in flight
        float va[4], vb[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int x = xb + i * js;
            va[i] = oka && x < n ? __ldg(ua + x) : 0.f;
            vb[i] = okb && x < n ? __ldg(ub + x) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int x = xb + i * js;
            if (x >= n) break;
            const float d = ((x + n / 2) & 1) ? -__ldg(dp + x) : __ldg(dp + x);
            gen_sh[Y + x * C + c] = make_float2(va[i] * (d * sy), vb[i] * (d * sy1));
        }
    }
    __syncthreads();
    gen::any_pass<-1, C, true>(Y, X, p, 0, tw, c, j0, js, n / 2, n);
    __syncthreads();
    const float2 *a = gen_sh + gen::passes<-1, C>(X, Y, 1, p, tw, c, j0, js) + c;
    if (!oka && !okb) return;
    float2 *row = spec + pl * g.vplane + ((long long)(y + n / 2 + kVH) * g.vp + kVH) * 16 + v0;
    for (int k = j0; k <= n; k += js) {
        const float2 zk = a[k * C], zm = a[(k ? P - k : 0) * C];
        const float4 o = make_float4(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y), 0.5f * (zk.y + zm.y),
                                     0.5f * (zm.x - zk.x));
        if constexpr (YP) {
            row[(long long)k * 16] = make_float2(o.x, o.y);
            if (okb) row[((long long)g.vp + k) * 16] = make_float2(o.z, o.w);
        } else {
            *reinterpret_cast<float4 *>(row + (long long)k * 16) = o;
        }
    }
}

template <int C>
void run_fwd(const float *u, float2 *spec, int zb, const float *deapod, const float2 *tw, const GenPlan &p,
             const UsGeo &g, cudaStream_t s) {
    const int n = g.n, npl = vec_planes(g, zb);
    const float inv4n2 = (float)(1.0 / (4.0 * n * (double)n));
    if (g.tg == 1)
        k_gen_rows_fwd<C, true><<<dim3((n + 1) / 2 * (16 / C), npl), kThr, gen_rows_smem(g.P, C), s>>>(u, spec, deapod, p,
                                                                                                 tw, g, zb, inv4n2);
    else
        k_gen_rows_fwd<C, false><<<dim3(n * (8 / C), npl), kThr, gen_rows_smem(g.P, C), s>>>(u, spec, deapod, p, tw, g, zb,
                                                                                       inv4n2);
    LAUNCH_CHECK("k_gen_rows_fwd");
    const size_t smem = gen_cols_smem(g.P, C);
    const int nlv = vec_groups(g, zb, C);
    const long long ntiles = (long long)npl * (n + 1) * nlv;
    if (ntiles > 2147483647LL - 65536) throw Error(1, "pad FFT: too many column tiles");
    const int grid = (int)std::min<long long>(ntiles, gen_resident(smem, kColThr));
    k_gen_cols_fwd<C><<<grid, kColThr, smem, s>>>(spec, p, tw, g, nlv, (int)ntiles);
    LAUNCH_CHECK("k_gen_cols_fwd");
}

}  // namespace

void gen_fft_fwd_prepare() {
    constexpr int most = 227 * 1024;
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_cols_fwd<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_cols_fwd<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_rows_fwd<4, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_rows_fwd<8, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_rows_fwd<4, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_rows_fwd<8, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
}

// Radices of P, at most six of 2 .. 13, 15, 16, 17, 19, as few as possible and then as
// even as possible; an odd one first where there is one (the first pass
// writes with the stride of its radix: odd strides are free of bank
// conflicts).  False when P has a larger prime factor or does not fit.
bool gen_fft_plan(int P, GenPlan *p) {
    static const int radix[] = {19, 17, 16, 15, 13, 12, 11, 10, 9, 8, 7, 6, 5, 4, 3, 2};
    if (P < 32 || P > 2048 || P % 2) return false;
    int best[6], nbest = 7, cur[6];
    long long cost = 0;
    // depth-first over non-increasing radices
    struct Rec {
        static void go(int rest, int from, int depth, int *cur, int *best, int &nbest, long long &cost) {
            if (rest == 1) {
                long long c = 0;
                for (int i = 0; i < depth; ++i) c += (long long)cur[i] * cur[i];
                if (depth < nbest || (depth == nbest && c < cost)) {
                    nbest = depth;
                    cost = c;
                    for (int i = 0; i < depth; ++i) best[i] = cur[i];
                }
                return;
            }
            if (depth == 6) return;
            for (int i = from; i < 16; ++i)
                if (rest % radix[i] == 0) {
                    cur[depth] = radix[i];
                    go(rest / radix[i], i, depth + 1, cur, best, nbest, cost);
                }
        }
    };
    Rec::go(P, 0, 0, cur, best, nbest, cost);
    if (nbest > 6) return false;
    std::stable_sort(best, best + nbest, [](int a, int b) { return (a % 2) > (b % 2); });
    if (best[0] % 2 == 0)  // no odd radix: the least power of two first
        std::stable_sort(best, best + nbest, [](int a, int b) { return (a & -a) < (b & -b); });
    p->P = P;
    p->np = nbest;
    int Ns = 1, off = 0;
    for (int i = 0; i < nbest; ++i) {
        p->R[i] = best[i];
        p->Ns[i] = Ns;
        p->magic[i] = Ns > 1 ? (uint32_t)((0x100000000ULL + Ns - 1) / Ns) : 0u;
        p->toff[i] = off;
        if (i > 0) off += (best[i] - 1) * Ns;  // the first pass has no twiddles
        Ns *= best[i];
    }
    return true;
}

std::vector<float2> gen_fft_twiddles(const GenPlan &p) {
    std::vector<float2> w;
    for (int i = 1; i < p.np; ++i)
        for (int r = 1; r < p.R[i]; ++r)
            for (int k = 0; k < p.Ns[i]; ++k) {
                const double a = -2.0 * 3.14159265358979323846 * r * k / ((double)p.Ns[i] * p.R[i]);
                w.push_back(make_float2((float)std::cos(a), (float)std::sin(a)));
            }
    return w;
}

size_t gen_rows_smem(int P, int C) { return (size_t)2 * P * C * sizeof(float2); }
size_t gen_cols_smem(int P, int C) { return (size_t)2 * P * C * sizeof(float2); }
// Eight values per tile (64-byte runs) while three blocks fit an SM, else four.
int gen_width(int P) { return gen_cols_smem(P, 8) <= 74 * 1024 ? 8 : 4; }
int gen_resident(size_t smem, int threads) {
    return sm_count() * std::max(1, std::min((int)((size_t)227 * 1024 / (smem + 1024)), 1024 / threads));
}

void launch_gen_fft_fwd(const float *u, float2 *spec, int zb, const float *deapod, const float2 *tw, const GenPlan &p,
                        const UsGeo &g, cudaStream_t s) {
    if (vec_planes(g, zb) > 65535) throw Error(1, "pad FFT: too many planes per batch");
    if (gen_width(g.P) == 8)
        run_fwd<8>(u, spec, zb, deapod, tw, p, g, s);
    else
        run_fwd<4>(u, spec, zb, deapod, tw, p, g, s);
}

}  // namespace rectv
