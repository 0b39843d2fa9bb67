// Inverse padded-grid FFT for grid sides that are no
// power of two (fft_general_fwd.cu): inverse columns of the Hermitian half
// planes, then rows, added into the volume.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>

#include "fft_general.cuh"

namespace rectv {

namespace {

// Threads per block.  Columns: 192 in three blocks per SM (four where a tile has eight
// values): the radix passes have P / R x C items, few more than the threads, and
// wider blocks left half of a last round idle (8 planes of 505 columns of 1008
// points 0.279 ms, 0.291 with 256, 0.332 with 352; 4 planes of 65 x 128 points 4.6
// us, 7.3 with 256).  Residual rows: 128 in six blocks (0.107 ms, 0.116 with 256 in three).
constexpr int kThr = 256, kColThr = 192, kResThr = 128;

template <int C>
__global__ void __launch_bounds__(kColThr, C == 8 ? 4 : 3)
    k_gen_cols_inv(float2 *__restrict__ spec, const __grid_constant__ GenPlan p, const float2 *__restrict__ tw, UsGeo g, int nlv, int ntiles) {
    gen::cols<C, 1>(spec, p, tw, g, nlv, ntiles);
}

// One row y of C value pairs of a plane: the Hermitian extension of the two
// half rows as one complex inverse transform A + i B, the centre outputs
// modulated, deapodised, scaled and added into u (YP: as the forward's).
template <int C, bool YP>
__global__ void __launch_bounds__(kThr, 3)
    k_gen_rows_inv(const float2 *__restrict__ spec, float *__restrict__ u, const float *__restrict__ dp, const __grid_constant__ GenPlan p,
                   const float2 *__restrict__ tw, UsGeo g, int zb, float cscale) {
    using gen::gen_sh;
    const int n = g.n, P = g.P;
    const int c = threadIdx.x % C, j0 = threadIdx.x / C;
    constexpr int js = kThr / C;
    constexpr int G = YP ? 16 / C : 8 / C;  // blocks per row (pair)
    const int y = (YP ? 2 : 1) * (blockIdx.x / G), y1 = YP ? min(y + 1, n - 1) : y, pl = blockIdx.y;
    const int v0 = (YP ? 1 : 2) * ((blockIdx.x % G) * C + c), v1 = YP ? v0 : v0 + 1;
    if (!vec_live(g, zb, pl, v0 - (YP ? 1 : 2) * c)) return;  // the block's values hold no data
    const float2 *row = spec + pl * g.vplane + ((long long)(y + n / 2 + kVH) * g.vp + kVH) * 16 + v0;
    auto load = [&](int k) {  // column k of the pair's two half rows
        if constexpr (YP) {
            const float2 a = __ldg(row + (long long)k * 16), b = __ldg(row + ((long long)(y1 - y) * g.vp + k) * 16);
            return make_float4(a.x, a.y, b.x, b.y);
        } else {
            return __ldg(reinterpret_cast<const float4 *>(row + (long long)k * 16));
        }
    };
    for (int kb = j0; kb <= n; kb += 4 * js) {  // four loads in flight
        float4 f[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = kb + i * js;
            if (k <= n) f[i] = load(k);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int k = kb + i * js;
            if (k > n) break;
            if (k == 0 || k == n) {
                f[i].y = f[i].w = 0.f;  // columns 0 and n of a real image's spectrum
            } else {
                gen_sh[(P - k) * C + c] = make_float2(f[i].x + f[i].w, f[i].z - f[i].y);
            }
            gen_sh[k * C + c] = make_float2(f[i].x - f[i].w, f[i].y + f[i].z);
        }
    }
    __syncthreads();
    const float2 *a = gen_sh + gen::passes<1, C>(0, P * C, 0, p, tw, c, j0, js) + c;
    const int za = vec_slice(g, pl, v0), ta = vec_time(g, pl, v0);
    const int zc = vec_slice(g, pl, v1), tb = vec_time(g, pl, v1);
    const bool oka = za < zb && ta < g.m, okb = zc < zb && tb < g.m && !(YP && y + 1 >= n);
    float *ua = u + (((long long)(oka ? za : 0) * g.m + (oka ? ta : 0)) * n + y) * n;
    float *ub = u + (((long long)(okb ? zc : 0) * g.m + (okb ? tb : 0)) * n + y1) * n;
    const float sy = (((y + n / 2) & 1) ? -dp[y] : dp[y]) * cscale;
    const float sy1 = YP ? (((y1 + n / 2) & 1) ? -dp[y1] : dp[y1]) * cscale : sy;
    for (int xb = j0; xb < n; xb += 4 * js) {
        float va[4], vb[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int x = xb + i * js;
            va[i] = oka && x < n ? ua[x] : 0.f;
            vb[i] = okb && x < n ? ub[x] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int x = xb + i * js;
            if (x >= n) break;
            const float d = ((x + n / 2) & 1) ? -__ldg(dp + x) : __ldg(dp + x);
            const float2 o = a[(x + n / 2) * C];
            if (oka) ua[x] = va[i] + o.x * (d * sy);
            if (okb) ub[x] = vb[i] + o.y * (d * sy1);
        }
    }
}

template <int C>
void run_inv(float2 *spec, float *u, int zb, float cscale, const float *deapod, const float2 *tw, const GenPlan &p,
             const UsGeo &g, cudaStream_t s) {
    const int n = g.n, npl = vec_planes(g, zb);
    const size_t smem = gen_cols_smem(g.P, C);
    const int nlv = vec_groups(g, zb, C);
    const long long ntiles = (long long)npl * (n + 1) * nlv;
    if (ntiles > 2147483647LL - 65536) throw Error(1, "pad FFT: too many column tiles");
    const int grid = (int)std::min<long long>(ntiles, gen_resident(smem, kColThr));
    k_gen_cols_inv<C><<<grid, kColThr, smem, s>>>(spec, p, tw, g, nlv, (int)ntiles);
    LAUNCH_CHECK("k_gen_cols_inv");
    if (g.tg == 1)
        k_gen_rows_inv<C, true><<<dim3((n + 1) / 2 * (16 / C), npl), kThr, gen_rows_smem(g.P, C), s>>>(spec, u, deapod, p,
                                                                                                 tw, g, zb, cscale);
    else
        k_gen_rows_inv<C, false><<<dim3(n * (8 / C), npl), kThr, gen_rows_smem(g.P, C), s>>>(spec, u, deapod, p, tw, g, zb,
                                                                                       cscale);
    LAUNCH_CHECK("k_gen_rows_inv");
}

// ---------------------------------------------------------------------------
// Residual rows of the inner step (k_resid_rows of fft_kernels.cu on the
// mixed-radix core): two rows are one complex transform, C pairs per block;
// blockIdx.y: runs of nrows rows (launch_resid_rows).
// HALF: the rows hold their Hermitian half (direction path), else the whole
// row, of which the Hermitian part counts.  FWD: the forward operator of the
// direction path, fout = tau R u (k_resid_rows).
// ---------------------------------------------------------------------------
template <int C, bool HALF, bool FWD>
__global__ void __launch_bounds__(kResThr, 6)
    k_gen_resid(const float2 *__restrict__ rows, const float *__restrict__ gdata, float2 *__restrict__ out,
                const __grid_constant__ GenPlan p, const float2 *__restrict__ tw, long long nrows, float scale,
                float *__restrict__ fout, float tau) {
    using gen::gen_sh;
    const int n = p.P, hn = n / 2 + 1;
    const int c = threadIdx.x % C, j0 = threadIdx.x / C;
    constexpr int js = kResThr / C;
    const long long ra = 2 * ((long long)blockIdx.x * C + c), rb = ra + 1;
    const bool oka = ra < nrows, okb = rb < nrows;
    const int rn = HALF ? hn : n;  // values per row
    rows += blockIdx.y * nrows * rn;
    if constexpr (FWD) {
        fout += blockIdx.y * nrows * n;
    } else {
        gdata += blockIdx.y * nrows * n;
        out += blockIdx.y * nrows * hn;
    }
    const float2 *ga = rows + (oka ? ra : 0) * rn, *gb = rows + (okb ? rb : 0) * rn;
    const float2 zero = make_float2(0.f, 0.f);
    auto load = [&](const float2 *r, int k) {
        const float2 v = __ldg(r + k);
        if (HALF) return v;
        const float2 w = __ldg(r + (k ? n - k : 0));
        return make_float2(0.5f * (v.x + w.x), 0.5f * (v.y - w.y));
    };
    for (int kb = j0; kb < hn; kb += 2 * js) {
        float2 a[2], b[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int k = kb + i * js;
            a[i] = oka && k < hn ? load(ga, k) : zero;
            b[i] = okb && k < hn ? load(gb, k) : zero;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int k = kb + i * js;
            if (k >= hn) break;
            if (2 * k == n) {
                a[i].y = b[i].y = 0.f;  // the transform's output is real: its Nyquist bin is too
            } else if (k > 0) {
                gen_sh[(n - k) * C + c] = make_float2(a[i].x + b[i].y, b[i].x - a[i].y);
            }
            gen_sh[k * C + c] = make_float2(a[i].x - b[i].y, a[i].y + b[i].x);
        }
    }
    __syncthreads();
    const int f = gen::passes<1, C>(0, n * C, 0, p, tw, c, j0, js);
    if constexpr (FWD) {
        for (int x = j0; x < n; x += js) {
            const float2 v = gen_sh[f + x * C + c];
            const float sc = (x & 1) ? scale : -scale;
            if (oka) fout[ra * n + x] = tau * (v.x * sc);
            if (okb) fout[rb * n + x] = tau * (v.y * sc);
        }
        return;
    }
    const float *da = gdata + (oka ? ra : 0) * n, *db = gdata + (okb ? rb : 0) * n;
    for (int sb = j0; sb < n; sb += 2 * js) {
        float va[2], vb[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int x = sb + i * js;
            va[i] = oka && x < n ? __ldg(da + x) : 0.f;
            vb[i] = okb && x < n ? __ldg(db + x) : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int x = sb + i * js;
            if (x >= n) break;
            const float2 v = gen_sh[f + x * C + c];
            const float sg = (x & 1) ? 1.f : -1.f;
            // as the separate passes: v = x (+-scale), r = v - g, w = (+-) r
            gen_sh[f + x * C + c] = make_float2(oka ? sg * (sg * (v.x * scale) - va[i]) : 0.f,
                                                okb ? sg * (sg * (v.y * scale) - vb[i]) : 0.f);
        }
    }
    __syncthreads();
    const float2 *z = gen_sh + gen::passes<-1, C>(f, n * C - f, 0, p, tw, c, j0, js) + c;
    for (int k = j0; k < hn; k += js) {
        const float2 zk = z[k * C], zm = z[(k ? n - k : 0) * C];
        if (oka) out[ra * hn + k] = make_float2(0.5f * (zk.x + zm.x), 0.5f * (zk.y - zm.y));
        if (okb) out[rb * hn + k] = make_float2(0.5f * (zk.y + zm.y), 0.5f * (zm.x - zk.x));
    }
}

}  // namespace

static void gen_resid_rows(const float2 *rows, const float *gdata, float2 *out, const float2 *tw, const GenPlan &p, int zb,
                           bool half, const UsGeo &g, float *fout, float tau, cudaStream_t s) {
    constexpr int C = 4;
    const int runs = resid_runs(zb, g.ntheta);
    const long long nrows = (long long)zb * g.ntheta / runs, nblk = (nrows + 2 * C - 1) / (2 * C);
    if (nblk > 2147483647LL) throw Error(1, "residual rows: too many rows");
    const float scale = (float)(1.0 / std::sqrt((double)g.n * (double)g.ntheta));
    const size_t smem = gen_rows_smem(g.n, C);
    const long long rn = half ? g.n / 2 + 1 : g.n;
    const auto kern = fout ? k_gen_resid<C, true, true> : half ? k_gen_resid<C, true, false> : k_gen_resid<C, false, false>;
    for (int y = 0; y < runs; y += 65535) {
        const long long r0 = y * nrows;
        const dim3 gr((unsigned)nblk, std::min(65535, runs - y));
        kern<<<gr, kResThr, smem, s>>>(rows + r0 * rn, fout ? nullptr : gdata + r0 * g.n,
                                       fout ? nullptr : out + r0 * (g.n / 2 + 1), p, tw, nrows, scale,
                                       fout ? fout + r0 * g.n : nullptr, tau);
        LAUNCH_CHECK("k_gen_resid");
    }
}

void launch_gen_resid(const float2 *rows, const float *gdata, float2 *out, const float2 *tw, const GenPlan &p, int zb,
                      bool half, const UsGeo &g, cudaStream_t s) {
    gen_resid_rows(rows, gdata, out, tw, p, zb, half, g, nullptr, 0.f, s);
}

void launch_gen_fwd_rows(const float2 *hrows, float *out, float tau, const float2 *tw, const GenPlan &p, int zb,
                         const UsGeo &g, cudaStream_t s) {
    gen_resid_rows(hrows, nullptr, nullptr, tw, p, zb, true, g, out, tau, s);
}

void gen_fft_inv_prepare() {
    constexpr int most = 227 * 1024;
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_resid<4, true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_resid<4, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_resid<4, true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_cols_inv<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_cols_inv<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_rows_inv<4, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_rows_inv<8, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_rows_inv<4, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
    CUDA_CHECK(cudaFuncSetAttribute(k_gen_rows_inv<8, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
}

void launch_gen_fft_inv_accum(float2 *spec, float *u, int zb, float tau, const float *deapod, const float2 *tw,
                              const GenPlan &p, const UsGeo &g, cudaStream_t s) {
    if (vec_planes(g, zb) > 65535) throw Error(1, "pad FFT: too many planes per batch");
    const double scale = 1.0 / std::sqrt((double)g.n * (double)g.ntheta);
    const float c = (float)(tau * scale / (4.0 * g.n * (double)g.n));
    if (gen_width(g.P) == 8)
        run_inv<8>(spec, u, zb, c, deapod, tw, p, g, s);
    else
        run_inv<4>(spec, u, zb, c, deapod, tw, p, g, s);
}

}  // namespace rectv
