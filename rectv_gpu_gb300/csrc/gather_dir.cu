// Forward USFFT gather for scans that revisit their directions (direction
// path; the geometry and the first-order offset correction are described in
// scatter_dir.cu).
//
// Only the real part of the inverse row FFT is used (addreal,
// kernels_operators.cuh:75-84), so a ray needs the Hermitian half of its row
// alone:  H(k) = (row(k) + conj row(n - k)) / 2,  0 <= k <= n/2.  Samples k
// and n - k of a ray lie at p and -p, and the spectrum of a real image is
// Hermitian, so with S1_j = sum over the 9x9 stencil of p and S2_j = sum over
// the mirrored stencil of -p (cells fx - 3 .. fx + 5 against fx - 4 .. fx + 4
// of p, per axis; the same cells where the coordinate is an integer)
//     row(k)          ~ f(k) sum_j K'(theta, j) S1_j
//     conj row(n - k) ~ f(k) sum_j conj K'(theta, j) S2_j,
// both with the weights w(p, c) of p.  S2 differs from S1 in the stencils'
// edge rows and columns alone: S2 = S1 + C, so a position pair costs the 100
// cells of the joint 10x10 window instead of 2 x 81, only the half plane of
// the spectrum is read, and each ray stores n/2 + 1 values instead of n:
//     H(k) = f(k)/2 sum_j [ 2 Re K' (S1_j + delta S1perp_j) + conj K' C_j ]
// (an opposite ray takes the conjugate sum).  The offset correction of C is
// left out: its weights are 1.1e-5 of the stencil's peak, they change by 5.7 of
// themselves per cell, and delta is below 2e-3 cells, so the term is below 1.2e-7 of
// the peak, at the outermost samples (carried along, it left the operator's
// error at width 1024 at 2.73e-7, where the other roundings stood then).
//
// The spectra come in the vector layout (UsGeo): 16 (slice, time sample)
// values of a cell are 128 contiguous bytes, so the 25x25-cell footprint of a
// 16x16 tile of stencil origins is one TMA box and a quarter-warp reads one
// whole cell per tap without bank conflicts.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>

#include <algorithm>

#include "rectv_internal.cuh"
#include "tcgen05.cuh"
#include "usfft_common.cuh"

namespace rectv {

namespace {

constexpr int kT = 16;
constexpr int kGW = kT + 2 * kR + 1;  // footprint side: origins 0..15, taps -4 .. +5
constexpr int kGTap = kTaps + 1;      // 10 taps of a pair's joint window
constexpr int kGThr = 256;
constexpr int kGCap = 64;             // position pairs per item
// weights per pair, odd pitch (the four pairs of a warp on distinct banks):
constexpr int kWx = 0;       // [9] (-1)^b w_b of the x taps
constexpr int kWxd = 9;      // [9] their derivatives along x
constexpr int kE0 = 18;      // mirrored stencil minus direct one at columns 0 and 9
constexpr int kE9 = 19;
constexpr int kWy = 20;      // [9] (-1)^a w_a of the y taps times the origin's fftshift sign
constexpr int kWyd = 29;     // [9] their derivatives along y
constexpr int kEy0 = 38;     // mirrored minus direct at rows 0 and 9
constexpr int kEy9 = 39;
constexpr int kWy20 = 40;    // the mirrored stencil's weight of row 0
constexpr int kCos = 41;     // the direction's cos and -sin
constexpr int kSin = 42;
constexpr int kGPitch = 43;

struct GatherSmem {
    float4 fp[kGW * kGW * 8];     // footprint: 625 cells x 16 complex (TMA destination)
    float wt[kGCap][kGPitch];
    int org[kGCap];               // footprint cell of the joint window's first tap
    int pid[kGCap];               // d*(n/2) + q - 1, -1: none
    unsigned long long bar;
};
constexpr uint32_t kGBytes = kGW * kGW * 8 * sizeof(float4);

// The taps from the edges to the stencil's centre (tap 4): the weights fall by
// e^-11 to the edge, so that only the last three partial sums have the result's
// size and round at its unit (in order of position the last six have).
__host__ __device__ constexpr int col_order(int i) { return i & 1 ? 8 - i / 2 : i / 2; }                      // 0 8 1 7 2 6 3 5 4
__host__ __device__ constexpr int row_order(int i) { return i < 2 ? 9 * i : (i & 1 ? i / 2 : 9 - i / 2); }  // 0 9 8 1 7 ..

__device__ __forceinline__ float2 lo2(float4 f) { return make_float2(f.x, f.y); }
__device__ __forceinline__ float2 hi2(float4 f) { return make_float2(f.z, f.w); }
__device__ __forceinline__ float2 dup(float w) { return make_float2(w, w); }

}  // namespace

// ---------------------------------------------------------------------------
// One block (256 threads, two per SM) per (work item, planes); an item is at
// most 64 position pairs whose origins lie in one 16x16 tile.  Per plane the
// footprint lands by TMA while the other block of the SM computes; eight
// lanes per pair (two of the plane's 16 values each) sum the 100 cells and
// mix the pair's rays, eight per round: the lanes of a slice add their shares
// by recursive halving.
// Bound by the shared-memory wavefronts of the taps (100 per pair against
// 162 for separate stencils) and the footprint copies.  Measured at n = 1024,
// 360 directions x 8 rays, 16 time samples, 16 slices: 1.92 ms a launch; the
// kernel that gathered every position on its own (24x24 footprints of planar
// spectra through registers, whole rows) took 6.07 ms.  With 8 time samples
// (n = 504, 300 directions, 16 slices) 0.40 ms against 1.78 ms: two slices share
// a plane, where that kernel computed 8 empty samples.
// ---------------------------------------------------------------------------
template <int TG>
__global__ void __launch_bounds__(kGThr, 2)
    k_gather_dir(float2 *__restrict__ hrows, const __grid_constant__ CUtensorMap tmap,
                 const uint32_t *__restrict__ pos, const int4 *__restrict__ items, const float2 *__restrict__ dsincos,
                 const int *__restrict__ ray_start, const uint32_t *__restrict__ rays, const float *__restrict__ tau,
                 const float2 *__restrict__ dkmat, const float2 *__restrict__ shiftf, UsGeo g, int zb, int npz,
                 int per, int jgrp, int kstride, int *__restrict__ err) {
    extern __shared__ __align__(1024) unsigned char gd_smem[];
    GatherSmem &sm = *reinterpret_cast<GatherSmem *>(gd_smem);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int4 it = items[blockIdx.x];
    const int p0 = blockIdx.y * per, p1 = min(npz, p0 + per);
    const int tyi = it.x / g.NT, txi = it.x - tyi * g.NT;
    const int cnt = min(it.z, kGCap);
    const int nh = g.n / 2, hn = nh + 1;
    // footprint of plane group pz (plane pz jg + jgrp) into shared memory: one thread
    auto fetch = [&](int pz) {
        const uint32_t bar = tc::smem_addr(&sm.bar);
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(kGBytes) : "memory");
        asm volatile(
            "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, "
            "%5}], [%6];\n" ::"r"(tc::smem_addr(sm.fp)),
            "l"((unsigned long long)&tmap), "r"(0), "r"(txi * kT - kR + kVH), "r"(tyi * kT - kR + kVH),
            "r"(pz * g.jg + jgrp), "r"(bar)
            : "memory");
    };
    if (tid == 0) {
        tc::mbar_init(&sm.bar, 1);
        tc::fence_mbar_init();
        fetch(p0);
    }

    // ---- the item's position pairs (the same for every plane): thread = (pair, tap) ----
    const float c1 = 2.f * g.wexp / g.tn;  // d w / d position = c1 d w per grid cell
    for (int i = tid; i < cnt * 32; i += kGThr) {
        const int e = i >> 5, b = i & 15, ax = (i >> 4) & 1;
        const uint32_t id = __ldg(pos + it.y + e);
        const int d = id / (uint32_t)nh, q = id - d * nh + 1;
        const float2 sc = __ldg(dsincos + d);
        float x0, y0;
        int fx, fy;
        sample_pos(q, sc, g, x0, y0, fx, fy);
        const int lx0 = g.n + fx - txi * kT, ly0 = g.n + fy - tyi * kT;
        const bool ok = lx0 >= 0 && lx0 < kT && ly0 >= 0 && ly0 < kT;
        float *wt = sm.wt[e];
        if (b < kGTap) {
            const float p = ax ? y0 : x0;
            const int f = ax ? fy : fx;
            const float dd = (float)(f - kR + b) * g.inv2n - p;
            // (expf, not its fast form: with the sums' order the operator at width 1024 is 1.92e-7 off
            // its 64-bit value instead of 2.15e-7, at width 504 2.78e-7 instead of 3.24e-7)
            float w = expf(-g.wexp * dd * dd);
            if (b & 1) w = -w;
            if (ax && ((lx0 + ly0) & 1)) w = -w;  // fftshift sign of the stencil origin
            // the mirrored stencil starts one cell later, except at an integer coordinate
            const float v = __fmul_rn(g.tn, p);
            const bool mir = floorf(v) != v;
            if (b < kTaps) {
                wt[(ax ? kWy : kWx) + b] = w;
                wt[(ax ? kWyd : kWxd) + b] = c1 * dd * w;
                if (b == 0) {
                    wt[ax ? kEy0 : kE0] = mir ? -w : 0.f;
                    if (ax) wt[kWy20] = mir ? 0.f : w;
                }
            } else {
                wt[ax ? kEy9 : kE9] = mir ? w : 0.f;
            }
        } else if (b == 10 && ax == 0) {
            wt[kCos] = sc.y;
            wt[kSin] = -sc.x;
        } else if (b == 11 && ax == 0) {
            sm.pid[e] = ok ? (int)id : -1;
            sm.org[e] = ok ? ly0 * kGW + lx0 : 0;
            if (!ok) atomicAdd(err, 1);  // host/device bin disagreement
        }
    }
    __syncthreads();

    const int pi = lane >> 3, ci = lane & 7;  // pair of four, value pair of eight
    constexpr int L = TG >= 2 ? TG / 2 : 1;   // lanes per slice
    const int t0 = (2 * ci) & (TG - 1);       // time sample of this lane's first value
    const int j0 = 16 * jgrp + t0;
    bool ok = true;
    for (int pz = p0; pz < p1; ++pz) {
        ok = tc::mbar_wait(&sm.bar, (uint32_t)((pz - p0) & 1), ok) && ok;
        for (int e4 = 4 * wid; e4 < cnt; e4 += kGThr / 8) {
            const int e = min(e4 + pi, cnt - 1);
            const int id = (e4 + pi < cnt) ? sm.pid[e] : -1;
            const float4 *fq = sm.fp + sm.org[e] * 8 + ci;
            const float *wt = sm.wt[e];
            float wx[kTaps], wxd[kTaps];
#pragma unroll
            for (int b = 0; b < kTaps; ++b) {
                wx[b] = wt[kWx + b];
                wxd[b] = wt[kWxd + b];
            }
            const float ex0 = wt[kE0], ex9 = wt[kE9];
            // s: S1; dx, dy: the derivative sums; c: S2 - S1 (two values per lane)
            float2 s0 = dup(0.f), s1 = s0, dx0 = s0, dx1 = s0, dy0 = s0, dy1 = s0, c0 = s0, c1v = s0;
#pragma unroll
            for (int ia = 0; ia < kGTap; ++ia) {
                const int a = row_order(ia);
                float2 r0 = dup(0.f), r1 = r0, d0 = r0, d1 = r0;
                const float4 fa = fq[a * kGW * 8], fb = fq[(a * kGW + 9) * 8];
                float2 x0 = ffma2(dup(ex9), lo2(fb), make_float2(ex0 * fa.x, ex0 * fa.y));
                float2 x1 = ffma2(dup(ex9), hi2(fb), make_float2(ex0 * fa.z, ex0 * fa.w));
#pragma unroll
                for (int ib = 0; ib < kTaps; ++ib) {
                    const int b = col_order(ib);
                    const float4 f = b == 0 ? fa : fq[(a * kGW + b) * 8];
                    r0 = ffma2(dup(wx[b]), lo2(f), r0);
                    r1 = ffma2(dup(wx[b]), hi2(f), r1);
                    if (a < kTaps) {
                        d0 = ffma2(dup(wxd[b]), lo2(f), d0);
                        d1 = ffma2(dup(wxd[b]), hi2(f), d1);
                    }
                }
                if (a < kTaps) {
                    const float w = wt[kWy + a], wd = wt[kWyd + a];
                    s0 = ffma2(dup(w), r0, s0);
                    s1 = ffma2(dup(w), r1, s1);
                    dx0 = ffma2(dup(w), d0, dx0);
                    dx1 = ffma2(dup(w), d1, dx1);
                    dy0 = ffma2(dup(wd), r0, dy0);
                    dy1 = ffma2(dup(wd), r1, dy1);
                }
                if (a == 0 || a == 9) {
                    const float w = wt[a == 0 ? kEy0 : kEy9];
                    c0 = ffma2(dup(w), r0, c0);
                    c1v = ffma2(dup(w), r1, c1v);
                }
                const float w2 = wt[a == 0 ? kWy20 : (a == 9 ? kEy9 : kWy + a)];
                c0 = ffma2(dup(w2), x0, c0);
                c1v = ffma2(dup(w2), x1, c1v);
            }
            const float cs = wt[kCos], sn = wt[kSin];
            float2 q0 = make_float2(cs * dx0.x + sn * dy0.x, cs * dx0.y + sn * dy0.y);
            float2 q1 = make_float2(cs * dx1.x + sn * dy1.x, cs * dx1.y + sn * dy1.y);
            if (j0 >= g.m) s0 = q0 = c0 = dup(0.f);  // entries past the time samples hold no data
            if (TG > 1 && j0 + 1 >= g.m) s1 = q1 = c1v = dup(0.f);

            // ---- rays of the pair, eight per round ----
            int q = 0, rs = 0, nr = 0;
            if (id >= 0) {
                const int d = id / nh;
                q = id - d * nh + 1;
                rs = __ldg(ray_start + d);
                nr = __ldg(ray_start + d + 1) - rs;
            }
            const float qp = __fdiv_rn((float)(q - nh), (float)g.n);
            float cf = (q & 1) ? 0.5f * g.cw : -0.5f * g.cw;  // (-1)^(k+1) (pi/mu)/n / 2
            const float2 sh = __ldg(shiftf + q);
            const float2 fk = make_float2(sh.x * cf, sh.y * cf);
            auto put = [&](int ri, int z, float2 v) {  // ray ri of the pair, slice z
                if (ri >= nr || z >= zb) return;
                const uint32_t rv = __ldg(rays + rs + ri);
                if (rv >> 31) v.y = -v.y;
                float2 o = cmul(v, fk);
                float2 *dst = hrows + ((long long)z * g.ntheta + (rv & 0x7fffffffu)) * hn + q;
                if (jgrp > 0) {
                    const float2 p = *dst;
                    o.x += p.x;
                    o.y += p.y;
                } else if (q == 1) {
                    dst[-1] = dup(0.f);  // k = 0: zeroed by the reference (kernels_radonusfft.cuh:138-142)
                }
                *dst = o;
            };
            const int rounds = __reduce_max_sync(0xffffffffu, (nr + 7) >> 3);
            for (int rd = 0; rd < rounds; ++rd) {
                // lane ci fetches the offset of ray 8 rd + ci; the eight lanes share them by shuffles
                const float tv = (8 * rd + ci < nr) ? __ldg(tau + rs + 8 * rd + ci) : 0.f;
                float v[16], u[TG == 1 ? 16 : 1];
#pragma unroll
                for (int rr = 0; rr < 8; ++rr) {
                    const float dl = qp * __shfl_sync(0xffffffffu, tv, (lane & ~7) | rr);
                    float4 kv = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (8 * rd + rr < nr) {
                        const float2 *kr = dkmat + (long long)(rs + 8 * rd + rr) * kstride + j0;
                        if constexpr (TG == 1) {
                            const float2 k1 = __ldg(kr);
                            kv = make_float4(k1.x, k1.y, k1.x, k1.y);
                        } else {
                            kv = __ldg(reinterpret_cast<const float4 *>(kr));
                        }
                    }
                    // 2 Re K' (S1 + delta S1perp) + conj K' C = Re K' (2 (S1 + ..) + C) - i Im K' C
                    const float ax = fmaf(2.f, fmaf(dl, q0.x, s0.x), c0.x), ay = fmaf(2.f, fmaf(dl, q0.y, s0.y), c0.y);
                    const float bx = fmaf(2.f, fmaf(dl, q1.x, s1.x), c1v.x),
                                by = fmaf(2.f, fmaf(dl, q1.y, s1.y), c1v.y);
                    const float px = kv.x * ax + kv.y * c0.y, py = kv.x * ay - kv.y * c0.x;
                    const float rx = kv.z * bx + kv.w * c1v.y, ry = kv.z * by - kv.w * c1v.x;
                    if constexpr (TG == 1) {  // the two values are two slices
                        v[2 * rr] = px;
                        v[2 * rr + 1] = py;
                        u[2 * rr] = rx;
                        u[2 * rr + 1] = ry;
                    } else {
                        v[2 * rr] = px + rx;
                        v[2 * rr + 1] = py + ry;
                    }
                }
                // add over the L lanes of a slice: every step halves the rays a lane keeps
                int base = 8 * rd;
#pragma unroll
                for (int x = L / 2, h = 8; x >= 1; x >>= 1, h >>= 1) {
                    const bool up = ci & x;
#pragma unroll
                    for (int t = 0; t < h; ++t) {
                        const float send = up ? v[t] : v[h + t], keep = up ? v[h + t] : v[t];
                        v[t] = keep + __shfl_xor_sync(0xffffffffu, send, x);
                    }
                    base += up ? h / 2 : 0;
                }
                const int z = g.jg > 1 ? pz : pz * g.zs + (2 * ci) / TG;
#pragma unroll
                for (int i = 0; i < 8 / L; ++i) put(base + i, z, make_float2(v[2 * i], v[2 * i + 1]));
                if constexpr (TG == 1) {
#pragma unroll
                    for (int i = 0; i < 8; ++i) put(base + i, z + 1, make_float2(u[2 * i], u[2 * i + 1]));
                }
            }
        }
        __syncthreads();  // the footprint has been read
        if (tid == 0 && pz + 1 < p1) fetch(pz + 1);
    }
    if (!ok && lane == 0) atomicAdd(err, 1);
}

void make_vec_gather_map(CUtensorMap *map, float2 *spec, int npl, const UsGeo &g) {
    PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    cudaDriverEntryPointQueryResult q;
    CUDA_CHECK(cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", (void **)&encode, 12000, cudaEnableDefault,
                                                &q));
    if (q != cudaDriverEntryPointSuccess || !encode) throw Error(1, "cuTensorMapEncodeTiled unavailable");
    // float view: [planes][rows][cells][32]
    const cuuint64_t dims[4] = {32, (cuuint64_t)g.vp, (cuuint64_t)g.vrows, (cuuint64_t)npl};
    const cuuint64_t strides[3] = {128, 128ull * g.vp, 8ull * g.vplane};
    const cuuint32_t box[4] = {32, kGW, kGW, 1};
    const cuuint32_t es[4] = {1, 1, 1, 1};
    const CUresult r = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, spec, dims, strides, box, es,
                              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE,
                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) throw Error(1, "cuTensorMapEncodeTiled failed for the gather's footprints");
}

// ---------------------------------------------------------------------------
// Halo of the spectra in the vector layout: the ring of cells that stencils
// and footprints can reach (4 rows and columns before, 5 rows and `right`
// columns after the half plane) gets the periodic spectrum's values, through
// the Hermitian symmetry F(a, b) = conj F(-a, -b) outside the stored columns.
// One thread per 16 bytes (two values of a cell).
// ---------------------------------------------------------------------------
__global__ void k_vec_halo(float4 *__restrict__ spec, int right, UsGeo g) {
    constexpr int H0 = kR, H1 = kR + 1, HS = H0 + H1;
    const int P = g.P, n = g.n, side = H0 + right;
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int ci = (int)(i & 7);
    const long long e = i >> 3;
    const int wide = n + 1 + side;  // cells of a full halo row
    int y, x;
    if (e < (long long)HS * wide) {
        const int r = (int)(e / wide);
        x = (int)(e - (long long)r * wide) - H0;
        y = r < H0 ? r - H0 : P + r - H0;
    } else {
        const long long e2 = e - (long long)HS * wide;
        if (e2 >= (long long)P * side) return;
        y = (int)(e2 / side);
        const int c = (int)(e2 - (long long)y * side);
        x = c < H0 ? c - H0 : n + 1 + c - H0;
    }
    float4 *pl = spec + blockIdx.y * (g.vplane / 2);
    auto at = [&](int yy, int xx) { return pl + ((long long)(yy + kVH) * g.vp + xx + kVH) * 8 + ci; };
    const int a = (y % P + P) % P, b = (x % P + P) % P;
    float4 v;
    if (b <= n) {
        v = *at(a, b);
    } else {
        v = *at(a ? P - a : 0, P - b);
        v.y = -v.y;
        v.w = -v.w;
    }
    *at(y, x) = v;
}

void launch_vec_halo(float2 *spec, int npl, int right, const UsGeo &g, cudaStream_t s) {
    const int side = kR + right;
    const long long thr = 8 * ((long long)(2 * kR + 1) * (g.n + 1 + side) + (long long)g.P * side);
    if (npl > 65535) throw Error(1, "too many spectrum planes");
    k_vec_halo<<<dim3((unsigned)((thr + 255) / 256), npl), 256, 0, s>>>(reinterpret_cast<float4 *>(spec), right, g);
    LAUNCH_CHECK("k_vec_halo");
}

// ---------------------------------------------------------------------------
// Planar half planes [image][P][planar_pitch] (cuFFT's output for slices z0 .. z0 +
// nz - 1, image (z - z0) m + t) into the vector layout: one block per 128
// cells of a row, transposed through shared memory (eight loads of a thread in flight).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    k_planar_to_vec(const float2 *__restrict__ planar, float4 *__restrict__ spec, UsGeo g, int z0, int nz, int pl0) {
    __shared__ float2 sh[kLayoutCells][17];
    const int pl = pl0 + blockIdx.z, y = blockIdx.y, x0 = blockIdx.x * kLayoutCells;
    const int pitch = planar_pitch(g.n), lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const long long img = (long long)g.P * pitch;
    float2 f[2][kLayoutCells / 32];
#pragma unroll
    for (int h = 0; h < 2; ++h) {  // values w and w + 8
        const int v = w + 8 * h;
        const bool live = vec_live(g, z0 + nz, pl, v);
        const long long im = live ? (long long)(vec_slice(g, pl, v) - z0) * g.m + vec_time(g, pl, v) : 0;
        const float2 *src = planar + im * img + (long long)y * pitch + x0 + lane;
#pragma unroll
        for (int i = 0; i < kLayoutCells / 32; ++i)
            f[h][i] = live && x0 + lane + 32 * i <= g.n ? __ldg(src + 32 * i) : make_float2(0.f, 0.f);
    }
#pragma unroll
    for (int i = 0; i < kLayoutCells / 32; ++i) {
        sh[lane + 32 * i][w] = f[0][i];
        sh[lane + 32 * i][w + 8] = f[1][i];
    }
    __syncthreads();
    const int cell = threadIdx.x >> 3, ci = threadIdx.x & 7;
    float4 *dst = spec + pl * (g.vplane / 2) + ((long long)(y + kVH) * g.vp + kVH + x0 + cell) * 8 + ci;
    if (!vec_live(g, z0 + nz, pl, 2 * ci & ~3)) return;  // 32 bytes without data
#pragma unroll
    for (int i = 0; i < kLayoutCells / 32; ++i) {
        const float2 a = sh[cell + 32 * i][2 * ci], b = sh[cell + 32 * i][2 * ci + 1];
        if (x0 + cell + 32 * i <= g.n) dst[32 * 8 * i] = make_float4(a.x, a.y, b.x, b.y);
    }
}

void launch_planar_to_vec(const float2 *planar, float2 *spec, int z0, int nz, const UsGeo &g, cudaStream_t s) {
    const int pl0 = g.jg > 1 ? z0 * g.jg : z0 / g.zs, npl = vec_planes(g, nz);
    k_planar_to_vec<<<dim3(g.n / kLayoutCells + 1, g.P, npl), 256, 0, s>>>(planar, reinterpret_cast<float4 *>(spec), g, z0, nz,
                                                                    pl0);
    LAUNCH_CHECK("k_planar_to_vec");
}

template <int TG>
static void gather_dir_t(float2 *hrows, int zb, const GeoDev &gd, const UsGeo &g, const CUtensorMap &vmap,
                         cudaStream_t s) {
    const int npz = vec_planes(g, zb) / g.jg;
    // planes per block: all of them (the weights are built once) while there
    // are blocks for eight waves of two per SM, fewer for small problems
    const long long want = 16LL * sm_count();
    int per = (int)std::max<long long>(1, std::min<long long>(npz, (long long)gd.n_dfwd_items * npz / want));
    per = std::min(per, std::max(1, g.zper));
    const dim3 gs(gd.n_dfwd_items, (npz + per - 1) / per);
    const int kstride = g.jg > 1 ? 16 * g.jg : g.tg;
    for (int jg = 0; jg < g.jg; ++jg) {
        k_gather_dir<TG><<<gs, kGThr, sizeof(GatherSmem), s>>>(hrows, vmap, gd.dfwd_pos, gd.dfwd_items, gd.sincos,
                                                              gd.dray_start, gd.drays, gd.dtau, gd.dkmat, gd.shiftfwd,
                                                              g, zb, npz, per, jg, kstride, gd.err);
        LAUNCH_CHECK("k_gather_dir");
    }
}

int dir_fwd_capacity() { return kGCap; }

void gather_dir_prepare() {
    constexpr int bytes = (int)sizeof(GatherSmem);
    CUDA_CHECK(cudaFuncSetAttribute(k_gather_dir<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    CUDA_CHECK(cudaFuncSetAttribute(k_gather_dir<2>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    CUDA_CHECK(cudaFuncSetAttribute(k_gather_dir<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    CUDA_CHECK(cudaFuncSetAttribute(k_gather_dir<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
    CUDA_CHECK(cudaFuncSetAttribute(k_gather_dir<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
}

void launch_gather_dir(float2 *hrows, int zb, const GeoDev &gd, const UsGeo &g, const CUtensorMap &vmap,
                       cudaStream_t s) {
    if (gd.n_dfwd_items == 0) return;
    if (g.T != kT) throw Error(1, "tile size must be 16");
    switch (g.tg) {
        case 1: gather_dir_t<1>(hrows, zb, gd, g, vmap, s); break;
        case 2: gather_dir_t<2>(hrows, zb, gd, g, vmap, s); break;
        case 4: gather_dir_t<4>(hrows, zb, gd, g, vmap, s); break;
        case 8: gather_dir_t<8>(hrows, zb, gd, g, vmap, s); break;
        default: gather_dir_t<16>(hrows, zb, gd, g, vmap, s); break;
    }
}

}  // namespace rectv
