// USFFT for scans that revisit their directions: the formulation of both operators,
// and the adjoint scatter (the forward gather is gather_dir.cu).
//
// A scan over several half-turns sees every direction (theta modulo pi) more
// than once: rays theta, theta + pi, theta + 2 pi, ... sample the same points
// of the frequency plane (sample k of ray theta + pi is sample n - k of ray
// theta), and only their time weights K'(theta, j) differ.  The Gaussian
// interpolation (gather, kernels_radonusfft.cuh:81-144: 81 taps per sample)
// is linear and does not depend on a ray's time, so it is done once per
// position p = (direction d, 1 <= q < n) and time sample j, and the rays of
// the position are formed from it (the basis sums of operators.cu:143-152
// and 171-176 as the mixing K'):
//
//   forward:  S_j(p) = sum_taps w(p, c) F_j(c)
//             row(theta, k) = f(k) sum_j K'(theta, j) S_j(p)        (every ray theta of p)
//   adjoint:  E_j(p) = sum_{rays theta of p} conj K'(theta, j) f'(k) e(theta, k)
//             F_j(c) += sum_p w(p, c) E_j(p)
//
// with k = q for the rays of the representative's orientation and k = n - q
// for the opposite ones, f(k) = (-1)^(k+1) shiftfwd(k) (pi/mu)/n and f'(k) the
// same with shiftadj.
//
// The rays of a direction are grouped when their angles agree to the float32
// resolution of the input angles (2e-3 grid cells at the spectrum's edge);
// ray theta's own samples then lie delta = (q - n/2)/n tau_theta cells
// across the direction from the shared positions (DirPlan::tau).  Both
// kernels take that offset to first order: the forward interpolates S and
// its derivative across the direction, S_perp = sum_taps dw/dperp F, and ray
// theta reads S + delta S_perp; the adjoint scatters E and E_perp =
// sum_theta delta conj K' f' e with the weights w and dw/dperp.  The error
// left is O(delta^2) (the zeroth-order grouping alone errs by ~2e-4 relative
// at n = 1024 on white-noise spectra).
//
// At 2880 angles over 8 half-turns there are 360 directions: one eighth of
// the taps of the per-ray kernels, and the [ntheta x M] basis contraction
// becomes an 8-ray x 16-time-sample mix per position (FP32 on the CUDA
// cores: 16 complex products per ray sample, against 1296 for the taps of the
// per-ray formulation).
//
// Adjoint.  Only the real part of the inverse 2D FFT is used, i.e. the C2R of
// the Hermitian part H(k) = (X(k) + conj X(-k)) / 2 of the scattered grid X on
// the half plane.  Rows are spectra of real rows, so e(theta, n - k) =
// conj e(theta, k): the pair of positions p (sample q, 1 <= q <= n/2) and -p
// adds to H around p
//     w(p, c) [c in the stencil of p] (M0 - M2) + w(p, c) [c in the mirrored stencil of -p] M2,
//     M0_j = sum_theta Re K'(theta, j) v,   M2_j = 1/2 sum_theta K'(theta, j) v,
//     v = f'(k) e(theta, k) at k = q (conjugated for the opposite rays)
// (and its mirror image around -p, outside the half plane but for a border).
// The two stencils share 8 x 8 cells, where this is w M0; so
//     H(c) += wx1 (wy1 M0 + (wy2 - wy1) M2) + (wx2 - wx1) wy2 M2
// with the axis weights w1 on the stencil of p and w2 on the mirrored one, and
// to first order in the rays' offsets wx1 wy1' + wx1' wy1 times M0perp =
// sum_theta delta Re K' v (left out on the edges' M2 terms: below 1e-8 of M0).
// Against a scatter of every position this halves the entries, and every cell
// of the half plane belongs to one block, which stores it once: no atomics
// and no clearing.
#include <cuda_runtime.h>

#include <algorithm>

#include "rectv_internal.cuh"
#include "tcgen05.cuh"
#include "usfft_common.cuh"

namespace rectv {

namespace {

constexpr int kT = 16;
constexpr int kVec = 24;      // float4 per position pair: M0, M0perp, M2 of 16 values

// ---- mixing ----
constexpr int kMThr = 256;    // 32 position pairs x 8 lanes
constexpr int kMFly = 8;      // rays in flight per thread

// ---- scatter ----
constexpr int kSWarps = 8;               // consumer warps; one more warp issues the copies
constexpr int kSThr = 32 * (kSWarps + 1);
constexpr int kSChunk = 32;              // entries per stage
constexpr int kSStages = 4;
constexpr int kSCap = 192;               // entries whose weights are held

struct ScatSmem {
    float4 m[kSStages][kSChunk][kVec];   // the entries' M0, M0perp, M2 (bulk copies)
    float wx[kSCap][kT], wxd[kSCap][kT]; // wx1 and its first-order weight over the tile's columns
    float2 wy[kSCap][kT];                // (y weight of the joint 10 taps, first-order weight) over the rows
    float4 hd[kSCap];                    // first column and row of the joint window (int bits), wx2 - wx1 at its columns 0, 9
    uint32_t id[kSCap];
    uint32_t mask[kSCap / kSChunk][kSWarps];  // entries of a chunk whose window touches a warp's cells
    unsigned long long full[kSStages], empty[kSStages];
};

__device__ __forceinline__ float2 lo2(float4 f) { return make_float2(f.x, f.y); }
__device__ __forceinline__ float2 hi2(float4 f) { return make_float2(f.z, f.w); }
__device__ __forceinline__ float2 dup(float w) { return make_float2(w, w); }
__device__ __forceinline__ float2 mul2(float w, float2 a) { return make_float2(w * a.x, w * a.y); }

}  // namespace

// ---------------------------------------------------------------------------
// Adjoint, step 1: M0, M0perp, M2 of every position pair and plane.  Eight
// lanes per pair, two of the plane's 16 values each: a pair's 384 bytes leave
// as three full 128-byte lines.  The row values of eight rays are in flight
// per thread.  Out: emix[((pl ndir + d) n/2 + q - 1)][3][8] float4.
// Writes 1.13 GB at n = 1024, 360 directions, 16 slices: 0.92 ms a launch
// (1.46 ms for the kernel that mixed every position and cleared the half
// planes): bound by the latency of the ray -> row load chain.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kMThr)
    k_adj_mix(float4 *__restrict__ emix, const float2 *__restrict__ rowsc, const int *__restrict__ ray_start,
              const uint32_t *__restrict__ rays, const float *__restrict__ tau, const float2 *__restrict__ dkmat,
              const float2 *__restrict__ shifta, UsGeo g, int zb, int ndir, int jgrp, int kstride) {
    const int nh = g.n / 2, hn = nh + 1;
    const int ci = threadIdx.x & 7;
    const int q = 1 + blockIdx.x * (kMThr / 8) + (threadIdx.x >> 3), d = blockIdx.y, pz = blockIdx.z;
    if (q > nh) return;
    const int z0 = g.jg > 1 ? pz : pz * g.zs + (2 * ci) / g.tg;
    const int z1 = g.jg > 1 ? pz : pz * g.zs + (2 * ci + 1) / g.tg;
    const bool two = z1 != z0;  // one time sample: the two values are two slices
    const int j0 = 16 * jgrp + ((2 * ci) & (g.tg - 1));
    const int rs = __ldg(ray_start + d), nr = __ldg(ray_start + d + 1) - rs;
    const float qp = __fdiv_rn((float)(q - nh), (float)g.n);
    const float2 sh = __ldg(shifta + q);
    const float cf = ((q & 1) ? g.cw : -g.cw) * (q == nh ? 0.5f : 1.f);  // the pair q = n/2 is one position
    const float2 fk = make_float2(sh.x * cf, sh.y * cf);
    float2 a0 = dup(0.f), a1 = a0, p0 = a0, p1 = a0, i0 = a0, i1 = a0;  // sum h v, sum delta h v, sum g v (K' = h + i g)
    for (int r0 = 0; r0 < nr; r0 += kMFly) {
        float2 R0[kMFly], R1[kMFly];
#pragma unroll
        for (int i = 0; i < kMFly; ++i) {
            R0[i] = R1[i] = dup(0.f);
            if (r0 + i < nr) {
                const uint32_t rv = __ldg(rays + rs + r0 + i);
                const long long th = rv & 0x7fffffffu;
                if (z0 < zb) R0[i] = __ldg(rowsc + ((long long)z0 * g.ntheta + th) * hn + q);
                if (two && z1 < zb) R1[i] = __ldg(rowsc + ((long long)z1 * g.ntheta + th) * hn + q);
            }
        }
#pragma unroll
        for (int i = 0; i < kMFly; ++i) {
            if (r0 + i >= nr) break;
            const int r = rs + r0 + i;
            const uint32_t rv = __ldg(rays + r);
            const float dl = qp * __ldg(tau + r);  // this ray's offset across the direction
            float4 k;
            if (g.tg == 1) {
                const float2 k1 = __ldg(dkmat + (long long)r * kstride + j0);
                k = make_float4(k1.x, k1.y, k1.x, k1.y);
            } else {
                k = __ldg(reinterpret_cast<const float4 *>(dkmat + (long long)r * kstride + j0));
            }
            float2 v = cmul(R0[i], fk), w = two ? cmul(R1[i], fk) : v;
            if (rv >> 31) {
                v.y = -v.y;
                w.y = -w.y;
            }
            const float2 hv = mul2(k.x, v), hw = mul2(k.z, w);
            a0.x += hv.x;
            a0.y += hv.y;
            a1.x += hw.x;
            a1.y += hw.y;
            p0 = ffma2(dup(dl), hv, p0);
            p1 = ffma2(dup(dl), hw, p1);
            i0 = ffma2(dup(k.y), v, i0);
            i1 = ffma2(dup(k.w), w, i1);
        }
    }
    float4 *o = emix + (((long long)pz * ndir + d) * nh + q - 1) * kVec + ci;
    o[0] = make_float4(a0.x, a0.y, a1.x, a1.y);
    o[8] = make_float4(p0.x, p0.y, p1.x, p1.y);
    o[16] = make_float4(0.5f * (a0.x - i0.y), 0.5f * (a0.y + i0.x), 0.5f * (a1.x - i1.y), 0.5f * (a1.y + i1.x));
}

// ---------------------------------------------------------------------------
// Adjoint, step 2: one block (eight consumer warps and a copy warp, two
// blocks per SM) per (16x16 tile of the window, planes), the most work
// first.  The entries of a tile are the position pairs whose joint 10x10
// window touches it; their weights over the tile's columns and rows are
// computed once per block (per plane in the few tiles of more than 192
// entries).  Per plane the copy warp streams the entries' M0, M0perp, M2 (one
// 384-byte bulk copy each) through four stages of 32 entries; a warp owns 4
// rows x 8 columns of the tile and walks the entries that touch them, its
// lane (row, ci) two of the 16 values of the row's 8 cells:
//     U = wy1 M0 + wy1' M0perp + (wy2 - wy1) M2,  V = wy1 M0perp,
//     cell += wx1 U + wx1' V,  and wy2 M2 (wx2 - wx1) at the window's edge columns.
// So an entry costs a lane 3 16-byte loads of M for 8 cells.  Warps wait for
// copies only, never for each other.  All sums run in entry order; the cells
// leave as full 128-byte lines.  Measured at n = 1024, 360 directions, 16 time
// samples, 16 slices: 3.7 ms a launch, against 6.4 ms for a scatter of every
// position with float2 atomics into cleared half planes.  Bound by the latency
// of the shared loads and FMA chains (issue 54 % active, FMA pipe 42 %).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kSThr, 2)
    k_scatter_dir(const float4 *__restrict__ emix, float4 *__restrict__ spec, const uint32_t *__restrict__ pos,
                  const int4 *__restrict__ items, const float2 *__restrict__ dsincos, UsGeo g, int ndir, int jgrp,
                  int *__restrict__ err) {
    extern __shared__ __align__(128) unsigned char sd_smem[];
    ScatSmem &sm = *reinterpret_cast<ScatSmem *>(sd_smem);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int4 it = items[blockIdx.x];
    const int ntx = (g.vp + kT - 1) / kT;
    const int ty = it.x / ntx, Y0 = ty * kT, X0 = (it.x - ty * ntx) * kT;  // window cell (0, 0) of the tile
    const int p0 = it.w & 0xffff, p1 = it.w >> 16;
    const int nh = g.n / 2, nseg = (it.z + kSCap - 1) / kSCap;
    const long long rowp = (long long)g.vp * 8, plane = (long long)g.vrows * rowp;  // float4
    if (it.z == 0) {  // no entry: zeros
        for (int pz = p0; pz < p1; ++pz) {
            float4 *dst = spec + (long long)(pz * g.jg + jgrp) * plane;
            for (int i = tid; i < kT * kT * 8; i += kSThr) {
                const int Y = Y0 + (i >> 7), X = X0 + ((i >> 3) & (kT - 1));
                if (Y < g.vrows && X < g.vp) dst[Y * rowp + (long long)X * 8 + (i & 7)] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        return;
    }
    if (tid == 0) {
        for (int i = 0; i < kSStages; ++i) {
            tc::mbar_init(&sm.full[i], 1);
            tc::mbar_init(&sm.empty[i], kSWarps);
        }
        tc::fence_mbar_init();
    }
    const float c1 = 2.f * g.wexp / g.tn;  // d w / d position = c1 d w per grid cell
    // weights and warp masks of entries [s0, s0 + cnt)
    auto build = [&](int s0, int cnt) {
        for (int i = tid; i < cnt * 32; i += kSThr) {
            const int e = i >> 5, c = i & 15, ax = (i >> 4) & 1;
            const uint32_t id = __ldg(pos + it.y + s0 + e);
            const int d = id / (uint32_t)nh, q = id - d * nh + 1;
            const float2 sc = __ldg(dsincos + d);
            float x0, y0;
            int fx, fy;
            sample_pos(q, sc, g, x0, y0, fx, fy);
            const float p = ax ? y0 : x0;
            const int f = ax ? fy : fx;
            const int d0 = g.n + f - kR + kVH - (ax ? Y0 : X0);  // first tap of the window in the tile
            const float v = __fmul_rn(g.tn, p);
            const bool mir = floorf(v) != v;  // the mirrored stencil starts one cell later
            const int b = c - d0;
            float w = 0.f, wd = 0.f;
            if (b >= 0 && b <= kTaps) {
                w = tap_weight(f, b, p, g);
                if (b == kTaps) {
                    if (!mir) w = 0.f;
                } else {
                    wd = (ax ? -sc.x : sc.y) * c1 * ((float)(f - kR + b) * g.inv2n - p) * w;
                }
            }
            if (ax) {
                sm.wy[e][c] = make_float2(w, wd);
            } else {
                sm.wx[e][c] = b < kTaps ? w : 0.f;
                sm.wxd[e][c] = wd;
            }
            if (c == 0) {
                float *h = reinterpret_cast<float *>(&sm.hd[e]);
                if (ax) {
                    h[1] = __int_as_float(mir ? d0 : -1000);  // rows 0 and 9 of the window differ only when mirrored
                } else {
                    h[0] = __int_as_float(d0);
                    h[2] = mir ? -tap_weight(f, 0, p, g) : 0.f;
                    h[3] = mir ? tap_weight(f, kTaps, p, g) : 0.f;
                    sm.id[e] = id;
                }
            }
        }
        if (wid < kSWarps) {
            const int ry0 = 4 * (wid >> 1), cx0 = 8 * (wid & 1);
            for (int ch = 0; ch * kSChunk < cnt; ++ch) {
                const int e = ch * kSChunk + lane;
                bool in = false;
                if (e < cnt) {
                    const uint32_t id = __ldg(pos + it.y + s0 + e);
                    const int d = id / (uint32_t)nh, q = id - d * nh + 1;
                    float x0, y0;
                    int fx, fy;
                    sample_pos(q, __ldg(dsincos + d), g, x0, y0, fx, fy);
                    const int dx = g.n + fx - kR + kVH - X0, dy = g.n + fy - kR + kVH - Y0;
                    in = dx + kTaps >= cx0 && dx < cx0 + 8 && dy + kTaps >= ry0 && dy < ry0 + 4;
                }
                const uint32_t mk = __ballot_sync(0xffffffffu, in);
                if (lane == 0) sm.mask[ch][wid] = mk;
            }
        }
    };
    const int ci = lane & 7, ry = 4 * (wid >> 1) + (lane >> 3), cx0 = 8 * (wid & 1);
    float2 acc[8][2];
#pragma unroll
    for (int c = 0; c < 8; ++c) acc[c][0] = acc[c][1] = dup(0.f);
    bool ok = true;
    int k = 0;  // stages issued (copy warp) or consumed
    for (int pz = p0; pz < p1; ++pz) {
        for (int seg = 0; seg < nseg; ++seg) {
            const int s0 = seg * kSCap, cnt = min(kSCap, it.z - s0);
            if (nseg > 1 || pz == p0) {
                __syncthreads();  // the previous entries are done (and the barriers initialised)
                build(s0, cnt);
                __syncthreads();
            }
            const int nch = (cnt + kSChunk - 1) / kSChunk;
            if (wid == kSWarps) {
                for (int ch = 0; ch < nch; ++ch, ++k) {
                    const int slot = k % kSStages, ne = min(kSChunk, cnt - ch * kSChunk);
                    if (k >= kSStages) ok = tc::mbar_wait(&sm.empty[slot], (uint32_t)((k / kSStages - 1) & 1), ok) && ok;
                    const uint32_t bar = tc::smem_addr(&sm.full[slot]);
                    if (lane == 0)
                        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar),
                                     "r"((uint32_t)(ne * kVec * sizeof(float4)))
                                     : "memory");
                    __syncwarp();
                    if (lane < ne) {
                        const float4 *src = emix + ((long long)pz * ndir * nh + sm.id[ch * kSChunk + lane]) * kVec;
                        asm volatile(
                            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                                tc::smem_addr(sm.m[slot][lane])),
                            "l"(src), "r"((uint32_t)(kVec * sizeof(float4))), "r"(bar)
                            : "memory");
                    }
                }
                continue;
            }
            for (int ch = 0; ch < nch; ++ch, ++k) {
                const int slot = k % kSStages;
                ok = tc::mbar_wait(&sm.full[slot], (uint32_t)((k / kSStages) & 1), ok) && ok;
                for (uint32_t mk = sm.mask[ch][wid]; mk; mk &= mk - 1) {
                    const int el = __ffs(mk) - 1, e = ch * kSChunk + el;
                    const float4 m0 = sm.m[slot][el][ci], mp = sm.m[slot][el][8 + ci], m2 = sm.m[slot][el][16 + ci];
                    const float2 wy = sm.wy[e][ry];
                    const float4 h = sm.hd[e];
                    const float4 xa = *reinterpret_cast<const float4 *>(&sm.wx[e][cx0]),
                                 xb = *reinterpret_cast<const float4 *>(&sm.wx[e][cx0 + 4]),
                                 da = *reinterpret_cast<const float4 *>(&sm.wxd[e][cx0]),
                                 db = *reinterpret_cast<const float4 *>(&sm.wxd[e][cx0 + 4]);
                    const int a = ry - __float_as_int(h.y);
                    const float w1 = a == kTaps ? 0.f : wy.x, w2 = a == 0 ? 0.f : wy.x, we = w2 - w1;
                    const float2 U0 = ffma2(dup(we), lo2(m2), ffma2(dup(wy.y), lo2(mp), mul2(w1, lo2(m0))));
                    const float2 U1 = ffma2(dup(we), hi2(m2), ffma2(dup(wy.y), hi2(mp), mul2(w1, hi2(m0))));
                    const float2 V0 = mul2(w1, lo2(mp)), V1 = mul2(w1, hi2(mp));
                    const float wx[8] = {xa.x, xa.y, xa.z, xa.w, xb.x, xb.y, xb.z, xb.w};
                    const float wd[8] = {da.x, da.y, da.z, da.w, db.x, db.y, db.z, db.w};
#pragma unroll
                    for (int c = 0; c < 8; ++c) {
                        acc[c][0] = ffma2(dup(wd[c]), V0, ffma2(dup(wx[c]), U0, acc[c][0]));
                        acc[c][1] = ffma2(dup(wd[c]), V1, ffma2(dup(wx[c]), U1, acc[c][1]));
                    }
                    // edge columns of the window inside this warp's columns (at most one: they are 9 apart)
                    int ce = __float_as_int(h.x) - cx0;
                    float wv = h.z;
                    if (ce < 0) {
                        ce += kTaps;
                        wv = h.w;
                    }
                    const float2 E0 = mul2(wv * w2, lo2(m2)), E1 = mul2(wv * w2, hi2(m2));
                    switch (ce) {
#define RECTV_EDGE(c)                                                        \
    case c:                                                                  \
        acc[c][0] = make_float2(acc[c][0].x + E0.x, acc[c][0].y + E0.y);     \
        acc[c][1] = make_float2(acc[c][1].x + E1.x, acc[c][1].y + E1.y);     \
        break;
                        RECTV_EDGE(0)
                        RECTV_EDGE(1)
                        RECTV_EDGE(2)
                        RECTV_EDGE(3)
                        RECTV_EDGE(4)
                        RECTV_EDGE(5)
                        RECTV_EDGE(6)
                        RECTV_EDGE(7)
#undef RECTV_EDGE
                        default: break;
                    }
                }
                __syncwarp();
                if (lane == 0)
                    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc::smem_addr(&sm.empty[slot]))
                                 : "memory");
            }
        }
        if (wid < kSWarps) {  // the pre-IFFT fftshift sign is applied here
            float4 *dst = spec + (long long)(pz * g.jg + jgrp) * plane;
            const int Y = Y0 + ry;
            if (Y < g.vrows) {
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const int X = X0 + cx0 + c;
                    const float sg = ((X + Y) & 1) ? -1.f : 1.f;
                    if (X < g.vp)
                        dst[Y * rowp + (long long)X * 8 + ci] =
                            make_float4(sg * acc[c][0].x, sg * acc[c][0].y, sg * acc[c][1].x, sg * acc[c][1].y);
                }
            }
#pragma unroll
            for (int c = 0; c < 8; ++c) acc[c][0] = acc[c][1] = dup(0.f);
        }
    }
    if (!ok && lane == 0) atomicAdd(err, 1);
}

// ---------------------------------------------------------------------------
// Adjoint, step 3: the window's border folds back into the half plane (the
// adjoint of k_vec_halo): rows wrap modulo P, and the cells past the half
// plane's columns are mirror images, H(k) += conj A(-k); columns 0 and n are
// their own mirror columns.  One thread per 16 bytes of a target cell, or of
// the two cells k and -k in columns 0 and n.
// ---------------------------------------------------------------------------
__global__ void k_vec_fold(float4 *__restrict__ spec, UsGeo g) {
    constexpr int HL = kR, HR = kR + 1;  // window cells before and after the half plane that hold values
    const int P = g.P, n = g.n;
    const long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    const int ci = (int)(i & 7);
    const long long e = i >> 3;
    const int nside = HL + 1 + HR + 1;  // columns 0 .. 4 and n-5 .. n
    float4 *pl = spec + blockIdx.y * (g.vplane / 2);
    auto at = [&](int y, int x) { return pl + ((long long)(y + kVH) * g.vp + x + kVH) * 8 + ci; };
    auto add = [](float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); };
    auto rowsum = [&](int y, int x) {  // cell y of column x with its images P rows away
        float4 v = *at(y, x);
        if (y < HR) v = add(v, *at(y + P, x));
        if (y >= P - HL) v = add(v, *at(y - P, x));
        return v;
    };
    auto conj4 = [](float4 a) { return make_float4(a.x, -a.y, a.z, -a.w); };
    if (e < (long long)P * nside) {
        const int y = (int)(e / nside), c = (int)(e - (long long)y * nside);
        const int x = c <= HL ? c : n - HR + (c - HL - 1);
        const int ym = y ? P - y : 0;
        if (x == 0 || x == n) {
            if (y > ym) return;
            const float4 a = rowsum(y, x), b = rowsum(ym, x);
            *at(y, x) = add(a, conj4(b));
            if (ym != y) *at(ym, x) = add(b, conj4(a));
        } else {
            *at(y, x) = add(rowsum(y, x), conj4(rowsum(ym, x <= HL ? -x : 2 * n - x)));
        }
    } else {
        const long long e2 = e - (long long)P * nside;
        const int w = n + 1 - nside;
        if (e2 >= (long long)(HL + HR) * w) return;
        const int r = (int)(e2 / w), x = HL + 1 + (int)(e2 - (long long)r * w);
        const int y = r < HR ? r : P - HL + (r - HR);
        *at(y, x) = rowsum(y, x);
    }
}

// ---------------------------------------------------------------------------
// The vector layout's half planes of slices z0 .. z0 + nz - 1 into planar ones
// (rows of n + 2 complex) for cuFFT's C2R: k_planar_to_vec reversed.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    k_vec_to_planar(const float4 *__restrict__ spec, float2 *__restrict__ planar, UsGeo g, int z0, int nz, int pl0) {
    __shared__ float2 sh[32][17];
    const int pl = pl0 + blockIdx.z, y = blockIdx.y, x0 = blockIdx.x * 32;
    const int cell = threadIdx.x >> 3, ci = threadIdx.x & 7;
    if (x0 + cell <= g.n) {
        const float4 f = spec[pl * (g.vplane / 2) + ((long long)(y + kVH) * g.vp + x0 + cell + kVH) * 8 + ci];
        sh[cell][2 * ci] = lo2(f);
        sh[cell][2 * ci + 1] = hi2(f);
    }
    __syncthreads();
    const long long img = (long long)g.P * (g.n + 2);
    const int lane = threadIdx.x & 31, x = x0 + lane;
    for (int v = threadIdx.x >> 5; v < 16; v += 8) {
        const int z = vec_slice(g, pl, v), t = vec_time(g, pl, v);
        if (x <= g.n && z < z0 + nz && t < g.m)
            planar[((long long)(z - z0) * g.m + t) * img + (long long)y * (g.n + 2) + x] = sh[lane][v];
    }
}

void launch_vec_to_planar(const float2 *spec, float2 *planar, int z0, int nz, const UsGeo &g, cudaStream_t s) {
    const int pl0 = g.jg > 1 ? z0 * g.jg : z0 / g.zs, npl = vec_planes(g, nz);
    k_vec_to_planar<<<dim3((g.n + 32) / 32, g.P, npl), 256, 0, s>>>(reinterpret_cast<const float4 *>(spec), planar, g,
                                                                    z0, nz, pl0);
    LAUNCH_CHECK("k_vec_to_planar");
}

void scatter_dir_prepare() {
    CUDA_CHECK(cudaFuncSetAttribute(k_scatter_dir, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ScatSmem)));
}

size_t dir_mix_bytes(const UsGeo &g, int zb, int ndir) {
    return (size_t)(vec_planes(g, zb) / g.jg) * ndir * (g.n / 2) * kVec * sizeof(float4);
}

void launch_scatter_dir(const float2 *rowsc, float2 *spec, int zb, const GeoDev &gd, const UsGeo &g, cudaStream_t s) {
    if (g.T != kT) throw Error(1, "tile size must be 16");
    if (!gd.demix || gd.n_adj_items == 0) throw Error(1, "adjoint direction plan missing");
    if (zb > gd.demix_slices) throw Error(1, "adjoint direction mixing buffer too small");
    const int npl = vec_planes(g, zb), npz = npl / g.jg, nh = g.n / 2;
    if (npl > 32767) throw Error(1, "too many spectrum planes");  // plane ranges are packed in 16 bits
    const dim3 gm((nh + kMThr / 8 - 1) / (kMThr / 8), gd.ndir, npz);
    const int kstride = g.jg > 1 ? 16 * g.jg : g.tg;
    for (int jg = 0; jg < g.jg; ++jg) {
        k_adj_mix<<<gm, kMThr, 0, s>>>(gd.demix, rowsc, gd.dray_start, gd.drays, gd.dtau, gd.dkmat, gd.shiftadj, g, zb,
                                       gd.ndir, jg, kstride);
        LAUNCH_CHECK("k_adj_mix");
        k_scatter_dir<<<gd.n_adj_items, kSThr, sizeof(ScatSmem), s>>>(gd.demix, reinterpret_cast<float4 *>(spec),
                                                                     gd.adj_pts, gd.adj_items, gd.sincos, g, gd.ndir,
                                                                     jg, gd.err);
        LAUNCH_CHECK("k_scatter_dir");
    }
    const long long thr = 8 * ((long long)g.P * (2 * kR + 3) + (long long)(2 * kR + 1) * (g.n + 1 - (2 * kR + 3)));
    k_vec_fold<<<dim3((unsigned)((thr + 255) / 256), npl), 256, 0, s>>>(reinterpret_cast<float4 *>(spec), g);
    LAUNCH_CHECK("k_vec_fold");
}

}  // namespace rectv
