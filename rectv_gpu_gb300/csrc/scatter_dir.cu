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
// sum_theta delta Re K' v (left out on the edges' M2 terms: below 1.2e-7 of the
// stencil's peak at the outermost samples, as in gather_dir.cu).
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
constexpr int kMRays = 64;    // rays of a direction in shared memory

// ---- scatter ----
constexpr int kSWarps = 8;               // consumer warps; one more warp issues the copies
constexpr int kSThr = 32 * (kSWarps + 1);
constexpr int kSChunk = 32;              // entries per stage
constexpr int kSStages = 3;
constexpr int kSCap = 128;               // entries whose weights are held

struct SEntry {
    float wx[kT], wxd[kT];  // wx1 and its first-order weight over the tile's columns
    float2 wy[kT];          // (y weight of the joint 10 taps, first-order weight) over the rows
    float4 hd;              // first column and row of the joint window (int bits), wx2 - wx1 at its columns 0, 9
};

struct ScatSmem {
    float4 m[kSStages][kSChunk][kVec];   // the entries' M0, M0perp, M2 (bulk copies)
    SEntry ent[kSCap];
    uint32_t id[kSCap];
    uint32_t mask[kSCap / kSChunk][8];   // entries of a chunk whose window touches a pair of rows
    unsigned long long full[kSStages], empty[kSStages];
};

__device__ __forceinline__ float2 lo2(float4 f) { return make_float2(f.x, f.y); }
__device__ __forceinline__ float2 hi2(float4 f) { return make_float2(f.z, f.w); }
__device__ __forceinline__ float2 dup(float w) { return make_float2(w, w); }
__device__ __forceinline__ float2 mul2(float w, float2 a) { return make_float2(w * a.x, w * a.y); }

}  // namespace

// ---------------------------------------------------------------------------
// Adjoint, step 1: M0, M0perp, M2 of every position pair and plane.  One block
// per (32 pairs of a direction, planes); eight lanes per pair, two of the
// plane's 16 values each, so that a pair's 384 bytes leave as three full
// 128-byte lines.  The direction's rays (index, offset, K' rows) sit in shared
// memory for all planes of the block; a thread has the row values of eight
// rays in flight.
// Writes 1.13 GB at n = 1024, 360 directions, 16 slices: 0.45 ms a launch
// (0.92 ms with one plane per block, where every block waits through the chain
// of loads from the ray index to the row).
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kMThr)
    k_adj_mix(float4 *__restrict__ emix, const float2 *__restrict__ rowsc, const int *__restrict__ ray_start,
              const uint32_t *__restrict__ rays, const float *__restrict__ tau, const float2 *__restrict__ dkmat,
              const float2 *__restrict__ shifta, UsGeo g, int zb, int ndir, int npz, int per, int jgrp, int kstride) {
    __shared__ float4 ks[kMRays][8];   // K' of the plane's 16 values
    __shared__ uint32_t rvs[kMRays];
    __shared__ float tvs[kMRays];
    const int nh = g.n / 2, hn = nh + 1;
    const int ci = threadIdx.x & 7;
    const int d = blockIdx.y, q = min(nh, 1 + (int)blockIdx.x * (kMThr / 8) + (int)(threadIdx.x >> 3));
    const bool live = 1 + (int)blockIdx.x * (kMThr / 8) + (int)(threadIdx.x >> 3) <= nh;
    const int p0 = blockIdx.z * per, p1 = min(npz, p0 + per);
    const int rs = __ldg(ray_start + d), nr = __ldg(ray_start + d + 1) - rs;
    const float qp = __fdiv_rn((float)(q - nh), (float)g.n);
    const float2 sh = __ldg(shifta + q);
    const float cf = ((q & 1) ? g.cw : -g.cw) * (q == nh ? 0.5f : 1.f);  // the pair q = n/2 is one position
    const float2 fk = make_float2(sh.x * cf, sh.y * cf);
    const int s0 = g.jg > 1 ? 0 : (2 * ci) / g.tg;  // slice of this lane's first value
    const bool two = g.tg == 1;  // one time sample: the two values are two slices
    for (int r0 = 0; r0 < nr; r0 += kMRays) {
        const int nc = min(kMRays, nr - r0);
        if (r0 > 0) __syncthreads();
        for (int i = threadIdx.x; i < nc * 8; i += kMThr) {
            const int r = i >> 3, c = i & 7;
            const float2 *k = dkmat + (long long)(rs + r0 + r) * kstride + 16 * jgrp + ((2 * c) & (g.tg - 1));
            if (two) {
                const float2 k1 = __ldg(k);
                ks[r][c] = make_float4(k1.x, k1.y, k1.x, k1.y);
            } else {
                ks[r][c] = __ldg(reinterpret_cast<const float4 *>(k));
            }
            if (c == 0) {
                rvs[r] = __ldg(rays + rs + r0 + r);
                tvs[r] = __ldg(tau + rs + r0 + r);
            }
        }
        __syncthreads();
        for (int pz = p0; pz < p1; ++pz) {
            const int z0 = g.jg > 1 ? pz : pz * g.zs + s0;
            const bool ok0 = live && z0 < zb, ok1 = two && live && z0 + 1 < zb;
            const float2 *row = rowsc + (long long)z0 * g.ntheta * hn + q;
            float4 *o = emix + (((long long)pz * ndir + d) * nh + q - 1) * kVec + ci;
            // sums of h v, delta h v, g v (K' = h + i g); a later chunk of rays adds to the stored ones
            float2 a0 = dup(0.f), a1 = a0, e0 = a0, e1 = a0, i0 = a0, i1 = a0;
            if (r0 > 0 && live) {
                const float4 A = o[0], P = o[8], M = o[16];
                a0 = lo2(A), a1 = hi2(A), e0 = lo2(P), e1 = hi2(P);
                i0 = make_float2(2.f * M.y - A.y, A.x - 2.f * M.x);
                i1 = make_float2(2.f * M.w - A.w, A.z - 2.f * M.z);
            }
            for (int rb = 0; rb < nc; rb += kMFly) {
                float2 R0[kMFly], R1[kMFly];
#pragma unroll
                for (int i = 0; i < kMFly; ++i) {
                    R0[i] = R1[i] = dup(0.f);
                    if (rb + i < nc) {
                        const long long off = (long long)(rvs[rb + i] & 0x7fffffffu) * hn;
                        if (ok0) R0[i] = __ldg(row + off);
                        if (ok1) R1[i] = __ldg(row + off + (long long)g.ntheta * hn);
                    }
                }
#pragma unroll
                for (int i = 0; i < kMFly; ++i) {
                    if (rb + i >= nc) break;
                    const float dl = qp * tvs[rb + i];  // this ray's offset across the direction
                    const float4 k = ks[rb + i][ci];
                    float2 v = cmul(R0[i], fk), w = v;
                    if (two) w = cmul(R1[i], fk);
                    if (rvs[rb + i] >> 31) {
                        v.y = -v.y;
                        w.y = -w.y;
                    }
                    const float2 hv = mul2(k.x, v), hw = mul2(k.z, w);
                    a0.x += hv.x;
                    a0.y += hv.y;
                    a1.x += hw.x;
                    a1.y += hw.y;
                    e0 = ffma2(dup(dl), hv, e0);
                    e1 = ffma2(dup(dl), hw, e1);
                    i0 = ffma2(dup(k.y), v, i0);
                    i1 = ffma2(dup(k.w), w, i1);
                }
            }
            if (live) {
                o[0] = make_float4(a0.x, a0.y, a1.x, a1.y);
                o[8] = make_float4(e0.x, e0.y, e1.x, e1.y);
                o[16] = make_float4(0.5f * (a0.x - i0.y), 0.5f * (a0.y + i0.x), 0.5f * (a1.x - i1.y), 0.5f * (a1.y + i1.x));
            }
        }
    }
}

// ---------------------------------------------------------------------------
// Adjoint, step 2: one block (eight consumer warps and a copy warp, three
// blocks per SM) per (16x16 tile of the window, planes), the most work first.
// The entries of a tile are the position pairs whose joint 10x10 window
// touches it; the weights of up to 128 of them over the tile's columns and
// rows are computed once for all planes of the block (a tile with more takes
// them in turn and adds to its cells).  Per plane the copy warp streams the
// entries' M0, M0perp, M2 (384 bytes each, one bulk copy per run of
// consecutive samples) through three stages of 32 entries; a warp owns two
// rows of the tile and walks the entries that touch them, its lane (row, v)
// one of the 16 values of the row's 16 cells:
//     U = wy1 M0 + wy1' M0perp + (wy2 - wy1) M2,  V = wy1 M0perp,
//     cell += wx1 U + wx1' V,  and wy2 M2 (wx2 - wx1) at the window's edge columns,
// the left and the right eight cells each only if the window reaches them.
// Warps wait for copies only, never for each other.  All sums run in entry
// order; the cells leave as full 128-byte lines.
// Split items (item.x % 16 > 0): a block has four (two) rows of the tile, its
// warps take every fourth (eighth) entry each and add up at the end in warp
// order: four (eight) times the blocks for problems whose tiles would leave SMs
// idle (dir_adj_work).
// Measured at n = 1024, 360 directions, 16 time samples, 16 slices: 3.23 ms a
// launch (a scatter of every position with float2 atomics into cleared half
// planes: 6.4 ms).  Bound by instruction issue (59 % active; 105 instructions
// per entry and row pair, 22 of them the packed FMAs of the cells) and the
// latency of the shared loads.  Other splits of a tile measured: 4 rows x 8
// columns per warp with two values per lane and 16 consumer warps per SM
// 3.71 ms (3.95 ms with the next entry's loads in flight), 4 rows x 16
// columns, 128 registers, 12 consumer warps per SM 3.85 ms: fewer
// instructions, but too few warps to hide their latency.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(kSThr, 3)
    k_scatter_dir(const float4 *__restrict__ emix, float4 *__restrict__ spec, const uint32_t *__restrict__ pos,
                  const int4 *__restrict__ items, const float2 *__restrict__ dsincos, UsGeo g, int ndir, int jgrp,
                  int *__restrict__ err) {
    extern __shared__ __align__(128) unsigned char sd_smem[];
    ScatSmem &sm = *reinterpret_cast<ScatSmem *>(sd_smem);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int4 it = items[blockIdx.x];
    const int ntx = (g.vp + kT - 1) / kT;
    const int tile = it.x >> 4, sub = it.x & 15;  // sub 1..4: rows 4 (sub - 1) .. alone; 5..12: rows 2 (sub - 5) ..
    const int ty = tile / ntx, Y0 = ty * kT, X0 = (tile - ty * ntx) * kT;  // window cell (0, 0) of the tile
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
    // weights and row masks of entries [s0, s0 + cnt): thread = (entry, axis)
    auto build = [&](int s0, int cnt) {
        for (int i = tid; i < 2 * kSCap; i += kSThr) {
            const int e = i & (kSCap - 1), ax = i / kSCap;  // a warp: 32 entries of one chunk, one axis
            int d0 = 100;
            if (e < cnt) {
                const uint32_t id = __ldg(pos + it.y + s0 + e);
                const int d = id / (uint32_t)nh, q = id - d * nh + 1;
                const float2 sc = __ldg(dsincos + d);
                float x0, y0;
                int fx, fy;
                sample_pos(q, sc, g, x0, y0, fx, fy);
                const float p = ax ? y0 : x0, cd = (ax ? -sc.x : sc.y) * c1;
                const int f = ax ? fy : fx;
                d0 = g.n + f - kR + kVH - (ax ? Y0 : X0);  // first tap of the window in the tile
                const float v = __fmul_rn(g.tn, p);
                const bool mir = floorf(v) != v;  // the mirrored stencil starts one cell later
                SEntry &en = sm.ent[e];
                const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
                float4 *zero = reinterpret_cast<float4 *>(ax ? reinterpret_cast<float *>(en.wy) : en.wx);
#pragma unroll
                for (int k = 0; k < 8; ++k) zero[k] = z4;
#pragma unroll
                for (int b = 0; b <= kTaps; ++b) {
                    float w = tap_weight(f, b, p, g);
                    if (b == kTaps && !mir) w = 0.f;
                    const int c = d0 + b;
                    const float wd = cd * ((float)(f - kR + b) * g.inv2n - p) * w;
                    if (ax == 0 && b == 0) en.hd.z = mir ? -w : 0.f;
                    if (ax == 0 && b == kTaps) en.hd.w = w;
                    if (c < 0 || c >= kT) continue;
                    if (ax) {
                        en.wy[c] = make_float2(w, b < kTaps ? wd : 0.f);
                    } else if (b < kTaps) {
                        en.wx[c] = w;
                        en.wxd[c] = wd;
                    }
                }
                if (ax) {
                    en.hd.y = __int_as_float(mir ? d0 : -1000);  // rows 0 and 9 of the window differ only when mirrored
                } else {
                    en.hd.x = __int_as_float(d0);
                    sm.id[e] = id;
                }
            }
            if (ax && e - lane < cnt) {
#pragma unroll
                for (int r = 0; r < 8; ++r) {
                    const uint32_t mk = __ballot_sync(0xffffffffu, d0 + kTaps >= 2 * r && d0 < 2 * r + 2);
                    if (lane == 0) sm.mask[e / kSChunk][r] = mk;
                }
            }
        }
    };
    // this warp's pair of rows and its entries; the first nl warps sum a pair's warps
    const int nl = sub == 0 ? kSWarps : (sub < 5 ? 2 : 1);
    const int rg = sub == 0 ? wid & 7 : (sub < 5 ? 2 * (sub - 1) + (wid & 1) : sub - 5);
    const uint32_t part = sub == 0 ? 0xffffffffu : (sub < 5 ? 0x11111111u << ((wid >> 1) & 3) : 0x01010101u << (wid & 7));
    const int vi = lane & 15, ry = 2 * rg + (lane >> 4);
    float2 acc[2][8];  // [re, im][cell pair]
    bool ok = true;
    int k = 0;  // stages issued (copy warp) or consumed
    for (int seg = 0; seg < nseg; ++seg) {
        const int s0 = seg * kSCap, cnt = min(kSCap, it.z - s0), nch = (cnt + kSChunk - 1) / kSChunk;
        __syncthreads();  // the previous entries are done (and the barriers initialised)
        build(s0, cnt);
        __syncthreads();
        for (int pz = p0; pz < p1; ++pz) {
            float2 *dst = reinterpret_cast<float2 *>(spec + (long long)(pz * g.jg + jgrp) * plane +
                                                     (long long)(Y0 + ry) * rowp + (long long)X0 * 8) + vi;
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
                    // runs of consecutive pairs (a direction's samples inside the tile) are contiguous: one copy each
                    const uint32_t id = lane < ne ? sm.id[ch * kSChunk + lane] : 0u;
                    const uint32_t before = __shfl_up_sync(0xffffffffu, id, 1);
                    const bool first = lane < ne && (lane == 0 || id != before + 1);
                    const uint32_t rest = __ballot_sync(0xffffffffu, first) & ~((2u << lane) - 1u);
                    if (first) {
                        const int len = (rest ? __ffs(rest) - 1 : ne) - lane;
                        const float4 *src = emix + ((long long)pz * ndir * nh + id) * kVec;
                        asm volatile(
                            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                                tc::smem_addr(sm.m[slot][lane])),
                            "l"(src), "r"((uint32_t)(len * kVec * sizeof(float4))), "r"(bar)
                            : "memory");
                    }
                }
            } else {
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[i >> 3][i & 7] = dup(0.f);
                for (int ch = 0; ch < nch; ++ch, ++k) {
                    const int slot = k % kSStages;
                    ok = tc::mbar_wait(&sm.full[slot], (uint32_t)((k / kSStages) & 1), ok) && ok;
                    const float2 *mb = reinterpret_cast<const float2 *>(sm.m[slot][0]) + vi;
                    const SEntry *eb = &sm.ent[ch * kSChunk];
                    for (uint32_t mk = sm.mask[ch][rg] & part; mk; mk &= mk - 1) {
                        const int el = __ffs(mk) - 1;
                        const SEntry &en = eb[el];
                        const float2 m0 = mb[el * 2 * kVec], mp = mb[el * 2 * kVec + 16], m2 = mb[el * 2 * kVec + 32];
                        const float2 wy = en.wy[ry];
                        const float4 h = en.hd;
                        const float4 *x4 = reinterpret_cast<const float4 *>(en.wx);
                        const int a = ry - __float_as_int(h.y);
                        const float w1 = a == kTaps ? 0.f : wy.x, w2 = a == 0 ? 0.f : wy.x, we = w2 - w1;
                        const float U[2] = {fmaf(we, m2.x, fmaf(wy.y, mp.x, w1 * m0.x)),
                                            fmaf(we, m2.y, fmaf(wy.y, mp.y, w1 * m0.y))};
                        const float V[2] = {w1 * mp.x, w1 * mp.y};
                        const float E[2] = {w2 * m2.x, w2 * m2.y};
                        // (the same in every lane; the reduction's result is known to be, so the
                        // branches on it need no reconvergence: 3.23 instead of 3.32 ms)
                        const int dx = __reduce_max_sync(0xffffffffu, __float_as_int(h.x));
                        auto half = [&](int c0) {  // cells 2 c0 .. 2 c0 + 7 (pairs c0 ..)
                            const float4 xa = x4[c0 / 2], xb = x4[c0 / 2 + 1];
                            const float4 da = x4[kT / 4 + c0 / 2], db = x4[kT / 4 + c0 / 2 + 1];
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                acc[i][c0] = ffma2(lo2(xa), dup(U[i]), acc[i][c0]);
                                acc[i][c0 + 1] = ffma2(hi2(xa), dup(U[i]), acc[i][c0 + 1]);
                                acc[i][c0 + 2] = ffma2(lo2(xb), dup(U[i]), acc[i][c0 + 2]);
                                acc[i][c0 + 3] = ffma2(hi2(xb), dup(U[i]), acc[i][c0 + 3]);
                            }
#pragma unroll
                            for (int i = 0; i < 2; ++i) {
                                acc[i][c0] = ffma2(lo2(da), dup(V[i]), acc[i][c0]);
                                acc[i][c0 + 1] = ffma2(hi2(da), dup(V[i]), acc[i][c0 + 1]);
                                acc[i][c0 + 2] = ffma2(lo2(db), dup(V[i]), acc[i][c0 + 2]);
                                acc[i][c0 + 3] = ffma2(hi2(db), dup(V[i]), acc[i][c0 + 3]);
                            }
                        };
                        if (dx < 8) half(0);
                        if (dx + kTaps >= 8) half(4);
                        // the window's edge columns dx and dx + 9: one jump for both
                        switch (dx) {
#define RECTV_E0(c)                                                                         \
    _Pragma("unroll") for (int i = 0; i < 2; ++i) {                                         \
        if ((c) & 1) acc[i][(c) / 2].y = fmaf(h.z, E[i], acc[i][(c) / 2].y);                \
        else acc[i][(c) / 2].x = fmaf(h.z, E[i], acc[i][(c) / 2].x);                        \
    }
#define RECTV_E9(c)                                                                         \
    _Pragma("unroll") for (int i = 0; i < 2; ++i) {                                         \
        if ((c) & 1) acc[i][(c) / 2].y = fmaf(h.w, E[i], acc[i][(c) / 2].y);                \
        else acc[i][(c) / 2].x = fmaf(h.w, E[i], acc[i][(c) / 2].x);                        \
    }
#define RECTV_LEFT(c) case c - 9: RECTV_E9(c) break;
#define RECTV_BOTH(c) case c: RECTV_E0(c) RECTV_E9(c + 9) break;
#define RECTV_RIGHT(c) case c: RECTV_E0(c) break;
                            RECTV_LEFT(0) RECTV_LEFT(1) RECTV_LEFT(2) RECTV_LEFT(3) RECTV_LEFT(4) RECTV_LEFT(5)
                            RECTV_LEFT(6) RECTV_LEFT(7) RECTV_LEFT(8)
                            RECTV_BOTH(0) RECTV_BOTH(1) RECTV_BOTH(2) RECTV_BOTH(3) RECTV_BOTH(4) RECTV_BOTH(5)
                            RECTV_BOTH(6)
                            RECTV_RIGHT(7) RECTV_RIGHT(8) RECTV_RIGHT(9) RECTV_RIGHT(10) RECTV_RIGHT(11)
                            RECTV_RIGHT(12) RECTV_RIGHT(13) RECTV_RIGHT(14) RECTV_RIGHT(15)
#undef RECTV_E0
#undef RECTV_E9
#undef RECTV_LEFT
#undef RECTV_BOTH
#undef RECTV_RIGHT
                            default: break;
                        }
                    }
                    __syncwarp();
                    if (lane == 0)
                        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc::smem_addr(&sm.empty[slot]))
                                     : "memory");
                }
            }
            if (sub) {  // add the four or eight warps' sums, in warp order, through the (idle) stages
                __syncthreads();
                float2 *red = reinterpret_cast<float2 *>(sm.m);
                static_assert(sizeof(sm.m) >= 7 * 16 * 32 * sizeof(float2), "seven warps' sums");
                if (wid >= nl && wid < kSWarps) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) red[((wid - nl) * 16 + i) * 32 + lane] = acc[i >> 3][i & 7];
                }
                __syncthreads();
                if (wid < nl) {
                    for (int w = wid; w < kSWarps - nl; w += nl)
#pragma unroll
                        for (int i = 0; i < 16; ++i) {
                            const float2 o = red[(w * 16 + i) * 32 + lane];
                            acc[i >> 3][i & 7].x += o.x;
                            acc[i >> 3][i & 7].y += o.y;
                        }
                }
                tc::fence_proxy_async();  // before the next copies into the stages
                __syncthreads();
            }
            if (wid < nl && Y0 + ry < g.vrows) {  // the pre-IFFT fftshift sign is applied here
                const float sy = ((X0 + Y0 + ry) & 1) ? -1.f : 1.f;
#pragma unroll
                for (int c = 0; c < kT; ++c) {
                    if (X0 + c >= g.vp) continue;
                    const float2 r = acc[0][c >> 1], i = acc[1][c >> 1];
                    float2 o = (c & 1) ? make_float2(-sy * r.y, -sy * i.y) : make_float2(sy * r.x, sy * i.x);
                    if (seg > 0) {  // this thread's own earlier store
                        const float2 q = dst[c * 16];
                        o = make_float2(o.x + q.x, o.y + q.y);
                    }
                    dst[c * 16] = o;
                }
            }
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
// (rows of planar_pitch complex) for cuFFT's C2R: k_planar_to_vec reversed.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256)
    k_vec_to_planar(const float4 *__restrict__ spec, float2 *__restrict__ planar, UsGeo g, int z0, int nz, int pl0) {
    __shared__ float2 sh[kLayoutCells][17];
    const int pl = pl0 + blockIdx.z, y = blockIdx.y, x0 = blockIdx.x * kLayoutCells;
    const int cell = threadIdx.x >> 3, ci = threadIdx.x & 7;
    const bool any = vec_live(g, z0 + nz, pl, 2 * ci);  // (or the pair holds no data)
    const float4 *src = spec + pl * (g.vplane / 2) + ((long long)(y + kVH) * g.vp + kVH + x0 + cell) * 8 + ci;
    float4 f[kLayoutCells / 32];
#pragma unroll
    for (int i = 0; i < kLayoutCells / 32; ++i)
        f[i] = any && x0 + cell + 32 * i <= g.n ? __ldg(src + 32 * 8 * i) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int i = 0; i < kLayoutCells / 32; ++i) {
        sh[cell + 32 * i][2 * ci] = lo2(f[i]);
        sh[cell + 32 * i][2 * ci + 1] = hi2(f[i]);
    }
    __syncthreads();
    const int pitch = planar_pitch(g.n), lane = threadIdx.x & 31;
    const long long img = (long long)g.P * pitch;
    for (int v = threadIdx.x >> 5; v < 16; v += 8) {
        if (!vec_live(g, z0 + nz, pl, v)) continue;
        float2 *dst = planar + ((long long)(vec_slice(g, pl, v) - z0) * g.m + vec_time(g, pl, v)) * img +
                      (long long)y * pitch + x0 + lane;
#pragma unroll
        for (int i = 0; i < kLayoutCells / 32; ++i)
            if (x0 + lane + 32 * i <= g.n) dst[32 * i] = sh[lane + 32 * i][v];
    }
}

void launch_vec_to_planar(const float2 *spec, float2 *planar, int z0, int nz, const UsGeo &g, cudaStream_t s) {
    const int pl0 = g.jg > 1 ? z0 * g.jg : z0 / g.zs, npl = vec_planes(g, nz);
    k_vec_to_planar<<<dim3(g.n / kLayoutCells + 1, g.P, npl), 256, 0, s>>>(reinterpret_cast<const float4 *>(spec), planar, g,
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
    // the mix: up to eight planes per block while there are blocks for ten waves
    const int qb = (nh + kMThr / 8 - 1) / (kMThr / 8);
    const int per = (int)std::max<long long>(1, std::min<long long>(8, (long long)qb * gd.ndir * npz / 10000));
    const dim3 gm(qb, gd.ndir, (npz + per - 1) / per);
    const int kstride = g.jg > 1 ? 16 * g.jg : g.tg;
    for (int jg = 0; jg < g.jg; ++jg) {
        k_adj_mix<<<gm, kMThr, 0, s>>>(gd.demix, rowsc, gd.dray_start, gd.drays, gd.dtau, gd.dkmat, gd.shiftadj, g, zb,
                                       gd.ndir, npz, per, jg, kstride);
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
