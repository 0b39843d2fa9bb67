// 4D total-variation and ADMM kernels (x, y, time, z) for sm_103a.
//
// The reference builds an extended copy of the chunk (extendf), writes the
// float4 gradient (gradf), then runs separate axpby passes and the divergence
// (kernels_operators.cuh:4-73, admm.cu:5-122).  Here the inner step
//   u <- u - 1/2 div( rho (G u - psi) + mu )          (admm.cu:85-95)
// is one kernel that forms each needed gradient component on the fly, and the
// end-of-iteration shrink / dual update / residual norms (admm.cu:101-117)
// are another.  The norms are reduced in float64 in a fixed order so the rho
// rule (rectv.cu:223-232) is deterministic.
//
// Chunk semantics (rectv.cu:161-173, extendf): chunk c covers slices
// [c nzp, (c+1) nzp); the slice below/above a chunk is read from the previous
// outer iterate u_old (never the one being updated) and at the volume ends the
// border value is replicated.  Each chunk owns a dual grid of
// (n+1)^2 (m+1)(nzp+1) points whose point q sees voxel q-1 (clamped).
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>

#include "rectv_internal.cuh"

namespace rectv {

namespace {

__device__ __forceinline__ int clampi(int a, int lo, int hi) { return a < lo ? lo : (a > hi ? hi : a); }

__device__ __forceinline__ void prefetch_l2(const void *p) {
    asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p));
}

// the value d bytes from p
__device__ __forceinline__ const float &at(const float *p, long long d) {
    return *reinterpret_cast<const float *>(reinterpret_cast<const char *>(p) + d);
}
template <int V>
__device__ __forceinline__ void ldv(const float *p, float (&v)[V]) {
    if constexpr (V == 2) {
        const float2 a = *reinterpret_cast<const float2 *>(p);
        v[0] = a.x;
        v[1] = a.y;
    } else {
        v[0] = *p;
    }
}
__device__ __forceinline__ void put(float *p, long long d, float v) {
    *reinterpret_cast<float *>(reinterpret_cast<char *>(p) + d) = v;
}

// FP64 sums of the first cnt floats of each of sm's three rows, in a fixed order:
// warp w sums row w, a lane every 32nd value.  (One FP64 addition of a warp takes
// 16 cycles of the SM: all warps reducing their threads' doubles by shuffles
// cost 18 of them per warp, this 20 + cnt / 16 per block and row.)
template <int CAP>
__device__ __forceinline__ void block_sums3(const float (&sm)[3][CAP], int cnt, double *out) {
    __syncthreads();
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (w >= 3) return;
    double s = 0.;
    for (int i = lane; i < cnt; i += 32) s += (double)sm[w][i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) out[w] = s;
}

}  // namespace

// ---------------------------------------------------------------------------
// Fused inner step (gradient, lin4, divergent of admm.cu:85-95 with tau=-0.5):
//   u_out(v) = u_in(v) + tau sd sum_d [h_d(q-e_d) - h_d(q)],  q = v+1,
//   h = rho (G u_in - psi) + mu = rho G u_in + w,  w = mu - rho psi.
// psi, mu and rho change only at the end of an outer iteration, so the first
// inner step (MODE 1) reads psi and mu and also stores w for every dual point
// the step reads, and the later ones (MODE 2) read w alone (half the dual
// bytes); MODE 0 reads psi and mu only.
// One thread per (V neighbouring x, y, slice), marching along t: h_t(q - e_t) is
// the previous time point's h_t(q), kept in a register.  The grid runs over (x
// blocks, slices, rows) in that order, so the blocks that read a block's z-1 and
// y-1 dual neighbours run at the same time (L2 hits rather than second HBM reads).
// Bound by HBM (24 bytes a voxel in MODE 2, 56 in MODE 1) as far as enough loads
// are in flight: 512 x 512 x 16 x 16 voxels take 0.283 ms in MODE 2 (5.7 TB/s)
// and 0.705 in MODE 1.  Two voxels per thread share the loads' addresses and the
// h_x between them (110 instead of 152 instructions a voxel), and 40 warps per SM
// with the next time point's lines prefetched into L2 hide more latency than 32
// (24) warps that hold the next point's loads in registers: 0.397 (0.781) ms.
// ---------------------------------------------------------------------------
template <int MODE, int V>
__global__ void __launch_bounds__(256, V == 2 ? (MODE == 2 ? 5 : 3) : (MODE == 2 ? 6 : 4))
    k_graddiv(const float *__restrict__ uin, const float *__restrict__ uold, float *__restrict__ uout,
              const float *__restrict__ psi, const float *__restrict__ mu, float *__restrict__ w,
              const float *__restrict__ rhop, TvGeo t, int c0, int nch_total, float tau) {
    const int x = V * (blockIdx.x * blockDim.x + threadIdx.x);
    const int zr = blockIdx.y;
    const int y = blockIdx.z * blockDim.y + threadIdx.y;
    if (x >= t.n || y >= t.n) return;
    const int n = t.n, m = t.m, nzp = t.nzp;
    const int c = c0 + zr / nzp, zl = zr % nzp;
    const long long slab = t.vol_slab, nn = (long long)n * n;
    const long long v0 = ((long long)c * nzp + zl) * slab + (long long)y * n + x;  // voxel (x, y, t = 0)
    const float rho = *rhop;
    const long long sy = n + 1, st = (long long)(n + 1) * (n + 1), sz = st * (m + 1);
    const long long cs = t.comp_stride;
    const long long q0 = (long long)c * t.gp + (zl + 1) * sz + st + (y + 1) * sy + (x + 1);  // q of t = 0
    const float sg = t.sg, sgt = t.sg * t.lambda1;
    // Everything a time point reads lies at block-uniform byte distances from
    // the thread's voxel and from its dual point: a thread carries two pointers along t.
    const float *u = uin + v0;  // the voxel at the time point the next load() is for
    const bool xp = x + V < n, xm = x > 0, yp = y < n - 1, ym = y > 0;
    // z neighbours: inside the chunk, else the previous outer iterate, else replicated
    const long long alt = reinterpret_cast<const char *>(uold) - reinterpret_cast<const char *>(uin);
    const long long dzp = zl < nzp - 1 ? 4 * slab : (c < nch_total - 1 ? alt + 4 * slab : 0);
    const long long dzm = zl > 0 ? -4 * slab : (c > 0 ? alt - 4 * slab : 0);
    float *out = uout + v0;
    const float *pq = (MODE == 2 ? w : psi) + q0;  // its dual point
    const long long dmu = reinterpret_cast<const char *>(mu) - reinterpret_cast<const char *>(psi);
    float *pw = w + q0;
    const long long ci[4] = {0, 4 * cs, 8 * cs, 12 * cs}, cy = 4 * (cs - sy), cz = 4 * (3 * cs - sz);
    // one time point: u at y+1, y-1, z+1, z-1, t+1 and right and left of the
    // V voxels; the dual values (psi and mu, or w) at q (4 components) and of
    // component x at q-1, y at q-sy, z at q-sz
    constexpr int S = MODE == 2 ? 1 : 2;
    struct Pt {
        float up[V], um[V], uzp[V], uzm[V], ut[V], xr, xl;
        float p[S][4][V], py[S][V], pz[S][V], px[S];
    };
    auto load = [&](int tt, const float(&f)[V], Pt &a) {
        a.xr = xp ? u[V] : f[V - 1];
        a.xl = xm ? u[-1] : f[0];
#pragma unroll
        for (int v = 0; v < V; ++v) a.up[v] = a.um[v] = a.ut[v] = f[v];
        if (yp) ldv<V>(u + n, a.up);
        if (ym) ldv<V>(u - n, a.um);
        ldv<V>(&at(u, dzp), a.uzp);
        ldv<V>(&at(u, dzm), a.uzm);
        if (tt < m - 1) ldv<V>(u + nn, a.ut);
#pragma unroll
        for (int s = 0; s < S; ++s) {
            const long long d = s ? dmu : 0;
            a.px[s] = at(pq, d - 4);
#pragma unroll
            for (int v = 0; v < V; ++v) {
#pragma unroll
                for (int i = 0; i < 4; ++i) a.p[s][i][v] = at(pq + v, d + ci[i]);
                a.py[s][v] = at(pq + v, d + cy);
                a.pz[s][v] = at(pq + v, d + cz);
            }
        }
    };
    // h of one component from the gradient term g and the dual values
    auto hval = [&](float g, float p, float mv) {
        if constexpr (MODE == 2)
            return rho * g + p;
        else
            return rho * (g - p) + mv;
    };
    float f0[V], hmt[V];  // hmt: h_t at q - st; for t = 0 the clamped backward difference is zero
    ldv<V>(u, f0);
#pragma unroll
    for (int v = 0; v < V; ++v) {
        const float p0 = at(pq + v, ci[2] - 4 * st), m0 = MODE == 2 ? 0.f : at(pq + v, dmu + ci[2] - 4 * st);
        hmt[v] = hval(sgt * (f0[v] - f0[v]), p0, m0);
        if constexpr (MODE == 1) put(pw + v, ci[2] - 4 * st, m0 - rho * p0);
    }
#pragma unroll 1
    for (int tt = 0; tt < m; ++tt) {
        // the lines only this thread's column brings from HBM (its own dual
        // values and u at the next time point; the neighbours' are other
        // threads' own), into L2 two time points ahead of their load
        if (tt + 1 < m) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                prefetch_l2(&at(pq, 4 * st + ci[i]));
                if constexpr (MODE != 2) prefetch_l2(&at(pq, dmu + 4 * st + ci[i]));
            }
        }
        if (tt + 2 < m) prefetch_l2(u + 2 * nn);
        Pt cur;
        load(tt, f0, cur);
        if constexpr (MODE == 1) {  // w at q, and at the lower boundary planes these voxels read
#pragma unroll
            for (int v = 0; v < V; ++v) {
#pragma unroll
                for (int i = 0; i < 4; ++i) put(pw + v, ci[i], cur.p[S - 1][i][v] - rho * cur.p[0][i][v]);
                if (v == 0 && x == 0) put(pw, -4, cur.px[S - 1] - rho * cur.px[0]);
                if (y == 0) put(pw + v, cy, cur.py[S - 1][v] - rho * cur.py[0][v]);
                if (zl == 0) put(pw + v, cz, cur.pz[S - 1][v] - rho * cur.pz[0][v]);
            }
        }
        u += nn;
        pq += st;
        pw += st;
        float r[V], hx = hval(sg * (f0[0] - cur.xl), cur.px[0], cur.px[S - 1]);  // h_x left of the voxel
#pragma unroll
        for (int v = 0; v < V; ++v) {
            float d;
            {  // x
                const float hq = hval(sg * ((v < V - 1 ? f0[v + 1 < V ? v + 1 : v] : cur.xr) - f0[v]), cur.p[0][0][v],
                                      cur.p[S - 1][0][v]);
                d = hx - hq;
                hx = hq;
            }
            {  // y
                const float hq = hval(sg * (cur.up[v] - f0[v]), cur.p[0][1][v], cur.p[S - 1][1][v]);
                const float hm = hval(sg * (f0[v] - cur.um[v]), cur.py[0][v], cur.py[S - 1][v]);
                d += hm - hq;
            }
            {  // t (scaled by lambda1 in both gradient and divergence)
                const float hq = hval(sgt * (cur.ut[v] - f0[v]), cur.p[0][2][v], cur.p[S - 1][2][v]);
                d += t.lambda1 * (hmt[v] - hq);
                hmt[v] = hq;
            }
            {  // z
                const float hq = hval(sg * (cur.uzp[v] - f0[v]), cur.p[0][3][v], cur.p[S - 1][3][v]);
                const float hm = hval(sg * (f0[v] - cur.uzm[v]), cur.pz[0][v], cur.pz[S - 1][v]);
                d += hm - hq;
            }
            r[v] = f0[v] + tau * t.sd * d;
        }
        if constexpr (V == 2)
            *reinterpret_cast<float2 *>(out) = make_float2(r[0], r[1]);
        else
            *out = r[0];
        out += nn;
#pragma unroll
        for (int v = 0; v < V; ++v) f0[v] = cur.ut[v];  // u at t+1
    }
}

template <int V>
static void graddiv_v(const float *u_in, const float *u_old, float *u_out, const float *psi, const float *mu, float *w,
                      int mode, const float *rho, int c0, int nch, const TvGeo &t, cudaStream_t s) {
    const int bx = std::min(256, ((t.n + V - 1) / V + 31) / 32 * 32);
    const dim3 bs(bx, 256 / bx), gs((t.n + V * bx - 1) / (V * bx), t.nchunks * t.nzp, (t.n + bs.y - 1) / bs.y);
    if (gs.y > 65535u || gs.z > 65535u) throw Error(1, "graddiv: grid too large");
    if (mode == 1)
        k_graddiv<1, V><<<gs, bs, 0, s>>>(u_in, u_old, u_out, psi, mu, w, rho, t, c0, nch, -0.5f);
    else if (mode == 2)
        k_graddiv<2, V><<<gs, bs, 0, s>>>(u_in, u_old, u_out, psi, mu, w, rho, t, c0, nch, -0.5f);
    else
        k_graddiv<0, V><<<gs, bs, 0, s>>>(u_in, u_old, u_out, psi, mu, w, rho, t, c0, nch, -0.5f);
    LAUNCH_CHECK("k_graddiv");
}

void launch_graddiv(const float *u_in, const float *u_old, float *u_out, const float *psi,
                    const float *mu, float *w, int mode, const float *rho, int c0, int nchunks_total,
                    const TvGeo &t, cudaStream_t s) {
    if (mode != 0 && !w) throw Error(1, "graddiv: no w buffer");
    // two voxels per thread where the rows' voxels come in aligned pairs and the
    // threads still fill the chip
    const bool even = t.n % 2 == 0 && t.vol_slab % 2 == 0 && (long long)t.n * t.n * t.nchunks * t.nzp >= 152 * 2048 &&
                      ((uintptr_t)u_in | (uintptr_t)u_old | (uintptr_t)u_out) % 8 == 0;
    if (even)
        graddiv_v<2>(u_in, u_old, u_out, psi, mu, w, mode, rho, c0, nchunks_total, t, s);
    else
        graddiv_v<1>(u_in, u_old, u_out, psi, mu, w, mode, rho, c0, nchunks_total, t, s);
}

// ---------------------------------------------------------------------------
// End of outer iteration for one chunk (admm.cu:101-117):
//   h = G u_cur, ho = G u_old (the reference's h2stored),
//   psi = shrink(h + mu/rho, lambda0/rho), mu += rho h - rho psi,
//   sums of |h-psi|^2, |ho-h|^2 and, for q >= 1, (u_cur-u_old)^2.
// One thread per (qx, qy, qz) marching along qt; the squares along its qt column
// are summed in FP32 (at most m+1 = 17 terms for m = 16) and the column sums
// are accumulated in FP64 in a fixed order; one FP64 partial triple per block.
// Blocks of 256 threads over a plane's (qy, qx) in that order, the planes
// (chunk, qz) fastest, so that the blocks reading a slice twice run together.
// At 9 x 17 x 513 x 513 points per chunk, two chunks: 0.83 ms (the planes slowest
// 0.92; the next time point's values held in registers in place of the L2
// prefetch, blocks of 32 x 8 points: 1.00; two points per thread 1.06).
// ---------------------------------------------------------------------------
// What a thread's column of points (qx, qy, qz) reads: the extended chunk's slabs
// at z0 = qz-1 and z1 = qz (extendf, kernels_operators.cuh:14-19) and, as in
// k_graddiv, block-uniform byte distances from its lower voxel (x0, y0, z0) in
// the new iterate.
struct ShrinkCol {
    const float *u;          // (x0, y0, t = 0, z0) of the new iterate
    float *pm, *pp;          // mu and psi at qt = 0
    long long dz[2], du[2];  // z1 of the new and the old iterate; z0 of the same
    long long nn, st, ci[4];
    bool xin, yin, inner;    // the upper neighbour is another voxel; q - 1 is inside the chunk
    float sg, sgt, rho, thr, rinv;
    __device__ __forceinline__ void init(const float *ucur, const float *uold, float *psi, float *mu, float r,
                                         float lambda0, const TvGeo &t, int c, int nch_total, int qx, int qy, int qz) {
        const int n = t.n, nzp = t.nzp;
        const long long slab = t.vol_slab, zc = (long long)c * nzp;
        auto slab_of = [&](const float *v, int zl) -> const char * {
            const float *p;
            if (zl < 0) p = (c > 0) ? uold + (zc - 1) * slab : v + zc * slab;
            else if (zl >= nzp) p = (c < nch_total - 1) ? uold + (zc + nzp) * slab : v + (zc + nzp - 1) * slab;
            else p = v + (zc + zl) * slab;
            return reinterpret_cast<const char *>(p);
        };
        const char *b0 = slab_of(ucur, qz - 1);
        dz[0] = slab_of(ucur, qz) - b0;
        dz[1] = slab_of(uold, qz) - b0;
        du[0] = 0;
        du[1] = slab_of(uold, qz - 1) - b0;
        nn = (long long)n * n;
        st = (long long)(n + 1) * (n + 1);
#pragma unroll
        for (int i = 0; i < 4; ++i) ci[i] = 4 * i * t.comp_stride;
        u = reinterpret_cast<const float *>(b0) + (long long)clampi(qy - 1, 0, n - 1) * n + clampi(qx - 1, 0, n - 1);
        const long long q = (long long)c * t.gp + (long long)qz * (t.m + 1) * st + (long long)qy * (n + 1) + qx;
        pm = mu + q;
        pp = psi + q;
        xin = qx > 0 && qx < n;
        yin = qy > 0 && qy < n;
        inner = qx >= 1 && qy >= 1 && qz >= 1;
        sg = t.sg;
        sgt = t.sg * t.lambda1;
        rho = r;
        thr = lambda0 / rho;
        rinv = 1.0f / rho;
    }
    __device__ __forceinline__ void grad(float f, float fx, float fy, float fz, float ft, float (&g)[4]) const {
        g[0] = sg * (fx - f);
        g[1] = sg * (fy - f);
        g[2] = sgt * (ft - f);
        g[3] = sg * (fz - f);
    }
};

// One point: g = (G u_new, G u_old); stores psi and mu, returns its squares.
__device__ __forceinline__ void shrink_point(const float (&g)[2][4], float *pm, float *pp, const ShrinkCol &k,
                                             const float (&mv)[4], float &r2, float &s2) {
    float ps[4], za2 = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        ps[i] = g[0][i] + mv[i] * k.rinv;  // solve_reg_ker, admm.cu:49-52
        za2 += ps[i] * ps[i];
    }
    const float za = sqrtf(za2);
    const float shr = (za <= k.thr) ? 0.f : 1.0f - k.thr / za;  // shrink factor of the 4-vector
    r2 = s2 = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float h = g[0][i];
        ps[i] = ps[i] * shr;
        put(pp, k.ci[i], ps[i]);
        put(pm, k.ci[i], mv[i] + k.rho * h - k.rho * ps[i]);  // lin4(mu,h2,psi,1,rho,-rho)
        const float dr = h - ps[i], ds = g[1][i] - h;
        r2 += dr * dr;
        s2 += ds * ds;
    }
}

__global__ void __launch_bounds__(256, 4)
    k_shrink(const float *__restrict__ ucur, const float *__restrict__ uold, float *__restrict__ psi,
             float *__restrict__ mu, const float *__restrict__ rhop, float rho, float lambda0, TvGeo t, int c0,
             int nch_total, double *__restrict__ partials) {
    __shared__ float cs[3][256];
    const int n = t.n, m = t.m;
    const int planes = t.nchunks * (t.nzp + 1), pl = blockIdx.x % planes;  // the block's (chunk, qz)
    const int e = blockIdx.x / planes * 256 + threadIdx.x;
    const int qy = e / (n + 1);
    float a0 = 0.f, a1 = 0.f, a2 = 0.f;
    if (qy <= n) {
        ShrinkCol k;
        k.init(ucur, uold, psi, mu, rhop ? *rhop : rho, lambda0, t, c0 + pl / (t.nzp + 1), nch_total, e - qy * (n + 1),
               qy, pl % (t.nzp + 1));
        const float *u = k.u;  // at t0 = clamp(qt-1)
        float *pm = k.pm, *pp = k.pp;
        float f[2] = {u[0], at(u, k.du[1])};  // values at t0 of the new and the old iterate
#pragma unroll 1
        for (int qt = 0; qt <= m; ++qt) {
            // the lines only this thread's column brings from HBM, into L2 ahead of their loads
            if (qt + 2 <= m) {
#pragma unroll
                for (int i = 0; i < 4; ++i) prefetch_l2(&at(pm, k.ci[i] + 8 * k.st));
                if (qt > 0 && qt + 2 < m) {
                    prefetch_l2(u + 3 * k.nn);
                    prefetch_l2(&at(u, k.du[1] + 12 * k.nn));
                }
            }
            float mv[4], g[2][4], ft[2], r2, s2;
#pragma unroll
            for (int i = 0; i < 4; ++i) mv[i] = at(pm, k.ci[i]);
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                const float *us = &at(u, k.du[s]);
                const float fx = k.xin ? us[1] : f[s], fy = k.yin ? us[n] : f[s], fz = at(u, k.dz[s]);
                ft[s] = qt > 0 && qt < m ? us[k.nn] : f[s];
                k.grad(f[s], fx, fy, fz, ft[s], g[s]);
            }
            shrink_point(g, pm, pp, k, mv, r2, s2);
            a0 += r2;
            a1 += s2;
            if (qt >= 1 && k.inner) {  // voxel q-1 = (x0, y0, t0, z0)
                const float dd = f[0] - f[1];
                a2 = fmaf(dd, dd, a2);
            }
            f[0] = ft[0];
            f[1] = ft[1];
            if (qt > 0) u += k.nn;
            pm += k.st;
            pp += k.st;
        }
    }
    cs[0][threadIdx.x] = a0;
    cs[1][threadIdx.x] = a1;
    cs[2][threadIdx.x] = a2;
    block_sums3(cs, 256, partials + 3LL * blockIdx.x);
}

// Grids of at most two blocks per SM, where a column costs m+1 memory latencies:
// the same with the loads of five points at a time in flight (a grid this small
// leaves the registers for it).  9 x 9 x 65 x 65 points: 7.4 us, 10.6 one point at a time.
__global__ void __launch_bounds__(256, 2)
    k_shrink_few(const float *__restrict__ ucur, const float *__restrict__ uold, float *__restrict__ psi,
                 float *__restrict__ mu, const float *__restrict__ rhop, float rho, float lambda0, TvGeo t, int c0,
                 int nch_total, double *__restrict__ partials) {
    constexpr int G = 5;
    __shared__ float cs[3][256];
    const int n = t.n, m = t.m;
    const int planes = t.nchunks * (t.nzp + 1), pl = blockIdx.x % planes;
    const int e = blockIdx.x / planes * 256 + threadIdx.x;
    const int qy = e / (n + 1);
    float a0 = 0.f, a1 = 0.f, a2 = 0.f;
    if (qy <= n) {
        ShrinkCol k;
        k.init(ucur, uold, psi, mu, rhop ? *rhop : rho, lambda0, t, c0 + pl / (t.nzp + 1), nch_total, e - qy * (n + 1),
               qy, pl % (t.nzp + 1));
        const float *u = k.u;
        float *pm = k.pm, *pp = k.pp;
        float f[2] = {u[0], at(u, k.du[1])};
#pragma unroll 1
        for (int q0 = 0; q0 <= m; q0 += G) {
            float mv[G][4], fx[G][2], fy[G][2], fz[G][2], ft[G][2];
#pragma unroll
            for (int j = 0; j < G; ++j) {
                if (q0 + j > m) break;
                const float *v = u;  // (x0, y0, t0, z0) of the point
                if (j > 0) v += (j - (q0 == 0 ? 1 : 0)) * k.nn;
#pragma unroll
                for (int s = 0; s < 2; ++s) {  // (neighbours a clamp maps to the voxel itself stay unset)
                    const float *us = &at(v, k.du[s]);
                    if (k.xin) fx[j][s] = us[1];
                    if (k.yin) fy[j][s] = us[n];
                    fz[j][s] = at(v, k.dz[s]);
                    if (q0 + j > 0 && q0 + j < m) ft[j][s] = us[k.nn];
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) mv[j][i] = at(pm + j * k.st, k.ci[i]);
            }
#pragma unroll
            for (int j = 0; j < G; ++j) {
                if (q0 + j > m) break;
                float g[2][4], r2, s2;
#pragma unroll
                for (int s = 0; s < 2; ++s) {
                    if (q0 + j == 0 || q0 + j == m) ft[j][s] = f[s];
                    k.grad(f[s], k.xin ? fx[j][s] : f[s], k.yin ? fy[j][s] : f[s], fz[j][s], ft[j][s], g[s]);
                }
                shrink_point(g, pm, pp, k, mv[j], r2, s2);
                a0 += r2;
                a1 += s2;
                if (q0 + j >= 1 && k.inner) {
                    const float dd = f[0] - f[1];
                    a2 = fmaf(dd, dd, a2);
                }
                f[0] = ft[j][0];
                f[1] = ft[j][1];
                if (q0 + j > 0) u += k.nn;
                pm += k.st;
                pp += k.st;
            }
        }
    }
    cs[0][threadIdx.x] = a0;
    cs[1][threadIdx.x] = a1;
    cs[2][threadIdx.x] = a2;
    block_sums3(cs, 256, partials + 3LL * blockIdx.x);
}

int shrink_blocks(const TvGeo &t, int nchunks) {
    return (int)(((long long)(t.n + 1) * (t.n + 1) + 255) / 256) * nchunks * (t.nzp + 1);
}

int launch_shrink(const float *u_cur, const float *u_old, float *psi, float *mu, const float *rho_d, float rho,
                  float lambda0, int c0, int nchunks_total, const TvGeo &t, double *partials,
                  cudaStream_t s) {
    const int nb = shrink_blocks(t, t.nchunks);
    if (nb <= 152 * 2)
        k_shrink_few<<<nb, 256, 0, s>>>(u_cur, u_old, psi, mu, rho_d, rho, lambda0, t, c0, nchunks_total, partials);
    else
        k_shrink<<<nb, 256, 0, s>>>(u_cur, u_old, psi, mu, rho_d, rho, lambda0, t, c0, nchunks_total, partials);
    LAUNCH_CHECK("k_shrink");
    return nb;
}

// ---------------------------------------------------------------------------
// Fixed-order FP64 sum of the shrink partials and the rho rule
// (rectv.cu:223-232): r = sum |h-psi|^2, s = rho^2 sum |dG u|^2;
// r > 10 s -> rho *= 2, s > 10 r -> rho *= 0.5.
// stats row = (||u_new - u_old||^2, rho_new, r, s); *iter_ctr counts rows.
// ---------------------------------------------------------------------------
__global__ void k_reduce_rho(const double *__restrict__ partials, int nparts, float *rho,
                             double *stats, int *iter_ctr, int stats_cap) {
    __shared__ double sh[3][256];
    double a = 0, b = 0, c = 0;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) {
        a += partials[3 * i];
        b += partials[3 * i + 1];
        c += partials[3 * i + 2];
    }
    sh[0][threadIdx.x] = a;
    sh[1][threadIdx.x] = b;
    sh[2][threadIdx.x] = c;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            sh[0][threadIdx.x] += sh[0][threadIdx.x + o];
            sh[1][threadIdx.x] += sh[1][threadIdx.x + o];
            sh[2][threadIdx.x] += sh[2][threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const float r0 = *rho;
        const double r = sh[0][0];
        const double sv = (double)r0 * (double)r0 * sh[1][0];
        float rn = r0;
        if (r > 10.0 * sv) rn = r0 * 2.0f;
        else if (sv > 10.0 * r) rn = r0 * 0.5f;
        *rho = rn;
        const int it = *iter_ctr;
        if (it < stats_cap) {
            stats[4 * it + 0] = sh[2][0];
            stats[4 * it + 1] = rn;
            stats[4 * it + 2] = r;
            stats[4 * it + 3] = sv;
        }
        *iter_ctr = it + 1;
    }
}

// First stage: block b sums its contiguous share of the partials, in order.
__global__ void k_sum_stage1(const double *__restrict__ partials, int nparts, double *__restrict__ out) {
    __shared__ double sh[3][256];
    const int per = (nparts + gridDim.x - 1) / gridDim.x;
    const int lo = blockIdx.x * per, hi = min(nparts, lo + per);
    double a = 0, b = 0, c = 0;
    for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        a += partials[3 * i];
        b += partials[3 * i + 1];
        c += partials[3 * i + 2];
    }
    sh[0][threadIdx.x] = a;
    sh[1][threadIdx.x] = b;
    sh[2][threadIdx.x] = c;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            sh[0][threadIdx.x] += sh[0][threadIdx.x + o];
            sh[1][threadIdx.x] += sh[1][threadIdx.x + o];
            sh[2][threadIdx.x] += sh[2][threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        out[3 * blockIdx.x] = sh[0][0];
        out[3 * blockIdx.x + 1] = sh[1][0];
        out[3 * blockIdx.x + 2] = sh[2][0];
    }
}

int reduce_stage1_parts() { return 256; }

void launch_reduce_rho(const double *partials, int nparts, double *stage1, float *rho, double *stats, int *ctr,
                       int cap, cudaStream_t s) {
    k_sum_stage1<<<256, 256, 0, s>>>(partials, nparts, stage1);
    LAUNCH_CHECK("k_sum_stage1");
    k_reduce_rho<<<1, 256, 0, s>>>(stage1, 256, rho, stats, ctr, cap);
    LAUNCH_CHECK("k_reduce_rho");
}

// ---------------------------------------------------------------------------
// Reference-layout gradient (extendf + gradf, kernels_operators.cuh:4-44):
// fm [nzp+2][m][n][n] with halo slabs at 0 and nzp+1, h2 float4
// [nzp+1][m+1][n+1][n+1].
// ---------------------------------------------------------------------------
__global__ void k_gradient_ref(const float *__restrict__ fm, int zbase, float4 *__restrict__ h2, int flgl,
                               int flgr, TvGeo t) {
    const int qx = blockIdx.x * blockDim.x + threadIdx.x;
    const int qy = blockIdx.y * blockDim.y + threadIdx.y;
    const int pl = blockIdx.z;
    const int n = t.n, m = t.m, nzp = t.nzp;
    const int qt = pl % (m + 1), qz = pl / (m + 1);
    if (qx > n || qy > n) return;
    auto fe = [&](int a, int b, int c, int d) -> float {
        const int x = clampi(a - 1, 0, n - 1), y = clampi(b - 1, 0, n - 1), tt = clampi(c - 1, 0, m - 1);
        const int z = clampi(d - 1, -flgl, nzp - 1 + flgr) + zbase;
        return fm[(((long long)z * m + tt) * n + y) * n + x];
    };
    const float f0 = fe(qx, qy, qt, qz);
    const float s = t.sg;
    float4 h;
    h.x = (fe(qx + 1, qy, qt, qz) - f0) * s;
    h.y = (fe(qx, qy + 1, qt, qz) - f0) * s;
    h.z = (fe(qx, qy, qt + 1, qz) - f0) * s * t.lambda1;
    h.w = (fe(qx, qy, qt, qz + 1) - f0) * s;
    h2[(((long long)qz * (m + 1) + qt) * (n + 1) + qy) * (n + 1) + qx] = h;
}

void launch_gradient_ref(const float *fm, int zbase, float *h2, int flgl, int flgr, const TvGeo &t,
                         cudaStream_t s) {
    dim3 bs(32, 8), gs((t.n + 1 + 31) / 32, (t.n + 1 + 7) / 8, (t.nzp + 1) * (t.m + 1));
    k_gradient_ref<<<gs, bs, 0, s>>>(fm, zbase, reinterpret_cast<float4 *>(h2), flgl, flgr, t);
    LAUNCH_CHECK("k_gradient_ref");
}

// Reference-layout divergence (div, kernels_operators.cuh:46-73): four
// separately rounded accumulations, as in the reference.
__global__ void k_divergent_ref(float *__restrict__ fn, const float4 *__restrict__ h2, float tau,
                                TvGeo t) {
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y * blockDim.y + threadIdx.y;
    const int pl = blockIdx.z;
    const int n = t.n, m = t.m;
    const int tt = pl % m, z = pl / m;
    if (x >= n || y >= n) return;
    const long long v = (((long long)z * m + tt) * n + y) * n + x;
    const long long sy = n + 1, st = sy * (n + 1), sz = st * (m + 1);
    const long long q = (z + 1) * sz + (tt + 1) * st + (y + 1) * sy + (x + 1);
    const float s = t.sd;
    float f = fn[v];
    f += tau * (h2[q - 1].x - h2[q].x) * s;
    f += tau * (h2[q - sy].y - h2[q].y) * s;
    f += tau * (h2[q - st].z - h2[q].z) * s * t.lambda1;
    f += tau * (h2[q - sz].w - h2[q].w) * s;
    fn[v] = f;
}

void launch_divergent_ref(float *fn, const float *h2, float tau, const TvGeo &t, cudaStream_t s) {
    dim3 bs(32, 8), gs((t.n + 31) / 32, (t.n + 7) / 8, t.nzp * t.m);
    k_divergent_ref<<<gs, bs, 0, s>>>(fn, reinterpret_cast<const float4 *>(h2), tau, t);
    LAUNCH_CHECK("k_divergent_ref");
}

// ---------------------------------------------------------------------------
// FP64 dot product sum_i a_i b_i of float32 arrays, two fixed-order passes.
// ---------------------------------------------------------------------------
constexpr int kDotParts = 1024;
int dot_parts() { return kDotParts; }

__global__ void k_dot_part(const float *__restrict__ a, const float *__restrict__ b, long long count,
                           double *__restrict__ partials) {
    double acc = 0.0;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < count;
         i += (long long)gridDim.x * blockDim.x)
        acc += (double)a[i] * (double)b[i];
    __shared__ double sh[256];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) partials[blockIdx.x] = sh[0];
}

__global__ void k_dot_final(const double *__restrict__ partials, int nparts, double *out) {
    __shared__ double sh[256];
    double acc = 0.0;
    for (int i = threadIdx.x; i < nparts; i += blockDim.x) acc += partials[i];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out += sh[0];
}

void launch_dot(const float *a, const float *b, long long count, double *partials, int nparts,
                double *out, cudaStream_t s) {
    k_dot_part<<<nparts, 256, 0, s>>>(a, b, count, partials);
    LAUNCH_CHECK("k_dot_part");
    k_dot_final<<<1, 256, 0, s>>>(partials, nparts, out);
    LAUNCH_CHECK("k_dot_final");
}

}  // namespace rectv
