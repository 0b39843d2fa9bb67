// struct Handle: the device state, geometry, cuFFT plans, captured graphs
// and host logic of one reconstruction problem (one rectv object of the
// reference, src/include/rectv.cuh:7-55, src/cuda/rectv.cu), shared by the
// C ABI (rectv_host.cu) and the multi-problem engine (engine.cu).
#pragma once

#include <cuda_runtime.h>
#include <cufft.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "rectv_gb300.h"
#include "rectv_internal.cuh"

namespace rectv {

// Message of the last failing C-ABI call on this thread.
std::string &last_error();

// Runs f, mapping exceptions to the C ABI's status codes and message.
template <class F>
int guarded(F &&f) {
    try {
        f();
        last_error().clear();
        return RECTV_OK;
    } catch (const Error &e) {
        last_error() = e.what();
        return e.code;
    } catch (const std::bad_alloc &) {
        last_error() = "host out of memory";
        return RECTV_ERR_NOMEM;
    } catch (const std::exception &e) {
        last_error() = e.what();
        return RECTV_ERR_ARG;
    }
}

namespace detail {


template <class T>
T *dalloc(size_t count, std::vector<void *> &owned, cudaStream_t s) {
    void *p = nullptr;
    if (count == 0) count = 1;
    // stream-ordered: freeing (cudaFreeAsync) never synchronises the device,
    // so problems can come and go while others run (engine.cu)
    CUDA_CHECK(cudaMallocAsync(&p, count * sizeof(T), s));
    owned.push_back(p);
    return static_cast<T *>(p);
}

inline int usfft_radius(int n, float *mu_out) {
    // radonusfft.cu:10-11
    const float eps = 1e-3f;
    const float mu = (float)(-std::log((double)eps) / (2.0 * n * (double)n));
    const double r = std::ceil(2.0 * n / kPiUsfft *
                               std::sqrt(-(double)mu * std::log((double)eps) + ((double)mu * n) * ((double)mu * n) / 4.0));
    *mu_out = mu;
    return (int)r;
}

}  // namespace detail

// Sizes of one problem's device buffers and its slice batch: a function of
// the dimensions, the per-batch scratch budget and the environment overrides
// (RECTV_SCATTER=direct, RECTV_CUFFT=1, RECTV_BATCH_BYTES), used both to
// allocate a handle and to estimate its device memory before creating it.
struct Layout {
    int P = 0, nchunks = 0, nzc = 0, zb = 0, nbatch = 0;
    bool tc_scatter = false;  // time samples mixed on the tensor cores in the adjoint (k_scatter_tc)
    bool pad_fft = false;     // hand-written padded-grid 2D FFTs, 2n a power of two
    bool gen_fft = false;     // mixed-radix ones
    bool fused_rows = false;  // fused residual rows (k_resid_rows)
    bool gen_rows = false;    // mixed-radix ones (k_gen_resid)
    bool dirs = false;        // the direction path may run (a geometry decides)
    int tg = 1, zs = 1, jg = 1;  // vector layout of the spectra (UsGeo)
    int vec_slices = 0;       // slices per 2D cuFFT call (without the hand-written FFTs)
    long long slab = 0, gp = 0;
    size_t spec_elems = 0, planar_elems = 0;
    // estimate of all device memory, geometry included, for a geometry on the
    // per-ray kernels; direction_bytes() more where rays share directions
    double bytes = 0;
    int planes() const { return (jg > 1 ? zb * jg : (zb + zs - 1) / zs); }
};

inline Layout make_layout(int n, int ntheta, int m, int nz, int nzp, double batch_bytes) {
    Layout L;
    L.P = 2 * n;
    const long long P = L.P;
    L.nchunks = nz / nzp;
    L.nzc = L.nchunks * nzp;
    L.slab = (long long)n * n * m;
    L.gp = (long long)(n + 1) * (n + 1) * (m + 1) * (nzp + 1);
    // adjoint: tensor-core time-sample mixing (k_scatter_tc) from 8 time
    // samples up; RECTV_SCATTER=direct forces the FP32 scatter
    L.tc_scatter = m >= 8 && ntheta < 65536;  // ray index packed in 16 bits
    L.dirs = true;
    if (const char *e = std::getenv("RECTV_SCATTER"))
        if (!std::strcmp(e, "direct")) L.tc_scatter = L.dirs = false;
    {
        const char *e = std::getenv("RECTV_CUFFT");
        const bool own = !(e && std::atoi(e) != 0);
        GenPlan p;
        L.pad_fft = own && pad_fft_supported(L.P);
        L.gen_fft = own && !L.pad_fft && gen_fft_plan(L.P, &p);
        L.fused_rows = own && resid_rows_supported(n);
        L.gen_rows = own && !L.fused_rows && gen_fft_plan(n, &p);
    }
    if (m > 16) {
        L.tg = 16;
        L.jg = (m + 15) / 16;
    } else {
        while (L.tg < m) L.tg *= 2;
        L.zs = 16 / L.tg;
    }
    const long long vec_plane = (P + 2 * kVH) * (n + 1 + kVH + kVR) * 16;
    // batch size: largest zb = nzp*d, d | nchunks, with per-batch scratch under budget
    double budget = batch_bytes;
    if (budget <= 0) {
        budget = 40.0 * (1ull << 30);
        if (const char *e = std::getenv("RECTV_BATCH_BYTES")) budget = std::atof(e);
    }
    const double per_slice = (double)vec_plane * L.jg / L.zs * 8.0 + (double)ntheta * n * 12.0;
    int d = 1;
    for (int cand = L.nchunks; cand >= 1; --cand) {
        if (L.nchunks % cand) continue;
        if (cand == 1 || per_slice * nzp * cand <= budget) {
            d = cand;
            break;
        }
    }
    L.zb = nzp * d;
    L.nbatch = L.nchunks / d;
    L.spec_elems = std::max<size_t>((size_t)(L.planes() * vec_plane), (size_t)2 * (n + 1) * (n + 1) * (m + 1) * (nzp + 1));
    if (!L.pad_fft && !L.gen_fft) {
        // 2D cuFFT calls over as many slices as keep the planar images near the L2 (whole planes
        // of the vector layout, but never more slices than there are), of equal size.  A slice
        // that takes most of the L2 gains nothing from it: there as many as 1 GB takes (5 slices
        // of width 736, 16 samples: 21.6 ms an iteration, 22.2 one at a time; 8 slices of width
        // 230: 3.6 ms in 64 MB, 3.7 in one call)
        const double img = (double)m * P * planar_pitch(n) * 8.0;
        const double group = img > 32e6 ? std::min(1e9, std::max(64e6, budget / 4)) : 64e6;
        const int most = (int)std::max(1.0, std::min((double)L.zb, group / img));
        const int calls = (L.zb + most - 1) / most, even = (L.zb + calls - 1) / calls;
        L.vec_slices = std::min(L.zb, (even + L.zs - 1) / L.zs * L.zs);
        L.planar_elems = (size_t)L.vec_slices * m * P * planar_pitch(n);
        // the per-ray adjoint's planar images of all slices lie in the spectra, whole calls of them
        L.spec_elems = std::max(L.spec_elems, (size_t)((L.zb + L.vec_slices - 1) / L.vec_slices) * L.planar_elems);
    }
    const double nt = (double)ntheta * n;
    double b = 3.0 * L.nzc * L.slab * 4 + (double)nz * nt * 4 + 3.0 * 4 * L.nchunks * L.gp * 4;
    b += (double)L.zb * nt * 4 + L.spec_elems * 8.0 + (double)L.zb * ntheta * std::max(n, n / 2 + 1) * 8.0;
    if (L.fused_rows || L.gen_rows) b += (double)L.zb * ntheta * (n / 2 + 1) * 8.0;
    b += 3.0 * 8 * (double)((n + 32) / 32) * ((n + 8) / 8) * d * (nzp + 1) * L.nbatch + (4 << 20);
    // geometry: angle plan, adjoint entries (about 2.25 tiles per sample) and records
    b += nt * (4 + 2.5 * 4 + (L.tc_scatter ? 2.5 * 144 + 12 : 0)) + 8.0 * ntheta * m + (1 << 20);
    if (L.pad_fft) b += 16.0 * P * 8;
    // cuFFT's planar images, and the work area that its plans share: as large as the images (twice
    // for small ones) and as the batch's rows at most
    const bool own_fft = L.pad_fft || L.gen_fft, own_rows = L.fused_rows || L.gen_rows;
    b += L.planar_elems * 8.0;
    if (!own_fft || !own_rows)
        b += std::max((n < 32 ? 2.0 : 1.0) * L.planar_elems * 8.0, (double)L.zb * nt * 8.0) * 1.01 + (1 << 20);
    L.bytes = b;
    return L;
}

// When a geometry may take the direction path: rays per direction at least
// *min_group (<= 0: never), rays grouped within *tol grid cells.  Used when the
// rays average at least 2.5 per direction (RECTV_DIRS=1: whenever it can run,
// RECTV_DIRS=0: never) and no FP32 scatter is asked for; RECTV_DIR_TOL sets the
// tolerance (2e-3).
inline void direction_rule(const Layout &L, double *min_group, double *tol) {
    *min_group = kDirMinGroup;
    *tol = kDirTolCells;
    if (const char *e = std::getenv("RECTV_DIRS")) {
        if (!std::strcmp(e, "0")) *min_group = -1.0;
        if (!std::strcmp(e, "1")) *min_group = 1.0;
    }
    if (const char *e = std::getenv("RECTV_DIR_TOL")) *tol = std::max(0.0, std::atof(e));
    if (!L.dirs) *min_group = -1.0;
}

// Device memory of a geometry of ndir directions: the mixing buffer, the
// position pairs (about 2.6 tiles each), their work items and K'.
inline double direction_bytes(const Layout &L, int n, int ntheta, int ndir) {
    if (ndir <= 0) return 0.0;
    const double npz = L.planes() / L.jg, pairs = (double)ndir * (n / 2);
    const double tiles = ((n + 1 + kVH + kVR) / 16 + 1.0) * ((L.P + 2 * kVH) / 16 + 1.0);
    return npz * pairs * 384.0 + pairs * 4 * 3.6 + tiles * npz * 16 * 2 +
           (double)ntheta * (L.jg > 1 ? 16.0 * L.jg : L.tg) * 8 + ntheta * 8.0 + (1 << 20);
}

struct Handle {
    // dimensions (rectv.cuh:43-47)
    int n, ntheta, m, nz, nzp, ngpus, nchunks, nzc;
    int device = 0;
    bool freed = false;
    bool verbose = true;
    bool use_graphs = true;
    cudaStream_t stream = nullptr;      // where work is queued (bind_stream)
    cudaStream_t own_stream = nullptr;  // created with the handle, owns its allocations
    std::vector<void *> owned;

    Layout lay;
    double batch_bytes = -1;  // per-batch scratch budget (<= 0: default / RECTV_BATCH_BYTES)
    size_t dev_bytes = 0;     // device memory owned (buffers), and ...
    size_t geo_bytes = 0;     // ... held by the geometry
    UsGeo ug{};
    TvGeo tv{};
    float mu_us = 0.f;
    int zb = 0;        // slices per batch (multiple of nzp, divides nzc)
    int nbatch = 0;
    long long slab = 0;  // n*n*m
    long long gp = 0;    // dual points per chunk

    // device buffers
    float *U[3] = {nullptr, nullptr, nullptr};
    float *gdata = nullptr;
    float *psi = nullptr, *mu = nullptr;
    float *wdual = nullptr;  // w = mu - rho psi of the current outer iteration (psi's layout)
    float *h1 = nullptr;
    float2 *spec = nullptr;
    float2 *rows = nullptr;
    double *partials = nullptr;
    double *stage1 = nullptr;
    int nparts_batch = 0;
    double *dot_part = nullptr;
    double *dot_out = nullptr;
    float *rho_d = nullptr;
    int *iter_ctr = nullptr;
    double *stats = nullptr;
    int stats_cap = 0;
    GeoDev gd;
    std::vector<void *> geo_owned;

    // cuFFT plans, made as a geometry's path needs them (ensure_plans)
    enum { kR2C2D, kC2R2D, kRowsC2C, kRowsR2C, kRowsC2R, kNPlans };
    cufftHandle plan[kNPlans] = {};
    bool plan_made[kNPlans] = {};
    size_t fft_work_bytes = 0;
    int vec_slices = 1;          // slices per 2D cuFFT call (Layout)
    float2 *planar = nullptr;    // their planar images [vec_slices m][P][planar_pitch]
    CUtensorMap dir_tmap, tc_tmap;  // footprint boxes of the direction gather and the tensor-core gather
    // key of the geometry on the device (set_geometry)
    bool geo_valid = false, geo_has_phi = false, geo_tc_scatter = false;
    float geo_center = 0.f, geo_tc_spr = 0.f;
    double geo_dir_min = 0.0, geo_dir_tol = 0.0;
    std::vector<float> geo_theta, geo_phi;
    // key of the captured graphs besides the geometry (setup)
    int graph_titer = -1;
    float graph_lambda0 = 0.f, graph_lambda1 = 0.f;
    void *fft_work = nullptr;
    // padded-grid FFTs: hand-written ones for P a power of two in [256, 2048],
    // mixed-radix ones for other lengths, else cuFFT with pad, crop and layout
    // passes (RECTV_CUFFT=1 selects cuFFT)
    bool pad_fft = false, gen_fft = false;
    float2 *fft_tw = nullptr;  // twiddle tables (pad_fft_twiddles, gen_fft_twiddles)
    GenPlan gen_plan{};
    CUtensorMap fft_map;       // TMA tiles of the column passes (pad_fft)
    // fused residual rows (inverse row FFT, residual, R2C in one kernel), n a
    // power of two in [256, 1024] or mixed-radix
    bool fused_rows = false, gen_rows = false;
    float2 *fft_tw_n = nullptr;  // twiddles of the n-point row transforms
    GenPlan gen_rplan{};
    float2 *rows_adj = nullptr;  // the adjoint's row spectra [zb][ntheta][n/2+1]
    bool own_rows() const { return fused_rows || gen_rows; }
    bool own_fft() const { return pad_fft || gen_fft; }
    // the per-ray scatters add straight into planar images (in spec) where cuFFT inverts them
    bool planar_adj() const { return !own_fft() && !gd.dirs; }

    // session
    bool session = false;
    int cur = 0;
    float lambda0 = 0.f, lambda1 = 1.f;
    int titer = 0;
    int iters_done = 0;
    int pending = 0;  // iterations queued by enqueue_iterations, not yet collected
    std::vector<double> h_rdiff, h_rho, h_r, h_s;
    double *stats_host = nullptr;  // pinned, allocated by the first iterate()
    int stats_host_cap = 0;
    cudaGraphExec_t graphs[3] = {nullptr, nullptr, nullptr};

    Handle(int n_, int ntheta_, int m_, int nz_, int nzp_, int ngpus_, double batch_bytes_ = -1) {
        batch_bytes = batch_bytes_;
        n = n_;
        ntheta = ntheta_;
        m = m_;
        nz = nz_;
        nzp = nzp_;
        if (n < 2 || ntheta < 1 || m < 1 || nz < 1 || nzp < 1)
            throw Error(RECTV_ERR_ARG, "rectv: n>=2, ntheta>=1, m>=1, nz>=1, nzp>=1 required");
        if (nzp > nz) throw Error(RECTV_ERR_ARG, "rectv: nzp must not exceed nz");
        if ((long long)n * ntheta >= (1LL << 32)) throw Error(RECTV_ERR_ARG, "rectv: n*ntheta too large");
        nchunks = nz / nzp;
        nzc = nchunks * nzp;
        ngpus = std::max(1, std::min(ngpus_, nchunks));  // rectv.cu:9
        CUDA_CHECK(cudaGetDevice(&device));
        const int r = detail::usfft_radius(n, &mu_us);
        if (r != kR) throw Error(RECTV_ERR_ARG, "rectv: USFFT radius " + std::to_string(r) + " != 4");
        try {
            init();
        } catch (...) {
            release();
            throw;
        }
    }

    ~Handle() { release(); }

    void init() {
        CUDA_CHECK(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
        own_stream = stream;
        usfft_prepare();
        gather_tc_prepare();
        scatter_tc_prepare();
        gather_dir_prepare();
        scatter_dir_prepare();
        pad_fft_prepare();
        gen_fft_fwd_prepare();
        gen_fft_inv_prepare();
        const int P = 2 * n;
        ug.n = n;
        ug.ntheta = ntheta;
        ug.m = m;
        ug.P = P;
        ug.tn = (float)(2 * n);
        ug.inv2n = (float)(1.0 / (2.0 * n));
        ug.wexp = (float)(kPiUsfft * kPiUsfft / (double)mu_us);
        ug.cw = (float)(kPiUsfft / (double)mu_us / (double)n);
        ug.T = 16;
        ug.NT = (P + ug.T - 1) / ug.T;
        ug.zper = 64;
        ug.sc_grid = 0;

        lay = make_layout(n, ntheta, m, nz, nzp, batch_bytes);
        ug.tg = lay.tg;
        ug.zs = lay.zs;
        ug.jg = lay.jg;
        ug.vp = n + 1 + kVH + kVR;
        ug.vrows = P + 2 * kVH;
        ug.vplane = (long long)ug.vrows * ug.vp * 16;
        slab = lay.slab;
        gp = lay.gp;
        zb = lay.zb;
        nbatch = lay.nbatch;
        const int d = zb / nzp;

        for (int i = 0; i < 3; ++i) U[i] = alloc<float>((size_t)nzc * slab);
        gdata = alloc<float>((size_t)nz * ntheta * n);
        psi = alloc<float>((size_t)4 * nchunks * gp);
        mu = alloc<float>((size_t)4 * nchunks * gp);
        wdual = alloc<float>((size_t)4 * nchunks * gp);
        CUDA_CHECK(cudaMemsetAsync(wdual, 0, sizeof(float) * (size_t)4 * nchunks * gp, stream));
        h1 = alloc<float>((size_t)zb * ntheta * n);
        // spectra (forward and the adjoint's half planes); also the float4
        // gradient scratch of check_adjoints
        spec = alloc<float2>(lay.spec_elems);
        make_vec_gather_map(&dir_tmap, spec, vec_planes(ug, zb), ug);
        make_vec_gather_tc_map(&tc_tmap, spec, vec_planes(ug, zb), ug);
        rows = alloc<float2>((size_t)zb * ntheta * (size_t)std::max(n, n / 2 + 1));

        tv.n = n;
        tv.m = m;
        tv.nzp = nzp;
        tv.nchunks = d;
        tv.vol_slab = slab;
        tv.gp = gp;
        tv.comp_stride = (long long)nchunks * gp;
        set_lambda1(1.0f);
        nparts_batch = shrink_blocks(tv, d);
        partials = alloc<double>((size_t)3 * nparts_batch * nbatch);
        dot_part = alloc<double>((size_t)dot_parts());
        dot_out = alloc<double>(8);
        stage1 = alloc<double>((size_t)3 * reduce_stage1_parts());
        rho_d = alloc<float>(1);
        iter_ctr = alloc<int>(1);
        gd.err = alloc<int>(1);
        gd.sc_next = alloc<int>(1);
        CUDA_CHECK(cudaMemsetAsync(gd.err, 0, sizeof(int), stream));
        auto table = [&](const std::vector<float2> &w) {
            float2 *d = alloc<float2>(w.size());
            CUDA_CHECK(cudaMemcpyAsync(d, w.data(), sizeof(float2) * w.size(), cudaMemcpyHostToDevice, stream));
            CUDA_CHECK(cudaStreamSynchronize(stream));
            return d;
        };
        pad_fft = lay.pad_fft;
        gen_fft = lay.gen_fft && gen_fft_plan(P, &gen_plan);
        if (pad_fft) {
            fft_tw = table(pad_fft_twiddles(P));
            make_vec_fft_map(&fft_map, spec, vec_planes(ug, zb), ug);
        } else if (gen_fft) {
            fft_tw = table(gen_fft_twiddles(gen_plan));
        } else {
            vec_slices = lay.vec_slices;
            planar = alloc<float2>(lay.planar_elems);
        }
        fused_rows = lay.fused_rows;
        gen_rows = lay.gen_rows && gen_fft_plan(n, &gen_rplan);
        if (own_rows()) {
            fft_tw_n = table(fused_rows ? pad_fft_twiddles(n) : gen_fft_twiddles(gen_rplan));
            rows_adj = alloc<float2>((size_t)zb * ntheta * (size_t)(n / 2 + 1));
        }
        CUDA_CHECK(cudaStreamSynchronize(stream));
    }

    // cuFFT plans are made on first need (never during stream capture): the
    // outer iteration needs them only where the hand-written transforms do not
    // run, the operator API, check_adjoints and FBP always (rows).  The geometry
    // must be set: its path decides which plans run.
    void ensure_plans() {
        bool need[kNPlans] = {};
        need[kRowsR2C] = true;
        need[gd.dirs ? kRowsC2R : kRowsC2C] = !(gd.dirs && own_rows());
        need[kR2C2D] = need[kC2R2D] = !own_fft();
        make_fft_plans(need);
    }

    template <class T>
    T *alloc(size_t count) {
        T *p = detail::dalloc<T>(count, owned, stream);
        dev_bytes += std::max<size_t>(count, 1) * sizeof(T);
        return p;
    }

    size_t device_bytes() const { return dev_bytes + geo_bytes; }

    void set_lambda1(float l1) {
        lambda1 = l1;
        tv.lambda1 = l1;
        // kernels_operators.cuh:40-43 and 69-72
        tv.sg = (float)(1.0 / (2.0 * std::cbrt(2.0) * ((double)l1 / 2.0)));
        tv.sd = (float)(1.0 / (4.0 * std::cbrt(2.0) * ((double)l1 / 2.0)));
    }

    void make_fft_plans(const bool (&need)[kNPlans]) {
        const int P = 2 * n, nrows = zb * ntheta, hn = n / 2 + 1, pp = planar_pitch(n);
        size_t ws = fft_work_bytes;
        bool any = false;
        for (int i = 0; i < kNPlans; ++i) {
            if (!need[i] || plan_made[i]) continue;
            any = true;
            CUFFT_CHECK(cufftCreate(&plan[i]));
            plan_made[i] = true;
            CUFFT_CHECK(cufftSetAutoAllocation(plan[i], 0));
            size_t w1 = 0;
            // 2D (rows of iem / oem elements, images of idist / odist) or rows of n
            auto make = [&](int rank, int len, int iem, int idist, int oem, int odist, cufftType type, int batch) {
                int nn[2] = {len, len}, in[2] = {len, iem}, on[2] = {len, oem};
                if (rank == 1) {
                    in[0] = iem;
                    on[0] = oem;
                }
                CUFFT_CHECK(cufftMakePlanMany(plan[i], rank, nn, in, 1, idist, on, 1, odist, type, batch, &w1));
            };
            switch (i) {
                case kR2C2D:  // in place in the planar images
                    make(2, P, 2 * pp, 2 * pp * P, pp, pp * P, CUFFT_R2C, vec_slices * m);
                    break;
                case kC2R2D: make(2, P, pp, pp * P, 2 * pp, 2 * pp * P, CUFFT_C2R, vec_slices * m); break;
                case kRowsC2C: make(1, n, n, n, n, n, CUFFT_C2C, nrows); break;
                case kRowsR2C: make(1, n, 2 * hn, 2 * hn, hn, hn, CUFFT_R2C, nrows); break;  // in place (adjoint)
                case kRowsC2R: make(1, n, hn, hn, 2 * hn, 2 * hn, CUFFT_C2R, nrows); break;  // in place (forward)
            }
            CUFFT_CHECK(cufftSetStream(plan[i], stream));
            ws = std::max(ws, w1);
        }
        if (!any) return;
        if (ws > fft_work_bytes) {
            if (fft_work) {
                drop_graphs();  // they hold the work area's address
                cudaFreeAsync(fft_work, stream);
                owned.erase(std::find(owned.begin(), owned.end(), fft_work));
                dev_bytes -= fft_work_bytes;
            }
            fft_work = alloc<char>(ws);
            fft_work_bytes = ws;
        }
        for (int i = 0; i < kNPlans; ++i)
            if (plan_made[i]) CUFFT_CHECK(cufftSetWorkArea(plan[i], fft_work));
    }

    void drop_graphs() {
        for (auto &g : graphs)
            if (g) {
                cudaGraphExecDestroy(g);
                g = nullptr;
            }
    }

    void free_geo() {
        geo_valid = false;
        for (void *p : geo_owned) cudaFreeAsync(p, stream);
        geo_owned.clear();
        geo_bytes = 0;
        int *err = gd.err, *next = gd.sc_next;
        gd = GeoDev();
        gd.err = err;
        gd.sc_next = next;
    }

    // Queue this handle's work on s (a stream of the same device) from now on;
    // nullptr returns to the handle's own stream.  The caller orders s after
    // the handle's earlier work (the engine binds only idle handles).
    void bind_stream(cudaStream_t s) {
        stream = s ? s : own_stream;
        for (int i = 0; i < kNPlans; ++i)
            if (plan_made[i]) CUFFT_CHECK(cufftSetStream(plan[i], stream));
    }

    void release() {
        if (stream) cudaStreamSynchronize(stream);
        if (own_stream && own_stream != stream) cudaStreamSynchronize(own_stream);
        stream = own_stream;
        drop_graphs();
        free_geo();
        for (int i = 0; i < kNPlans; ++i)
            if (plan_made[i]) {
                cufftDestroy(plan[i]);
                plan_made[i] = false;
            }
        for (void *p : owned) cudaFreeAsync(p, stream);
        owned.clear();
        if (stats_host) cudaFreeHost(stats_host);
        stats_host = nullptr;
        stats_host_cap = 0;
        if (own_stream) cudaStreamDestroy(own_stream);
        stream = own_stream = nullptr;
        freed = true;
        session = false;
    }

    // 16 time samples per gather pass (the tensor-core gather's K)
    bool mp16() const { return m >= 8; }

    void check_live() const {
        if (freed) throw Error(RECTV_ERR_STATE, "rectv: object was freed");
    }

    // ---- geometry: angle plan, basis mixing matrix, centre shifts ----
    // Returns true when the geometry was (re)built: plan, K', shifts and
    // records are a function of (theta, phi, center) and of the kernel choice,
    // so a call with the same values keeps them (and the captured graphs).
    bool set_geometry(const float *theta_h, const float *phi_h, float center) {
        // gather items hold at most one sample table; scatter items are whole
        // tiles (one block owns each tile, so tiles are stored, never added)
        // forward items with >= 2 samples per ray use the tensor-core gather
        // (time samples are mixed once per ray); RECTV_GATHER=direct|tc forces
        // one kernel (A/B comparisons).  Below 8 time samples the direct
        // kernel's shared-memory rows are short and it stays the only one.
        float tc_min_spr = (mp16() ? 2.0f : -1.0f);
        if (const char *e = std::getenv("RECTV_GATHER")) {
            if (!std::strcmp(e, "direct")) tc_min_spr = -1.0f;
            if (!std::strcmp(e, "tc") && mp16()) tc_min_spr = 0.0f;
        }
        // adjoint: tensor-core time-sample mixing (k_scatter_tc) as fixed by
        // the layout at creation
        const bool tc_scatter = lay.tc_scatter;
        // direction path (scatter_dir.cu): rays that revisit a direction over
        // several half-turns share its sample positions, so the USFFT
        // interpolates once per position
        double dir_min = 0.0, dir_tol = 0.0;
        direction_rule(lay, &dir_min, &dir_tol);
        const size_t nphi = phi_h ? (size_t)2 * m * ntheta : 0;
        if (geo_valid && center == geo_center && tc_min_spr == geo_tc_spr && tc_scatter == geo_tc_scatter &&
            dir_min == geo_dir_min && dir_tol == geo_dir_tol &&
            (phi_h != nullptr) == geo_has_phi && !std::memcmp(theta_h, geo_theta.data(), sizeof(float) * ntheta) &&
            (!phi_h || !std::memcmp(phi_h, geo_phi.data(), sizeof(float) * nphi)))
            return false;
        drop_graphs();
        free_geo();
        DirPlan dplan;
        const bool dirs =
            dir_min > 0 && build_dir_plan(theta_h, n, ntheta, ug.T, dir_fwd_capacity(), dir_tol, dir_min, dplan);
        HostPlan hp;
        if (dirs) {  // per-direction sincos and adjoint entries; no per-ray items
            hp.sincos = dplan.sincos;
            hp.adj_pts = std::move(dplan.adj_pos);
            hp.adj_items = dir_adj_work(dplan.adj_items, vec_planes(ug, zb) / ug.jg);
            dplan.fwd_items = dir_fwd_work(dplan.fwd_items, vec_planes(ug, zb) / ug.jg);
        } else {
            hp = build_plan(theta_h, n, ntheta, ug.T, table_capacity(), tc_min_spr);
        }
        auto up = [&](const void *src, size_t bytes) -> void * {
            void *p = nullptr;
            CUDA_CHECK(cudaMallocAsync(&p, std::max<size_t>(bytes, 16), stream));
            geo_owned.push_back(p);
            geo_bytes += std::max<size_t>(bytes, 16);
            if (bytes) CUDA_CHECK(cudaMemcpyAsync(p, src, bytes, cudaMemcpyHostToDevice, stream));
            return p;
        };
        gd.sincos = (float2 *)up(hp.sincos.data(), hp.sincos.size() * sizeof(float2));
        gd.fwd_pts = (uint32_t *)up(hp.fwd_pts.data(), hp.fwd_pts.size() * 4);
        gd.fwd_items = (int4 *)up(hp.fwd_items.data(), hp.fwd_items.size() * sizeof(int4));
        gd.n_fwd_items = (int)hp.fwd_items.size();
        gd.fwd_tc_items = (int4 *)up(hp.fwd_tc_items.data(), hp.fwd_tc_items.size() * sizeof(int4));
        gd.n_fwd_tc_items = (int)hp.fwd_tc_items.size();
        gd.adj_pts = (uint32_t *)up(hp.adj_pts.data(), hp.adj_pts.size() * 4);
        gd.adj_items = (int4 *)up(hp.adj_items.data(), hp.adj_items.size() * sizeof(int4));
        gd.n_adj_items = (int)hp.adj_items.size();
        gd.n_adj_busy = 0;
        while (gd.n_adj_busy < gd.n_adj_items && hp.adj_items[gd.n_adj_busy].z > 0) ++gd.n_adj_busy;
        gd.tc_scatter = tc_scatter;
        if (dirs) {
            gd.dirs = true;
            gd.ndir = dplan.ndir;
            gd.dray_start = (int *)up(dplan.ray_start.data(), dplan.ray_start.size() * sizeof(int));
            gd.drays = (uint32_t *)up(dplan.rays.data(), dplan.rays.size() * 4);
            gd.dtau = (float *)up(dplan.tau.data(), dplan.tau.size() * 4);
            gd.dfwd_pos = (uint32_t *)up(dplan.fwd_pos.data(), dplan.fwd_pos.size() * 4);
            gd.dfwd_items = (int4 *)up(dplan.fwd_items.data(), dplan.fwd_items.size() * sizeof(int4));
            gd.n_dfwd_items = (int)dplan.fwd_items.size();
            {  // the adjoint's mixed rays per (plane, position pair) of one batch
                const size_t bytes = dir_mix_bytes(ug, zb, dplan.ndir);
                void *p = nullptr;
                CUDA_CHECK(cudaMallocAsync(&p, bytes, stream));
                geo_owned.push_back(p);
                geo_bytes += bytes;
                gd.demix = (float4 *)p;
                gd.demix_slices = zb;
            }
        }
        std::vector<int> tab_base(1, 0);  // uploaded asynchronously: kept until the stream sync below
        std::vector<int4> tabs;
        if (tc_scatter && !dirs) {
            void *p = nullptr;
            CUDA_CHECK(cudaMallocAsync(&p, std::max<size_t>(hp.adj_pts.size() * sizeof(AdjRec), 16), stream));
            geo_owned.push_back(p);
            geo_bytes += std::max<size_t>(hp.adj_pts.size() * sizeof(AdjRec), 16);
            gd.adj_recs = (AdjRec *)p;
            // tables of the busy items and the size of their ray segmentation
            const int cap = scatter_tc_table_capacity();
            long long words = 0;
            // a table holds whole rays (runs of equal theta), at most one MMA
            // batch of them (scatter_tc_batch_rays()) and at most cap entries
            const int max_rays = scatter_tc_batch_rays();
            for (int i = 0; i < gd.n_adj_busy; ++i) {
                const int4 it = hp.adj_items[i];
                const uint32_t *pts = hp.adj_pts.data() + it.y;
                int c0 = 0;
                while (c0 < it.z) {
                    int c1 = c0, nseg = 0;
                    while (c1 < it.z) {
                        int r = c1 + 1;  // end of the ray starting at c1
                        while (r < it.z && pts[r] / (uint32_t)n == pts[c1] / (uint32_t)n) ++r;
                        if (nseg > 0 && (nseg == max_rays || r - c0 > cap)) break;
                        if (r - c0 > cap) r = c0 + cap;  // a ray longer than a table is split
                        c1 = r;
                        ++nseg;
                    }
                    const int w = scatter_tc_info_words(nseg);
                    tabs.push_back(make_int4(it.y + c0, c1 - c0, (int)words, w));
                    words += w;
                    if (words > 2147483647LL) throw Error(RECTV_ERR_ARG, "rectv: adjoint plan too large");
                    c0 = c1;
                }
                tab_base.push_back((int)tabs.size());
            }
            gd.n_adj_tabs = (int)tabs.size();
            gd.adj_tabs = (int4 *)up(tabs.data(), tabs.size() * sizeof(int4));
            gd.adj_tab_base = (int *)up(tab_base.data(), tab_base.size() * sizeof(int));
            void *q = nullptr;
            CUDA_CHECK(cudaMallocAsync(&q, std::max<size_t>((size_t)words * 4, 16), stream));
            geo_owned.push_back(q);
            geo_bytes += std::max<size_t>((size_t)words * 4, 16);
            gd.adj_info = (uint32_t *)q;
        }
        if (gd.n_fwd_items > 2147483647 || gd.n_adj_items > 2147483647)
            throw Error(RECTV_ERR_ARG, "rectv: plan too large");

        // K'(theta, j) = ntheta/sqrt(m) sum_i phi_i(theta) conj(phi_i(t_j)),
        // t_j = j*ntheta/m: decphi/mulphi/recphi (kernels_operators.cuh:99-149)
        // phi_h == nullptr: the plain (static) Radon transform into time sample 0,
        // K'(theta, 0) = 1, K'(theta, j > 0) = 0 (filtered backprojection)
        std::vector<float2> kmat((size_t)ntheta * m, make_float2(0.f, 0.f));
        const double cphi = (double)ntheta / std::sqrt((double)m);
        if (!phi_h)
            for (int th = 0; th < ntheta; ++th) kmat[(size_t)th * m] = make_float2(1.f, 0.f);
        for (int th = 0; phi_h && th < ntheta; ++th)
            for (int j = 0; j < m; ++j) {
                const int tj = (int)(((long long)j * ntheta) / m);
                std::complex<double> acc(0.0, 0.0);
                for (int i = 0; i < m; ++i) {
                    const std::complex<double> a(phi_h[(size_t)i * 2 * ntheta + 2 * th],
                                                 phi_h[(size_t)i * 2 * ntheta + 2 * th + 1]);
                    const std::complex<double> b(phi_h[(size_t)i * 2 * ntheta + 2 * tj],
                                                 phi_h[(size_t)i * 2 * ntheta + 2 * tj + 1]);
                    acc += a * std::conj(b);
                }
                acc *= cphi;
                kmat[(size_t)th * m + j] = make_float2((float)acc.real(), (float)acc.imag());
            }
        gd.kmat = (float2 *)up(kmat.data(), kmat.size() * sizeof(float2));
        std::vector<float2> dk;  // K' in direction order, rows padded to whole groups of time samples
        if (dirs) {
            const int ks = ug.jg > 1 ? 16 * ug.jg : ug.tg;
            dk.assign((size_t)ntheta * ks, make_float2(0.f, 0.f));
            for (int r = 0; r < ntheta; ++r) {
                const size_t th = dplan.rays[r] & 0x7fffffffu;
                std::copy(kmat.begin() + th * m, kmat.begin() + (th + 1) * m, dk.begin() + (size_t)r * ks);
            }
            gd.dkmat = (float2 *)up(dk.data(), dk.size() * sizeof(float2));
        }
        // set_center (radonusfft.cu:70-75, takeshift kernels_radonusfft.cuh:191-198)
        std::vector<float2> sf(n), sa(n);
        for (int k = 0; k < n; ++k) {
            const double cf = -((double)center - n / 2.0), ca = (double)center - n / 2.0;
            const double af = 2 * kPiUsfft * cf * (k - n / 2.0) / n;
            const double aa = 2 * kPiUsfft * ca * (k - n / 2.0) / n;
            sf[k] = make_float2((float)std::cos(af), (float)std::sin(af));
            sa[k] = make_float2((float)std::cos(aa), (float)std::sin(aa));
        }
        gd.shiftfwd = (float2 *)up(sf.data(), n * sizeof(float2));
        gd.shiftadj = (float2 *)up(sa.data(), n * sizeof(float2));
        // 1/phi of divphi (kernels_radonusfft.cuh:11), separable
        std::vector<float> dp(n);
        for (int x = 0; x < n; ++x) {
            const double d = (double)(x - n / 2);
            dp[x] = (float)std::exp((double)mu_us * d * d);
        }
        gd.deapod = (float *)up(dp.data(), n * sizeof(float));
        if (gd.tc_scatter && !gd.dirs) {
            launch_adj_records(gd.adj_recs, gd, ug, stream);
            launch_adj_tabinfo(gd, stream);
        }
        CUDA_CHECK(cudaStreamSynchronize(stream));  // host vectors go out of scope
        geo_theta.assign(theta_h, theta_h + ntheta);
        geo_phi.assign(phi_h, phi_h + nphi);
        geo_has_phi = phi_h != nullptr;
        geo_center = center;
        geo_tc_spr = tc_min_spr;
        geo_tc_scatter = tc_scatter;
        geo_dir_min = dir_min;
        geo_dir_tol = dir_tol;
        geo_valid = true;
        return true;
    }

    // ---- operators on one batch of zb slices ----
    // out = tau R_apr u  (residual: out = R_apr u - gb)
    void forward(const float *u, const float *gb, float *out, float tau, int residual) {
        forward_rows(u);
        if (gd.dirs && own_rows() && !residual) {  // Hermitian half rows, two per transform
            if (fused_rows)
                launch_fwd_rows(rows, out, tau, fft_tw_n, zb, ug, stream);
            else
                launch_gen_fwd_rows(rows, out, tau, fft_tw_n, gen_rplan, zb, ug, stream);
            return;
        }
        if (gd.dirs) {
            CUFFT_CHECK(cufftExecC2R(plan[kRowsC2R], reinterpret_cast<cufftComplex *>(rows),
                                     reinterpret_cast<cufftReal *>(rows)));
            launch_finish_fwd_real(reinterpret_cast<const float *>(rows), gb, out, zb, tau, residual, ug, stream);
            return;
        }
        CUFFT_CHECK(cufftExecC2C(plan[kRowsC2C], reinterpret_cast<cufftComplex *>(rows),
                                 reinterpret_cast<cufftComplex *>(rows), CUFFT_INVERSE));
        launch_finish_fwd(rows, gb, out, zb, tau, residual, ug, stream);
    }

    // the gathered row spectra of R_apr u (before the inverse row FFT) in rows:
    // whole rows, or their Hermitian halves on the direction path
    void forward_rows(const float *u) {
        if (pad_fft) {
            launch_pad_fft_fwd(u, spec, zb, gd.deapod, fft_tw, fft_map, gd.err, ug, stream);
        } else if (gen_fft) {
            launch_gen_fft_fwd(u, spec, zb, gd.deapod, fft_tw, gen_plan, ug, stream);
        } else {
            for (int z = 0; z < zb; z += vec_slices) {
                const int nzg = std::min(vec_slices, zb - z);
                launch_deapod_pad(u + (long long)z * slab, reinterpret_cast<float *>(planar), nzg * m, gd.deapod, ug,
                                  stream);
                CUFFT_CHECK(cufftExecR2C(plan[kR2C2D], reinterpret_cast<cufftReal *>(planar),
                                         reinterpret_cast<cufftComplex *>(planar)));
                launch_planar_to_vec(planar, spec, z, nzg, ug, stream);
            }
        }
        launch_vec_halo(spec, vec_planes(ug, zb), gd.dirs ? kR + 1 : kVR, ug, stream);
        launch_gather_fwd(spec, rows, zb, gd, ug, gd.dirs ? &dir_tmap : &tc_tmap, stream);
    }

    // u += tau R_apr^T h
    void adjoint(const float *h, float *u, float tau, const float *row_filter = nullptr) {
        launch_adj_prep(h, reinterpret_cast<float *>(rows), zb, ug, stream);
        CUFFT_CHECK(cufftExecR2C(plan[kRowsR2C], reinterpret_cast<cufftReal *>(rows),
                                 reinterpret_cast<cufftComplex *>(rows)));
        if (row_filter) launch_filter_rows(rows, row_filter, (long long)zb * ntheta, n, stream);
        adjoint_rows(rows, u, tau);
    }

    // u += tau R_apr^T of the row spectra rowsc [zb][ntheta][n/2+1]
    void adjoint_rows(const float2 *rowsc, float *u, float tau) {
        // Re IFFT2 of the scattered grids as a C2R of their Hermitian part
        launch_scatter_adj(rowsc, spec, zb, gd, ug, planar_adj(), stream);
        if (pad_fft) {
            launch_pad_fft_inv_accum(spec, u, zb, tau, gd.deapod, fft_tw, fft_map, gd.err, ug, stream);
        } else if (gen_fft) {
            launch_gen_fft_inv_accum(spec, u, zb, tau, gd.deapod, fft_tw, gen_plan, ug, stream);
        } else {
            for (int z = 0; z < zb; z += vec_slices) {
                const int nzg = std::min(vec_slices, zb - z);
                float2 *img = planar_adj() ? spec + (long long)z * m * ug.P * planar_pitch(n) : planar;
                if (!planar_adj()) launch_vec_to_planar(spec, planar, z, nzg, ug, stream);
                CUFFT_CHECK(cufftExecC2R(plan[kC2R2D], reinterpret_cast<cufftComplex *>(img),
                                         reinterpret_cast<cufftReal *>(img)));
                launch_crop_accum_real(reinterpret_cast<const float *>(img), u + (long long)z * slab, nzg, tau, gd.deapod,
                                       ug, stream);
            }
        }
    }

    // ---- one outer ADMM iteration (rectv.cu:140-245 for all chunks) ----
    void enqueue_outer(int old) {
        const int a = (old + 1) % 3, b = (old + 2) % 3;
        int src = old;
        const int dpb = zb / nzp;  // chunks per batch
        for (int k = 0; k < titer; ++k) {
            const int dst = (k % 2 == 0) ? a : b;
            for (int bb = 0; bb < nbatch; ++bb) {
                const long long z0 = (long long)bb * zb;
                const int c0 = bb * dpb;
                if (own_rows()) {  // residual rows straight into the adjoint's row spectra
                    forward_rows(U[src] + z0 * slab);
                    if (fused_rows)
                        launch_resid_rows(rows, gdata + z0 * ntheta * n, rows_adj, fft_tw_n, zb, gd.dirs, ug, stream);
                    else
                        launch_gen_resid(rows, gdata + z0 * ntheta * n, rows_adj, fft_tw_n, gen_rplan, zb, gd.dirs, ug,
                                         stream);
                } else {
                    forward(U[src] + z0 * slab, gdata + z0 * ntheta * n, h1, 1.0f, 1);
                }
                // first inner step: psi, mu in, w = mu - rho psi out; later steps: w in
                const int gmode = titer > 1 ? (k == 0 ? 1 : 2) : 0;
                launch_graddiv(U[src], U[old], U[dst], psi, mu, wdual, gmode, rho_d, c0, nchunks, tv, stream);
                if (own_rows())
                    adjoint_rows(rows_adj, U[dst] + z0 * slab, -0.5f);
                else
                    adjoint(h1, U[dst] + z0 * slab, -0.5f);
            }
            src = dst;
        }
        for (int bb = 0; bb < nbatch; ++bb) {
            launch_shrink(U[src], U[old], psi, mu, rho_d, 0.f, lambda0, bb * dpb, nchunks, tv,
                          partials + (size_t)3 * nparts_batch * bb, stream);
        }
        launch_reduce_rho(partials, nparts_batch * nbatch, stage1, rho_d, stats, iter_ctr, stats_cap, stream);
    }

    int next_cur(int old) const {
        if (titer == 0) return old;
        return (titer % 2 == 1) ? (old + 1) % 3 : (old + 2) % 3;
    }

    void launch_outer() {
        const int old = cur;
        if (use_graphs) {
            if (!graphs[old]) {
                cudaGraph_t g = nullptr;
                CUDA_CHECK(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
                try {
                    enqueue_outer(old);
                } catch (...) {
                    cudaStreamEndCapture(stream, &g);
                    if (g) cudaGraphDestroy(g);
                    throw;
                }
                CUDA_CHECK(cudaStreamEndCapture(stream, &g));
                cudaGraphExec_t ge = nullptr;
                cudaError_t e = cudaGraphInstantiate(&ge, g, 0);
                cudaGraphDestroy(g);
                CUDA_CHECK(e);
                graphs[old] = ge;
            }
            CUDA_CHECK(cudaGraphLaunch(graphs[old], stream));
        } else {
            enqueue_outer(old);
        }
        cur = next_cur(old);
    }

    void setup(const float *theta_h, const float *phi_h, float center, float lambda0_, float lambda1_,
               int titer_, const float *init = nullptr, cudaMemcpyKind init_kind = cudaMemcpyHostToDevice) {
        check_live();
        if (titer_ < 0) throw Error(RECTV_ERR_ARG, "rectv: titer must be >= 0");
        if (!phi_h) throw Error(RECTV_ERR_ARG, "rectv: phi is required");
        const bool rebuilt = set_geometry(theta_h, phi_h, center);
        if (!own_rows() || !own_fft()) ensure_plans();
        lambda0 = lambda0_;
        set_lambda1(lambda1_);
        titer = titer_;
        // graphs bake in the geometry, titer and the two lambdas
        if (rebuilt || titer != graph_titer || lambda0 != graph_lambda0 || lambda1 != graph_lambda1) {
            drop_graphs();
            graph_titer = titer;
            graph_lambda0 = lambda0;
            graph_lambda1 = lambda1;
        }
        // initial guess (zero, as rectv.cu:119-120, unless given) and ADMM state (rectv.cu:121-125)
        cur = 0;
        if (init)
            CUDA_CHECK(cudaMemcpyAsync(U[0], init, sizeof(float) * (size_t)nzc * slab, init_kind, stream));
        else
            CUDA_CHECK(cudaMemsetAsync(U[0], 0, sizeof(float) * (size_t)nzc * slab, stream));
        CUDA_CHECK(cudaMemsetAsync(psi, 0, sizeof(float) * (size_t)4 * nchunks * gp, stream));
        CUDA_CHECK(cudaMemsetAsync(mu, 0, sizeof(float) * (size_t)4 * nchunks * gp, stream));
        const float rho0 = 0.5f;
        CUDA_CHECK(cudaMemcpyAsync(rho_d, &rho0, sizeof(float), cudaMemcpyHostToDevice, stream));
        CUDA_CHECK(cudaStreamSynchronize(stream));
        iters_done = 0;
        h_rdiff.clear();
        h_rho.clear();
        h_r.clear();
        h_s.clear();
        session = true;
    }

    void ensure_stats(int cap) {
        if (cap <= stats_cap) return;
        drop_graphs();  // graphs hold the stats pointer
        if (stats) {
            cudaFreeAsync(stats, stream);
            owned.erase(std::find(owned.begin(), owned.end(), (void *)stats));
            dev_bytes -= sizeof(double) * (size_t)4 * stats_cap;
        }
        stats = alloc<double>((size_t)4 * cap);
        stats_cap = cap;
    }

    void report(int it, int niter_total, const double *row) {
        h_rdiff.push_back(row[0]);
        h_rho.push_back(row[1]);
        h_r.push_back(row[2]);
        h_s.push_back(row[3]);
        if (verbose) {
            std::fprintf(stderr, "iter (%d/%d), rdiff ||f(k+1)-f(k)||:%f \n", it, niter_total, row[0]);
            std::fflush(stderr);
        }
    }

    void iterate(int niter) {
        check_live();
        if (!session) throw Error(RECTV_ERR_STATE, "rectv: setup must precede iterate");
        if (niter < 0) throw Error(RECTV_ERR_ARG, "rectv: niter must be >= 0");
        if (niter == 0) return;
        ensure_stats(niter);
        if (stats_host_cap < niter) {
            if (stats_host) cudaFreeHost(stats_host);
            stats_host = nullptr;
            stats_host_cap = 0;
            CUDA_CHECK(cudaMallocHost(&stats_host, sizeof(double) * 4 * niter));
            stats_host_cap = niter;
        }
        CUDA_CHECK(cudaMemsetAsync(iter_ctr, 0, sizeof(int), stream));
        std::vector<cudaEvent_t> ev;
        if (verbose) {
            ev.resize(niter);
            for (auto &e : ev) CUDA_CHECK(cudaEventCreateWithFlags(&e, cudaEventDisableTiming));
        }
        int reported = 0;
        try {
            for (int it = 0; it < niter; ++it) {
                launch_outer();
                if (verbose) {
                    CUDA_CHECK(cudaMemcpyAsync(stats_host + 4 * it, stats + 4 * it, 4 * sizeof(double),
                                               cudaMemcpyDeviceToHost, stream));
                    CUDA_CHECK(cudaEventRecord(ev[it], stream));
                    // report the previous iteration while this one runs
                    while (reported < it) {
                        CUDA_CHECK(cudaEventSynchronize(ev[reported]));
                        report(iters_done + reported, niter, stats_host + 4 * reported);
                        ++reported;
                    }
                }
            }
            if (verbose) {
                while (reported < niter) {
                    CUDA_CHECK(cudaEventSynchronize(ev[reported]));
                    report(iters_done + reported, niter, stats_host + 4 * reported);
                    ++reported;
                }
            } else {
                CUDA_CHECK(cudaMemcpyAsync(stats_host, stats, 4 * sizeof(double) * niter, cudaMemcpyDeviceToHost,
                                           stream));
                CUDA_CHECK(cudaStreamSynchronize(stream));
                for (int it = 0; it < niter; ++it) {
                    h_rdiff.push_back(stats_host[4 * it]);
                    h_rho.push_back(stats_host[4 * it + 1]);
                    h_r.push_back(stats_host[4 * it + 2]);
                    h_s.push_back(stats_host[4 * it + 3]);
                }
            }
        } catch (...) {
            for (auto &e : ev) cudaEventDestroy(e);
            throw;
        }
        for (auto &e : ev) cudaEventDestroy(e);
        iters_done += niter;
        check_device_errors();
    }

    // Queues niter outer iterations on the handle's stream and returns
    // without waiting; their statistics stay on the device until
    // collect_history().  (The engine's asynchronous form of iterate().)
    void enqueue_iterations(int niter) {
        check_live();
        if (!session) throw Error(RECTV_ERR_STATE, "rectv: setup must precede iterate");
        if (niter < 0) throw Error(RECTV_ERR_ARG, "rectv: niter must be >= 0");
        pending = niter;
        if (niter == 0) return;
        ensure_stats(niter);
        CUDA_CHECK(cudaMemsetAsync(iter_ctr, 0, sizeof(int), stream));
        for (int it = 0; it < niter; ++it) launch_outer();
    }

    // After the stream has finished the queued iterations: appends their
    // statistics to the history (pageable host copy, no pinned buffer) and
    // raises if a kernel recorded an error.
    void collect_history() {
        if (pending > 0) {
            std::vector<double> row((size_t)4 * pending);
            CUDA_CHECK(cudaMemcpyAsync(row.data(), stats, sizeof(double) * row.size(), cudaMemcpyDeviceToHost, stream));
            CUDA_CHECK(cudaStreamSynchronize(stream));
            for (int it = 0; it < pending; ++it) {
                h_rdiff.push_back(row[4 * it]);
                h_rho.push_back(row[4 * it + 1]);
                h_r.push_back(row[4 * it + 2]);
                h_s.push_back(row[4 * it + 3]);
            }
            iters_done += pending;
        }
        pending = 0;
        check_device_errors();
    }

    // Waits for the stream and raises if a kernel recorded an error on the
    // device since the handle was created: a host/device plan disagreement
    // or a bounded TMA / tensor-core wait that gave up.
    void check_device_errors() {
        int errs = 0;
        CUDA_CHECK(cudaMemcpyAsync(&errs, gd.err, sizeof(int), cudaMemcpyDeviceToHost, stream));
        CUDA_CHECK(cudaStreamSynchronize(stream));
        if (errs)
            throw Error(RECTV_ERR_STATE,
                        "rectv: internal kernel error (plan/stencil mismatch or a TMA / tensor-core wait timed out)");
    }

    // ---- operator API helpers: any number of slices via zero-padded batches ----
    void op_forward(float *out, const float *u, int nslices, float tau) {
        ensure_plans();
        for (int z0 = 0; z0 < nslices; z0 += zb) {
            const int nb = std::min(zb, nslices - z0);
            const float *src = u + (size_t)z0 * slab;
            float *dst = out + (size_t)z0 * ntheta * n;
            if (nb == zb) {
                forward(src, nullptr, dst, tau, 0);
            } else {
                float *tmp = U[2];
                CUDA_CHECK(cudaMemsetAsync(tmp, 0, sizeof(float) * zb * slab, stream));
                CUDA_CHECK(cudaMemcpyAsync(tmp, src, sizeof(float) * nb * slab, cudaMemcpyDeviceToDevice, stream));
                forward(tmp, nullptr, h1, tau, 0);
                CUDA_CHECK(cudaMemcpyAsync(dst, h1, sizeof(float) * nb * ntheta * n, cudaMemcpyDeviceToDevice,
                                           stream));
            }
        }
    }

    void op_adjoint(float *u, const float *g, int nslices, float tau) {
        ensure_plans();
        for (int z0 = 0; z0 < nslices; z0 += zb) {
            const int nb = std::min(zb, nslices - z0);
            const float *src = g + (size_t)z0 * ntheta * n;
            float *dst = u + (size_t)z0 * slab;
            if (nb == zb) {
                adjoint(src, dst, tau);
            } else {
                CUDA_CHECK(cudaMemsetAsync(h1, 0, sizeof(float) * zb * ntheta * n, stream));
                CUDA_CHECK(cudaMemcpyAsync(h1, src, sizeof(float) * nb * ntheta * n, cudaMemcpyDeviceToDevice,
                                           stream));
                float *tmp = U[2];
                CUDA_CHECK(cudaMemsetAsync(tmp, 0, sizeof(float) * zb * slab, stream));
                adjoint(h1, tmp, 1.0f);
                launch_axpy(dst, tmp, tau, (long long)nb * slab);
            }
        }
    }

    void launch_axpy(float *y, const float *x, float a, long long count);

    // ---- filtered backprojection (static object), per slice ----
    // frec[z] = circ( pi/4 * R^T( applyfilter(g[z]) ) ): the USFFT adjoint with
    // the reference's ramp filter (kernels_radonusfft.cuh:173-189) on the
    // centred row spectrum and its circular mask (kernels_radonusfft.cuh:
    // 146-159, r = 0).  pi/4 makes R^T W R the identity on band-limited,
    // zero-mean objects for this operator's 1/sqrt(n ntheta) normalisation.
    void fbp(float *frec_h, const float *g_h, const float *theta_h, float center) {
        check_live();
        session = false;
        drop_graphs();
        set_geometry(theta_h, nullptr, center);
        ensure_plans();
        std::vector<float> w(n / 2 + 1);
        for (int k = 0; k <= n / 2; ++k) {
            const float rho = (float)(k - n / 2) / (float)n;
            w[k] = (rho == 0.f) ? 0.f : (float)(std::fabs((double)rho) * n * 4 * std::sin((double)rho) / rho);
        }
        float *w_d = nullptr;
        CUDA_CHECK(cudaMallocAsync(&w_d, w.size() * sizeof(float), stream));
        geo_owned.push_back(w_d);
        CUDA_CHECK(cudaMemcpyAsync(w_d, w.data(), w.size() * sizeof(float), cudaMemcpyHostToDevice, stream));
        const float scale = (float)(kPiUsfft / 4.0);
        float *tmp = U[2], *out = U[1];
        for (int z0 = 0; z0 < nz; z0 += zb) {
            const int nb = std::min(zb, nz - z0);
            CUDA_CHECK(cudaMemsetAsync(h1, 0, sizeof(float) * (size_t)zb * ntheta * n, stream));
            CUDA_CHECK(cudaMemcpyAsync(h1, g_h + (size_t)z0 * ntheta * n, sizeof(float) * (size_t)nb * ntheta * n,
                                       cudaMemcpyHostToDevice, stream));
            CUDA_CHECK(cudaMemsetAsync(tmp, 0, sizeof(float) * (size_t)zb * slab, stream));
            adjoint(h1, tmp, scale, w_d);
            launch_fbp_mask(tmp, out, nb, n, m, 0.f, stream);
            CUDA_CHECK(cudaMemcpyAsync(frec_h + (size_t)z0 * n * n, out, sizeof(float) * (size_t)nb * n * n,
                                       cudaMemcpyDeviceToHost, stream));
            CUDA_CHECK(cudaStreamSynchronize(stream));
        }
        free_geo();  // the FBP geometry is not the reconstruction's
    }

    // ---- instrumentation ----
    int jgroups() const { return (m + 15) / 16; }
    void launch_counts(int *kern, int *ffts) const {
        const int ng = jgroups();
        const int calls = (zb + vec_slices - 1) / vec_slices;  // 2D cuFFT calls without the hand-written FFTs
        // forward: rows and columns (deapodise/pad and the layout change per
        // cuFFT call), halo, then per group of 16 time samples the direction
        // gather, or after the zeroing of the k = 0 samples the tensor-core
        // gather (8+ time samples) and the direct one (items with few samples
        // per ray), then the residual rows or the forward epilogue
        const int gather_k =
            gd.dirs ? (gd.n_dfwd_items > 0 ? ng : 0)
                    : 1 + ng * (((m >= 8 && gd.n_fwd_tc_items > 0) ? 1 : 0) + (gd.n_fwd_items > 0 ? 1 : 0));
        const int fwd_k = (own_fft() ? 2 : 2 * calls) + 1 + gather_k + 1;
        const int fwd_f = (own_fft() ? 0 : calls) + (own_rows() ? 0 : 1);
        // adjoint: [row preparation], [zeros where planes are partly filled], one scatter
        // per group (direction path: the mixing and the scatter, and the fold of the
        // border), then columns and rows (per cuFFT call the layout change, on the
        // direction path, and the crop)
        const int zero_k = !gd.dirs && !planar_adj() && vec_groups(ug, zb, 4) < 4 ? 1 : 0;
        const int adj_k = (own_rows() ? 0 : 1) + zero_k + (gd.dirs ? 2 * ng + 1 : ng) +
                          (own_fft() ? 2 : (gd.dirs ? 2 : 1) * calls);
        const int adj_f = (own_rows() ? 0 : 1) + (own_fft() ? 0 : calls);
        // per outer iteration: titer inner steps per batch (forward, graddiv,
        // adjoint), one shrink per batch, the two-stage rho reduction
        *kern = titer * nbatch * (fwd_k + 1 + adj_k) + nbatch + 2;
        *ffts = titer * nbatch * (fwd_f + adj_f);
    }

    void kernel_cost(int which, double *bytes, double *flops) const {
        const double P = 2.0 * n;
        const double npts = (double)ntheta * (n - 1) * zb;  // polar samples per launch
        const int dpb = zb / nzp;
        switch (which) {
            case 0:  // gather: half-plane spectra in, complex rows out
                *bytes = (double)zb * m * P * (P / 2 + 1) * 8.0 + (double)zb * ntheta * n * 8.0;
                *flops = npts * (81.0 * 2.0 * m * 2.0 + 8.0 * m + 18.0 * 4.0);
                break;
            case 1:  // scatter: half row spectra in, Hermitian half planes out
                *bytes = (double)zb * ntheta * (n / 2 + 1) * 8.0 +
                         (double)zb * m * P * (P / 2 + 1) * 8.0;
                *flops = npts * (81.0 * 2.0 * m * 2.0 + 8.0 * m + 18.0 * 4.0);
                break;
            case 2:  // graddiv after the first inner step: u in, u out, w in (psi and mu when titer = 1)
                *bytes = (double)zb * slab * 8.0 + (titer > 1 ? 1.0 : 2.0) * 4.0 * dpb * gp * 4.0;
                *flops = (double)zb * slab * 60.0;
                break;
            case 6:  // graddiv of the first inner step: u in, u out, psi and mu in, w out
                *bytes = (double)zb * slab * 8.0 + (titer > 1 ? 3.0 : 2.0) * 4.0 * dpb * gp * 4.0;
                *flops = (double)zb * slab * 60.0;
                break;
            case 3:  // shrink: u_cur, u_old in, mu in, psi and mu out
                *bytes = (double)zb * slab * 8.0 + 3.0 * 4.0 * dpb * gp * 4.0;
                *flops = (double)dpb * gp * 80.0;
                break;
            case 4:    // padded forward FFT: u in; half rows of the n centre rows out, in again; P rows out
            case 5: {  // padded inverse FFT: P rows in; n centre rows out, in again; u read and written
                const double nimg = (double)zb * m, hp = (double)n + 1.0;
                const double half_rows = (double)n * hp * 8.0;
                *bytes = which == 4 ? nimg * (4.0 * n * n + 2.0 * half_rows + P * hp * 8.0)
                                    : nimg * (P * hp * 8.0 + 2.0 * half_rows + 8.0 * n * n);
                // 5 P log2 P flops per complex P-point transform: n/2 row pairs and n+1 columns
                *flops = nimg * (n / 2 + n + 1) * 5.0 * P * std::log2(P);
                break;
            }
            default:
                throw Error(RECTV_ERR_ARG, "rectv_kernel_cost: unknown kernel id");
        }
    }

    void launch_kernel(int which, int reps) {
        check_live();
        if (!session) throw Error(RECTV_ERR_STATE, "rectv_launch_kernel: needs a set-up session");
        if (which < 0 || which > 6) throw Error(RECTV_ERR_ARG, "rectv_launch_kernel: unknown kernel id");
        if ((which == 4 || which == 5) && !own_fft())
            throw Error(RECTV_ERR_ARG, "rectv_launch_kernel: no padded-grid FFT at this size");
        for (int r = 0; r < reps; ++r) {
            switch (which) {
                case 0: launch_gather_fwd(spec, rows, zb, gd, ug, gd.dirs ? &dir_tmap : &tc_tmap, stream); break;
                case 1: launch_scatter_adj(own_rows() ? rows_adj : rows, spec, zb, gd, ug, planar_adj(), stream); break;
                case 2:  // the inner steps after the first (w = mu - rho psi as stored by the last iteration)
                    launch_graddiv(U[cur], U[cur], U[(cur + 1) % 3], psi, mu, wdual, titer > 1 ? 2 : 0, rho_d, 0,
                                   nchunks, tv, stream);
                    break;
                case 3:  // overwrites the session's dual variables
                    launch_shrink(U[cur], U[cur], psi, mu, rho_d, 0.f, lambda0, 0, nchunks, tv, partials, stream);
                    break;
                case 4:  // padded-grid forward FFT of the batch (rows + columns)
                    if (pad_fft)
                        launch_pad_fft_fwd(U[cur], spec, zb, gd.deapod, fft_tw, fft_map, gd.err, ug, stream);
                    else
                        launch_gen_fft_fwd(U[cur], spec, zb, gd.deapod, fft_tw, gen_plan, ug, stream);
                    break;
                case 6:  // the first inner step (psi, mu in; stores w = mu - rho psi, unchanged values)
                    launch_graddiv(U[cur], U[cur], U[(cur + 1) % 3], psi, mu, wdual, titer > 1 ? 1 : 0, rho_d, 0,
                                   nchunks, tv, stream);
                    break;
                case 5:  // padded-grid inverse FFT (columns + rows), added into the scratch iterate
                    if (pad_fft)
                        launch_pad_fft_inv_accum(spec, U[(cur + 1) % 3], zb, 0.f, gd.deapod, fft_tw, fft_map, gd.err, ug,
                                                 stream);
                    else
                        launch_gen_fft_inv_accum(spec, U[(cur + 1) % 3], zb, 0.f, gd.deapod, fft_tw, gen_plan, ug,
                                                 stream);
                    break;
                default: throw Error(RECTV_ERR_ARG, "rectv_launch_kernel: unknown kernel id");
            }
        }
    }

    void check_adjoints(double *res, const float *g_h, const float *theta_h, const float *phi_h,
                        float lambda1_, float center) {
        check_live();
        if (nz != nzp)
            throw Error(RECTV_ERR_ARG, "rectv: check_adjoints needs nz == nzp (one chunk), as in rectv.cu:258");
        session = false;
        drop_graphs();
        set_geometry(theta_h, phi_h, center);
        ensure_plans();
        set_lambda1(lambda1_);
        CUDA_CHECK(cudaMemcpyAsync(gdata, g_h, sizeof(float) * (size_t)nz * ntheta * n, cudaMemcpyHostToDevice,
                                   stream));
        float *f = U[0], *fn = U[1];
        CUDA_CHECK(cudaMemsetAsync(f, 0, sizeof(float) * (size_t)nzc * slab, stream));
        CUDA_CHECK(cudaMemsetAsync(fn, 0, sizeof(float) * (size_t)nzc * slab, stream));
        CUDA_CHECK(cudaMemsetAsync(dot_out, 0, sizeof(double) * 8, stream));
        // rectv.cu:266-275
        adjoint(gdata, f, 1.0f);
        forward(f, nullptr, h1, 1.0f, 0);
        const long long nf = (long long)nzc * slab, ng = (long long)nz * ntheta * n;
        launch_dot(f, f, nf, dot_part, dot_parts(), dot_out + 0, stream);
        launch_dot(gdata, h1, ng, dot_part, dot_parts(), dot_out + 1, stream);
        launch_dot(h1, h1, ng, dot_part, dot_parts(), dot_out + 2, stream);
        // rectv.cu:278-288 (gradient into the spectrum scratch, float4 layout)
        float *h2 = reinterpret_cast<float *>(spec);
        TvGeo t1 = tv;
        t1.nchunks = 1;
        launch_gradient_ref(f, 0, h2, 0, 0, t1, stream);
        launch_divergent_ref(fn, h2, 1.0f, t1, stream);
        launch_dot(f, fn, nf, dot_part, dot_parts(), dot_out + 3, stream);
        const long long npts = (long long)(n + 1) * (n + 1) * (m + 1) * (nz + 1);
        launch_dot(h2, h2, npts, dot_part, dot_parts(), dot_out + 4, stream);
        launch_dot(fn, fn, nf, dot_part, dot_parts(), dot_out + 5, stream);
        double r[8];
        CUDA_CHECK(cudaMemcpyAsync(r, dot_out, sizeof(double) * 8, cudaMemcpyDeviceToHost, stream));
        CUDA_CHECK(cudaStreamSynchronize(stream));
        for (int i = 0; i < 6; ++i) res[i] += r[i];
    }
};

// Launch shapes chosen by the autotuner (engine.cu): slices per block of the
// tensor-core gather and persistent blocks of the tensor-core scatter (0: one
// per SM), with the measured times of the chosen shapes.
struct Tune {
    int zper = 64;
    int sc_grid = 0;
    double gather_ms = 0, scatter_ms = 0;
};

// Times the candidate launch shapes on a handle with a set-up session,
// applies the fastest (dropping captured graphs) and returns them; cached per
// (device, n, ntheta, m, slices per launch) unless force.
Tune autotune(Handle &h, bool force);

}  // namespace rectv
