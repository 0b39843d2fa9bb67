// Internal declarations shared by the CUDA translation units of librectv_gb300.
//
// Data layout in HBM (all float32 unless stated):
//   volume  u  [z][t][y][x]            z < nz, t < m (time samples), y,x < n
//   data    g  [z][theta][s]           s < n (detector)
//   dual    psi, mu: SoA [4][chunk][qz][qt][qy][qx], qz<=nzp, qt<=m, qy,qx<=n
//   spectra half planes of P x (n+1) complex, P = 2n, 16 (slice, time sample)
//           values per cell (UsGeo)
//   rows    [z][theta][n] complex (forward), [z][theta][n+2] real / n/2+1
//           complex in-place R2C (adjoint)
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <cufft.h>
#include <cstdint>
#include <stdexcept>
#include <string>
#include <vector>

namespace rectv {

// USFFT interpolation radius.  radonusfft.cu:11 evaluates to 4 for every n;
// kernels are specialised for it and the host checks the formula.
constexpr int kR = 4;
constexpr int kTaps = 2 * kR + 1;
// The USFFT kernels of the reference use this truncated value of pi
// (kernels_radonusfft.cuh:1).
constexpr double kPiUsfft = 3.1415926535;

struct Error : std::runtime_error {
    int code;
    Error(int c, const std::string &m) : std::runtime_error(m), code(c) {}
};

void cuda_check(cudaError_t e, const char *what, const char *file, int line);
void cufft_check(cufftResult e, const char *what, const char *file, int line);
#define CUDA_CHECK(x) ::rectv::cuda_check((x), #x, __FILE__, __LINE__)
#define CUFFT_CHECK(x) ::rectv::cufft_check((x), #x, __FILE__, __LINE__)
#define LAUNCH_CHECK(what) ::rectv::cuda_check(cudaGetLastError(), what, __FILE__, __LINE__)

// Geometry of the USFFT kernels.
struct UsGeo {
    int n, ntheta, m;   // detector width, projections, time samples
    int P;              // oversampled grid side 2n
    float tn;           // (float)(2n)
    float inv2n;        // 1/(2n)
    float wexp;         // pi^2/mu
    float cw;           // (pi/mu)/n : gather weight scale and 1/n of gather
    int T;              // tile core side
    int NT;             // tiles per side P/T
    // launch shapes chosen per problem (tunable): slices per block of the
    // tensor-core gather (1..64), and blocks of the persistent tensor-core
    // scatter (0: one per SM)
    int zper;
    int sc_grid;
    // Vector layout of the spectra: the half planes of 16 (slice, time sample)
    // pairs are stored together, cell by cell: [plane][row][column][16] complex
    // over the window rows [-kVH, P + kVH) x columns [-kVH, n + kVR].  One plane
    // holds tg time samples (1, 2, 4, 8 or 16, at least m) of zs = 16 / tg
    // slices; with m > 16 a slice takes jg = ceil(m / 16) planes of 16 samples.
    // The halo around rows [0, P) x columns [0, n] holds the periodic
    // spectrum's wrapped and Hermitian-mirrored cells, so that every tile's
    // footprint is one rectangular box.
    int tg, zs, jg;
    int vp;             // row pitch in cells: n + 1 + kVH + kVR
    int vrows;          // P + 2 kVH
    long long vplane;   // complex elements per plane
};

// halo cells of the vector layout: a stencil and its mirror image reach from 4
// cells before to 5 cells after the origin; the per-ray gather's footprints
// read up to 16 columns past the half plane
constexpr int kVH = 8, kVR = 16;
__host__ __device__ inline int vec_planes(const UsGeo &g, int zb) {  // planes of zb slices
    return g.jg > 1 ? zb * g.jg : (zb + g.zs - 1) / g.zs;
}
// planes of slice z, group jgrp of 16 time samples, and the slice's first entry there
__host__ __device__ inline long long vec_plane_of(const UsGeo &g, int z, int jgrp) {
    return g.jg > 1 ? (long long)z * g.jg + jgrp : z / g.zs;
}
__host__ __device__ inline int vec_entry(const UsGeo &g, int z) { return g.jg > 1 ? 0 : (z % g.zs) * g.tg; }
// floats per row of the planar images cuFFT transforms (even: 16-byte rows), in complex
__host__ __device__ inline int planar_pitch(int n) { return n + 2 + (n & 1); }
// slice and time sample of entry v of plane pl
__host__ __device__ inline int vec_slice(const UsGeo &g, int pl, int v) {
    return g.jg > 1 ? pl / g.jg : pl * g.zs + v / g.tg;
}
__host__ __device__ inline int vec_time(const UsGeo &g, int pl, int v) {
    return g.jg > 1 ? (pl % g.jg) * 16 + v : v & (g.tg - 1);
}

// whether entry v of plane pl holds data (of zb slices); a run of 2, 4, 8 or 16
// entries from a multiple of its length on holds some where its first one does
__host__ __device__ inline bool vec_live(const UsGeo &g, int zb, int pl, int v) {
    return g.jg > 1 ? (pl % g.jg) * 16 + v < g.m : v < (zb - pl * g.zs) * g.tg && (v & (g.tg - 1)) < g.m;
}
// groups of C entries of a cell that hold data in any plane: fewer than all with
// 9 .. 15 time samples, or with less than a plane's slices
inline int vec_groups(const UsGeo &g, int zb, int C) {
    return g.jg > 1 ? 16 / C : (((zb < g.zs ? zb : g.zs) - 1) * g.tg + g.m + C - 1) / C;
}

// Weights of one polar sample restricted to one 16x16 tile of the adjoint
// plan (zero outside the sample's 9x9 stencil), with its ray and the mask of
// tile rows its stencil covers (thm = theta << 16 | mask, theta < 65536),
// its detector index and row factor (-1)^(k+1) shiftadj(k) (pi/mu)/n.
struct AdjRec {
    float wx[16];
    float wy[16];
    int thm;
    int k;
    float2 sf;
};

// Per-angle constants uploaded at geometry set-up.
struct GeoDev {
    float2 *sincos = nullptr;    // [ntheta] (sin, cos) of theta
    float2 *kmat = nullptr;      // [ntheta][m]  K'(theta,j) = ntheta/sqrt(m) sum_i phi_i(theta) conj(phi_i(t_j))
    float2 *shiftfwd = nullptr;  // [n]
    float2 *shiftadj = nullptr;  // [n]
    float *deapod = nullptr;     // [n] exp(mu (x-n/2)^2)
    uint32_t *fwd_pts = nullptr; // point ids theta*n+k sorted by tile
    int4 *fwd_items = nullptr;   // (tile, start, count, 0): direct gather (k_gather_fwd)
    int n_fwd_items = 0;
    int4 *fwd_tc_items = nullptr; // (tile, start, count, rays): tensor-core gather (k_gather_tc)
    int n_fwd_tc_items = 0;
    uint32_t *adj_pts = nullptr; // point ids, one entry per tile a stencil touches
    int4 *adj_items = nullptr;   // (tile, start, count, 0), whole tiles
    int n_adj_items = 0;
    int *err = nullptr;          // device counter of host/device bin disagreements
    int *sc_next = nullptr;      // unit counter of the tensor-core scatter, zeroed by each launch
    bool tc_scatter = false;     // adjoint time-sample mixing on the tensor cores (k_scatter_tc)
    AdjRec *adj_recs = nullptr;  // geometry records of adj_pts (tensor-core scatter only)
    int n_adj_busy = 0;          // leading adj_items with samples (items are sorted by count)
    // tensor-core scatter tables: each busy item's entries in runs of whole
    // rays (at most one MMA batch of rays and scatter_tc_table_capacity()
    // entries); item i owns tables [adj_tab_base[i],
    // adj_tab_base[i+1]); adj_tabs = (first entry, count, segmentation offset
    // and size in 32-bit words); adj_info = the tables' ray segmentation
    int4 *adj_tabs = nullptr;
    int *adj_tab_base = nullptr;
    uint32_t *adj_info = nullptr;
    int n_adj_tabs = 0;
    // direction path (gather_dir.cu, scatter_dir.cu, DirPlan): sincos then holds
    // one (sin, cos) per direction, adj_pts / adj_items the position pairs
    // touching each 16x16 tile of the window
    bool dirs = false;
    int ndir = 0;
    int *dray_start = nullptr;    // [ndir + 1]
    uint32_t *drays = nullptr;    // theta | opposite << 31
    float *dtau = nullptr;        // per ray: offset across the direction (DirPlan::tau)
    float2 *dkmat = nullptr;      // K' in the order of drays, [ray][max(tg, 16 jg)], zero past m
    float4 *demix = nullptr;      // the adjoint's mixed rays per (plane, position pair): dir_mix_bytes
    int demix_slices = 0;
    uint32_t *dfwd_pos = nullptr; // position pairs d*(n/2) + q - 1 sorted by origin tile
    int4 *dfwd_items = nullptr;   // (tile, start, count, 0)
    int n_dfwd_items = 0;
};

// Host-side angle plan (built in plan.cpp).
struct HostPlan {
    std::vector<float2> sincos;
    std::vector<uint32_t> fwd_pts;
    std::vector<int4> fwd_items;
    std::vector<int4> fwd_tc_items;
    std::vector<uint32_t> adj_pts;
    std::vector<int4> adj_items;
};

// Forward work items hold whole rays of one tile and at most fwd_cap samples;
// an item with at least tc_min_spr samples per ray goes to the tensor-core
// gather (tc_min_spr < 0: none does).
HostPlan build_plan(const float *theta, int n, int ntheta, int T, int fwd_cap, float tc_min_spr);

// Rays grouped by direction (theta modulo pi), for scans that revisit their
// angles over several half-turns: the rays of one direction sample the same
// positions, so the USFFT interpolates once per position (scatter_dir.cu).
struct DirPlan {
    int ndir = 0;
    std::vector<float2> sincos;     // [ndir] (sin, cos) of each direction's representative ray
    std::vector<int> ray_start;     // [ndir + 1]: rays of direction d are rays[ray_start[d] .. ray_start[d+1])
    std::vector<uint32_t> rays;     // theta index | opposite << 31 (sample k of an opposite ray is position n - k)
    std::vector<float> tau;         // per ray (order of rays): its samples' offset across the direction, in
                                    // grid cells per unit of (q - n/2)/n
    std::vector<uint32_t> fwd_pos;  // position pairs d*(n/2) + q - 1 (1 <= q <= n/2) sorted by the tile of the stencil origin
    std::vector<int4> fwd_items;    // (tile, start, count, 0): at most fwd_cap positions of one tile
    std::vector<uint32_t> adj_pos;  // pairs, one entry per tile of the vector layout's window their cells touch
    std::vector<int4> adj_items;    // (tile, start, count, 0), one per tile
};
// Defaults of the direction path: rays are grouped when their samples agree
// within kDirTolCells grid cells, and the path is taken when the rays average
// at least kDirMinGroup per direction.
constexpr double kDirTolCells = 2e-3;
constexpr double kDirMinGroup = 2.5;
// Groups rays whose sample positions agree within tol_cells grid cells.
// Returns false (plan unused) when the rays average fewer than min_group per
// direction or there are 65536 directions or more.
bool build_dir_plan(const float *theta, int n, int ntheta, int T, int fwd_cap, double tol_cells, double min_group,
                    DirPlan &dp);
// its first step, the rays of each direction (no positions)
bool group_directions(const float *theta, int n, int ntheta, double tol_cells, double min_group, DirPlan &dp);

// 32-bit words of an adjoint table's ray segmentation with nseg rays: [0]
// nseg, [4 + 8 s + w] the table rows [lo, hi) of ray s that cover rows 2w,
// 2w+1 of the tile (lo | hi << 16), then the first row of every ray and the
// table size as 16-bit values; padded to 16 bytes.
__host__ __device__ constexpr int adj_info_words(int nseg) { return (4 + 8 * nseg + (nseg + 2) / 2 + 3) & ~3; }

int sm_count();  // of the current device (fft_kernels.cu)

// ---- USFFT kernel launchers (usfft_kernels.cu) ----
// deapodised, padded and modulated images for cuFFT's R2C (planar_pitch)
void launch_deapod_pad(const float *u, float *planar, int nimg, const float *deapod, const UsGeo &g,
                       cudaStream_t s);
void launch_gather_fwd(const float2 *spec, float2 *rows, int zb, const GeoDev &gd, const UsGeo &g,
                       const CUtensorMap *tmap, cudaStream_t s);
void launch_finish_fwd(const float2 *rows, const float *gdata, float *out, int zb, float tau,
                       int residual, const UsGeo &g, cudaStream_t s);
// the same from the real output of the rows' C2R inverse (rows of 2 (n/2+1) floats)
void launch_finish_fwd_real(const float *rows, const float *gdata, float *out, int zb, float tau, int residual,
                            const UsGeo &g, cudaStream_t s);
void launch_adj_prep(const float *h, float *rowsr, int zb, const UsGeo &g, cudaStream_t s);
// the adjoint's Hermitian half planes from the row spectra; planar (per-ray kernels
// only): as planar images [zb m][P][planar_pitch] for cuFFT
void launch_scatter_adj(const float2 *rowsc, float2 *spec, int zb, const GeoDev &gd,
                        const UsGeo &g, bool planar, cudaStream_t s);
// cropped, deapodised and added into u, from cuFFT's C2R output (rows of 2 planar_pitch floats)
void launch_crop_accum_real(const float *out, float *u, int zb, float tau, const float *deapod, const UsGeo &g,
                            cudaStream_t s);
// tensor-core gather (gather_tc.cu): items of fwd_tc_items, time samples
// [16 jgrp, 16 jgrp + 16)
void launch_gather_tc(float2 *rows, int zb, const GeoDev &gd, const UsGeo &g, const CUtensorMap &tmap, int jgrp,
                      cudaStream_t s);
void gather_tc_prepare();
// tensor-core scatter (scatter_tc.cu): all adjoint items, time samples [16 jgrp, 16 jgrp + 16),
// added into the zeroed Hermitian half planes of the C2R inverse
void launch_scatter_tc(const float2 *rowsc, float2 *spec, int zb, const GeoDev &gd, const UsGeo &g, int jgrp,
                       bool planar, cudaStream_t s);
void scatter_tc_prepare();
void launch_adj_records(AdjRec *recs, const GeoDev &gd, const UsGeo &g, cudaStream_t s);
// entries per scatter table, and the 32-bit words of a table's segmentation
// with nseg rays (count, per-warp sample ranges, ray starts)
int scatter_tc_table_capacity();
int scatter_tc_batch_rays();  // rays per tensor-core batch
int scatter_tc_info_words(int nseg);
// fill adj_info from the records (after launch_adj_records)
void launch_adj_tabinfo(const GeoDev &gd, cudaStream_t s);
// direction path (gather_dir.cu, scatter_dir.cu): the Hermitian half rows
// [z][theta][n/2+1] of all rays from the spectra in the vector layout, and the
// adjoint: half rows into the Hermitian half planes in the vector layout
void launch_gather_dir(float2 *hrows, int zb, const GeoDev &gd, const UsGeo &g, const CUtensorMap &vmap,
                       cudaStream_t s);
void launch_scatter_dir(const float2 *rowsc, float2 *spec, int zb, const GeoDev &gd, const UsGeo &g, cudaStream_t s);
// TMA descriptors of the gathers' footprints in the vector layout (npl planes):
// the direction path's 25x25 cells, the per-ray tensor-core gather's 24x24
// cells with 128-byte swizzle
void make_vec_gather_map(CUtensorMap *map, float2 *spec, int npl, const UsGeo &g);
void make_vec_gather_tc_map(CUtensorMap *map, float2 *spec, int npl, const UsGeo &g);
// fills the halo of the forward spectra (right: columns past the half plane, 5
// on the direction path, kVR per ray)
void launch_vec_halo(float2 *spec, int npl, int right, const UsGeo &g, cudaStream_t s);
// cuFFT's spectra of slices z0 .. z0 + nz - 1 (planar, rows of planar_pitch
// complex, image (z - z0) m + t) into the vector layout, and back
void launch_planar_to_vec(const float2 *planar, float2 *spec, int z0, int nz, const UsGeo &g, cudaStream_t s);
constexpr int kLayoutCells = 128;  // cells of a row per block of either
void launch_vec_to_planar(const float2 *spec, float2 *planar, int z0, int nz, const UsGeo &g, cudaStream_t s);
void gather_dir_prepare();    // kernel attributes; once, outside stream capture
void scatter_dir_prepare();
int dir_fwd_capacity();       // position pairs per forward item
// work items of the adjoint over npz planes: (tile, start, count, first plane |
// end plane << 16) of a plan's (tile, start, count), the most work first
std::vector<int4> dir_adj_work(const std::vector<int4> &tiles, int npz);
std::vector<int4> dir_fwd_work(const std::vector<int4> &items, int npz);  // and of the forward gather
size_t dir_mix_bytes(const UsGeo &g, int zb, int ndir);  // the adjoint's per-position mixing buffer
// hand-written 2D FFTs of the zero-padded grids in the vector layout
// (fft_kernels.cu), P = 2n a power of two in [256, 2048]: forward =
// deapodise/pad/modulate + R2C (halo not filled); inverse = C2R of the
// Hermitian half planes (overwritten) + crop/deapodise, u += tau * ...
bool pad_fft_supported(int P);
void pad_fft_prepare();
std::vector<float2> pad_fft_twiddles(int P);
// TMA descriptor of the column passes over the spectra (npl planes)
void make_vec_fft_map(CUtensorMap *map, float2 *spec, int npl, const UsGeo &g);
void launch_pad_fft_fwd(const float *u, float2 *spec, int zb, const float *deapod, const float2 *tw,
                        const CUtensorMap &map, int *err, const UsGeo &g, cudaStream_t s);
void launch_pad_fft_inv_accum(float2 *spec, float *u, int zb, float tau, const float *deapod, const float2 *tw,
                              const CUtensorMap &map, int *err, const UsGeo &g, cudaStream_t s);
// mixed-radix passes for grid sides that are no power of two (fft_general.cuh,
// fft_general_fwd.cu, fft_general_inv.cu): even lengths 32 .. 2048 with prime
// factors up to 13, 17 or 19
struct GenPlan {
    int P, np;           // length, passes
    int R[6], Ns[6];     // radix of a pass, product of the radices before it
    uint32_t magic[6];   // ceil(2^32 / Ns): j / Ns = mulhi(j, magic) for j < 2^16
    int toff[6];         // first twiddle of a pass: exp(-2 pi i r k / (Ns R)) at toff + (r - 1) Ns + k
};
bool gen_fft_plan(int P, GenPlan *p);
std::vector<float2> gen_fft_twiddles(const GenPlan &p);
void gen_fft_fwd_prepare();
void gen_fft_inv_prepare();
size_t gen_rows_smem(int P, int C);
size_t gen_cols_smem(int P, int C);
int gen_width(int P);
int gen_resident(size_t smem, int threads);
void launch_gen_fft_fwd(const float *u, float2 *spec, int zb, const float *deapod, const float2 *tw, const GenPlan &p,
                        const UsGeo &g, cudaStream_t s);
void launch_gen_fft_inv_accum(float2 *spec, float *u, int zb, float tau, const float *deapod, const float2 *tw,
                              const GenPlan &p, const UsGeo &g, cudaStream_t s);
// launch_resid_rows, p and tw of length n
void launch_gen_resid(const float2 *rows, const float *gdata, float2 *out, const float2 *tw, const GenPlan &p, int zb,
                      bool half, const UsGeo &g, cudaStream_t s);
// fused residual rows of the inner step (fft_kernels.cu), n a power of two in
// [256, 1024]: gathered rows [z][theta][n] and data g -> the adjoint's row
// spectra [z][theta][n/2+1] (inverse row FFT, residual, fftshift, R2C)
bool resid_rows_supported(int n);
int resid_runs(int zb, int ntheta);  // runs of rows that are paired among themselves
// half: the rows hold the Hermitian half k = 0 .. n/2 (direction path)
void launch_resid_rows(const float2 *rows, const float *gdata, float2 *out, const float2 *tw_n, int zb, bool half,
                       const UsGeo &g, cudaStream_t s);
// out = tau R u from the Hermitian half rows, on the same transforms
void launch_fwd_rows(const float2 *hrows, float *out, float tau, const float2 *tw_n, int zb, const UsGeo &g,
                     cudaStream_t s);
void launch_gen_fwd_rows(const float2 *hrows, float *out, float tau, const float2 *tw, const GenPlan &p, int zb,
                         const UsGeo &g, cudaStream_t s);
size_t gather_tc_smem();
int gather_tc_table_capacity();
void usfft_prepare();  // kernel attributes; call once, outside stream capture
int table_capacity();  // samples per gather work item

// ---- TV / ADMM kernel launchers (tv_kernels.cu) ----
struct TvGeo {
    int n, m, nzp, nchunks;  // chunks processed: nchunks of nzp slices
    long long vol_slab;      // n*n*m
    long long gp;            // grid points per chunk (n+1)^2 (m+1)(nzp+1)
    long long comp_stride;   // elements between SoA components = nchunks_total*gp
    float sg;                // gradient scale 1/(2 cbrt2 lambda1/2)
    float sd;                // divergence scale 1/(4 cbrt2 lambda1/2)
    float lambda1;
};

// u_out = u_in - 0.5 * div(rho (G u_in - psi) + mu) for chunks [c0, c0+nchunks);
// mode 0 reads psi and mu, mode 1 also stores w = mu - rho psi (psi's layout),
// mode 2 reads w only (psi, mu and rho unchanged since the mode-1 step)
void launch_graddiv(const float *u_in, const float *u_old, float *u_out, const float *psi,
                    const float *mu, float *w, int mode, const float *rho, int c0, int nchunks_total,
                    const TvGeo &t, cudaStream_t s);
// shrink + dual update + residual sums into per-block partials
// (rho is read from rho_d, or is the argument where rho_d is null)
int launch_shrink(const float *u_cur, const float *u_old, float *psi, float *mu, const float *rho_d, float rho,
                  float lambda0, int c0, int nchunks_total, const TvGeo &t, double *partials,
                  cudaStream_t s);
int shrink_blocks(const TvGeo &t, int nchunks);
// sum partials in fixed order, apply the rho rule, append a stats row at *ctr
// (two fixed-order stages; stage1 holds 3*reduce_stage1_parts() doubles)
void launch_reduce_rho(const double *partials, int nparts, double *stage1, float *rho, double *stats, int *ctr,
                       int cap, cudaStream_t s);
int reduce_stage1_parts();
// reference-layout gradient / divergence for the operator API and check_adjoints
// fm points at slab zbase-1 of the extended chunk (zbase = 1 when fm holds
// the two halo slabs, 0 when it holds the chunk only and flgl = flgr = 0)
void launch_gradient_ref(const float *fm, int zbase, float *h2, int flgl, int flgr, const TvGeo &t,
                         cudaStream_t s);
void launch_divergent_ref(float *fn, const float *h2, float tau, const TvGeo &t, cudaStream_t s);
// FP64 dot products: out[0] += sum a*b over count (a==b allowed); deterministic two-pass
void launch_dot(const float *a, const float *b, long long count, double *partials, int nparts,
                double *out, cudaStream_t s);
int dot_parts();

// ---- filtered backprojection helpers (io_kernels.cu) ----
void launch_filter_rows(float2 *rowsc, const float *w, long long nrows, int n, cudaStream_t s);
void launch_fbp_mask(const float *u, float *out, int nslices, int n, int m, float r, cudaStream_t s);

// ---- data ingest (io_kernels.cu) ----
void preprocess(float *out, const void *data, const void *dark, const void *flat, int dtype, int ntheta, int nz,
                int n, int ndark, int nflat);

}  // namespace rectv
