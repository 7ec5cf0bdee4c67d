// Periodic cell-list radius graph for B200 (sm_100a).
//
// Replaces the reference's radius_graph_pbc_cuda_impl_ex
// (dynamis_state/src/csrc/graph/radius_graph_kernels.cu:479-934) behind the C ABI in dynb.h.
//
// Pipeline (one stream, no host synchronisation inside the plan):
//   rg_wrap        wrap positions into the unit cell, classify which periodic images each atom
//                  needs, bounding box of all images                     (ref :596-605, :18-67)
//   rg_target_bbox bounding box of the targets (only with a target subset)
//                  the last block of these two chooses the cell grid, unless the host could (ref :662-692)
//   rg_bin_count   histogram of images / targets per cell (atomics; part of rg_wrap with a grid from the host)
//                                                                        (ref :146-171)
//   scan           cell starts
//   rg_bin_scatter provisional slot inside each cell (atomic rank)
//   rg_bin_finalize deterministic order inside each cell, write packed source / target records
//   rg_count       per-target degree and hit bits                        (ref :197-258)
//   scan           edge offsets + total
//   rg_fillmask    edges from the hit bits of the count pass             (ref :282-442)
//   rg_pair        edges of groups whose candidate list is too long for hit bits
//
// The edge SET is fixed by three predicates that are kept expression-for-expression identical to
// the reference (same operand order, compiled with the same default FMA contraction): the wrap,
// the periodic-image test with the image position, and d2 <= r2 && d2 > 1e-8f.  The cell grid
// only decides which pairs are examined and is free to differ.
//
// Work decomposition of the cell scan: one warp owns a group of group_cells x group_cells_y cells (x, y)
// and all targets inside.  It flattens the contiguous runs of neighbouring source records (one run
// per (y, z) row, one lane per run) into one list, the same in every pass.  rg_count tests the targets one at a time against
// candidates in registers; the writers find the edges in its hit bits; rg_pair tests the targets of long lists two at a time
// against candidates in shared memory (ballot + popc compaction, hits parked in per-target lists).  Edges are written 32 at
// a time so that the 8-byte index stores of a warp cover one contiguous 256-byte run.  With a target subset the
// source images are first clipped to the targets' bounding box grown by the cutoff.

#include "common.cuh"
#include "clear.cuh"
#include "scan.cuh"

#include <math.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

namespace dynb {

// ------------------------------------------------------------------------------------------
// Device-resident plan header.  The first 64 bytes mirror dynb_rg_header.
// ------------------------------------------------------------------------------------------
struct DevHeader {
    unsigned long long E;
    unsigned long long M;
    uint32_t status;
    uint32_t max_degree;
    int32_t nx, ny, nz;
    int32_t group_cells;
    unsigned long long num_groups;
    long long reserved[2];
    // ---- internal -----------------------------------------------------------------------
    uint32_t ncell_plus1;
    int32_t pad;
    int32_t gx;
    int32_t group_cells_y;  // cells per warp work item along y (1 or 2)
    unsigned long long bb_min[3];  // ordered-integer images of the bounding box
    unsigned long long bb_max[3];
    unsigned long long tb_min[3];  // the same of the wrapped targets (target subsets only)
    unsigned long long tb_max[3];
    uint32_t arrived;              // blocks of the pass that chooses the grid that are done
    double gmin[3];
    double res_inv;
    double clip_lo[3];  // source images outside [clip_lo, clip_hi] cannot reach any target and are dropped
    double clip_hi[3];
    uint32_t active_groups;  // entries of the list of groups that hold targets (target subsets only)
    uint32_t halo_groups;    // halo marking: entries of halo_list
    float test_near, test_lo, test_hi;  // double positions: thresholds of the float test (float_test)
    uint32_t test_equal_is_near;
    uint32_t count_next;      // count pass: groups taken behind every warp's first
};
static_assert(offsetof(DevHeader, ncell_plus1) == sizeof(dynb_rg_header), "public header prefix mismatch");

constexpr uint32_t RG_FATAL = DYNB_RG_SRC_OVERFLOW | DYNB_RG_BAD_TARGET | DYNB_RG_NONFINITE | DYNB_RG_SHIFT_RANGE;

template <typename T> struct Geom {
    T inv[9];
    T cell[9];
    T cf[3];
    int rep[3];
    int pbc[3];
};

// Rounded-once helpers (no contraction across them).
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float floor_t(float a) { return floorf(a); }
__device__ __forceinline__ double floor_t(double a) { return floor(a); }
__device__ __forceinline__ bool finite_t(float a) { return isfinite(a); }
__device__ __forceinline__ bool finite_t(double a) { return isfinite(a); }

__device__ __forceinline__ unsigned long long ordered_any(float v) { return (unsigned long long)ordered_u32(v); }
__device__ __forceinline__ unsigned long long ordered_any(double v) { return ordered_u64(v); }
// the same keys in their natural width: 32 bits for float (one REDUX instruction reduces them over a warp)
__device__ __forceinline__ uint32_t ordered_key(float v) { return ordered_u32(v); }
__device__ __forceinline__ unsigned long long ordered_key(double v) { return ordered_u64(v); }
template <typename T> __device__ __forceinline__ double unordered_any(unsigned long long u);
template <> __device__ __forceinline__ double unordered_any<float>(unsigned long long u) { return (double)unordered_f32((uint32_t)u); }
template <> __device__ __forceinline__ double unordered_any<double>(unsigned long long u) { return unordered_f64(u); }

// K = 3 inner product exactly as an fp32/fp64 GEMM accumulates it: k-sequential FMA chain.
// The reference wraps positions with two at::mm calls (radius_graph_kernels.cu:602,605).
template <typename T> __device__ __forceinline__ T dot3_gemm(T a0, T b0, T a1, T b1, T a2, T b2)
{
    return fma_rn(a2, b2, fma_rn(a1, b1, mul_rn(a0, b0)));
}

// Image position, same expression shape as the reference's write_pbc_images_kernel (:122-128).
template <typename T>
__device__ __forceinline__ void image_pos(const Geom<T>& g, T px, T py, T pz, int dx, int dy, int dz, T& x, T& y, T& z)
{
    T shift_x = (T)dx * g.cell[0] + (T)dy * g.cell[3] + (T)dz * g.cell[6];
    T shift_y = (T)dx * g.cell[1] + (T)dy * g.cell[4] + (T)dz * g.cell[7];
    T shift_z = (T)dx * g.cell[2] + (T)dy * g.cell[5] + (T)dz * g.cell[8];
    x = px + shift_x;
    y = py + shift_y;
    z = pz + shift_z;
}

// image flags of an atom: bit d = "may be shifted up along d", bit 3+d = "may be shifted down along d"

template <typename T>
__device__ __forceinline__ uint32_t cell_of(const DevHeader& h, T x, T y, T z)
{
    const T ri = (T)h.res_inv;
    int cx = (int)floor_t((x - (T)h.gmin[0]) * ri);
    int cy = (int)floor_t((y - (T)h.gmin[1]) * ri);
    int cz = (int)floor_t((z - (T)h.gmin[2]) * ri);
    cx = max(0, min(cx, h.nx - 1));
    cy = max(0, min(cy, h.ny - 1));
    cz = max(0, min(cz, h.nz - 1));
    return (uint32_t)cx + (uint32_t)h.nx * ((uint32_t)cy + (uint32_t)h.ny * (uint32_t)cz);
}

constexpr int RG_MASK_SLOTS = 16;  // hit bits kept per lane and target (candidate lists up to 512 records)

// The cell grid of a plan and the shape of a warp's work item.  Chosen on the device from the bounding box of
// the data (rg_choose_grid_device), or on the host from the cell when the box is periodic in all directions and every
// atom is a target (the images then fill a known box and the first two passes run as one).
struct GridChoice {
    int nx, ny, nz, pad, group_cells, group_cells_y, gx;
    uint32_t ncell_plus1;
    unsigned long long num_groups;
    double gmin[3];
    double res_inv;
};

// Cells of edge radius/1.99 scanned +-2 (as the reference, :662,776) unless that would need more than
// cell_capacity cells; then the cells grow, and once they are wider than the cutoff the scan shrinks to +-1.
__host__ __device__ inline void rg_choose_shape(GridChoice& gc, double avg, int cand_capacity, bool allow_wide);
// avg: expected sources per cell, for the shape of the work items.
__host__ __device__ inline void rg_choose_grid(const double lo[3], const double ext[3], double radius, long long cell_capacity,
                                               int cand_capacity, double M, double sources_per_volume, bool allow_wide, GridChoice& gc)
{
    double res = radius / 1.99;
    long long n[3];
    for (int it = 0; it < 400; it++) {
        double tot = 1.0;
        for (int k = 0; k < 3; k++) {
            double c = ceil(ext[k] / res);
            if (!(c >= 1.0)) c = 1.0;
            if (c > 2.0e9) c = 2.0e9;
            n[k] = (long long)c;
            tot *= c;
        }
        if (tot + 1.0 <= (double)cell_capacity) break;
        res *= 1.2;
        if (it == 399) { n[0] = n[1] = n[2] = 1; }
    }
    gc.nx = (int)n[0]; gc.ny = (int)n[1]; gc.nz = (int)n[2];
    const long long ncell = n[0] * n[1] * n[2];
    gc.ncell_plus1 = (uint32_t)(ncell + 1);
    const int pad = (res >= radius * 1.001) ? 1 : 2;
    gc.pad = pad;
    for (int k = 0; k < 3; k++) gc.gmin[k] = lo[k];
    gc.res_inv = 1.0 / res;
    rg_choose_shape(gc, sources_per_volume > 0.0 ? sources_per_volume * res * res * res : M / (double)ncell, cand_capacity, allow_wide);
}

// cells per warp work item (Sx along x, Sy along y): as many target cells as possible while the
// expected dense candidate list stays within 1.5 shared-memory lists
// allow_wide: the mean is taken over a box that the sources fill.  With a target subset the grid can span far more
// cells than hold sources (a subdomain whose wrapped targets sit on both sides of the periodic box), the mean then
// says nothing about the lists, and the wide shapes — which sit just under the limit of the hit bits — stay out.
constexpr int RG_SHAPES = 5;   // 4 x 2, 3 x 2, 2 x 2, 2 x 1, 1 x 1
__host__ __device__ inline void rg_shape(int c, int& sx, int& sy)
{
    sx = c == 0 ? 4 : (c == 1 ? 3 : (c < 4 ? 2 : 1));
    sy = c < 3 ? 2 : 1;
}
__host__ __device__ inline bool rg_shape_fits(int c, int pad, double avg, int cand_capacity, bool allow_wide)
{
    int sx, sy;
    rg_shape(c, sx, sy);
    if ((sy + 2 * pad) * (2 * pad + 1) > 32) return false;  // one lane per candidate run
    if (sx > 2 && !allow_wide) return false;
    const double Lexp = (double)(sx + 2 * pad) * (double)(sy + 2 * pad) * (double)(2 * pad + 1) * (avg > 1e-6 ? avg : 1e-6);
    return (sx > 2) ? (1.15 * Lexp + 4.0 * sqrt(Lexp) <= (double)(RG_MASK_SLOTS * 32)) : (Lexp <= 1.5 * (double)cand_capacity);
}
__host__ __device__ inline void rg_set_shape(GridChoice& gc, int c)
{
    int sx, sy;
    rg_shape(c, sx, sy);
    if (sx > gc.nx) sx = gc.nx;
    if (sy > gc.ny) sy = gc.ny;
    gc.group_cells = sx;
    gc.group_cells_y = sy;
    gc.gx = (gc.nx + sx - 1) / sx;
    const int gy = (gc.ny + sy - 1) / sy;
    gc.num_groups = (unsigned long long)gc.gx * (unsigned long long)gy * (unsigned long long)gc.nz;
}
__host__ __device__ inline void rg_choose_shape(GridChoice& gc, double avg, int cand_capacity, bool allow_wide)
{
    // measured on B200 (1 M-atom liquid, 1 M-atom fcc): 2 x 2 cells per warp beat 2 x 1 and 1 x 1 even when the
    // candidate list then needs a second chunk, and wider groups (3 or 4 cells along x, which lengthens every
    // candidate run instead of adding runs) beat 2 x 2 as long as the list keeps its hit bits: the work per group
    // (decode, run table, staging) is shared by more targets.  A list longer than the hit bits sends its group to
    // the slow writer, so the wide shapes are taken only with a margin (15 % on the mean density, four standard
    // deviations of a Poisson count) under that limit.
    int best = 0;
    while (best < RG_SHAPES - 1 && !rg_shape_fits(best, gc.pad, avg, cand_capacity, allow_wide)) best++;
    rg_set_shape(gc, best);
}

__host__ __device__ inline void rg_store_grid(DevHeader& h, const GridChoice& gc)
{
    h.nx = gc.nx; h.ny = gc.ny; h.nz = gc.nz;
    h.ncell_plus1 = gc.ncell_plus1;
    h.pad = gc.pad;
    for (int k = 0; k < 3; k++) h.gmin[k] = gc.gmin[k];
    h.res_inv = gc.res_inv;
    h.group_cells = gc.group_cells;
    h.group_cells_y = gc.group_cells_y;
    h.gx = gc.gx;
    h.num_groups = gc.num_groups;
}

// cell_of for a grid that travels as a kernel argument: the same expression on the same numbers
template <typename T>
__device__ __forceinline__ uint32_t cell_of(const GridChoice& h, T x, T y, T z)
{
    const T ri = (T)h.res_inv;
    int cx = (int)floor_t((x - (T)h.gmin[0]) * ri);
    int cy = (int)floor_t((y - (T)h.gmin[1]) * ri);
    int cz = (int)floor_t((z - (T)h.gmin[2]) * ri);
    cx = max(0, min(cx, h.nx - 1));
    cy = max(0, min(cy, h.ny - 1));
    cz = max(0, min(cz, h.nz - 1));
    return (uint32_t)cx + (uint32_t)h.nx * ((uint32_t)cy + (uint32_t)h.ny * (uint32_t)cz);
}

// ------------------------------------------------------------------------------------------
// rg_wrap
// ------------------------------------------------------------------------------------------
// Squared distance with the rounding every pass must share (the contraction nvcc applies to
// dx*dx + dy*dy + dz*dz, written out so that no pass depends on the compiler's choice):
// fma(dz, dz, fma(dx, dx, dy * dy)).
template <typename T> __device__ __forceinline__ T dist2(T ax, T ay, T az, T sx, T sy, T sz)
{
    const T dx = sub_rn(ax, sx), dy = sub_rn(ay, sy), dz = sub_rn(az, sz);
    return fma_rn(dz, dz, fma_rn(dx, dx, mul_rn(dy, dy)));
}
// The same for two fp32 candidates at once with the packed fp32 instructions of sm_100 (each half is an
// IEEE round-to-nearest operation, so the halves equal dist2<float> bit for bit); one instruction issue
// per two tests.
__device__ __forceinline__ unsigned long long f32x2_pack(float lo, float hi)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
// The candidate comes negated: a - s = a + (-s).
__device__ __forceinline__ unsigned long long dist2_x2(unsigned long long ax2, unsigned long long ay2, unsigned long long az2,
                                                       unsigned long long minus_sx2, unsigned long long minus_sy2, unsigned long long minus_sz2)
{
    unsigned long long dx, dy, dz, d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(dx) : "l"(ax2), "l"(minus_sx2));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(dy) : "l"(ay2), "l"(minus_sy2));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(dz) : "l"(az2), "l"(minus_sz2));
    asm("mul.rn.f32x2 %0, %1, %1;" : "=l"(d) : "l"(dy));
    asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(d) : "l"(dx), "l"(d));
    asm("fma.rn.f32x2 %0, %1, %1, %2;" : "=l"(d) : "l"(dz), "l"(d));
    return d;
}

// The grid when the host cannot choose it: from the bounding boxes of the images and, with a target subset, of the targets,
// by one thread of the block that finishes last of the pass that gathers the last of them.  Cells of edge radius/1.99 scanned
// +-2 (as the reference, :662,776) unless that would need more than cell_capacity cells; then the cells grow, and once they
// are wider than the cutoff the scan shrinks to +-1.  As a launch of its own, reducing per-block partial results: 22 us (1.6 M atoms, a subset of 1 M).
struct GridArgs { double radius; long long src_capacity, cell_capacity; int cand_capacity; };
template <typename T>
__device__ void rg_choose_grid_device(DevHeader* h, const GridArgs& a, bool subset)
{
    const double radius = a.radius;
    const long long src_capacity = a.src_capacity, cell_capacity = a.cell_capacity;
    const int cand_capacity = a.cand_capacity;
    // written by the atomics of other blocks: read at L2
    const unsigned long long M = __ldcg(&h->M);
    const uint32_t status = __ldcg(&h->status);
    if (M > (unsigned long long)src_capacity) atomicOr(&h->status, DYNB_RG_SRC_OVERFLOW);
    for (int k = 0; k < 3; k++) { h->clip_lo[k] = -1.0e300; h->clip_hi[k] = 1.0e300; }
    if (M == 0 || M > (unsigned long long)src_capacity || (status & RG_FATAL)) {
        h->nx = h->ny = h->nz = 1;
        h->ncell_plus1 = 2;
        h->pad = 1;
        h->group_cells = 1;
        h->group_cells_y = 1;
        h->gx = 1;
        h->num_groups = 0;
        h->gmin[0] = h->gmin[1] = h->gmin[2] = 0.0;
        h->res_inv = 1.0;
        return;
    }
    double lo[3], ext[3];
    for (int k = 0; k < 3; k++) {
        lo[k] = unordered_any<T>(__ldcg(&h->bb_min[k])) - 0.01;
        double hi = unordered_any<T>(__ldcg(&h->bb_max[k])) + 0.01;
        const unsigned long long tmin = __ldcg(&h->tb_min[k]), tmax = __ldcg(&h->tb_max[k]);
        if (subset && tmin <= tmax) {
            // clip to the targets' box grown by the cutoff (with slack far above any rounding)
            const double margin = radius * 1.001 + 0.02;
            const double tlo = unordered_any<T>(tmin) - margin, thi = unordered_any<T>(tmax) + margin;
            if (tlo > lo[k]) lo[k] = tlo;
            if (thi < hi) hi = thi;
            h->clip_lo[k] = lo[k];
            h->clip_hi[k] = hi;
            if (hi < lo[k]) hi = lo[k];
        }
        ext[k] = hi - lo[k];
    }
    GridChoice gc;
    rg_choose_grid(lo, ext, radius, cell_capacity, cand_capacity, (double)M, 0.0, !subset, gc);
    rg_store_grid(*h, gc);
}
template <typename T>
__device__ __forceinline__ void rg_last_block_chooses(DevHeader* h, const GridArgs& a, bool subset)
{
    __threadfence();
    __syncthreads();
    if (threadIdx.x != 0) return;
    if (atomicAdd(&h->arrived, 1u) != gridDim.x - 1) return;
    __threadfence();
    rg_choose_grid_device<T>(h, a, subset);
}

constexpr int WRAP_THREADS = 256;

// FUSED: the grid is known before the launch (gc, chosen on the host), so the images and the targets are counted
// into their cells here; the bounding box then only steers the shape of the work items.
template <typename T, bool FUSED>
__global__ void __launch_bounds__(WRAP_THREADS)
rg_wrap_kernel(const T* pos, int64_t N, Geom<T> g, int vec_ok, Vec4<T>* posw,
               int4* aff, DevHeader* h, const GridArgs ga, int subset,
               const GridChoice gc, uint32_t* ccount, uint32_t* tccount)
{
    chain_begin();
    __shared__ T stage[WRAP_THREADS * 3];
    __shared__ unsigned long long red[6][WRAP_THREADS / 32];
    __shared__ unsigned int red_cnt[WRAP_THREADS / 32];

    const int64_t block_base = (int64_t)blockIdx.x * WRAP_THREADS;
    const int64_t i = block_base + threadIdx.x;
    const int64_t nblock = min((int64_t)WRAP_THREADS, N - block_base);

    // Coalesced 16-byte loads of this block's 3*nblock reals, then a conflict-free stride-3 read.
    {
        const T* src = pos + block_base * 3;
        const int nreal = (int)nblock * 3;
        constexpr int PER = 16 / (int)sizeof(T);
        if (vec_ok && nblock == WRAP_THREADS) {
            using V = typename std::conditional<sizeof(T) == 4, float4, double2>::type;
            const V* src4 = reinterpret_cast<const V*>(src);
            V* dst4 = reinterpret_cast<V*>(stage);
            for (int k = threadIdx.x; k < nreal / PER; k += WRAP_THREADS) dst4[k] = src4[k];
        } else {
            for (int k = threadIdx.x; k < nreal; k += WRAP_THREADS) stage[k] = src[k];
        }
    }
    __syncthreads();

    using Key = typename std::conditional<sizeof(T) == 4, uint32_t, unsigned long long>::type;
    Key mn[3] = {~(Key)0, ~(Key)0, ~(Key)0}, mx[3] = {0, 0, 0};
    unsigned int count = 0;
    uint32_t status = 0;

    if (i < N) {
        const T px = stage[threadIdx.x * 3 + 0], py = stage[threadIdx.x * 3 + 1], pz = stage[threadIdx.x * 3 + 2];
        T f[3], m[3];
#pragma unroll
        for (int k = 0; k < 3; k++) f[k] = floor_t(dot3_gemm(px, g.inv[k], py, g.inv[3 + k], pz, g.inv[6 + k]));
#pragma unroll
        for (int k = 0; k < 3; k++) m[k] = dot3_gemm(f[0], g.cell[k], f[1], g.cell[3 + k], f[2], g.cell[6 + k]);
        const T wx = sub_rn(px, m[0]), wy = sub_rn(py, m[1]), wz = sub_rn(pz, m[2]);

        if (!(finite_t(wx) && finite_t(wy) && finite_t(wz))) status |= DYNB_RG_NONFINITE;
        const T lim = (T)1048576.0;
        if (!(fabs(f[0]) < lim && fabs(f[1]) < lim && fabs(f[2]) < lim)) status |= DYNB_RG_SHIFT_RANGE;

        // Fractional coordinates of the wrapped position, reference expression (:36-38).
        T s[3];
        s[0] = wx * g.inv[0] + wy * g.inv[3] + wz * g.inv[6];
        s[1] = wx * g.inv[1] + wy * g.inv[4] + wz * g.inv[7];
        s[2] = wx * g.inv[2] + wy * g.inv[5] + wz * g.inv[8];
        uint32_t flags = 0;
#pragma unroll
        for (int d = 0; d < 3; d++) {
            if (g.pbc[d]) {
                if (!(s[d] >= g.cf[d])) flags |= (1u << d);                 // :55
                if (!(s[d] <= (T)1.0f - g.cf[d])) flags |= (8u << d);       // :58
            }
        }
        if (!(status & DYNB_RG_NONFINITE) && flags == 0) {
            // interior atom: only its own (0,0,0) image
            T x, y, z;
            image_pos(g, wx, wy, wz, 0, 0, 0, x, y, z);
            if (FUSED) atomicAdd(&ccount[cell_of(gc, x, y, z)], 1u);
            mn[0] = mx[0] = ordered_key(x);
            mn[1] = mx[1] = ordered_key(y);
            mn[2] = mx[2] = ordered_key(z);
            count = 1;
        } else if (!(status & DYNB_RG_NONFINITE)) {
            // the images an atom needs form a box of shifts (the flags are per axis and direction): walk
            // that box only, so that a warp runs as many rounds as its busiest atom has images, not (2 rep + 1)^3
            const int lo0 = (flags & 8u) ? -g.rep[0] : 0, hi0 = (flags & 1u) ? g.rep[0] : 0;
            const int lo1 = (flags & 16u) ? -g.rep[1] : 0, hi1 = (flags & 2u) ? g.rep[1] : 0;
            const int lo2 = (flags & 32u) ? -g.rep[2] : 0, hi2 = (flags & 4u) ? g.rep[2] : 0;
            for (int dx = lo0; dx <= hi0; dx++)
                for (int dy = lo1; dy <= hi1; dy++)
                    for (int dz = lo2; dz <= hi2; dz++) {
                        T x, y, z;
                        image_pos(g, wx, wy, wz, dx, dy, dz, x, y, z);
                        if (FUSED) atomicAdd(&ccount[cell_of(gc, x, y, z)], 1u);
                        const Key ox = ordered_key(x), oy = ordered_key(y), oz = ordered_key(z);
                        mn[0] = min(mn[0], ox); mx[0] = max(mx[0], ox);
                        mn[1] = min(mn[1], oy); mx[1] = max(mx[1], oy);
                        mn[2] = min(mn[2], oz); mx[2] = max(mx[2], oz);
                        count++;
                    }
        }
        Vec4<T> w;
        w.x = wx; w.y = wy; w.z = wz; w.w = bits_to_real((int32_t)flags, T());
        posw[i] = w;
        aff[i] = make_int4((int)f[0], (int)f[1], (int)f[2], (int)count);
        // every atom is a target, binned by its wrapped position (as rg_bin_kernel does)
        if (FUSED && !(status & DYNB_RG_NONFINITE)) atomicAdd(&tccount[cell_of(gc, wx, wy, wz)], 1u);
    }

    // block reduction
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if constexpr (sizeof(T) == 4) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            mn[k] = (Key)__reduce_min_sync(0xffffffffu, (unsigned)mn[k]);
            mx[k] = (Key)__reduce_max_sync(0xffffffffu, (unsigned)mx[k]);
        }
        count = __reduce_add_sync(0xffffffffu, count);
        status = __reduce_or_sync(0xffffffffu, status);
    } else {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
#pragma unroll
            for (int k = 0; k < 3; k++) {
                mn[k] = min(mn[k], (Key)__shfl_xor_sync(0xffffffffu, mn[k], o));
                mx[k] = max(mx[k], (Key)__shfl_xor_sync(0xffffffffu, mx[k], o));
            }
            count += __shfl_xor_sync(0xffffffffu, count, o);
            status |= __shfl_xor_sync(0xffffffffu, status, o);
        }
    }
    if (lane == 0) {
#pragma unroll
        for (int k = 0; k < 3; k++) {
            // "no image" stays the 64-bit identity of the minimum
            red[k][warp] = (mn[k] == ~(Key)0) ? ~0ull : (unsigned long long)mn[k];
            red[3 + k][warp] = (unsigned long long)mx[k];
        }
        red_cnt[warp] = count;
        if (status) atomicOr(&h->status, status);
    }
    __syncthreads();
    // the bounding box goes straight to the header: six fire-and-forget atomics per block (with a grid chosen on the host it
    // only steers the shape of the work items, which is settled three launches later)
    if (threadIdx.x < 6) {
        unsigned long long v = red[threadIdx.x][0];
        for (int w = 1; w < WRAP_THREADS / 32; w++)
            v = (threadIdx.x < 3) ? min(v, red[threadIdx.x][w]) : max(v, red[threadIdx.x][w]);
        if (threadIdx.x < 3) atomicMin(&h->bb_min[threadIdx.x], v);
        else atomicMax(&h->bb_max[threadIdx.x - 3], v);
    } else if (!FUSED && threadIdx.x == 6) {
        unsigned long long c = 0;
        for (int w = 0; w < WRAP_THREADS / 32; w++) c += red_cnt[w];
        atomicAdd(&h->M, c);
    }
    if (!FUSED && !subset) rg_last_block_chooses<T>(h, ga, false);
}

// Bounding box of the wrapped TARGET positions (only when a target subset is given), then the grid.  Sources farther than the cutoff from that box are never
// needed, which keeps the grid and the image count small when a rank builds edges for its own
// atoms only.
template <typename T>
__global__ void __launch_bounds__(256)
rg_target_bbox_kernel(const int64_t* targets, int64_t Nt, int64_t N, const Vec4<T>* posw,
                      DevHeader* h, const GridArgs ga)
{
    chain_begin();
    __shared__ unsigned long long red[6][8];
    unsigned long long v[6] = {~0ull, ~0ull, ~0ull, 0ull, 0ull, 0ull};
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < Nt) {
        const int64_t a = targets[i];
        if (a >= 0 && a < N) {
            const Vec4<T> w = posw[a];
            v[0] = v[3] = ordered_any(w.x);
            v[1] = v[4] = ordered_any(w.y);
            v[2] = v[5] = ordered_any(w.z);
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 3; k++) {
            v[k] = min(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
            v[3 + k] = max(v[3 + k], __shfl_xor_sync(0xffffffffu, v[3 + k], o));
        }
    if ((threadIdx.x & 31) == 0)
        for (int k = 0; k < 6; k++) red[k][threadIdx.x >> 5] = v[k];
    __syncthreads();
    if (threadIdx.x < 6) {
        unsigned long long a = red[threadIdx.x][0];
        for (int w = 1; w < 8; w++) a = (threadIdx.x < 3) ? min(a, red[threadIdx.x][w]) : max(a, red[threadIdx.x][w]);
        if (threadIdx.x < 3) atomicMin(&h->tb_min[threadIdx.x], a);
        else atomicMax(&h->tb_max[threadIdx.x - 3], a);
    }
    rg_last_block_chooses<T>(h, ga, true);
}

// ------------------------------------------------------------------------------------------
// binning
// ------------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t pack_shift_code(int ex, int ey, int ez)
{
    return (uint32_t)(ex + 512) | ((uint32_t)(ey + 512) << 10) | ((uint32_t)(ez + 512) << 20);
}

// What the scatter pass leaves in the provisional slot of a source image (key: image order, id: atom, code: shift - floor)
// or of a target of a subset (key: atom, id: entry, code: floor).  In single precision the position goes along: the ordering
// pass then reads its own slot and its cell's slots and gathers nothing by atom number, and a slot is one 32-byte sector,
// written by one store.  In double precision it would be two sectors (48 bytes: 27 us slower for 500 k atoms); there the
// ordering pass fetches the wrapped position.  Without a subset no target is scattered: the targets of a cell are its images
// at shift zero, in the same order.  Atoms in random order, scatter and ordering, before and after: 263 + 218 -> 144 + 82 us
// (4 M), 47 + 37 -> 37 + 20 us (1 M); bound by the sectors of the random writes and the cursors' atomics.
template <typename T> struct SlotRec;
template <> struct __align__(32) SlotRec<float> { uint32_t key, id, cell, code; float x, y, z, pad; };
template <> struct __align__(16) SlotRec<double> { uint32_t key, id, cell, code; };
__device__ __forceinline__ void store_slot(SlotRec<float>* at, uint32_t key, uint32_t id, uint32_t cell, uint32_t code, float x, float y, float z)
{
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(at), "r"(key), "r"(id), "r"(cell), "r"(code),
                 "r"(__float_as_uint(x)), "r"(__float_as_uint(y)), "r"(__float_as_uint(z)), "r"(0u) : "memory");
}
__device__ __forceinline__ void store_slot(SlotRec<double>* at, uint32_t key, uint32_t id, uint32_t cell, uint32_t code, double, double, double)
{
    *reinterpret_cast<uint4*>(at) = make_uint4(key, id, cell, code);
}
template <typename T, bool SCATTER>
__global__ void __launch_bounds__(256, 4)
rg_bin_kernel(int64_t N, int64_t Nt, const int64_t* targets, Geom<T> g,
              const Vec4<T>* posw, const int4* aff, DevHeader* hp,
              uint32_t* ccount, uint32_t* cfill,
              uint32_t* tccount, uint32_t* tcfill,
              SlotRec<T>* srec, SlotRec<T>* trec, long long src_capacity, int shape_cand_capacity)
{
    chain_begin();
    const DevHeader h = *hp;
    // the counting pass still runs when only the image capacity is short (it writes nothing but the cell counters): the
    // prefix sum's total then leaves the true number of images in header.M for the caller's second attempt
    if (h.status & (SCATTER ? RG_FATAL : (RG_FATAL & ~(uint32_t)DYNB_RG_SRC_OVERFLOW))) return;
    if (SCATTER && h.M > (unsigned long long)src_capacity) {
        // more images than the caller's buffers hold (header.M is the prefix sum's total by now; with a grid chosen on
        // the host this is the first place that knows): nothing is placed, the plan is repeated with a larger capacity
        if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&hp->status, DYNB_RG_SRC_OVERFLOW);
        return;
    }
    if (SCATTER && shape_cand_capacity > 0 && blockIdx.x == 0 && threadIdx.x < 32) {
        // grid chosen on the host: the shape of the work items is settled here, from the number of images and the
        // bounding box they really fill (gathered while wrapping) — an atom cluster in a large periodic box is as
        // dense in its cells as it is, whatever the volume of the cell.  One lane per axis, then one per shape: the divisions
        // and square roots of the five shapes are in flight together (scatter of a thousand atoms 10.1 -> 9.3 us).
        const int lane = threadIdx.x;
        double cells = 1.0;
        if (lane < 3) {
            const int n = lane == 0 ? h.nx : (lane == 1 ? h.ny : h.nz);
            cells = ceil((unordered_any<T>(hp->bb_max[lane]) - unordered_any<T>(hp->bb_min[lane]) + 0.02) / (1.0 / h.res_inv));
            if (!(cells >= 1.0)) cells = 1.0;
            if (cells > (double)n) cells = (double)n;
        }
        const double vol_cells = __shfl_sync(0xffffffffu, cells, 0) * __shfl_sync(0xffffffffu, cells, 1) * __shfl_sync(0xffffffffu, cells, 2);
        const bool fits = lane >= RG_SHAPES - 1 || rg_shape_fits(lane, h.pad, (double)h.M / vol_cells, shape_cand_capacity, true);
        const int best = __ffs((int)__ballot_sync(0xffffffffu, fits)) - 1;
        if (lane == 0) {
            GridChoice gc;
            gc.nx = h.nx; gc.ny = h.ny; gc.nz = h.nz;
            rg_set_shape(gc, best);
            hp->group_cells = gc.group_cells;
            hp->group_cells_y = gc.group_cells_y;
            hp->gx = gc.gx;
            hp->num_groups = gc.num_groups;
        }
    }
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < N) {
        const Vec4<T> w = posw[i];
        int4 f = make_int4(0, 0, 0, 0);
        if (SCATTER) f = aff[i];
        const uint32_t flags = (uint32_t)real_to_bits(w.w);
        const int k1 = 2 * g.rep[1] + 1, k2 = 2 * g.rep[2] + 1;
        // box of needed shifts (see rg_wrap_kernel); same (dx, dy, dz) order as a full walk
        const int lo0 = (flags & 8u) ? -g.rep[0] : 0, hi0 = (flags & 1u) ? g.rep[0] : 0;
        const int lo1 = (flags & 16u) ? -g.rep[1] : 0, hi1 = (flags & 2u) ? g.rep[1] : 0;
        const int lo2 = (flags & 32u) ? -g.rep[2] : 0, hi2 = (flags & 4u) ? g.rep[2] : 0;
        // Four images at a time: their cursors' atomics are in flight together before the first slot is written.  One by one a
        // corner atom's eight images are eight round trips to L2 in a row: 2 us of a call with a thousand atoms, 5 us of one
        // with a million.
        constexpr int U = SCATTER ? 4 : 1;
        int dx = lo0, dy = lo1, dz = lo2;
        const int total = (hi0 - lo0 + 1) * (hi1 - lo1 + 1) * (hi2 - lo2 + 1);
        for (int m = 0; m < total; m += U) {
            T x[U], y[U], z[U];
            uint32_t cell[U], slot[U], image[U], code[U];
            bool there[U];
#pragma unroll
            for (int u = 0; u < U; u++) {
                there[u] = m + u < total;
                if (!there[u]) continue;
                image_pos(g, w.x, w.y, w.z, dx, dy, dz, x[u], y[u], z[u]);
                // farther than the cutoff from every target: dropped
                there[u] = !((double)x[u] < h.clip_lo[0] || (double)x[u] > h.clip_hi[0] || (double)y[u] < h.clip_lo[1] ||
                             (double)y[u] > h.clip_hi[1] || (double)z[u] < h.clip_lo[2] || (double)z[u] > h.clip_hi[2]);
                if (there[u]) {
                    cell[u] = cell_of(h, x[u], y[u], z[u]);
                    if (!SCATTER) {
                        atomicAdd(&ccount[cell[u]], 1u);
                    } else {
                        // the fill cursors start at the cells' first slots (the prefix sum wrote them there too):
                        // one atomic and one record per image; (atom, image) orders the images of a cell
                        slot[u] = atomicAdd(&cfill[cell[u]], 1u);
                        image[u] = (uint32_t)(((dx + g.rep[0]) * k1 + (dy + g.rep[1])) * k2 + (dz + g.rep[2]));
                        const int ex = dx - f.x, ey = dy - f.y, ez = dz - f.z;
                        if (max(max(abs(ex), abs(ey)), abs(ez)) > 511) atomicOr(&hp->status, DYNB_RG_SHIFT_RANGE);
                        code[u] = pack_shift_code(ex, ey, ez);
                    }
                }
                if (++dz > hi2) {
                    dz = lo2;
                    if (++dy > hi1) { dy = lo1; dx++; }
                }
            }
            if (SCATTER) {
#pragma unroll
                for (int u = 0; u < U; u++)
                    if (there[u]) store_slot(&srec[slot[u]], image[u], (uint32_t)i, cell[u], code[u], x[u], y[u], z[u]);
            }
        }
    }
    // without a subset the targets are the images at shift zero: the ordering pass finds them among the sources
    if (i < Nt && (!SCATTER || targets != nullptr)) {
        const int64_t a = targets ? targets[i] : i;
        if (a < 0 || a >= N) {
            atomicOr(&hp->status, DYNB_RG_BAD_TARGET);
        } else {
            const Vec4<T> w = posw[a];
            const uint32_t c = cell_of(h, w.x, w.y, w.z);
            if (!SCATTER) {
                atomicAdd(&tccount[c], 1u);
            } else {
                const int4 f = aff[a];
                const uint32_t slot = atomicAdd(&tcfill[c], 1u);
                // a floor that does not fit its ten bits: the atom's own image has raised the range status
                store_slot(&trec[slot], (uint32_t)a, (uint32_t)i, c, pack_shift_code(f.x, f.y, f.z), w.x, w.y, w.z);
            }
        }
    }
}

// Coordinates as the count pass tests them: float positions as they are, double positions as floats from the grid's origin.
__device__ __forceinline__ float scan_coord(float x, double) { return x; }
__device__ __forceinline__ float scan_coord(double x, double origin) { return (float)(x - origin); }

// The count pass in double precision tests floats first.  A float distance d from coordinates relative to the grid's origin
// (scan_coord) decides a pair when it lies clear of the cutoff; the few others are tested on the double records:
//   lo >= d > near: a neighbour;   d > hi: none;   else the double test decides (exact_hits).
// With u = 2^-24 and X the largest coordinate a difference of two coordinates is off by at most eta = 2 u X, so for
// |delta| near t the float result differs from the true t^2 by less than 2 sqrt(3) t eta + 6 u t^2 + 3 (eta + u t)^2
// (conversion, three subtractions, three roundings of the sum); twice that is the margin around r^2 and above the
// self-distance limit.  The thresholds are rounded outwards, a distance that is not a number is never decided here, and
// coordinates near the end of the float range are left to the double test altogether.
// A float distance of zero means coordinates within 2 u X of one another along each axis (equal floats, or ones so close to
// zero that the square underflows): when that puts them inside the self-distance limit, the pair (every target meets itself)
// is no neighbour and needs no double test.  500 k atoms of silicon, 6 A: 364 us with a double test for every candidate, 228
// with this one.
__device__ __forceinline__ void float_test(double r2, double X, float& near, float& lo, float& hi, uint32_t& equal_is_near)
{
    const double u = 5.9604644775390625e-8, eta = 2.0 * u * X, eps = (double)1e-8f;
    double margin[2];
    const double t2[2] = {eps, r2};
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const double t = sqrt(t2[k]), e = eta + u * t;
        margin[k] = 2.0 * (3.5 * t * eta + 6.0 * u * t2[k] + 3.0 * e * e);
    }
    const bool in_range = X < 1.0e15 && r2 < 1.0e30;
    near = __double2float_ru(eps + margin[0]);
    lo = in_range ? __double2float_rd(r2 - margin[1]) : -1.0f;
    hi = in_range ? __double2float_ru(r2 + margin[1]) : __int_as_float(0x7f800000);
    equal_is_near = 3.1 * eta * eta < eps ? 1u : 0u;
}

// Deterministic order inside each cell (ascending key) and the packed records.
template <typename T>
__global__ void __launch_bounds__(256)
rg_bin_finalize_kernel(int64_t Nt, int subset, Geom<T> g, const Vec4<T>* posw, DevHeader* hp,
                       const uint32_t* cstart, const uint32_t* tcstart,
                       const SlotRec<T>* srec, const SlotRec<T>* trec,
                       Vec4<T>* spos, float4* sscan,
                       uint2* smeta, Vec4<T>* tpos, float4* tscan,
                       int4* tmeta, double r2, uint4* header_host)
{
    chain_begin();
    // a plan that ends here: its header is complete
    if (header_host != nullptr && blockIdx.x == 0 && threadIdx.x == 0) publish_64_bytes(reinterpret_cast<const uint4*>(hp), header_host);
    if (hp->status & RG_FATAL) return;
    if (sizeof(T) == 8 && blockIdx.x == 0 && threadIdx.x == 0)
        float_test(r2, 1.01 * (double)max(hp->nx, max(hp->ny, hp->nz)) / hp->res_inv + 0.02, hp->test_near, hp->test_lo, hp->test_hi,
                   hp->test_equal_is_near);
    const unsigned long long M = hp->M;
    const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const bool has_s = j < (int64_t)M, has_t = subset && j < Nt;
    auto put_target = [&](uint32_t at, T x, T y, T z, uint32_t entry, uint32_t atom, int fx, int fy, int fz) {
        Vec4<T> r;
        r.x = x; r.y = y; r.z = z; r.w = bits_to_real((int32_t)entry, T());
        tpos[at] = r;
        if (sizeof(T) == 8)
            tscan[at] = make_float4(scan_coord(x, hp->gmin[0]), scan_coord(y, hp->gmin[1]), scan_coord(z, hp->gmin[2]), __int_as_float((int)entry));
        tmeta[at] = make_int4((int)atom, fx, fy, fz);
    };
    // The loads are issued level by level for the source image and the target of this thread together: the two
    // slots, then the cell ranges, then the slots of the cell for the rank; the kernel waits for memory, not for arithmetic.
    SlotRec<T> s{}, t{};
    if (has_s) s = srec[j];
    if (has_t) t = trec[j];
    uint32_t sb = 0, se = 0, tb = 0, te = 0;
    const int k1 = 2 * g.rep[1] + 1, k2 = 2 * g.rep[2] + 1;
    const uint32_t center = (uint32_t)((g.rep[0] * k1 + g.rep[1]) * k2 + g.rep[2]);  // the image at shift zero
    Vec4<T> sw{}, tw{};
    if (has_s) {
        sb = cstart[s.cell];
        se = cstart[s.cell + 1];
        if (!subset && s.key == center) tb = tcstart[s.cell];
        if constexpr (sizeof(T) == 8) {
            sw = posw[s.id];
            unsigned image = s.key;
            const int dz = (int)(image % k2) - g.rep[2]; image /= k2;
            const int dy = (int)(image % k1) - g.rep[1]; image /= k1;
            image_pos(g, sw.x, sw.y, sw.z, (int)image - g.rep[0], dy, dz, sw.x, sw.y, sw.z);
        } else {
            sw.x = s.x; sw.y = s.y; sw.z = s.z;
        }
    }
    if (has_t) {
        tb = tcstart[t.cell];
        te = tcstart[t.cell + 1];
        if constexpr (sizeof(T) == 8) tw = posw[t.key];
        else { tw.x = t.x; tw.y = t.y; tw.z = t.z; }
    }
    if (has_s) {
        // place in the cell: images in front of this one; and, of those, the ones at shift zero
        const unsigned long long mine = ((unsigned long long)s.id << 32) | s.key;
        uint32_t rank = 0, trank = 0;
        for (uint32_t q = sb; q < se; q++) {
            const uint2 kq = *reinterpret_cast<const uint2*>(&srec[q]);
            const bool before = ((((unsigned long long)kq.y << 32) | kq.x) < mine);
            rank += before ? 1u : 0u;
            trank += (before && kq.x == center) ? 1u : 0u;
        }
        const uint32_t at = sb + rank;
        Vec4<T> r;
        r.x = sw.x; r.y = sw.y; r.z = sw.z; r.w = bits_to_real((int32_t)s.id, T());
        spos[at] = r;
        if (sizeof(T) == 8)
            sscan[at] = make_float4(scan_coord(sw.x, hp->gmin[0]), scan_coord(sw.y, hp->gmin[1]), scan_coord(sw.z, hp->gmin[2]), 0.0f);
        smeta[at] = make_uint2(s.id, s.code);
        // its shift is zero: the code is minus the floor
        if (!subset && s.key == center)
            put_target(tb + trank, sw.x, sw.y, sw.z, s.id, s.id, 512 - (int)(s.code & 1023u), 512 - (int)((s.code >> 10) & 1023u),
                       512 - (int)((s.code >> 20) & 1023u));
    }
    if (has_t) {
        uint32_t rank = 0;
        for (uint32_t q = tb; q < te; q++) rank += (trec[q].id < t.id) ? 1u : 0u;
        put_target(tb + rank, tw.x, tw.y, tw.z, t.id, t.key, (int)(t.code & 1023u) - 512, (int)((t.code >> 10) & 1023u) - 512,
                   (int)((t.code >> 20) & 1023u) - 512);
    }
}

// ------------------------------------------------------------------------------------------
// rg_pair: the cell scan.
// ------------------------------------------------------------------------------------------
constexpr int PAIR_WARPS = 8;
constexpr int PAIR_THREADS = PAIR_WARPS * 32;
constexpr int PAIR_CAND_BYTES = 5120;  // dense candidate records per warp (320 float4 / 160 double4)
constexpr int PAIR_CODE_BYTES = 1280;  // packed shift code per candidate (up to 320)
constexpr int PAIR_LIST = 128;         // parked hits per target (uint16 each, two targets per warp)
// The pair kernels are launched with this many times the CTAs that fit the device at once: SMs do not
// all drain their share at the same speed, and a static one-wave split left the slowest SM 20-30 %
// behind the average; with several short waves the block scheduler evens that out.
constexpr int PAIR_GRID_WAVES = 8;
constexpr int PAIR_SHARE = 8;          // warps that share a listed group's targets when few groups are listed
constexpr int RUN_FLAG_WORDS = 16;     // run-start bitmap of one staged chunk (up to 512 records)
constexpr int RUN_INDEX_BYTES = 32 * 4 + RUN_FLAG_WORDS * 4;
constexpr int PAIR_WARP_BYTES = PAIR_CAND_BYTES + PAIR_CODE_BYTES + PAIR_LIST * 4 + RUN_INDEX_BYTES;

// Flattened candidate list of a warp: lane r owns source run r (run_a = first record, run_off = place
// of the run in the flattened list).  To find the record behind flattened index jj, the non-empty
// runs are compacted into delta[] (record = delta[rank] + jj) and every chunk of the list gets a bitmap
// of the places where a run starts; the rank of the run that covers jj is then a population count.
__device__ __forceinline__ void runs_compact(int* delta, int run_a, int run_off, int run_len, uint32_t lt)
{
    const uint32_t nem = __ballot_sync(0xffffffffu, run_len > 0);
    if (run_len > 0) delta[__popc(nem & lt)] = run_a - run_off;
}
// Asynchronous global -> shared copies (LDGSTS): the records of a whole chunk are requested back to back
// without passing through registers; cp_async_wait_all() before the warp reads them.
template <int BYTES>
__device__ __forceinline__ void cp_async(void* smem_dst, const void* gsrc)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(d), "l"(gsrc), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// returns the number of non-empty runs that start before cbeg; flags covers [cbeg, cbeg + 32 * RUN_FLAG_WORDS)
__device__ __forceinline__ int runs_flags(uint32_t* flags, int run_off, int run_len, int lane, int cbeg)
{
    if (lane < RUN_FLAG_WORDS) flags[lane] = 0u;
    __syncwarp();
    const int rel = run_off - cbeg;
    if (run_len > 0 && rel >= 0 && rel < 32 * RUN_FLAG_WORDS) atomicOr(&flags[rel >> 5], 1u << (rel & 31));
    const uint32_t before = __ballot_sync(0xffffffffu, run_len > 0 && rel < 0);
    __syncwarp();
    return __popc(before);
}

// The mask of the lanes below, likewise: read again where it is used it was 24 of 530 instructions a target.
__device__ __forceinline__ uint32_t lanes_below()
{
    uint32_t m;
    asm volatile("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}
__device__ __forceinline__ int lane_id()
{
    int l;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(l));  // volatile: kept in a register instead of read again
    return l;
}
__device__ __forceinline__ uint32_t warp_incl_scan_u32(uint32_t x)
{
    // the shuffle's own predicate says whether there is a lane to add
#pragma unroll
    for (int o = 1; o < 32; o <<= 1)
        asm volatile("{\n\t.reg .pred q;\n\t.reg .b32 y;\n\tshfl.sync.up.b32 y|q, %0, %1, 0, 0xffffffff;\n\t@q add.u32 %0, %0, y;\n\t}" : "+r"(x) : "r"(o));
    return x;
}
// What a warp keeps to find the record behind a place of its candidate list (one chunk of up to 512 places).
struct RunIndex {
    int delta[32];                  // per non-empty run: record = delta + place
    uint32_t flags[RUN_FLAG_WORDS]; // places of the chunk where a run starts
    uint2 word[RUN_FLAG_WORDS];     // the same word, and the number of runs that start in front of it, minus one
    // lane r owns run r (run_a = first record, run_off = place in the list); the chunk starts at place cbeg
    __device__ __forceinline__ void set(int run_a, int run_off, int run_len, int cbeg, int lane, uint32_t lt)
    {
        runs_compact(delta, run_a, run_off, run_len, lt);
        const int before = runs_flags(flags, run_off, run_len, lane, cbeg);
        const uint32_t f = lane < RUN_FLAG_WORDS ? flags[lane] : 0u;
        const uint32_t own = (uint32_t)__popc(f), rank = (uint32_t)before + warp_incl_scan_u32(own) - own;
        if (lane < RUN_FLAG_WORDS) word[lane] = make_uint2(f, rank - 1u);
        __syncwarp();
    }
    // the same for a list of up to 64 places: its first two words, from registers (that gas: 826 -> 800 us)
    __device__ __forceinline__ void set_short(int run_a, int run_off, int run_len, int lane, uint32_t lt)
    {
        runs_compact(delta, run_a, run_off, run_len, lt);
        const uint32_t start = run_len > 0 ? 1u << (run_off & 31) : 0u;
        const uint32_t f0 = __reduce_or_sync(0xffffffffu, run_off < 32 ? start : 0u), f1 = __reduce_or_sync(0xffffffffu, run_off < 32 ? 0u : start);
        if (lane < 2) word[lane] = lane == 0 ? make_uint2(f0, 0xffffffffu) : make_uint2(f1, (uint32_t)__popc(f0) - 1u);
        __syncwarp();
    }
    // record - place, for place 32 s + lane of the chunk
    __device__ __forceinline__ int record(int s, uint32_t le) const
    {
        const uint2 f = word[s];
        return delta[(int)f.y + __popc(f.x & le)];
    }
};

// Optional extras of the edge writers for the model-side glue: the shifts written with the caller's sign
// and the Cartesian shift of every edge, unit_shift @ cell, rounded like a K = 3 float GEMM
// (products and sums of torch.matmul(unit_shifts, cell): fma(u2, c2, fma(u1, c1, u0 * c0))).
struct GlueArgs {
    float* cart;              // [E,3] or nullptr
    const long long* id_map;  // [n_atoms] ids to write instead of the atom indices (local -> global), or nullptr
    int negate;               // 1: write -shift
    float c[9];               // cell, row-major
};
__device__ __forceinline__ void glue_write(const GlueArgs& g, float* __restrict__ shifts, long long e, int ix, int iy, int iz)
{
    if (g.negate) { ix = -ix; iy = -iy; iz = -iz; }
    const float u0 = (float)ix, u1 = (float)iy, u2 = (float)iz;
    shifts[3 * e + 0] = u0;
    shifts[3 * e + 1] = u1;
    shifts[3 * e + 2] = u2;
    if (g.cart != nullptr) {
#pragma unroll
        for (int k = 0; k < 3; k++)
            g.cart[3 * e + k] = __fmaf_rn(u2, g.c[6 + k], __fmaf_rn(u1, g.c[3 + k], __fmul_rn(u0, g.c[k])));
    }
}

// The grid and the shape of the groups, and one group: its targets (one contiguous run a cell row, at most two rows) and this
// lane's run of source records.  Both cell-scan kernels keep the grid in shared memory and read it where a group is looked
// up: in registers it left too few for the loops.
struct __align__(16) GroupShape { uint32_t gx, by_gx, gy, by_gy; int nx, ny, nz, sx; int sy, pad, unused[2]; };
// As loaded (nothing waits for the loads until the group's turn): lanes below 30 have their run of source records, the two last lanes the
// targets of the group's two rows.
struct GroupDesc { int run_a, run_e; };
constexpr int GROUP_ROW_LANE = 30;
__device__ __forceinline__ GroupShape group_shape(const DevHeader* hp)
{
    const uint32_t gx = (uint32_t)hp->gx, gy = (uint32_t)((hp->ny + hp->group_cells_y - 1) / hp->group_cells_y);
    return {gx, 0xffffffffu / gx, gy, 0xffffffffu / gy, hp->nx, hp->ny, hp->nz, hp->group_cells, hp->group_cells_y, hp->pad, {0, 0}};
}
// v / d and the remainder, from by_d = floor((2^32 - 1) / d) >= 2^32 / d - 1: v by_d / 2^32 lies above v / d - 1, so the upper half
// of the product is the quotient or one less.  (The compiler's division is three times as many instructions.)
__device__ __forceinline__ uint32_t group_divide(uint32_t v, uint32_t d, uint32_t by_d, uint32_t& rest)
{
    uint32_t q = __umulhi(v, by_d);
    rest = v - q * d;
    if (rest >= d) { rest -= d; q++; }
    return q;
}
// Which cells a lane looks up: (y, z) row relative to the group's first, and how far beyond the group along x; -1: none
__device__ __forceinline__ int group_lane(const GroupShape& g, int lane)
{
    const int wy = g.sy + 2 * g.pad;
    if (lane >= GROUP_ROW_LANE) return (8 + lane - GROUP_ROW_LANE) | (8 << 8);
    return lane < wy * (2 * g.pad + 1) ? ((8 + lane % wy - g.pad) | ((8 + lane / wy - g.pad) << 8) | (g.pad << 16)) : -1;
}
__device__ __forceinline__ uint4 shared_words(const void* at)
{
    uint4 v;
    asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"((uint32_t)__cvta_generic_to_shared(at)));
    return v;
}
// cells: first records of the cells, of the sources, for the two last lanes of the targets.  Two loads a lane, and none of the
// branches that a row outside the grid would need: its lane reads an empty run.  Edge writer, before (every lane loaded the rows'
// targets, ten words of the grid were read one by one) and after: 309 -> 298 us (liquid, 1 M atoms), 162 -> 153 (silicon in double
// precision, 500 k), 25.3 -> 23.1 (copper, 32 k), 12.8 -> 10.7 (1 k), 605 -> 605 (a rank's copper with Cartesian shifts).
__device__ __forceinline__ GroupDesc fetch_group(const GroupShape& shape, const uint32_t* cells, uint32_t grp, int which)
{
    const uint4 g = shared_words(&shape.gx), n = shared_words(&shape.nx), s = shared_words(&shape.sy);
    const int nx = (int)n.x, ny = (int)n.y, nz = (int)n.z;
    uint32_t ix, iy;
    const uint32_t row = group_divide(grp, g.x, g.y, ix);
    const int cz = (int)group_divide(row, g.z, g.w, iy), cy0 = (int)(iy * s.x), cy1 = min(cy0 + (int)s.x, ny) - 1;
    GroupDesc d;
    const int cx0 = (int)(ix * n.w), cx1 = min(cx0 + (int)n.w, nx) - 1;
    const int beyond = which >> 16, yy = cy0 + (which & 255) - 8, zz = cz + ((which >> 8) & 255) - 8;
    const bool there = which >= 0 && yy >= 0 && yy <= min(cy1 + beyond, ny - 1) && zz >= 0 && zz < nz;
    const uint32_t first = ((uint32_t)zz * (uint32_t)ny + (uint32_t)yy) * (uint32_t)nx;
    const uint32_t a = there ? first + (uint32_t)max(cx0 - beyond, 0) : 0u, e = there ? first + (uint32_t)min(cx1 + beyond, nx - 1) + 1u : 0u;
    asm volatile("ld.global.b32 %0, [%1];" : "=r"(d.run_a) : "l"(cells + a));
    asm volatile("ld.global.b32 %0, [%1];" : "=r"(d.run_e) : "l"(cells + e));
    return d;
}

// The same for the count pass, which does not load ahead: every lane loads the rows' targets, and nothing is handed round behind the
// loads (a rank's copper: 265 us with this one, 270 with the other; the liquid 209 and 211).
struct GroupRows { uint32_t tb0, te0, tb1, te1; int run_a, run_e, cy0, cy1, cz; };
__device__ __forceinline__ int group_lane_run(const GroupShape& g, int lane)
{
    const int wy = g.sy + 2 * g.pad;
    return lane < wy * (2 * g.pad + 1) ? (((lane / wy) << 8) | (lane % wy)) : -1;
}
__device__ __forceinline__ GroupRows fetch_group_rows(const volatile GroupShape& g, const uint32_t* tcstart, const uint32_t* cstart, uint32_t grp, int lane_run)
{
    GroupRows d;
    const int nx = g.nx, ny = g.ny, pad = g.pad, sx = g.sx, sy = g.sy;
    const uint32_t gx = g.gx, gy = g.gy;
    uint32_t ix, iy;
    const uint32_t row = group_divide(grp, gx, g.by_gx, ix);
    const int cz = (int)group_divide(row, gy, g.by_gy, iy), cx0 = (int)ix * sx, cy0 = (int)iy * sy;
    const int cx1 = min(cx0 + sx, nx) - 1, cy1 = min(cy0 + sy, ny) - 1;
    d.cy0 = cy0;
    d.cy1 = cy1;
    d.cz = cz;
    const uint32_t* tcell = tcstart + ((uint32_t)cz * ny + cy0) * nx;
    d.tb0 = tcell[cx0];
    d.te0 = tcell[cx1 + 1];
    d.tb1 = d.te1 = 0;
    if (cy1 > cy0) {
        d.tb1 = tcell[nx + cx0];
        d.te1 = tcell[nx + cx1 + 1];
    }
    d.run_a = d.run_e = 0;
    if (lane_run >= 0) {
        const int yy = cy0 - pad + (lane_run & 255), zz = cz - pad + (lane_run >> 8);
        if (yy >= 0 && yy < ny && yy <= cy1 + pad && zz >= 0 && zz < g.nz) {
            const uint32_t* cell = cstart + ((uint32_t)zz * ny + yy) * nx;
            d.run_a = (int)cell[max(cx0 - pad, 0)];
            d.run_e = (int)cell[min(cx1 + pad, nx - 1) + 1];
        }
    }
    return d;
}

template <typename T> struct PairParams {
    DevHeader* h;
    const uint32_t* cstart;
    const uint32_t* tcstart;
    const Vec4<T>* spos;
    const float4* sscan;      // the source records' coordinates as the count pass tests them (float: the records themselves)
    const Vec4<T>* tpos;
    const float4* tscan;      // the targets' coordinates as the count pass tests them, and the entry
    const int4* tmeta;
    uint32_t* tcount;         // [Nt+1] degree per sorted target; running cursor of rg_pair_kernel
    const long long* toffset; // [Nt+1]
    unsigned short* hitmask;  // [Nt, 32] per lane: bit s set if candidate 32 s + lane is a neighbour (written by rg_count_kernel)
    const uint2* smeta;       // [M] {atom id, packed shift code} per source record
    int32_t* counts_out;      // [Nt] degrees in caller order, or nullptr
    const uint32_t* glist;    // groups that hold at least one target (h->active_groups entries), or nullptr = all groups
    uint32_t* long_list;      // groups whose candidate list exceeds the hit bits (h->reserved[1] entries, written by rg_count_kernel)
    long long n_targets;
    // halo marking only (rg_halo_*): owner of every source record and of every target, and a word for every candidate run
    unsigned short* sown;     // [M]; lies over the binning slots, which nothing reads behind the plan
    unsigned short* town;     // [n_targets]; likewise
    unsigned short* run_owner;  // [gx * ny * nz]
    uint32_t* halo_list;        // [n_targets] groups that can hold an edge of interest (h->halo_groups entries); behind sown
    T r2;
};
// The plan stores its PairParams inside the workspace (after the header) so that the fill call
// needs nothing but the workspace pointer.
constexpr int64_t RG_PARAMS_OFFSET = 512;
constexpr int64_t RG_HEADER_BYTES = 1024;

// With a target subset (a rank building edges for the atoms it owns) the grid may span far more cells than
// hold targets — a subdomain that touches the periodic boundary has wrapped targets on both sides of the box
// and its grid covers the whole box.  The cell-scan kernels then walk a list of the groups that hold targets
// instead of all groups.  The order of the list is not defined (it only distributes the work; every target's
// output place is fixed by the offsets).
template <typename T>
__global__ void __launch_bounds__(256)
rg_group_list_kernel(const PairParams<T>* params_dev, uint32_t* glist)
{
    chain_begin();
    const PairParams<T> p = *params_dev;
    DevHeader* hp = p.h;
    if (hp->status & RG_FATAL) return;
    const int nx = hp->nx, ny = hp->ny, S = hp->group_cells, Sy = hp->group_cells_y;
    const uint32_t gx = (uint32_t)hp->gx;
    const uint32_t gy = (uint32_t)((ny + Sy - 1) / Sy);
    const uint32_t num_groups = (uint32_t)hp->num_groups;
    const int lane = threadIdx.x & 31;
    for (uint32_t g0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; g0 < num_groups; g0 += gridDim.x * blockDim.x) {
        const uint32_t grp = g0 + lane;
        bool has = false;
        if (grp < num_groups) {
            const uint32_t row = grp / gx;
            const int ix = (int)(grp - row * gx);
            const int cz = (int)(row / gy), iy = (int)(row - (uint32_t)cz * gy);
            const int cx0 = ix * S, cx1 = min(cx0 + S, nx) - 1;
            const int cy0 = iy * Sy, cy1 = min(cy0 + Sy, ny) - 1;
            has = p.tcstart[((uint32_t)cz * ny + cy0) * nx + cx0] != p.tcstart[((uint32_t)cz * ny + cy0) * nx + cx1 + 1];
            if (!has && cy1 > cy0)
                has = p.tcstart[((uint32_t)cz * ny + cy1) * nx + cx0] != p.tcstart[((uint32_t)cz * ny + cy1) * nx + cx1 + 1];
        }
        const uint32_t m = __ballot_sync(0xffffffffu, has);
        uint32_t base = 0;
        if (lane == 0 && m) base = atomicAdd(&hp->active_groups, (uint32_t)__popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (has) glist[base + __popc(m & lanemask_lt())] = grp;
    }
}

// ------------------------------------------------------------------------------------------
// rg_count: degrees and hit bits.  Lane l holds the coordinates of candidates l, 32 + l, 64 + l, ... of its warp's list in
// registers, two candidates to a packed register pair, and the targets pass by one at a time, from shared memory: the test loop is
// unrolled over the whole list.  A warp takes the next group when it is done with one.
// Two tests a pair: d <= r^2, and d above the self-distance limit.  The second is made for the two blocks of 64 candidates only that
// hold the records of the targets' own cell rows, for records elsewhere are further away (targets next to the faces of these rows are
// tested again in full; lists whose own records touch three blocks, and lists of several chunks, take both tests everywhere); for these
// two blocks to be the same registers in every group the blocks are loaded in turned order.
// The bits of a target go to shared memory and leave it, with the degrees, for 16 targets together.
// Bound by the latency of its loads, its issue slots (60 % busy) and the FMA pipe (40 %): 156 instructions a target of the liquid, 56 of
// them tests; 207 without the items above.  Before and after: 266 -> 207 us (liquid, 1 M atoms, 5 A), 309 -> 259 (a rank's 1 M of the
// 8 M copper atoms), 177 -> 163 (silicon in double precision, 500 k atoms, 6 A), 46 -> 39 (liquid, 131 k), 9.5 -> 8.3 (1 k).
// Distances from the matrix units (halves of split coordinates, pairs near the cutoff again) took 482 us: operand moves and the
// 8 cycles of an m16n8k16.  The next group's look-up, or its candidates, copied ahead to shared memory: 218 and 231 us.
// ------------------------------------------------------------------------------------------
// Five blocks of four warps: 96 registers; float without spills, double with 104 bytes of stores and 112 of loads.  Six and 80: 213 us, 284 for
// the rank's copper.  Eight waves of blocks in place of the counter: 222.  Double with four, five, six and seven blocks, degrees of 200 k
// atoms of the liquid, whole call: 219, 222, 219 and 217 us at 6 A, 254, 259, 269 and 274 at 7 A; the crystal on a shell (exact_hits_call)
// 428, 400, 401 and 360.
constexpr int COUNT_WARPS = 4;
constexpr int COUNT_BLOCKS = 5;
constexpr int COUNT_TARGETS = 16;   // staged together

// A pair as the result of an instruction: pairs that are copies (of two words of different loads, of one word twice, of a
// uniform register) are made again in front of every use, two moves each time: 8 of 19 instructions a block.  nothing: {-0, -0}
__device__ __forceinline__ unsigned long long f32x2_kept(float lo, float hi, unsigned long long nothing)
{
    unsigned long long r = f32x2_pack(lo, hi);
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(r) : "l"(nothing));
    return r;
}

// Thresholds of a distance test, negated and twice: a bit is set when lo <= d < hi, where lo and hi are the floats behind the bounds
// of "d > near && d <= upto", and hi >= lo.  A difference of two floats is zero only for equal ones, so the signs of d - lo and
// d - hi are exact, and that of their product (which keeps it when it underflows) is set between the two.  Two packed
// additions, a packed product and a funnel shift a bit: as compares and selects the bits kept the ALU pipe busier than the
// distances the FMA pipe (289 us against 276, liquid of a million atoms).
struct SignTest { float2 lo, hi; };
__device__ __forceinline__ SignTest sign_test(float near, float upto)
{
    const float lo = nextafterf(near, INFINITY), hi = fmaxf(nextafterf(upto, INFINITY), lo);
    return {make_float2(-lo, -lo), make_float2(-hi, -hi)};
}
// From shared memory, every time: registers are short in the test loop.
__device__ __forceinline__ unsigned long long f32x2_load(const float2& at)
{
    unsigned long long r;
    asm volatile("ld.shared.b64 %0, [%1];" : "=l"(r) : "r"((uint32_t)__cvta_generic_to_shared(&at)));
    return r;
}
__device__ __forceinline__ unsigned long long f32x2_add(unsigned long long a, unsigned long long b)
{
    unsigned long long r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// bits = bits << 2 with the signs of the two halves of a (the upper one first)
__device__ __forceinline__ void push_signs(unsigned long long a, uint32_t& bits)
{
    uint32_t s0, s1;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(s0), "=r"(s1) : "l"(a));
    bits = __funnelshift_l(s1, bits, 1);
    bits = __funnelshift_l(s0, bits, 1);
}
__device__ __forceinline__ void test_x2(unsigned long long d, unsigned long long lo, unsigned long long hi, uint32_t& bits)
{
    unsigned long long a = f32x2_add(d, lo);
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(a) : "l"(f32x2_add(d, hi)));
    push_signs(a, bits);
}

struct CountTests {
    SignTest hit;                // single precision: decides; double: d decided to be a neighbour
    SignTest may;                // double: d may be one
    float2 middle;               // double: minus the middle of the undecided distances around the cutoff
    float half;                  //         and their reach on both sides
};
// What a warp keeps of its group, in shared memory.
struct CountGroup {
    uint32_t tb0, n0, tb1, ntot;   // targets of the two rows
    int cbeg, clen;                // chunk of the candidate list
    int turn;                      // block of 64 that the first registers hold
    float ylo, yhi, zlo, zhi;      // where a target's cell coordinates are clear of the faces of its rows
    int write_masks, first, last, all_exact;
    uint32_t unsettled;            // double: targets that the float tests outside the own rows (FULL: anywhere) leave open
    __device__ __forceinline__ uint32_t target(uint32_t k) const volatile { return k < n0 ? tb0 + k : tb1 + (k - n0); }
};
struct CountWarp {
    float4 target[COUNT_TARGETS][2];            // {x, x, y, y}, {z, z, entry, -}
    unsigned short mask[COUNT_TARGETS][32];
    RunIndex index;
    CountGroup group;
    int pad;
};
struct CountCells { float gmin_y, gmin_z, res_inv; };

// The candidates of a target given by `which` (bit s: place 32 s + lane of the chunk) by the expression that decides.
__device__ __forceinline__ uint32_t exact_hits(const Vec4<float>* spos, const Vec4<float>* target, const float r2, uint32_t which, const RunIndex& index, int cbeg,
                                               int clen, int lane, uint32_t le)
{
    uint32_t hits = 0;
    while (which) {
        const int s = __ffs((int)which) - 1, j = 32 * s + lane;
        which &= which - 1;
        if (j >= clen) continue;  // padding
        const Vec4<float> c = spos[index.record(s, le) + cbeg + j], a = *target;
        const float d = dist2<float>(a.x, a.y, a.z, c.x, c.y, c.z);
        if (d <= r2 && d > 1e-8f) hits |= 1u << s;
    }
    return hits;
}
// Out of line in double, where it is called for every target with an undecided candidate: the copies of the test loop overran the
// instruction cache (176 us against 160, silicon of 500 k atoms).  In single precision the call costs more (207 against 224, liquid of 1 M).
// Two records in flight: the crystal with its cutoff on a shell, below, takes 430 us with one, 402 with two, 418 with three, 446 with four.
__device__ __noinline__ uint32_t exact_hits_call(const Vec4<double>* spos, const Vec4<double>* target, const double r2, uint32_t which, const RunIndex& index,
                                                 int cbeg, int clen)
{
    const int lane = lane_id();
    const uint32_t le = 0xffffffffu >> (31 - lane);
    const Vec4<double> a = *target;
    uint32_t hits = 0;
    while (which) {
        // the second may be the first again; a padding place reads the last record
        const int s0 = __ffs((int)which) - 1;
        which &= which - 1;
        const int s1 = which ? __ffs((int)which) - 1 : s0, j0 = 32 * s0 + lane, j1 = 32 * s1 + lane;
        which &= which - 1;
        const Vec4<double> c0 = spos[index.record(s0, le) + cbeg + min(j0, clen - 1)], c1 = spos[index.record(s1, le) + cbeg + min(j1, clen - 1)];
        const double d0 = dist2<double>(a.x, a.y, a.z, c0.x, c0.y, c0.z), d1 = dist2<double>(a.x, a.y, a.z, c1.x, c1.y, c1.z);
        if (j0 < clen && d0 <= r2 && d0 > (double)1e-8f) hits |= 1u << s0;
        if (j1 < clen && d1 <= r2 && d1 > (double)1e-8f) hits |= 1u << s1;
    }
    return hits;
}

// The targets of a group against the chunk's candidates, at most 64 NB of them.  FULL: both tests for all blocks.
template <typename T, int NB, bool FULL>
__device__ __forceinline__ void count_group(const PairParams<T>& p, CountWarp& w, const volatile CountCells& cells, const CountTests& test, int& max_degree, const int lane,
                                            const uint32_t le)
{
    volatile CountGroup& g = w.group;
    constexpr int OWN = FULL ? NB : 2;
    constexpr uint32_t ALL_BITS = 0xffffu >> (16 - 2 * NB);
    unsigned long long cx[NB], cy[NB], cz[NB];
    {
        const float4* const src = p.sscan + g.cbeg;
        int b0 = g.turn;
        const int clen = g.clen;
        const unsigned long long nothing = 0x8000000080000000ull;
#pragma unroll
        for (int b = 0; b < NB; b++) {
            float4 v[2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                // a padding place reads the last record; x alone keeps it out of every cutoff, its distance is infinite
                const int j = 64 * b0 + 32 * i + lane;
                v[i] = src[w.index.record(2 * b0 + i, le) + min(j, clen - 1)];
                if (j >= clen) v[i].x = 3.0e38f;
            }
            cx[b] = f32x2_kept(-v[0].x, -v[1].x, nothing);
            cy[b] = f32x2_kept(-v[0].y, -v[1].y, nothing);
            cz[b] = f32x2_kept(-v[0].z, -v[1].z, nothing);
            b0 = b0 + 1 == NB ? 0 : b0 + 1;
        }
    }
    const unsigned long long upto = f32x2_load(sizeof(T) == 8 ? test.middle : test.hit.hi);
    const int turn = 2 * (NB - g.turn);
#pragma unroll 1
    for (uint32_t k0 = 0; k0 < g.ntot; k0 += COUNT_TARGETS) {
        const int n = (int)min(g.ntot - k0, (uint32_t)COUNT_TARGETS);
        uint32_t again = 0;   // targets to be tested again in full
        {
            const float4 v = p.tscan[g.target(k0 + min(lane, n - 1))];   // w = entry
            __syncwarp();
            if (lane < n) {
                w.target[lane][0] = make_float4(v.x, v.x, v.y, v.y);
                w.target[lane][1] = make_float4(v.z, v.z, v.w, 0.0f);
            }
            if constexpr (!FULL) {
                const float fy = (v.y - cells.gmin_y) * cells.res_inv, fz = (v.z - cells.gmin_z) * cells.res_inv;
                const bool clear = fy > g.ylo && fy < g.yhi && fz > g.zlo && fz < g.zhi;
                again = __ballot_sync(0xffffffffu, lane < n && !clear);
            }
            if (sizeof(T) == 8 && g.all_exact) again = 0xffffu >> (COUNT_TARGETS - n);
            __syncwarp();
        }
#pragma unroll 1
        for (int k = 0; k < n; k++) {
            const ulonglong2 axy = *reinterpret_cast<const ulonglong2*>(&w.target[k][0]);
            const unsigned long long az = *reinterpret_cast<const unsigned long long*>(&w.target[k][1]);
            uint32_t bits = 0, maybe = 0;
            float closest = INFINITY;
            const unsigned long long lo = f32x2_load(test.hit.lo);
            unsigned long long hi = 0, may_lo = 0, may_hi = 0;
            if (sizeof(T) == 8) {
                hi = f32x2_load(test.hit.hi);
                may_lo = f32x2_load(test.may.lo);
                may_hi = f32x2_load(test.may.hi);
            }
#pragma unroll
            for (int b = NB - 1; b >= 0; b--) {
                const unsigned long long d = dist2_x2(axy.x, axy.y, az, cx[b], cy[b], cz[b]);
                if (b < OWN) {
                    test_x2(d, lo, sizeof(T) == 8 ? hi : upto, bits);
                    if (sizeof(T) == 8) test_x2(d, may_lo, may_hi, maybe);
                } else {
                    const unsigned long long a = f32x2_add(d, upto);
                    push_signs(a, bits);
                    if (sizeof(T) == 8) {
                        float a0, a1;
                        asm("mov.b64 {%0, %1}, %2;" : "=f"(a0), "=f"(a1) : "l"(a));
                        asm("min.f32 %0, %0, %1, %2;" : "+f"(closest) : "f"(fabsf(a0)), "f"(fabsf(a1)));
                    }
                }
            }
            // bit 2 b + i of the registers is bit 2 (b + turn mod NB) + i of the list
            auto turned = [&](uint32_t v) { return ((v | (v << (2 * NB))) >> turn) & ALL_BITS; };
            bits = turned(bits);
            if constexpr (sizeof(T) == 8) {
                const uint32_t undecided = turned(maybe) & ~bits & turned(0xffffu >> (16 - 2 * OWN));
                if (!g.all_exact) {
                    if (undecided) bits |= exact_hits_call(p.spos, p.tpos + g.target(k0 + k), p.r2, undecided, w.index, g.cbeg, g.clen);
                }
                if (FULL ? undecided != 0u : closest <= test.half) again |= 1u << k;
            }
            w.mask[k][lane] = (unsigned short)bits;
        }
        __syncwarp();
        if (sizeof(T) == 8) {
            again = __reduce_or_sync(0xffffffffu, again);
            if (again && lane == 0) g.unsettled = g.unsettled + __popc(again);
            if (FULL && !g.all_exact) again = 0u;
        }
#pragma unroll 1
        for (; !(FULL && sizeof(T) == 4) && again; again &= again - 1) {
            const int k = __ffs((int)again) - 1;
            uint32_t bits;
            if constexpr (sizeof(T) == 8) bits = exact_hits_call(p.spos, p.tpos + g.target(k0 + k), p.r2, ALL_BITS, w.index, g.cbeg, g.clen);
            else bits = exact_hits(p.spos, p.tpos + g.target(k0 + k), p.r2, ALL_BITS, w.index, g.cbeg, g.clen, lane, le);
            w.mask[k][lane] = (unsigned short)bits;
            __syncwarp();
        }
        // degrees, and the bits to memory: four lanes a target
#pragma unroll 1
        for (int i0 = 0; i0 < 4 * n; i0 += 32) {
            const int i = i0 + lane, k = min(i >> 2, n - 1);
            const uint4 m = reinterpret_cast<const uint4*>(w.mask[k])[i & 3];
            const uint32_t t = g.target(k0 + k);
            int degree = __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
            degree += __shfl_xor_sync(0xffffffffu, degree, 1);
            degree += __shfl_xor_sync(0xffffffffu, degree, 2);
            if (i < 4 * n) {
                if (g.write_masks) reinterpret_cast<uint4*>(p.hitmask + (size_t)t * 32)[i & 3] = m;
                if ((i & 3) == 0) {
                    if (!g.first) degree += (int)p.tcount[t];
                    p.tcount[t] = (uint32_t)degree;
                    if (g.last) {
                        if (p.counts_out != nullptr) p.counts_out[__float_as_int(w.target[k][1].z)] = degree;  // in caller order
                        max_degree = max(max_degree, degree);
                    }
                }
            }
        }
        __syncwarp();
    }
}

template <typename T>
__global__ void __launch_bounds__(COUNT_WARPS * 32, COUNT_BLOCKS)
rg_count_kernel(const PairParams<T> p)
{
    chain_begin();
    __shared__ CountWarp warps[COUNT_WARPS];
    __shared__ GroupShape shape;
    __shared__ CountCells cells;
    __shared__ CountTests test;
    constexpr bool ONE_BLOCK = sizeof(T) == 4;   // a copy of the loop for one block of 64
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    CountWarp& w = warps[warp];
    const uint32_t lt = lanemask_lt(), le = lt | (1u << lane);
    DevHeader* hp = p.h;
    if (hp->status & RG_FATAL) return;
    int warp_max_slots = 0, max_degree = 0;
    if (lane == 0) w.group.unsettled = w.group.ntot = 0u;
    if (threadIdx.x == 0) {
        shape = group_shape(hp);
        // double positions are scanned relative to the grid's origin
        cells.gmin_y = sizeof(T) == 8 ? 0.0f : (float)hp->gmin[1];
        cells.gmin_z = sizeof(T) == 8 ? 0.0f : (float)hp->gmin[2];
        cells.res_inv = (float)hp->res_inv;
    }
    if (threadIdx.x == 32) {
        test.hit = sizeof(T) == 8 ? sign_test(hp->test_near, hp->test_lo) : sign_test(1e-8f, (float)p.r2);
        test.may = sizeof(T) == 8 ? sign_test(hp->test_equal_is_near ? 0.0f : -1.0f, hp->test_hi) : test.hit;
        const float middle = 0.5f * (hp->test_lo + hp->test_hi);
        test.middle = make_float2(-middle, -middle);
        test.half = 1.001f * fmaxf(middle - hp->test_lo, hp->test_hi - middle);
    }
    const uint32_t num_groups = p.glist ? hp->active_groups : (uint32_t)hp->num_groups;  // < 2^31: never more groups than cells
    // Groups are taken one by one, or, from 128 a warp on, several in a row (a power of two, 64 to 128 takings a warp): every taking is an
    // addition to one address, and a thin gas has a group for every atom or two.  Degrees of 1 M atoms, 0.001 per A^3, 5 A, whole call: 937 us one by
    // one, 876 so; 300 k atoms in dense pockets of a gas 402 and 295.
    if (threadIdx.x == 0) shape.unused[0] = 1 << (31 - __clz((int)max(num_groups / (64u * COUNT_WARPS * gridDim.x), 1u)));
    __syncthreads();
    const int lane_run = group_lane_run(shape, lane);
    const bool all_exact = sizeof(T) == 8 && hp->test_lo < 0.0f;  // coordinates out of the float test's range (float_test)
    // Records within the self-distance limit of a target (1e-4, or what the float test calls near) lie in the target's cell row
    // but for targets this close to its faces, in cells: the distance, and the rounding of the two cell coordinates.
    const float skin = 1.01f * sqrtf(sizeof(T) == 8 ? hp->test_near : 1e-8f) * (float)hp->res_inv + 1e-6f * (float)(16 + max(hp->ny, hp->nz));

    const uint32_t nwarps = gridDim.x * COUNT_WARPS;
    const volatile int& in_a_row = shape.unused[0];
    uint32_t gi = (blockIdx.x * COUNT_WARPS + warp) * (uint32_t)in_a_row;
#pragma unroll 1
    while (gi < num_groups) {
        const uint32_t grp = p.glist ? p.glist[gi] : gi;
        uint32_t following = gi + 1u;
        if (lane == 0) {
            const uint32_t taken = (uint32_t)in_a_row;
            if ((following & (taken - 1u)) == 0u) following = nwarps * taken + atomicAdd(&hp->count_next, taken);
        }
        const GroupRows d = fetch_group_rows(shape, p.tcstart, p.cstart, grp, lane_run);
        const int run_a = d.run_a, run_len = d.run_e - d.run_a;
        volatile CountGroup& g = w.group;   // all lanes write the same
        const uint32_t n0 = d.te0 - d.tb0, ntot = n0 + (d.te1 - d.tb1);
        if (ntot != 0) {
            // Double: a target that is tested again takes three or four times the loop (all places of its list by the deciding expression), so both tests
            // everywhere where more than one in 16 of the warp's group before were.  Degrees of 512 k atoms of an ideal silicon crystal with the cutoff on
            // a shell of neighbours, whole call: 865 us without this line, 402 with it (253 off the shell, with and without).
            const bool unsettled = sizeof(T) == 8 && 16u * g.unsettled > g.ntot;
            __syncwarp();
            if (sizeof(T) == 8) g.unsettled = 0u;
            g.tb0 = d.tb0;
            g.tb1 = d.tb1;
            g.n0 = n0;
            g.ntot = ntot;
            const int run_end = (int)warp_incl_scan_u32((uint32_t)run_len), run_off = run_end - run_len, L = __shfl_sync(0xffffffffu, run_end, 31);
            const int nslots = (L + 31) >> 5;
            g.write_masks = nslots <= RG_MASK_SLOTS;
            g.all_exact = all_exact;
            warp_max_slots = max(warp_max_slots, nslots);
            if (nslots > RG_MASK_SLOTS && lane == 0) p.long_list[atomicAdd(reinterpret_cast<uint32_t*>(&hp->reserved[1]), 1u)] = grp;
            g.ylo = (float)d.cy0 + skin;
            g.yhi = (float)(d.cy1 + 1) - skin;
            g.zlo = (float)d.cz + skin;
            g.zhi = (float)(d.cz + 1) - skin;
            int own_beg, own_end;
            {
                // the runs that hold the targets' own rows
                const volatile GroupShape& f = shape;
                const int own = f.pad * (f.sy + 2 * f.pad) + f.pad;
                own_beg = __shfl_sync(0xffffffffu, run_off, own);
                own_end = __shfl_sync(0xffffffffu, run_end, own + d.cy1 - d.cy0);
            }
#pragma unroll 1
            for (int cbeg = 0; cbeg < L; cbeg += RG_MASK_SLOTS * 32) {
                const int clen = min(RG_MASK_SLOTS * 32, L - cbeg);
                // both tests everywhere where the own records are not in two blocks, and in lists of several chunks
                const bool everywhere = unsettled || L > RG_MASK_SLOTS * 32 || ((own_end - 1) >> 6) - (own_beg >> 6) > 1;
                __syncwarp();
                g.cbeg = cbeg;
                g.clen = clen;
                g.first = cbeg == 0;
                g.last = cbeg + RG_MASK_SLOTS * 32 >= L;
                g.turn = everywhere ? 0 : own_beg >> 6;
                if (ONE_BLOCK && L <= 64) w.index.set_short(run_a, run_off, run_len, lane, lt);   // no more than its two words are read below
                else w.index.set(run_a, run_off, run_len, cbeg, lane, lt);
                auto run = [&](auto nb, auto full) {
                    count_group<T, decltype(nb)::value, decltype(full)::value>(p, w, cells, test, max_degree, lane, le);
                };
                // Copies of the test loop for 1 (float), 2, 4, 5, 6, 7 and 8 blocks of 64, with both tests everywhere for 1, 2, 4 and 8; a chunk takes the
                // smallest that holds it, with padding.  The last chunk of a list is often short: 200 k atoms of the liquid, degrees
                // alone, at 7 A (512 + 32 places) 222 us with the copy for 8 blocks for all chunks and 199 so, at 9 A (512 + 512 + 131) 247
                // and 224.  No copies for 5, 6 and 7: what the loop saves the instruction cache loses (8 A, 512 + 300: 212 us with
                // one for 5, 207 without; in double 287 and 266; 245 and 355 with the copy for 8 inlined twice).  The one for 1, that gas: 876 ->
                // 826; in double it costs the others (jittered silicon of 500 k atoms 268 -> 278 us).
                const int blocks = (clen + 63) >> 6;
                switch (everywhere && blocks > 2 ? (blocks > 4 ? 10 : 9) : blocks) {
                case 1: if constexpr (ONE_BLOCK) { run(std::integral_constant<int, 1>(), std::true_type()); break; }
                case 2: run(std::integral_constant<int, 2>(), std::true_type()); break;
                case 3:
                case 4: run(std::integral_constant<int, 4>(), std::false_type()); break;
                case 5: run(std::integral_constant<int, 5>(), std::false_type()); break;
                case 6: run(std::integral_constant<int, 6>(), std::false_type()); break;
                case 7: run(std::integral_constant<int, 7>(), std::false_type()); break;
                case 8: run(std::integral_constant<int, 8>(), std::false_type()); break;
                case 9: run(std::integral_constant<int, 4>(), std::true_type()); break;
                default: run(std::integral_constant<int, 8>(), std::true_type()); break;
                }
            }
            // a group whose neighbourhood holds no source at all still owes its targets a zero
            if (L == 0)
                for (uint32_t k = lane; k < ntot; k += 32) p.tcount[g.target(k)] = 0;
        }
        gi = __shfl_sync(0xffffffffu, following, 0);
    }
    // largest degree; a candidate list too long for the hit bits: the edge writer has to recompute distances
    max_degree = __reduce_max_sync(0xffffffffu, max_degree);
    if (lane == 0 && max_degree > (int)__ldcg(&hp->max_degree)) atomicMax(&hp->max_degree, (uint32_t)max_degree);
    if (lane == 0 && warp_max_slots > RG_MASK_SLOTS) atomicMax(&hp->reserved[0], (long long)warp_max_slots);
}

template <typename T>
__global__ void __launch_bounds__(PAIR_THREADS, 4)
rg_pair_kernel(const PairParams<T>* params_dev, long long* ei,
               float* shifts, T* d2out, const long long E, const GlueArgs glue, const int all_groups,
               long long* total)
{
    chain_begin();
    const PairParams<T> p = *params_dev;
    extern __shared__ __align__(32) unsigned char smem_raw[];
    constexpr int CAP = PAIR_CAND_BYTES / (int)sizeof(Vec4<T>);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char* wbase = smem_raw + warp * PAIR_WARP_BYTES;
    Vec4<T>* cand = reinterpret_cast<Vec4<T>*>(wbase);
    uint32_t* codes = reinterpret_cast<uint32_t*>(wbase + PAIR_CAND_BYTES);
    unsigned short* listA = reinterpret_cast<unsigned short*>(wbase + PAIR_CAND_BYTES + PAIR_CODE_BYTES);
    unsigned short* listB = listA + PAIR_LIST;
    int* delta = reinterpret_cast<int*>(wbase + PAIR_CAND_BYTES + PAIR_CODE_BYTES + PAIR_LIST * 4);
    uint32_t* flags = reinterpret_cast<uint32_t*>(delta + 32);
    const uint32_t le = lanemask_lt() | (1u << (threadIdx.x & 31));

    DevHeader* hp = p.h;
    if (hp->status & RG_FATAL) return;
    // behind rg_fillmask_kernel the writing pass has only the groups whose candidate list was too long for the hit bits
    const bool long_only = !all_groups;
    if (long_only && hp->reserved[1] == 0) return;
    if (total != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *total = E;
    const int nx = hp->nx, ny = hp->ny, nz = hp->nz, S = hp->group_cells, Sy = hp->group_cells_y, pad = hp->pad;
    const uint32_t gx = (uint32_t)hp->gx;
    const uint32_t gy = (uint32_t)((ny + Sy - 1) / Sy);
    const uint32_t num_groups = long_only ? (uint32_t)hp->reserved[1]
                                          : (p.glist ? hp->active_groups : (uint32_t)hp->num_groups);  // < 2^31: never more groups than cells
    const int Wd = 2 * pad + 1, Wy = Sy + 2 * pad, nrun = Wy * Wd;
    const int lane_dy = (lane % Wy) - pad, lane_dz = (lane / Wy) - pad;
    const T r2 = p.r2;
    const T eps = (T)1e-8f;
    const uint32_t lt = lanemask_lt();

    const uint32_t nwarps = gridDim.x * PAIR_WARPS;
    // A few listed groups leave the chip idle but for the chain of one warp each: then eight warps share a group's targets (graph
    // calls of a liquid at 6 A, where one list in some hundred is long: 8 k atoms 166 -> 117 us, 20 k 179 -> 129, 60 k 160 -> 153).
    const uint32_t parts = long_only && num_groups * (uint32_t)PAIR_SHARE <= nwarps ? (uint32_t)PAIR_SHARE : 1u;
    for (uint32_t item = blockIdx.x * PAIR_WARPS + warp; item < num_groups * parts; item += nwarps) {
        const uint32_t gi = item / parts, part = item - gi * parts;
        const uint32_t grp = long_only ? p.long_list[gi] : (p.glist ? p.glist[gi] : gi);
        const uint32_t row = grp / gx;
        const int ix = (int)(grp - row * gx);
        const int cz = (int)(row / gy), iy = (int)(row - (uint32_t)cz * gy);
        const int cx0 = ix * S, cx1 = min(cx0 + S, nx) - 1;
        const int cy0 = iy * Sy, cy1 = min(cy0 + Sy, ny) - 1;
        // targets: one contiguous run per target row
        uint32_t tb[2], te[2];
        tb[0] = p.tcstart[((uint32_t)cz * ny + cy0) * nx + cx0];
        te[0] = p.tcstart[((uint32_t)cz * ny + cy0) * nx + cx1 + 1];
        tb[1] = te[1] = 0;
        if (cy1 > cy0) {
            tb[1] = p.tcstart[((uint32_t)cz * ny + cy1) * nx + cx0];
            te[1] = p.tcstart[((uint32_t)cz * ny + cy1) * nx + cx1 + 1];
        }
        if (tb[0] == te[0] && tb[1] == te[1]) continue;

        // contiguous source runs: lane r owns run (y row, z row)
        int run_a = 0, run_len = 0;
        if (lane < nrun) {
            const int yy = cy0 + lane_dy, zz = cz + lane_dz;
            if (yy >= 0 && yy < ny && yy <= cy1 + pad && zz >= 0 && zz < nz) {
                const uint32_t b = ((uint32_t)zz * ny + yy) * nx;
                const uint32_t a = p.cstart[b + max(cx0 - pad, 0)];
                const uint32_t e = p.cstart[b + min(cx1 + pad, nx - 1) + 1];
                run_a = (int)a;
                run_len = (int)(e - a);
            }
        }
        int L;
        const int run_off = warp_excl_scan(run_len, lane, &L);
        __syncwarp();
        runs_compact(delta, run_a, run_off, run_len, lt);

        for (int cbeg = 0, chunk = 0; cbeg < L; cbeg += CAP, chunk++) {
            const int clen = min(CAP, L - cbeg);
            const int clen32 = (clen + 31) & ~31;
            const bool more_chunks = cbeg + CAP < L;
            // dense staging: slot j of the list holds flattened candidate cbeg + j; all loads of a chunk are
            // independent
            int rank_base = runs_flags(flags, run_off, run_len, lane, cbeg);
            for (int j = lane, sw = 0; j < clen32; j += 32, sw++) {
                const uint32_t word = flags[sw];
                const int r = rank_base + __popc(word & le) - 1;
                rank_base += __popc(word);
                if (j < clen) {
                    const int gidx = delta[r] + cbeg + j;
                    if (sizeof(Vec4<T>) == 16) {
                        cp_async<16>(&cand[j], &p.spos[gidx]);  // w = atom id
                    } else {
                        cp_async<16>(&cand[j], &p.spos[gidx]);
                        cp_async<16>(reinterpret_cast<char*>(&cand[j]) + 16, reinterpret_cast<const char*>(&p.spos[gidx]) + 16);
                    }
                    cp_async<4>(&codes[j], &p.smeta[gidx].y);
                }
            }
            if (clen + lane < clen32) {
                Vec4<T> c;
                c.x = c.y = c.z = (T)3.0e38f;  // never within the cutoff
                c.w = (T)0;
                cand[clen + lane] = c;
            }
            cp_async_wait_all();
            __syncwarp();

#pragma unroll
          for (int yr = 0; yr < 2; yr++) {
            const uint32_t t0 = tb[yr], t1 = te[yr];
            // two targets share every candidate load
            for (uint32_t t = t0 + 2 * part; t < t1; t += 2 * parts) {
                const bool has2 = (t + 1 < t1);
                const Vec4<T> tpA = p.tpos[t];
                const Vec4<T> tpB = p.tpos[has2 ? t + 1 : t];
                const T ax = tpA.x, ay = tpA.y, az = tpA.z, bx = tpB.x, by = tpB.y, bz = tpB.z;
                int prodA = 0, prodB = 0;
                if (chunk != 0) {
                    prodA = (int)p.tcount[t];
                    prodB = has2 ? (int)p.tcount[t + 1] : 0;
                }
                {
                    int4 tmA = p.tmeta[t];
                    int4 tmB = p.tmeta[has2 ? t + 1 : t];
                    const long long baseA = p.toffset[t], baseB = p.toffset[has2 ? t + 1 : t];
                    int n = 0, nB = 0;  // parked hits of target A / target B
                    for (int k = 0; k < clen32; k += 32) {
                        const int j = k + lane;
                        const Vec4<T> c = cand[j];
                        const T dA = dist2<T>(ax, ay, az, c.x, c.y, c.z);
                        const T dB = dist2<T>(bx, by, bz, c.x, c.y, c.z);
                        const bool hitA = (dA <= r2) && (dA > eps);
                        const bool hitB = has2 && (dB <= r2) && (dB > eps);
                        {
                            // each target parks the slots of its hits in its own half of the list; the index in
                            // the half is the position inside the target's edge run since the last write-out
                            const uint32_t mA = __ballot_sync(0xffffffffu, hitA);
                            const uint32_t mB = __ballot_sync(0xffffffffu, hitB);
                            if (hitA) listA[n + __popc(mA & lt)] = (unsigned short)j;
                            if (hitB) listB[nB + __popc(mB & lt)] = (unsigned short)j;
                            n += __popc(mA);
                            nB += __popc(mB);
                            if (n > PAIR_LIST - 32 || nB > PAIR_LIST - 32 || k + 32 >= clen32) {
                                __syncwarp();
#pragma unroll
                                for (int sel = 0; sel < 2; sel++) {
                                    const int cntX = sel ? nB : n;
                                    const unsigned short* lx = sel ? listB : listA;
                                    const int4 tm = sel ? tmB : tmA;
                                    const long long bX = (sel ? baseB + prodB : baseA + prodA);
                                    for (int i = lane; i < cntX; i += 32) {
                                        const int jh = lx[i];
                                        const Vec4<T> ch = cand[jh];
                                        const uint32_t code = codes[jh];
                                        const long long e = bX + i;
                                        const long long sa = (long long)real_to_bits(ch.w);
                                        ei[e] = glue.id_map ? glue.id_map[sa] : sa;
                                        ei[E + e] = glue.id_map ? glue.id_map[tm.x] : (long long)tm.x;
                                        glue_write(glue, shifts, e, (int)(code & 1023u) - 512 + tm.y, (int)((code >> 10) & 1023u) - 512 + tm.z,
                                                   (int)((code >> 20) & 1023u) - 512 + tm.w);
                                        if (d2out != nullptr) {
                                            const T tx = sel ? bx : ax, ty = sel ? by : ay, tz = sel ? bz : az;
                                            d2out[e] = dist2<T>(tx, ty, tz, ch.x, ch.y, ch.z);
                                        }
                                    }
                                }
                                prodA += n;
                                prodB += nB;
                                n = 0;
                                nB = 0;
                                __syncwarp();
                            }
                        }
                    }
                    if (more_chunks && lane == 0) {
                        p.tcount[t] = (uint32_t)prodA;
                        if (has2) p.tcount[t + 1] = (uint32_t)prodB;
                    }
                }
            }
          }
        }
    }
}

// ------------------------------------------------------------------------------------------
// Edge writer driven by the hit bits of the counting pass, for the groups whose candidate list is not longer than
// RG_MASK_SLOTS * 32 records (the usual case: about 27 cells of 8-16 atoms).  No distance is tested again.
//
// The 64 bytes of a target are 512 bits: bit 16 l + s belongs to the candidate at place 32 s + l.  The targets of a cell row
// follow one another, and so do their edges: the bits of a row that are set, in order, ARE its edges.  A lane takes 64 bits
// (eight lanes a target, both rows of the group in one go), a prefix sum gives it the place of its first edge, and it puts
// what belongs to its bits into the warp's buffer; the buffer goes out 32 edges at a time.
// In most groups all candidates have one shift code, and then all shifts are zero (the targets are candidates too): zeros are
// written 32 bytes a lane, and a group's edges need the two indices only.
// Bound by the latency of its loads and by instructions (4 an edge, issue slots 57 % busy), not by the 1.47 GB it writes (4.9 TB/s).  Target by target, with a prefix sum, a list and two rounds of 32 edges for each of them, and three
// stores with a stride of 12 bytes for the shifts: 240 M.  Before and after: 381 -> 308 us (liquid, 1 M atoms), 742 -> 611 (a
// rank's 1 M of the 8 M copper atoms, with Cartesian shifts), 189 -> 160 (silicon, double precision), 15 -> 13 (1 k atoms, where
// every group is at the boundary), 25 -> 25 (32 k atoms).  What is loaded ahead is not touched until its turn: a subtraction
// behind the loads of the next group's runs or of the rows' places in the output waits for them (322 -> 308 us).  298 with the look-up by
// two loads a lane (fetch_group).
// Bulk copies of a block of zeros for the shifts: no gain.
// ------------------------------------------------------------------------------------------
constexpr int FM_TABLE = 33 * (RG_MASK_SLOTS * 32 / 32);   // a word of padding every 32 bits: the lanes of a slot fall into 32 banks
// Seven blocks of four warps: 72 registers, and 177 of the 228 KB of shared memory, which leaves L1 for the records that neighbouring
// groups share (liquid, 1 M atoms: 320 us; eight blocks 338, six 336; ten blocks of 48 registers and hardly any L1, with an earlier
// form of the loop, 445 against 368).  Small blocks and eight waves of them even out the SMs (four waves 367, eight 350).
constexpr int EDGE_WARPS = 4, EDGE_BLOCKS = 7, EDGE_WAVES = 8;
constexpr int FM_EDGES = 384;                              // edges collected before they are written (512: 315 us against 306)
struct EdgeWarp {
    union {
        uint2 edge[FM_EDGES];             // plain groups: {atom, atom of the target}
        struct {
            uint32_t mixed[FM_EDGES];     // others: table place | lane of the target << 16
            uint32_t code[FM_TABLE];      //         per bit of a target: shift code of the candidate
        };
    };
    uint32_t table[FM_TABLE];             // per bit of a target: atom of the candidate
    RunIndex index;
};

// The highest set bit s of `bits`, if there is one: table word s goes in front of `at` (bytes of shared memory), which moves back.
__device__ __forceinline__ void put_edge(uint32_t& bits, uint32_t& at, uint32_t table, uint32_t tag)
{
    asm volatile("{\n\t.reg .pred q;\n\t.reg .b32 s, m, a, v;\n\t"
                 "setp.ne.u32 q, %0, 0;\n\t"
                 "bfind.u32 s, %0;\n\t"
                 "shl.b32 m, 1, s;\n\t"
                 "xor.b32 %0, %0, m;\n\t"
                 "mad.lo.u32 a, s, 4, %2;\n\t"
                 "@q ld.shared.u32 v, [a];\n\t"
                 "@q add.u32 %1, %1, -8;\n\t"
                 "@q st.shared.v2.u32 [%1], {v, %3};\n\t}"
                 : "+r"(bits), "+r"(at) : "r"(table), "r"(tag) : "memory");
}
// The same with s itself in place of what the table holds.
__device__ __forceinline__ void put_mixed(uint32_t& bits, uint32_t& at, uint32_t tag)
{
    asm volatile("{\n\t.reg .pred q;\n\t.reg .b32 s, m;\n\t"
                 "setp.ne.u32 q, %0, 0;\n\t"
                 "bfind.u32 s, %0;\n\t"
                 "shl.b32 m, 1, s;\n\t"
                 "xor.b32 %0, %0, m;\n\t"
                 "add.u32 s, s, %2;\n\t"
                 "@q add.u32 %1, %1, -4;\n\t"
                 "@q st.shared.u32 [%1], s;\n\t}"
                 : "+r"(bits), "+r"(at) : "r"(tag) : "memory");
}
// n floats of zero: whole 32-byte sectors, single words at the ends
__device__ __forceinline__ void zero_floats(float* at, int n, int lane)
{
    const int head = min((int)((0u - (uint32_t)(reinterpret_cast<uintptr_t>(at) >> 2)) & 7u), n);
    const int body = (n - head) & ~7, tail = n - head - body;
    if (lane < head) at[lane] = 0.0f;
    at += head;
#pragma unroll 1
    for (int i = 8 * lane; i < body; i += 256)
        asm volatile("st.global.v8.b32 [%0], {%1, %1, %1, %1, %1, %1, %1, %1};" ::"l"(at + i), "r"(0u) : "memory");
    if (lane < tail) at[body + lane] = 0.0f;
}

template <typename T, bool GLUE>
__global__ void __launch_bounds__(EDGE_WARPS * 32, EDGE_BLOCKS)
rg_fillmask_kernel(const PairParams<T>* params_dev, long long* ei, float* shifts, const long long E,
                const GlueArgs glue, long long* total)
{
    chain_begin();
    // the plan's pointers are read where they are used, too
    __shared__ PairParams<T> params;
    __shared__ GroupShape shape;
    const DevHeader* hp = params_dev->h;
    if (hp->status & RG_FATAL) return;
    for (int i = threadIdx.x; i < (int)(sizeof(PairParams<T>) / 4); i += EDGE_WARPS * 32)
        reinterpret_cast<uint32_t*>(&params)[i] = reinterpret_cast<const uint32_t*>(params_dev)[i];
    if (threadIdx.x == 0) shape = group_shape(hp);
    const uint32_t num_groups = params_dev->glist ? hp->active_groups : (uint32_t)hp->num_groups;
    __syncthreads();
    const volatile PairParams<T>& p = params;
    extern __shared__ __align__(32) unsigned char smem_raw[];
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    EdgeWarp& w = reinterpret_cast<EdgeWarp*>(smem_raw)[warp];
    const uint32_t lt = lanemask_lt(), le = lt | (1u << lane);

    if (total != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *total = E;
    const int which = group_lane(shape, lane);
    // Candidates of one shift code: the targets, which are among them, have it too, and every shift of the group is zero.
    // Left out: mapped ids, and Cartesian shifts of which a zero is a negative zero (a column of the cell that is all negative).
    bool may_be_plain = true;
    if constexpr (GLUE) {
        may_be_plain = glue.id_map == nullptr;
        if (glue.cart != nullptr) {
#pragma unroll
            for (int k = 0; k < 3; k++)
                may_be_plain = may_be_plain && __float_as_uint(__fmaf_rn(0.0f, glue.c[6 + k], __fmaf_rn(0.0f, glue.c[3 + k], __fmul_rn(0.0f, glue.c[k])))) == 0u;
        }
    }
    // this lane's place in the table as a lane of the candidate list, and as the holder of 64 bits
    uint32_t* const my_table = w.table + 33 * (lane >> 1) + 16 * (lane & 1);
    const uint32_t my_bits = (uint32_t)__cvta_generic_to_shared(w.table) + 4u * 66u * (uint32_t)(lane & 7);
    const uint32_t edges_at = (uint32_t)__cvta_generic_to_shared(w.edge);

    // the next group is looked up while the current one is written, so that one round trip to memory per group (the candidate
    // records) stays exposed
    static_assert(offsetof(PairParams<T>, tcstart) == offsetof(PairParams<T>, cstart) + sizeof(void*), "read as a pair");
    auto fetch = [&](uint32_t i) {
        const uint32_t* cells = reinterpret_cast<const uint32_t* const volatile*>(&params.cstart)[lane >= GROUP_ROW_LANE ? 1 : 0];
        return fetch_group(shape, cells, p.glist ? p.glist[i] : i, which);
    };

    const uint32_t nwarps = gridDim.x * EDGE_WARPS;
    uint32_t gi = blockIdx.x * EDGE_WARPS + warp;
    if (gi >= num_groups) return;
    GroupDesc nd = fetch(gi);
#pragma unroll 1
    for (; gi < num_groups; gi += nwarps) {
        const GroupDesc d = nd;
        if (gi + nwarps < num_groups) nd = fetch(gi + nwarps);
        const uint32_t tb0 = __shfl_sync(0xffffffffu, (uint32_t)d.run_a, GROUP_ROW_LANE), te0 = __shfl_sync(0xffffffffu, (uint32_t)d.run_e, GROUP_ROW_LANE);
        const uint32_t tb1 = __shfl_sync(0xffffffffu, (uint32_t)d.run_a, GROUP_ROW_LANE + 1), te1 = __shfl_sync(0xffffffffu, (uint32_t)d.run_e, GROUP_ROW_LANE + 1);
        const int n0 = (int)(te0 - tb0), pieces = 8 * (n0 + (int)(te1 - tb1));
        if (pieces == 0) continue;
        // the first bits and the rows' places in the output do not depend on the candidate records: ask for them now
        const uint32_t second = tb1 - (uint32_t)n0;   // + number of a target of the second row among all
        auto target = [&](int i) { return (uint32_t)(i >> 3) + ((i >> 3) < n0 ? tb0 : second); };
        uint2 next_bits = make_uint2(0u, 0u);
        int next_dst = 0;
        if (lane < pieces) {
            const uint32_t t = target(lane);
            next_bits = reinterpret_cast<const uint2*>(p.hitmask + (size_t)t * 32)[lane & 7];
            next_dst = p.tmeta[t].x;
        }
        const long long base0 = p.toffset[tb0], base1 = p.toffset[tb1], end0 = p.toffset[te0], end1 = p.toffset[te1];
        const int run_len = lane < GROUP_ROW_LANE ? d.run_e - d.run_a : 0, run_end = (int)warp_incl_scan_u32((uint32_t)run_len), run_off = run_end - run_len, L = __shfl_sync(0xffffffffu, run_end, 31);
        const int nslots = (L + 31) >> 5;
        if (nslots == 0 || nslots > RG_MASK_SLOTS) continue;  // a longer list has no hit bits: rg_pair_kernel writes that group
        // one or two targets are often without neighbours (a gas of a million atoms, 0.001 per A^3: 433 us without this line, 357
        // with it, 399 target by target); more of them hardly ever are, and the test waits for the bits
        if (pieces <= 16 && !__any_sync(0xffffffffu, (next_bits.x | next_bits.y) != 0u)) continue;

        __syncwarp();
        w.index.set(d.run_a, run_off, run_len, 0, lane, lt);
        // four slots at a time: the four gathers are in flight together before the first is stored
        uint32_t all = 0xffffffffu, any = 0u;
#pragma unroll 1
        for (int s0 = 0; s0 < nslots; s0 += 4) {
            uint2 m[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int j = (s0 + u) * 32 + lane;
                if (j < L) {
                    m[u] = p.smeta[w.index.record(s0 + u, le) + j];
                    all &= m[u].y;
                    any |= m[u].y;
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++)
                if ((s0 + u) * 32 + lane < L) my_table[s0 + u] = m[u].x;
        }
        const bool plain = may_be_plain && __reduce_and_sync(0xffffffffu, all) == __reduce_or_sync(0xffffffffu, any);
        const int edges0 = (int)(end0 - base0), edges1 = (int)(end1 - base1);
        if (plain) {
            zero_floats(shifts + 3 * base0, 3 * edges0, lane);
            zero_floats(shifts + 3 * base1, 3 * edges1, lane);
            if (GLUE && glue.cart != nullptr) {
                zero_floats(glue.cart + 3 * base0, 3 * edges0, lane);
                zero_floats(glue.cart + 3 * base1, 3 * edges1, lane);
            }
        } else {
            uint32_t* const my_code = w.code + (my_table - w.table);
#pragma unroll 1
            for (int s0 = 0; s0 < nslots; s0 += 4) {
                uint32_t m[4];
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if ((s0 + u) * 32 + lane < L) m[u] = p.smeta[w.index.record(s0 + u, le) + (s0 + u) * 32 + lane].y;
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if ((s0 + u) * 32 + lane < L) my_code[s0 + u] = m[u];
            }
        }
        __syncwarp();

        int written = 0;   // edges of the group in front of this step
#pragma unroll 1
        for (int i0 = 0; i0 < pieces; i0 += 32) {
            uint32_t lo = next_bits.x, hi = next_bits.y;
            const int dst = next_dst;
            next_bits = make_uint2(0u, 0u);
            if (i0 + 32 + lane < pieces) {
                const uint32_t t = target(i0 + 32 + lane);
                next_bits = reinterpret_cast<const uint2*>(p.hitmask + (size_t)t * 32)[lane & 7];
                next_dst = p.tmeta[t].x;
            }
            const uint32_t clo = (uint32_t)__popc(lo), chi = (uint32_t)__popc(hi);
            const uint32_t incl = warp_incl_scan_u32(clo + chi);
            const int ntot = (int)__shfl_sync(0xffffffffu, incl, 31);
            int4 tm = make_int4(dst, 0, 0, 0);
            if (!plain && i0 + lane < pieces) tm = p.tmeta[target(i0 + lane)];
            // In one go, or two targets and two targets, or (targets with more neighbours than that) piece by piece.  Piece by
            // piece in place of two and two: 1043 us against 1021 a graph call (liquid of 1 M atoms, 6 A: 90 neighbours).
            const int half = (int)__shfl_sync(0xffffffffu, incl, 15);
            const bool whole = ntot <= FM_EDGES, halves = !whole && max(half, ntot - half) <= FM_EDGES;
            int n;
#pragma unroll 1
            for (int win = 0; win < ntot; win += n) {
                n = whole ? ntot : (halves ? (win == 0 ? half : ntot - half) : min(FM_EDGES, ntot - win));
                if (whole || halves) {
                    const bool mine = whole || (lane < 16) == (win == 0);
                    uint32_t l = mine ? lo : 0u, h = mine ? hi : 0u;
                    if (plain) {
                        uint32_t ahi = edges_at + 8u * (incl - (uint32_t)win), alo = ahi - 8u * chi;
                        do {
                            put_edge(l, alo, my_bits, (uint32_t)dst);
                            put_edge(h, ahi, my_bits + 4u * 33u, (uint32_t)dst);
                        } while (__any_sync(0xffffffffu, (l | h) != 0u));
                    } else {
                        const uint32_t tag = (uint32_t)(66 * (lane & 7)) | ((uint32_t)lane << 16);
                        uint32_t ahi = edges_at + 4u * (incl - (uint32_t)win), alo = ahi - 4u * chi;
                        do {
                            put_mixed(l, alo, tag);
                            put_mixed(h, ahi, tag + 33u);
                        } while (__any_sync(0xffffffffu, (l | h) != 0u));
                    }
                } else {
                    uint32_t at = incl - clo - chi - (uint32_t)win;
                    auto put = [&](uint32_t place) {
                        if (at < (uint32_t)FM_EDGES) {
                            if (plain) w.edge[at] = make_uint2(w.table[place], (uint32_t)dst);
                            else w.mixed[at] = place | ((uint32_t)lane << 16);
                        }
                        at++;
                    };
                    for (uint32_t b = lo; b; b &= b - 1) put(66 * (lane & 7) + __ffs((int)b) - 1);
                    for (uint32_t b = hi; b; b &= b - 1) put(66 * (lane & 7) + 33 + __ffs((int)b) - 1);
                }
                __syncwarp();
                const int first = written + win;
                // edges [0, mid) of the buffer belong to the first row, the others to the second
                const int mid = max(0, min(n, edges0 - first));
#pragma unroll 1
                for (int r = 0; r < 2; r++) {
                    const int a = r ? mid : 0, b = r ? n : mid;
                    const long long e0 = (r ? base1 - edges0 : base0) + first;
                    if (plain) {
                        long long *src = ei + e0, *to = src + E;
#pragma unroll 1
                        for (int i = a + lane; i < b; i += 32) {
                            const uint2 v = w.edge[i];
                            src[i] = (long long)v.x;
                            to[i] = (long long)v.y;
                        }
                    } else {
#pragma unroll 1
                        for (int i32 = a; i32 < b; i32 += 32) {
                            const int i = i32 + lane;
                            const uint32_t v = w.mixed[min(i, b - 1)], id = w.table[v & 0xffffu], code = w.code[v & 0xffffu];
                            const int from = (int)(v >> 16);
                            const int td = __shfl_sync(0xffffffffu, tm.x, from), tx = __shfl_sync(0xffffffffu, tm.y, from),
                                      ty = __shfl_sync(0xffffffffu, tm.z, from), tz = __shfl_sync(0xffffffffu, tm.w, from);
                            if (i < b) {
                                const long long e = e0 + i;
                                const int sx = (int)(code & 1023u) - 512 + tx, sy = (int)((code >> 10) & 1023u) - 512 + ty, sz = (int)((code >> 20) & 1023u) - 512 + tz;
                                ei[e] = (GLUE && glue.id_map) ? glue.id_map[id] : (long long)id;
                                ei[E + e] = (GLUE && glue.id_map) ? glue.id_map[td] : (long long)td;
                                if (GLUE) {
                                    glue_write(glue, shifts, e, sx, sy, sz);
                                } else {
                                    shifts[3 * e + 0] = (float)sx;
                                    shifts[3 * e + 1] = (float)sy;
                                    shifts[3 * e + 2] = (float)sz;
                                }
                            }
                        }
                    }
                }
                __syncwarp();
            }
            written += ntot;
        }
    }
}

// ------------------------------------------------------------------------------------------
// The same with squared distances: a warp stages {record number, shift code} of its group's candidates and reads each target's
// mask words; the position and the atom id of a hit come from the cell-sorted records (a group's few hundred records stay in
// L1), and the edges of a target are ordered by candidate place, as rg_pair_kernel writes them: a slot's hits are placed by one
// ballot and a predicated store.  Bound by instructions (the loop over the slots) and the latency of the records.  131 k atoms, 6.9 M
// edges: 158 us when every pair was tested again by that kernel, 118 us from the hit bits with a branch a slot and the lane mask read
// again every time, 96 without, 89 with the look-up by two loads a lane.
// ------------------------------------------------------------------------------------------
constexpr int FM_META = RG_MASK_SLOTS * 32;                       // staged candidate records per warp
// A place of the list at `at` (shared memory) if there is a hit: a predicated store, no branch.
__device__ __forceinline__ void put_place(uint32_t hit, uint32_t at, uint32_t place)
{
    asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %0, 0;\n\t@q st.shared.u16 [%1], %2;\n\t}" ::"r"(hit), "r"(at), "h"((unsigned short)place) : "memory");
}
constexpr int FM_WARP_BYTES = FM_META * 8 + FM_META * 2 + RUN_INDEX_BYTES;    // records + one parked slot per possible hit

template <typename T>
__global__ void __launch_bounds__(PAIR_THREADS, 4)
rg_fillmask_dist_kernel(const PairParams<T>* params_dev, long long* ei, float* shifts,
                   T* d2out, const long long E, long long* total)
{
    chain_begin();
    const PairParams<T> p = *params_dev;
    extern __shared__ __align__(32) unsigned char smem_raw[];
    const int lane = lane_id(), warp = threadIdx.x >> 5;
    unsigned char* wbase = smem_raw + warp * FM_WARP_BYTES;
    uint2* meta = reinterpret_cast<uint2*>(wbase);
    unsigned short* list = reinterpret_cast<unsigned short*>(wbase + FM_META * 8);
    int* delta = reinterpret_cast<int*>(wbase + FM_META * 8 + FM_META * 2);
    uint32_t* flags = reinterpret_cast<uint32_t*>(delta + 32);
    const uint32_t lt = lanes_below(), le = lt | (1u << lane), list_at = (uint32_t)__cvta_generic_to_shared(list);

    const DevHeader* hp = p.h;
    if (hp->status & RG_FATAL) return;
    if (total != nullptr && blockIdx.x == 0 && threadIdx.x == 0) *total = E;
    __shared__ GroupShape shape;
    if (threadIdx.x == 0) shape = group_shape(hp);
    const uint32_t num_groups = p.glist ? hp->active_groups : (uint32_t)hp->num_groups;
    __syncthreads();
    // the next group is looked up while the current one is written, so that one round trip to memory per group (the candidate
    // records) stays exposed
    const int which = group_lane(shape, lane);
    const uint32_t* const cells = lane >= GROUP_ROW_LANE ? p.tcstart : p.cstart;
    auto fetch = [&](uint32_t i) { return fetch_group(shape, cells, p.glist ? p.glist[i] : i, which); };

    const uint32_t nwarps = gridDim.x * PAIR_WARPS;
    uint32_t grp = blockIdx.x * PAIR_WARPS + warp;
    if (grp >= num_groups) return;
    GroupDesc nd = fetch(grp);
    for (; grp < num_groups; grp += nwarps) {
        const GroupDesc d = nd;
        if (grp + nwarps < num_groups) nd = fetch(grp + nwarps);
        const uint32_t tb[2] = {__shfl_sync(0xffffffffu, (uint32_t)d.run_a, GROUP_ROW_LANE), __shfl_sync(0xffffffffu, (uint32_t)d.run_a, GROUP_ROW_LANE + 1)};
        const uint32_t te[2] = {__shfl_sync(0xffffffffu, (uint32_t)d.run_e, GROUP_ROW_LANE), __shfl_sync(0xffffffffu, (uint32_t)d.run_e, GROUP_ROW_LANE + 1)};
        if (tb[0] == te[0] && tb[1] == te[1]) continue;
        const int run_a = d.run_a, run_len = lane < GROUP_ROW_LANE ? d.run_e - d.run_a : 0;
        // the first target's words do not depend on the candidate records: ask for them now
        int4 ntm;
        long long nbase;
        uint32_t nw;
        {
            const uint32_t t = tb[0] != te[0] ? tb[0] : tb[1];
            ntm = p.tmeta[t]; nbase = p.toffset[t]; nw = p.hitmask[(size_t)t * 32 + lane];
        }
        int L;
        const int run_off = warp_excl_scan(run_len, lane, &L);
        const int nslots = (L + 31) >> 5;
        if (nslots == 0 || nslots > RG_MASK_SLOTS) continue;  // a longer list has no hit bits: rg_pair_kernel writes that group

        __syncwarp();
        runs_compact(delta, run_a, run_off, run_len, lt);
        int rank_base = runs_flags(flags, run_off, run_len, lane, 0);
        // four slots at a time: the four gathers are in flight together before the first is stored (measured
        // against asynchronous 8-byte copies into shared memory: equal on sparse cells, faster on dense ones)
        for (int sw0 = 0; sw0 < nslots; sw0 += 4) {
            uint2 mv[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int sw = sw0 + u, j = sw * 32 + lane;
                const uint32_t word = (sw < nslots) ? flags[sw] : 0u;
                const int r = rank_base + __popc(word & le) - 1;
                rank_base += __popc(word);
                mv[u] = (j < L) ? make_uint2((uint32_t)(delta[r] + j), p.smeta[delta[r] + j].y) : make_uint2(0u, 0u);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int j = (sw0 + u) * 32 + lane;
                if (j < L) meta[j] = mv[u];
            }
        }
        __syncwarp();

        // Targets of both rows as one list, one at a time; the words of the next target are requested
        // before the current one is written.  Lane l holds the hit bits of candidates l, 32 + l, ...
        const int n0 = (int)(te[0] - tb[0]), nT = n0 + (int)(te[1] - tb[1]);
        for (int q = 0; q < nT; q++) {
            const int4 tm = ntm;
            const long long base = nbase;
            uint32_t w = nw;
            const Vec4<T> tp = p.tpos[q < n0 ? tb[0] + q : tb[1] + (q - n0)];
            if (q + 1 < nT) {
                const int qa = q + 1;
                const uint32_t t = qa < n0 ? tb[0] + qa : tb[1] + (qa - n0);
                ntm = p.tmeta[t]; nbase = p.toffset[t]; nw = p.hitmask[(size_t)t * 32 + lane];
            }
            __syncwarp();
            // the hits slot by slot, four slots a step: the mask has no bits behind the list's end
            uint32_t at = list_at, place = (uint32_t)lane;
#pragma unroll 1
            for (int s0 = 0; s0 < nslots; s0 += 4) {
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const uint32_t hit = w & (1u << u), m = __ballot_sync(0xffffffffu, hit != 0u);
                    put_place(hit, at + 2u * (uint32_t)__popc(m & lt), place + 32u * u);
                    at += 2u * (uint32_t)__popc(m);
                }
                w >>= 4;
                place += 128u;
            }
            const int cnt = (int)(at - list_at) >> 1;
            __syncwarp();
            const int sx = tm.y - 512, sy = tm.z - 512, sz = tm.w - 512;
            if (sizeof(T) == 4 && cnt > 32) {
                // two rounds of 32 edges, both rounds' records asked for before the first edge is written (103 -> 96 us; up to 32 edges
                // it is a round for nothing, and in double, with twice the registers to a record, 994 -> 1009 us a call of 500 k atoms at 5.5 A)
                for (int i0 = 0; i0 < cnt; i0 += 64) {
                    uint2 m[2];
                    Vec4<T> c[2];
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        m[k] = meta[list[min(i0 + 32 * k + lane, cnt - 1)]];
                        c[k] = p.spos[m[k].x];
                    }
#pragma unroll
                    for (int k = 0; k < 2; k++) {
                        const int i = i0 + 32 * k + lane;
                        if (i >= cnt) break;
                        const uint32_t code = m[k].y;
                        const long long e = base + i;
                        d2out[e] = dist2<T>(tp.x, tp.y, tp.z, c[k].x, c[k].y, c[k].z);
                        ei[e] = (long long)real_to_bits(c[k].w);
                        ei[E + e] = (long long)tm.x;
                        shifts[3 * e + 0] = (float)((int)(code & 1023u) + sx);
                        shifts[3 * e + 1] = (float)((int)((code >> 10) & 1023u) + sy);
                        shifts[3 * e + 2] = (float)((int)((code >> 20) & 1023u) + sz);
                    }
                }
            } else {
                for (int i = lane; i < cnt; i += 32) {
                    const uint2 m = meta[list[i]];
                    const uint32_t code = m.y;
                    const long long e = base + i;
                    const Vec4<T> c = p.spos[m.x];
                    d2out[e] = dist2<T>(tp.x, tp.y, tp.z, c.x, c.y, c.z);
                    ei[e] = (long long)real_to_bits(c.w);
                    ei[E + e] = (long long)tm.x;
                    shifts[3 * e + 0] = (float)((int)(code & 1023u) + sx);
                    shifts[3 * e + 1] = (float)((int)((code >> 10) & 1023u) + sy);
                    shifts[3 * e + 2] = (float)((int)((code >> 20) & 1023u) + sz);
                }
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// Halo marking: for every edge src -> dst whose endpoints have different owners, owner(dst) needs src (bit owner(dst)
// of needed[src]) and dst has a foreign neighbour.  This is the edge loop of the reference's halo-map builder
// (dynamis_state/src/csrc/build_halo_maps.cpp:50-58, 127-138) without materialising the graph.  With rank >= 0 only
// the edges that start or end at an atom of that rank are looked at: they are all its send and receive lists need.
//
// What matters is what is not tested: most of the volume lies inside one subdomain.  The owners of the cell-sorted records
// and targets are gathered once, and every candidate run (one per group column and (y, z) row) gets a word that says whether
// all its records have one owner; from these words the groups that can hold an edge of interest are listed (at 1 M
// atoms, 8 ranks: one of ten).  A warp lists a group's candidates that can matter to one of their targets and
// test distances for these alone — lane = candidate, targets broadcast from shared memory, one hit bit per target in a
// register of the lane, one atomic per candidate and group.  A million atoms, 8 ranks, 6 A, one rank's edges:
// 17 + 6 + 14 + 79 us (owners, runs, list, marking); without the list of groups 126 us for the last two, the same with one list of owners per group and no words took 338 us,
// and the pass that tested every pair for every rank 1034 us.
// ------------------------------------------------------------------------------------------
// Word of a candidate run: the one owner of its records, or EMPTY or MIXED; HALO_RANK is set when a record belongs to the rank
// of interest (or when all ranks are of interest).
constexpr int HALO_EMPTY = 0x7fff, HALO_MIXED = 0x7ffe, HALO_RANK = 0x8000;
// An owner that has no bit in the masks (below 0, or from 32 * words on) is gathered as the one owner 32 * words, "nobody":
// its atoms are foreign to every rank.  The number fits the 16 bits below the words above: at most 32000 ranks.
struct HaloArgs {
    const long long* owner;      // [n_atoms] rank of each atom
    uint32_t* needed;            // [n_atoms, words]
    unsigned char* has_foreign;  // [n_atoms]
    uint32_t* bad;               // set when an edge of interest ends at an atom of nobody; or nullptr
    int words;
    int rank;                    // -1: all ranks
};

template <typename T>
__global__ void __launch_bounds__(256)
rg_halo_owner_kernel(const PairParams<T>* params_dev, const HaloArgs halo)
{
    chain_begin();
    const PairParams<T> p = *params_dev;
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // for the marking behind this launch
        if (halo.bad != nullptr) *halo.bad = 0u;
        p.h->halo_groups = 0u;
    }
    if (p.h->status & RG_FATAL) return;
    const int64_t M = (int64_t)p.h->M;
    const int64_t end = max(M, (int64_t)p.n_targets);  // the plan's targets, whatever the number of owners
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < end; j += (int64_t)gridDim.x * blockDim.x) {
        int64_t sa = -1, ta = -1;
        if (j < M) sa = (int64_t)p.smeta[j].x;
        if (j < p.n_targets) ta = (int64_t)p.tmeta[j].x;
        const unsigned long long nobody = 32ull * (unsigned)halo.words;   // unsigned: negative owners are large
        if (sa >= 0) p.sown[j] = (unsigned short)min((unsigned long long)halo.owner[sa], nobody);
        if (ta >= 0) p.town[j] = (unsigned short)min((unsigned long long)halo.owner[ta], nobody);
    }
}

template <typename T>
__global__ void __launch_bounds__(256)
rg_halo_runs_kernel(const PairParams<T>* params_dev, const HaloArgs halo)
{
    chain_begin();
    const PairParams<T> p = *params_dev;
    const DevHeader* hp = p.h;
    if (hp->status & RG_FATAL) return;
    const int nx = hp->nx, S = hp->group_cells, pad = hp->pad;
    const uint32_t gx = (uint32_t)hp->gx, total = gx * (uint32_t)hp->ny * (uint32_t)hp->nz;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += gridDim.x * blockDim.x) {
        const uint32_t row = i / gx;
        const int cx0 = (int)(i - row * gx) * S, cx1 = min(cx0 + S, nx) - 1;
        const uint32_t a = p.cstart[row * nx + max(cx0 - pad, 0)], e = p.cstart[row * nx + min(cx1 + pad, nx - 1) + 1];
        int o = HALO_EMPTY;
        bool found = false;
        if (a < e) {
            o = (int)p.sown[a];
            found = halo.rank < 0 || o == halo.rank;
            for (uint32_t j = a + 1; j < e && !(found && o == HALO_MIXED); j += 4) {
                int v[4];
#pragma unroll
                for (int u = 0; u < 4; u++) v[u] = (int)p.sown[min(j + u, e - 1)];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    if (v[u] != o) o = HALO_MIXED;
                    if (v[u] == halo.rank) found = true;
                }
            }
        }
        p.run_owner[i] = (unsigned short)(o | (found ? HALO_RANK : 0));
    }
}

// The groups that the marking has to look at, as a list: those whose runs have several owners (the targets' own records are among
// them), with a record of the rank of interest, and with targets.  They lie together along the subdomains' boundary, one in ten
// of all: spread over the warps by their numbers some warps had several and most had none.  A lane takes a group; the words
// of its runs lie beside those of the lanes next to it.  A million atoms, 8 ranks, 6 A: marking 126 -> 14 (this pass, bound by the
// latency of its loads) + 79 us; with a warp a group here 31 us.
template <typename T>
__global__ void __launch_bounds__(128)
rg_halo_list_kernel(const PairParams<T>* params_dev)
{
    chain_begin();
    const PairParams<T> p = *params_dev;
    DevHeader* hp = p.h;
    if (hp->status & RG_FATAL) return;
    const int nx = hp->nx, ny = hp->ny, nz = hp->nz, S = hp->group_cells, Sy = hp->group_cells_y, pad = hp->pad;
    const uint32_t gx = (uint32_t)hp->gx, gy = (uint32_t)((ny + Sy - 1) / Sy), num_groups = (uint32_t)hp->num_groups;
    for (uint32_t g0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; g0 < num_groups; g0 += gridDim.x * blockDim.x) {
        const uint32_t grp = g0 + (threadIdx.x & 31);
        bool wanted = false;
        if (grp < num_groups) {
            const uint32_t row = grp / gx;
            const int ix = (int)(grp - row * gx);
            const int cz = (int)(row / gy), iy = (int)(row - (uint32_t)cz * gy);
            const int cy0 = iy * Sy, cy1 = min(cy0 + Sy, ny) - 1;
            int lo = HALO_EMPTY, hi = 0;
            bool rank = false;
            for (int zz = max(cz - pad, 0); zz <= min(cz + pad, nz - 1); zz++) {
                const unsigned short* word = p.run_owner + ((uint32_t)zz * ny) * gx + ix;
#pragma unroll 6
                for (int yy = max(cy0 - pad, 0); yy <= min(cy1 + pad, ny - 1); yy++) {
                    const int w = (int)word[(uint32_t)yy * gx], o = w & 0x7fff;
                    rank = rank || (w & HALO_RANK);
                    lo = min(lo, o);
                    hi = max(hi, o == HALO_EMPTY ? 0 : o);
                }
            }
            if (rank && (lo != hi || lo == HALO_MIXED)) {
                const int cx0 = ix * S, cx1 = min(cx0 + S, nx) - 1;
                const uint32_t* tcell = p.tcstart + ((uint32_t)cz * ny + cy0) * nx;
                wanted = tcell[cx0] != tcell[cx1 + 1] || (cy1 > cy0 && tcell[nx + cx0] != tcell[nx + cx1 + 1]);
            }
        }
        const uint32_t m = __ballot_sync(0xffffffffu, wanted);
        uint32_t base = 0;
        if ((threadIdx.x & 31) == 0 && m) base = atomicAdd(&hp->halo_groups, (uint32_t)__popc(m));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (wanted) p.halo_list[base + __popc(m & lanemask_lt())] = grp;
    }
}

constexpr int HALO_LIST = 256;     // candidates listed by owner before they are looked at more closely
constexpr int HALO_TARGETS = 32;   // targets of a group tested together
template <typename T> struct HaloWarp {
    Vec4<T> tgt[HALO_TARGETS];     // w = owner
    Vec4<T> cand[64];              // w = atom
    int cand_owner[64];
    int list[HALO_LIST];
};
struct HaloBatch {                 // the staged targets
    int nt, owner;                 // owner: of all targets, or -1 when they belong to several ranks
    uint32_t open;                 // targets of interest that are not known to have a foreign neighbour yet
    float lo[3], hi[3], reach2;    // bounding box of the targets; squared reach with room for rounding
};

// One warp tests 32 (or, at the end, fewer) near candidates against its staged targets.
template <typename T, bool WIDE>
__device__ __forceinline__ void halo_test(const PairParams<T>& p, const HaloArgs& halo, const HaloWarp<T>& w, int first, int n, HaloBatch& b,
                                          uint32_t& foreign, int lane)
{
    const T r2 = p.r2, eps = (T)1e-8f;
    const bool live = lane < n;
    const Vec4<T> c = w.cand[first + (live ? lane : 0)];
    uint32_t hits = 0;
#pragma unroll 4
    for (int q = 0; q < b.nt; q++) {
        const Vec4<T> t = w.tgt[q];
        const T d = dist2<T>(t.x, t.y, t.z, c.x, c.y, c.z);
        if ((d <= r2) && (d > eps)) hits |= 1u << q;
    }
    if (!live) hits = 0;
    uint32_t need = 0;
    if (!WIDE && (uint32_t)b.owner < 32u) {
        if (hits) need = 1u << b.owner;
    } else if (hits) {
        const int o = w.cand_owner[first + lane];
        for (uint32_t left = hits; left; left &= left - 1) {
            const int q = __ffs((int)left) - 1, ot = real_to_bits(w.tgt[q].w);
            if (o == ot || !(halo.rank < 0 || o == halo.rank || ot == halo.rank)) {
                hits &= ~(1u << q);
            } else if (ot >= 32 * halo.words) {
                if (halo.bad != nullptr) *halo.bad = 1u;
            } else if (!WIDE) {
                need |= 1u << ot;
            } else {
                uint32_t* wd = &halo.needed[(long long)real_to_bits(c.w) * halo.words + (ot >> 5)];
                const uint32_t bit = 1u << (ot & 31);
                if (!(*wd & bit)) atomicOr(wd, bit);
            }
        }
    }
    if (!WIDE && need) {
        uint32_t* wd = &halo.needed[real_to_bits(c.w)];
        if ((*wd & need) != need) atomicOr(wd, need);
    }
    const uint32_t f = __reduce_or_sync(0xffffffffu, hits);
    foreign |= f;
    b.open &= ~f;
}

// The listed candidates: those within reach of the targets' bounding box go on to the tests, unless all that a test could
// find is known already (a group nearby has marked the candidate, and no target waits for its first foreign neighbour).
template <typename T, bool WIDE>
__device__ __forceinline__ void halo_batch(const PairParams<T>& p, const HaloArgs& halo, HaloWarp<T>& w, int n, int& near, HaloBatch& b,
                                           uint32_t& foreign, int lane, uint32_t lt)
{
    for (int base = 0; base < n; base += 32) {
        bool keep = base + lane < n;
        const int rec = w.list[keep ? base + lane : 0];
        const Vec4<T> c = p.spos[rec];
        const float x = (float)c.x, y = (float)c.y, z = (float)c.z;
        const float dx = fmaxf(fmaxf(b.lo[0] - x, x - b.hi[0]), 0.0f), dy = fmaxf(fmaxf(b.lo[1] - y, y - b.hi[1]), 0.0f),
                    dz = fmaxf(fmaxf(b.lo[2] - z, z - b.hi[2]), 0.0f);
        keep = keep && dx * dx + dy * dy + dz * dz <= b.reach2;
        if (!WIDE && keep && (uint32_t)b.owner < 32u && b.open == 0u) keep = !((halo.needed[real_to_bits(c.w)] >> b.owner) & 1u);
        const uint32_t m = __ballot_sync(0xffffffffu, keep);
        if (keep) {
            const int at = near + __popc(m & lt);
            w.cand[at] = c;
            w.cand_owner[at] = (int)p.sown[rec];
        }
        near += __popc(m);
        __syncwarp();
        if (near >= 32) {
            near -= 32;
            halo_test<T, WIDE>(p, halo, w, near, 32, b, foreign, lane);
            __syncwarp();
        }
    }
}

template <typename T, bool WIDE>   // WIDE: more than 32 ranks, several words per atom
__global__ void __launch_bounds__(PAIR_THREADS, 4)
rg_halo_kernel(const PairParams<T>* params_dev, const HaloArgs halo)
{
    chain_begin();
    const PairParams<T> p = *params_dev;
    __shared__ HaloWarp<T> warps[PAIR_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    HaloWarp<T>& w = warps[warp];
    const DevHeader* hp = p.h;
    if (hp->status & RG_FATAL) return;
    const int nx = hp->nx, ny = hp->ny, nz = hp->nz, S = hp->group_cells, Sy = hp->group_cells_y, pad = hp->pad;
    const uint32_t gx = (uint32_t)hp->gx, gy = (uint32_t)((ny + Sy - 1) / Sy), num_groups = hp->halo_groups;
    const int Wd = 2 * pad + 1, Wy = Sy + 2 * pad, nrun = Wy * Wd;
    const int lane_dy = (lane % Wy) - pad, lane_dz = (lane / Wy) - pad;
    const uint32_t lt = lanemask_lt();
    const int rank = halo.rank;
    const float reach0 = sqrtf((float)p.r2) * 1.002f;

    const uint32_t nwarps = gridDim.x * PAIR_WARPS;
    for (uint32_t gi = blockIdx.x * PAIR_WARPS + warp; gi < num_groups; gi += nwarps) {
        const uint32_t grp = p.halo_list[gi];
        const uint32_t row = grp / gx;
        const int ix = (int)(grp - row * gx);
        const int cz = (int)(row / gy), iy = (int)(row - (uint32_t)cz * gy);
        const int cy0 = iy * Sy, cy1 = min(cy0 + Sy, ny) - 1;
        const int yy = cy0 + lane_dy, zz = cz + lane_dz;
        const bool has_run = lane < nrun && yy >= 0 && yy < ny && yy <= cy1 + pad && zz >= 0 && zz < nz;
        const int run_word = has_run ? (int)p.run_owner[((uint32_t)zz * ny + yy) * gx + ix] & 0x7fff : HALO_EMPTY;
        const int cx0 = ix * S, cx1 = min(cx0 + S, nx) - 1;
        const uint32_t tb0 = p.tcstart[((uint32_t)cz * ny + cy0) * nx + cx0], te0 = p.tcstart[((uint32_t)cz * ny + cy0) * nx + cx1 + 1];
        uint32_t tb1 = 0, te1 = 0;
        if (cy1 > cy0) {
            tb1 = p.tcstart[((uint32_t)cz * ny + cy1) * nx + cx0];
            te1 = p.tcstart[((uint32_t)cz * ny + cy1) * nx + cx1 + 1];
        }
        const int n0 = (int)(te0 - tb0), ntot = n0 + (int)(te1 - tb1);
        if (ntot == 0) continue;
        int run_a = 0, run_len = 0;
        if (has_run) {
            const uint32_t b = ((uint32_t)zz * ny + yy) * nx;
            run_a = (int)p.cstart[b + max(cx0 - pad, 0)];
            run_len = (int)(p.cstart[b + min(cx1 + pad, nx - 1) + 1]) - run_a;
        }
        for (int q0 = 0; q0 < ntot; q0 += HALO_TARGETS) {
            const int nt = min(HALO_TARGETS, ntot - q0);
            const uint32_t t = (q0 + lane < n0) ? tb0 + q0 + lane : tb1 + (q0 + lane - n0);
            const int ot = (lane < nt) ? (int)p.town[t] : 0;
            const int lo = __reduce_min_sync(0xffffffffu, lane < nt ? ot : 0x7fffffff), hi = __reduce_max_sync(0xffffffffu, ot);
            const bool uniform = lo == hi, any_rank = rank < 0 || __any_sync(0xffffffffu, lane < nt && ot == rank);
            HaloBatch b;
            b.nt = nt;
            b.owner = uniform ? lo : -1;
            b.open = __ballot_sync(0xffffffffu, lane < nt && (rank < 0 || ot == rank));
            {
                float x[3] = {0.0f, 0.0f, 0.0f};
                if (lane < nt) {
                    Vec4<T> v = p.tpos[t];
                    x[0] = (float)v.x; x[1] = (float)v.y; x[2] = (float)v.z;
                    v.w = bits_to_real(ot, T());
                    w.tgt[lane] = v;
                }
                float far = 0.0f;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    b.lo[k] = unordered_f32(__reduce_min_sync(0xffffffffu, lane < nt ? ordered_u32(x[k]) : 0xffffffffu));
                    b.hi[k] = unordered_f32(__reduce_max_sync(0xffffffffu, lane < nt ? ordered_u32(x[k]) : 0u));
                    far = fmaxf(far, fmaxf(fabsf(b.lo[k]), fabsf(b.hi[k])));
                }
                const float reach = reach0 + 1e-6f * far;
                b.reach2 = reach * reach;
            }
            uint32_t foreign = 0;
            int n = 0, near = 0;
            // eight records of every run at a time: their loads are in flight together; a run of the targets' own owner is left out
            const int len = (uniform && run_word == lo) ? 0 : run_len;
            const int longest = __reduce_max_sync(0xffffffffu, len);
            for (int i0 = 0; i0 < longest; i0 += 8) {
                int o[8];
#pragma unroll
                for (int u = 0; u < 8; u++) o[u] = (i0 + u < len) ? (int)p.sown[run_a + i0 + u] : -1;
                uint32_t keep = 0;
#pragma unroll
                for (int u = 0; u < 8; u++)
                    if (o[u] >= 0 && (any_rank || o[u] == rank) && !(uniform && o[u] == lo)) keep |= 1u << u;
                for (uint32_t any = __reduce_or_sync(0xffffffffu, keep); any; any &= any - 1) {
                    const int u = __ffs((int)any) - 1;
                    const bool mine = (keep >> u) & 1u;
                    const uint32_t m = __ballot_sync(0xffffffffu, mine);
                    if (mine) w.list[n + __popc(m & lt)] = run_a + i0 + u;
                    n += __popc(m);
                    if (n > HALO_LIST - 32) {
                        __syncwarp();
                        halo_batch<T, WIDE>(p, halo, w, n, near, b, foreign, lane, lt);
                        n = 0;
                        __syncwarp();
                    }
                }
            }
            __syncwarp();
            if (n > 0) halo_batch<T, WIDE>(p, halo, w, n, near, b, foreign, lane, lt);
            if (near > 0) halo_test<T, WIDE>(p, halo, w, 0, near, b, foreign, lane);
            if (lane < nt && ((foreign >> lane) & 1u)) halo.has_foreign[p.tmeta[t].x] = 1;
            __syncwarp();
        }
    }
}

// First launch of a plan: the header block (it travels as a kernel argument: no staging copy of a pageable host
// buffer), the cell counters, the degree counters and the caller's degree array in one pass.
struct HeaderBlock { uint32_t words[RG_HEADER_BYTES / 4]; };
__global__ void __launch_bounds__(256)
rg_init_kernel(uint32_t* hdr, const HeaderBlock blk, uint4* zero_a, int64_t n_a16,
               uint4* zero_b, int64_t n_b16, int32_t* counts_out, int64_t Nt)
{
    chain_begin();
    const int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
    if (i0 < RG_HEADER_BYTES / 4) hdr[i0] = blk.words[i0];
    const uint4 z = make_uint4(0u, 0u, 0u, 0u);
    for (int64_t i = i0; i < n_a16; i += stride) zero_a[i] = z;
    for (int64_t i = i0; i < n_b16; i += stride) zero_b[i] = z;
    if (counts_out != nullptr)
        for (int64_t i = i0; i < Nt; i += stride) counts_out[i] = 0;
}

// ------------------------------------------------------------------------------------------
// host side
// ------------------------------------------------------------------------------------------
struct RgLayout {
    int64_t hdr, posw, aff, ccount, cfill, tccount, tcfill, srec, spos, sscan, smeta, hitmask, trec, tpos, tscan, tmeta,
        tcount, toffset, runs, sums, total;
};

// The layout starts at the first 256-byte boundary of the caller's workspace: its records are read and written in pieces
// of up to 32 bytes, wherever the workspace lies.
constexpr int64_t RG_WS_ALIGN = 256;
static unsigned char* rg_base(const void* ws)
{
    return reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(ws) + RG_WS_ALIGN - 1) / RG_WS_ALIGN * RG_WS_ALIGN);
}

static RgLayout rg_layout(int64_t N, int64_t Nt, int64_t src_cap, int64_t cell_cap, int dtype)
{
    const int64_t v4 = dtype == DYNB_F64 ? 32 : 16;
    RgLayout L;
    int64_t o = 0;
    auto take = [&](int64_t bytes) { int64_t r = o; o = align_up(o + bytes, 256); return r; };
    L.hdr = take(RG_HEADER_BYTES);
    // cell counters, cleared in one pass; the fill cursors are written by the prefix sum
    L.ccount = take((cell_cap + 2) * 4);
    L.tccount = take((cell_cap + 2) * 4);
    L.cfill = take((cell_cap + 2) * 4);
    L.tcfill = take((cell_cap + 2) * 4);
    L.posw = take(N * v4);
    L.aff = take(N * 16);
    const int64_t slot = dtype == DYNB_F64 ? sizeof(SlotRec<double>) : sizeof(SlotRec<float>);
    L.srec = take(src_cap * slot);  // source images in slot order
    L.spos = take(src_cap * v4);
    L.sscan = dtype == DYNB_F64 ? take(src_cap * 16) : L.spos;  // float positions are tested as they are
    L.smeta = take(src_cap * 8);
    L.hitmask = take(Nt * 32 * 2);
    L.trec = take(Nt * slot);     // targets in slot order
    L.tpos = take(Nt * v4);
    L.tscan = dtype == DYNB_F64 ? take(Nt * 16) : L.tpos;  // float positions are tested as they are
    L.tmeta = take(Nt * 16);
    L.tcount = take((Nt + 1) * 4);
    L.toffset = take((Nt + 2) * 8);
    L.runs = take((cell_cap + 2) * 2);
    const int64_t tiles = std::max<int64_t>(scan_num_tiles(cell_cap + 2), scan_num_tiles(Nt + 2)) + 1;
    L.sums = take(tiles * 8 * 2);
    L.total = o;
    return L;
}

// Host cell geometry in the precision of the positions, following the reference's host code
// (radius_graph_kernels.cu:516-587): face distances, replication counts, cutoff fractions and
// the cofactor inverse.  This translation unit is compiled with -ffp-contract=off for the host.
template <typename T>
static void rg_geometry(const T* cell, const uint8_t* pbc, T radius, Geom<T>& g)
{
    const T* a0 = cell; const T* a1 = cell + 3; const T* a2 = cell + 6;
    T c12[3] = {a1[1] * a2[2] - a1[2] * a2[1], a1[2] * a2[0] - a1[0] * a2[2], a1[0] * a2[1] - a1[1] * a2[0]};
    T vol = a0[0] * c12[0] + a0[1] * c12[1] + a0[2] * c12[2];
    T abs_vol = std::abs(vol);
    T c20[3] = {a2[1] * a0[2] - a2[2] * a0[1], a2[2] * a0[0] - a2[0] * a0[2], a2[0] * a0[1] - a2[1] * a0[0]};
    T c01[3] = {a0[1] * a1[2] - a0[2] * a1[1], a0[2] * a1[0] - a0[0] * a1[2], a0[0] * a1[1] - a0[1] * a1[0]};
    T n12 = std::sqrt(c12[0] * c12[0] + c12[1] * c12[1] + c12[2] * c12[2]);
    T n20 = std::sqrt(c20[0] * c20[0] + c20[1] * c20[1] + c20[2] * c20[2]);
    T n01 = std::sqrt(c01[0] * c01[0] + c01[1] * c01[1] + c01[2] * c01[2]);
    T d_face[3] = {abs_vol / n12, abs_vol / n20, abs_vol / n01};
    for (int d = 0; d < 3; d++) {
        g.pbc[d] = pbc[d] ? 1 : 0;
        if (pbc[d]) {
            g.rep[d] = (int)std::ceil(radius / d_face[d]);
            g.cf[d] = radius / d_face[d];
        } else {
            g.rep[d] = 0;
            g.cf[d] = (T)0;
        }
    }
    T inv_vol = (T)1 / vol;
    g.inv[0] = (a1[1] * a2[2] - a1[2] * a2[1]) * inv_vol;
    g.inv[1] = (a0[2] * a2[1] - a0[1] * a2[2]) * inv_vol;
    g.inv[2] = (a0[1] * a1[2] - a0[2] * a1[1]) * inv_vol;
    g.inv[3] = (a1[2] * a2[0] - a1[0] * a2[2]) * inv_vol;
    g.inv[4] = (a0[0] * a2[2] - a0[2] * a2[0]) * inv_vol;
    g.inv[5] = (a0[2] * a1[0] - a0[0] * a1[2]) * inv_vol;
    g.inv[6] = (a1[0] * a2[1] - a1[1] * a2[0]) * inv_vol;
    g.inv[7] = (a0[1] * a2[0] - a0[0] * a2[1]) * inv_vol;
    g.inv[8] = (a0[0] * a1[1] - a0[1] * a1[0]) * inv_vol;
    for (int i = 0; i < 9; i++) g.cell[i] = cell[i];
}

template <typename T>
static int rg_geometry_checked(const void* cell_host, const uint8_t* pbc_host, double radius, Geom<T>& g)
{
    if (cell_host == nullptr || pbc_host == nullptr) return fail_arg("cell and pbc must not be null");
    if (!(radius > 0.0)) return fail_arg("radius must be positive");
    rg_geometry<T>(static_cast<const T*>(cell_host), pbc_host, (T)radius, g);
    for (int d = 0; d < 3; d++) {
        if (!(g.rep[d] >= 0 && g.rep[d] <= 64) || !std::isfinite((double)g.cf[d]))
            return fail_arg("degenerate cell: a periodic axis needs more than 64 image layers (or the cell is singular)");
    }
    for (int i = 0; i < 9; i++)
        if (!std::isfinite((double)g.inv[i])) return fail_arg("cell matrix is singular");
    return DYNB_OK;
}

template <typename T>
static int rg_suggest(int64_t N, const void* cell_host, const uint8_t* pbc_host, double radius, int64_t* src_cap,
                      int64_t* cell_cap)
{
    Geom<T> g;
    int rc = rg_geometry_checked<T>(cell_host, pbc_host, radius, g);
    if (rc) return rc;
    double full = 1.0, est = 1.0, ext[3] = {0, 0, 0};
    for (int d = 0; d < 3; d++) {
        double span = 1.0;
        if (g.pbc[d]) {
            full *= 2 * g.rep[d] + 1;
            const double reach = g.rep[d] == 1 ? std::min(1.0, (double)g.cf[d]) : (double)g.rep[d];
            est *= 1.0 + 2.0 * reach;
            span = 1.0 + 2.0 * reach;
        }
        for (int k = 0; k < 3; k++) ext[k] += std::fabs((double)g.cell[3 * d + k]) * span;
    }
    const double nmax = (double)N * full;
    double cap = std::min(nmax, (double)N * est * 1.25 + 4096.0);
    if (cap < 1.0) cap = 1.0;
    *src_cap = (int64_t)cap;
    const double res = radius / 1.99;
    double cells = 1.0;
    for (int k = 0; k < 3; k++) cells *= std::ceil((ext[k] + 0.02) / res) + 1.0;
    double ccap = std::min(cells * 1.02 + 64.0, std::max(8.0 * cap, 1048576.0));
    ccap = std::min(ccap, 268435456.0);
    *cell_cap = (int64_t)ccap;
    return DYNB_OK;
}

template <typename T>
static int rg_plan(const void* pos_dev, int64_t N, const void* cell_host, const uint8_t* pbc_host, double radius,
                   const int64_t* targets, int64_t Nt, void* ws, int64_t ws_bytes, int64_t src_cap, int64_t cell_cap,
                   int32_t* counts_out, dynb_rg_header* header_host, bool bins_only, cudaStream_t stream)
{
    // bins_only: the plan ends with the sorted records (all that the halo marking reads)
    Geom<T> g;
    int rc = rg_geometry_checked<T>(cell_host, pbc_host, radius, g);
    if (rc) return rc;
    const int dtype = sizeof(T) == 8 ? DYNB_F64 : DYNB_F32;
    const RgLayout L = rg_layout(N, Nt, src_cap, cell_cap, dtype);
    unsigned char* w = rg_base(ws);
    if (ws_bytes < L.total + (w - static_cast<unsigned char*>(ws))) return fail_arg("workspace too small (see dynb_rg_workspace_bytes)");
    DevHeader* h = reinterpret_cast<DevHeader*>(w + L.hdr);

    auto* posw = reinterpret_cast<Vec4<T>*>(w + L.posw);
    auto* aff = reinterpret_cast<int4*>(w + L.aff);
    auto* ccount = reinterpret_cast<uint32_t*>(w + L.ccount);
    auto* cfill = reinterpret_cast<uint32_t*>(w + L.cfill);
    auto* tccount = reinterpret_cast<uint32_t*>(w + L.tccount);
    auto* tcfill = reinterpret_cast<uint32_t*>(w + L.tcfill);
    auto* srec = reinterpret_cast<SlotRec<T>*>(w + L.srec);
    auto* spos = reinterpret_cast<Vec4<T>*>(w + L.spos);
    auto* sscan = reinterpret_cast<float4*>(w + L.sscan);
    auto* smeta = reinterpret_cast<uint2*>(w + L.smeta);
    auto* hitmask = reinterpret_cast<unsigned short*>(w + L.hitmask);
    auto* trec = reinterpret_cast<SlotRec<T>*>(w + L.trec);
    auto* tpos = reinterpret_cast<Vec4<T>*>(w + L.tpos);
    auto* tscan = reinterpret_cast<float4*>(w + L.tscan);
    auto* tmeta = reinterpret_cast<int4*>(w + L.tmeta);
    auto* tcount = reinterpret_cast<uint32_t*>(w + L.tcount);
    auto* toffset = reinterpret_cast<long long*>(w + L.toffset);
    auto* sums32 = reinterpret_cast<uint32_t*>(w + L.sums);
    auto* sums64 = reinterpret_cast<long long*>(w + L.sums);
    auto* params_dev = reinterpret_cast<PairParams<T>*>(w + L.hdr + RG_PARAMS_OFFSET);

    // The last kernel of the plan writes the header to the host itself where the caller's copy lies in pinned memory (a copy
    // behind it is a launch of another engine: 8 to 10 us of a call with a thousand atoms).
    static_assert(sizeof(dynb_rg_header) == 64, "the header is published in four pieces of 16 bytes");
    uint4* header_written = nullptr;
    if (header_host != nullptr && (bins_only || scan_publishes(Nt + 1))) header_written = static_cast<uint4*>(device_view_of_host(header_host));
    static_assert(sizeof(DevHeader) <= RG_PARAMS_OFFSET, "header overlaps params");
    static_assert(RG_PARAMS_OFFSET + sizeof(PairParams<T>) <= RG_HEADER_BYTES, "params overflow header block");
    unsigned char init[RG_HEADER_BYTES];
    memset(init, 0, sizeof(init));
    PairParams<T> pp_host;
    memset(&pp_host, 0, sizeof(pp_host));
    // Periodic in all directions and every atom a target: the images fill a box that follows from the cell alone
    // (fractional coordinates in [1 - cf - rep, cf + rep] per axis, see rg_wrap_kernel's flags), so the grid is
    // chosen here and the first pass counts the images into their cells while it wraps.  Positions that rounding
    // leaves a hair outside land in the outermost cells (cell_of clamps), which a scan window always includes.
    GridChoice gc_host;
    memset(&gc_host, 0, sizeof(gc_host));
    bool host_grid = (targets == nullptr) && g.pbc[0] && g.pbc[1] && g.pbc[2];
    if (host_grid) {
        double lo[3] = {0, 0, 0}, hi3[3] = {0, 0, 0};
        for (int d = 0; d < 3; d++) {
            const double fa = std::max(-(double)g.rep[d], std::min(0.0, 1.0 - (double)g.cf[d] - (double)g.rep[d]));
            const double fb = std::min(1.0 + (double)g.rep[d], std::max(1.0, (double)g.cf[d] + (double)g.rep[d]));
            for (int k = 0; k < 3; k++) {
                const double c = (double)g.cell[3 * d + k];
                lo[k] += std::min(fa * c, fb * c);
                hi3[k] += std::max(fa * c, fb * c);
            }
        }
        double ext[3];
        for (int k = 0; k < 3; k++) {
            const double slack = 0.01 + 1e-5 * (hi3[k] - lo[k]);
            lo[k] -= slack;
            ext[k] = hi3[k] + slack - lo[k];
        }
        const double* c = nullptr;
        double cd[9];
        for (int k = 0; k < 9; k++) cd[k] = (double)g.cell[k];
        c = cd;
        const double vol = std::fabs(c[0] * (c[4] * c[8] - c[5] * c[7]) - c[1] * (c[3] * c[8] - c[5] * c[6]) + c[2] * (c[3] * c[7] - c[4] * c[6]));
        const double density = vol > 0.0 ? (double)N / vol : 0.0;  // images repeat the atoms: the same density everywhere in the box
        rg_choose_grid(lo, ext, radius, (long long)cell_cap, PAIR_CAND_BYTES / (int)sizeof(Vec4<T>), (double)N, density, true, gc_host);
        // A grid over the whole cell that had to take coarser cells to fit the cell capacity (few atoms in a large
        // periodic box) is worse than the grid over the data's own bounding box: that case keeps the device path.
        if (gc_host.res_inv < 0.999 * 1.99 / radius) host_grid = false;
    }
    {
        DevHeader hi;
        memset(&hi, 0, sizeof(hi));
        for (int k = 0; k < 3; k++) { hi.bb_min[k] = hi.tb_min[k] = ~0ull; hi.bb_max[k] = hi.tb_max[k] = 0ull; }
        if (host_grid) {
            rg_store_grid(hi, gc_host);
            for (int k = 0; k < 3; k++) { hi.clip_lo[k] = -1.0e300; hi.clip_hi[k] = 1.0e300; }
        }
        memcpy(init, &hi, sizeof(hi));
        PairParams<T>& pp = pp_host;
        pp.h = h; pp.cstart = ccount; pp.tcstart = tccount; pp.spos = spos; pp.sscan = sscan; pp.smeta = smeta; pp.hitmask = hitmask; pp.counts_out = counts_out; pp.tpos = tpos;
        pp.tscan = tscan; pp.tmeta = tmeta; pp.tcount = tcount; pp.toffset = toffset; pp.r2 = (T)radius * (T)radius;
        // the targets' fill counters are free once the targets are binned: they hold the list of groups with targets
        pp.glist = (targets != nullptr) ? tcfill : nullptr;
        pp.long_list = cfill;   // likewise free once the sources are binned
        pp.n_targets = Nt;
        static_assert(sizeof(SlotRec<T>) >= sizeof(unsigned short), "owners lie over the binning slots");
        pp.sown = reinterpret_cast<unsigned short*>(srec);
        pp.town = reinterpret_cast<unsigned short*>(trec);
        pp.run_owner = reinterpret_cast<unsigned short*>(w + L.runs);
        // a listed group holds targets: no more groups than targets, and no more of those than source records
        static_assert(sizeof(SlotRec<T>) >= sizeof(unsigned short) + sizeof(uint32_t), "the list lies behind the owners over the binning slots");
        pp.halo_list = reinterpret_cast<uint32_t*>(srec) + (src_cap + 1) / 2;
        memcpy(init + RG_PARAMS_OFFSET, &pp, sizeof(pp));
    }
    {
        HeaderBlock blk;
        memcpy(blk.words, init, sizeof(init));
        // every region of the layout starts on a 256-byte boundary and is padded to one
        const int64_t n_a16 = (L.cfill - L.ccount) / 16, n_b16 = bins_only ? 0 : ((Nt + 1) * 4 + 15) / 16;
        launch_chained(rg_init_kernel, sm_count_cached() * 4, 256, 0, stream, reinterpret_cast<uint32_t*>(w + L.hdr), blk,
                                                                  reinterpret_cast<uint4*>(w + L.ccount), n_a16,
                                                                  reinterpret_cast<uint4*>(w + L.tcount), n_b16, counts_out, Nt);
    }

    const int vec_ok = (reinterpret_cast<uintptr_t>(pos_dev) % 16 == 0) ? 1 : 0;
    const int64_t nb = std::max(N, Nt);
    if (host_grid) {
        launch_chained(rg_wrap_kernel<T, true>, (unsigned)((N + WRAP_THREADS - 1) / WRAP_THREADS), WRAP_THREADS, 0, stream, static_cast<const T*>(pos_dev), N, g, vec_ok, posw, aff, h, GridArgs{}, 0, gc_host, ccount, tccount);
    } else {
        const GridArgs ga = {radius, (long long)src_cap, (long long)cell_cap, PAIR_CAND_BYTES / (int)sizeof(Vec4<T>)};
        launch_chained(rg_wrap_kernel<T, false>, (unsigned)((N + WRAP_THREADS - 1) / WRAP_THREADS), WRAP_THREADS, 0, stream, static_cast<const T*>(pos_dev), N, g, vec_ok, posw, aff, h, ga, targets != nullptr ? 1 : 0, gc_host, nullptr, nullptr);
        if (targets != nullptr)
            launch_chained(rg_target_bbox_kernel<T>, (unsigned)((Nt + 255) / 256), 256, 0, stream, targets, Nt, N, posw, h, ga);
        launch_chained(rg_bin_kernel<T, false>, (unsigned)((nb + 255) / 256), 256, 0, stream, N, Nt, targets, g, posw, aff, h, ccount, cfill, tccount, tcfill, srec, trec, (long long)src_cap, 0);
    }
    // cell starts of sources and targets in the same two launches (which also set the fill cursors); the total of the source counts is the
    // number of source images actually binned (<= the count of rg_wrap when clipping): it becomes header.M
    DYNB_CUDA_OK((exclusive_scan_pair<uint32_t, uint32_t>(ccount, ccount, reinterpret_cast<uint32_t*>(&h->M), tccount, tccount, nullptr,
                                                           &h->ncell_plus1, cell_cap + 1, sums32, stream, cfill, tcfill)));
    launch_chained(rg_bin_kernel<T, true>, (unsigned)((nb + 255) / 256), 256, 0, stream, N, Nt, targets, g, posw, aff, h, ccount, cfill, tccount, tcfill, srec, trec, (long long)src_cap,
        host_grid ? PAIR_CAND_BYTES / (int)sizeof(Vec4<T>) : 0);
    const int64_t nf = std::max(src_cap, Nt);
    launch_chained(rg_bin_finalize_kernel<T>, (unsigned)((nf + 255) / 256), 256, 0, stream, Nt, targets != nullptr ? 1 : 0, g, posw, h, ccount, tccount, srec, trec, spos, sscan, smeta, tpos, tscan, tmeta, (double)pp_host.r2, bins_only ? header_written : nullptr);

    if (bins_only) {
        DYNB_CUDA_OK(cudaGetLastError());
        if (header_host != nullptr && header_written == nullptr)
            DYNB_CUDA_OK(cudaMemcpyAsync(header_host, h, sizeof(dynb_rg_header), cudaMemcpyDeviceToHost, stream));
        return DYNB_OK;
    }
    if (targets != nullptr)
        launch_chained(rg_group_list_kernel<T>, sm_count_cached() * 8, 256, 0, stream, params_dev, tcfill);
    // there are no more groups than cells, and with a target subset no more of interest than targets
    const int64_t most_groups = std::min(host_grid ? (int64_t)gc_host.ncell_plus1 : cell_cap, targets != nullptr ? Nt : cell_cap);
    const int grid = (int)std::min<int64_t>((int64_t)sm_count_cached() * COUNT_BLOCKS, (most_groups + COUNT_WARPS - 1) / COUNT_WARPS);
    launch_chained(rg_count_kernel<T>, grid, COUNT_WARPS * 32, 0, stream, pp_host);
    DYNB_CUDA_OK((exclusive_scan<uint32_t, long long>(tcount, toffset, nullptr, Nt + 1, sums64,
                                                       reinterpret_cast<long long*>(&h->E), stream,
                                                       ScanPublish{reinterpret_cast<const uint4*>(h), header_written})));
    DYNB_CUDA_OK(cudaGetLastError());
    if (header_host != nullptr && header_written == nullptr)
        DYNB_CUDA_OK(cudaMemcpyAsync(header_host, h, sizeof(dynb_rg_header), cudaMemcpyDeviceToHost, stream));
    return DYNB_OK;
}

constexpr int64_t RG_GROUPS_UNKNOWN = INT64_MAX / 2;  // for a caller who has not read the plan's header
// Edges with distances when some lists are too long for the hit bits: one pass that tests every pair again, over all groups,
// instead of the writer from the bits and that pass over the listed groups behind it?  Liquid of 0.1 atoms per A^3, one pass
// against two, us (share of listed groups):
//   200 k atoms, float:  348 / 333 (0.03), 320 / 367 (0.18), 368 / 447 (0.44), 559 / 578 (0.70)
//   200 k atoms, double: 495 / 371 (0.03), 515 / 455 (0.18), 537 / 574 (0.44), 763 / 778 (0.70)
//   20 k atoms (10 k groups), two listed groups: 60 / 76 float, 80 / 89 double -- the second pass is then a single warp's
//   chain over its group, about 15 us with nothing beside it; 74 k groups, 148 listed: 338 / 318 and 474 / 353.
// The order of the edges is the same.
constexpr int64_t RG_AT_ONCE_GROUPS = 16384;
template <typename T> static bool rg_write_at_once(int64_t groups, int64_t long_lists)
{
    if (long_lists <= 0 || groups >= RG_GROUPS_UNKNOWN) return false;
    return groups <= RG_AT_ONCE_GROUPS || long_lists >= groups / (sizeof(T) == 8 ? 4 : 16);
}
template <typename T>
static int rg_fill(const void* ws, int64_t* ei, float* shifts, void* d2out, int64_t E, const GlueArgs* glue_opt, int64_t* total_dev,
                   int64_t groups, int64_t long_lists, cudaStream_t stream)
{
    const unsigned char* w = rg_base(ws);
    const auto* params_dev = reinterpret_cast<const PairParams<T>*>(w + RG_PARAMS_OFFSET);
    // A warp per group, up to the waves of PAIR_GRID_WAVES.  The groups are walked whether they hold edges or not, so their
    // number bounds the launch and the number of edges does not: with E / 256 blocks the writer of a gas of a million atoms
    // and 8 k edges took 4124 us against 324, of 200 k atoms and 28 k edges 283 against 97.
    const int64_t full = (int64_t)sm_count_cached() * 4 * PAIR_GRID_WAVES;
    const int grid = (int)std::max<int64_t>(std::min(full, (groups + PAIR_WARPS - 1) / PAIR_WARPS), 1);
    GlueArgs glue{};
    if (glue_opt != nullptr) glue = *glue_opt;
    // The edges come from the hit masks of the counting pass; the groups whose candidate list was too long for the masks
    // (listed on the device by the counting pass; usually none) are written by the distance-recomputing pass behind it.
    auto* ei64 = reinterpret_cast<long long*>(ei);
    auto* d2 = static_cast<T*>(d2out);
    const int smem = PAIR_WARPS * PAIR_WARP_BYTES;
    if (long_lists != 0) DYNB_CUDA_OK(cudaFuncSetAttribute(rg_pair_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    if (d2 != nullptr && rg_write_at_once<T>(groups, long_lists)) {
        launch_chained(rg_pair_kernel<T>, grid, PAIR_THREADS, smem, stream, params_dev, ei64, shifts, d2, (long long)E, glue,
                                                                                 1, reinterpret_cast<long long*>(total_dev));
        DYNB_CUDA_OK(cudaGetLastError());
        return DYNB_OK;
    }
    auto launch = [&](auto kernel, int blocks, int warps, int bytes, auto... out) -> int {
        DYNB_CUDA_OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes));
        launch_chained(kernel, blocks, warps * 32, bytes, stream, params_dev, ei64, shifts, out..., reinterpret_cast<long long*>(total_dev));
        return DYNB_OK;
    };
    const int esmem = EDGE_WARPS * (int)sizeof(EdgeWarp);
    const int egrid = (int)std::max<int64_t>(std::min<int64_t>((int64_t)sm_count_cached() * EDGE_BLOCKS * EDGE_WAVES, (groups + EDGE_WARPS - 1) / EDGE_WARPS), 1);
    const int rc = d2 != nullptr ? launch(rg_fillmask_dist_kernel<T>, grid, PAIR_WARPS, PAIR_WARPS * FM_WARP_BYTES, d2, (long long)E)
                                 : (glue_opt != nullptr ? launch(rg_fillmask_kernel<T, true>, egrid, EDGE_WARPS, esmem, (long long)E, glue)
                                                        : launch(rg_fillmask_kernel<T, false>, egrid, EDGE_WARPS, esmem, (long long)E, glue));
    if (rc) return rc;
    // the groups the counting pass listed; a caller who has read the plan's header knows whether there are any
    if (long_lists != 0) {
        // Two waves where the caller has not read the header and most likely nothing is listed, else as many as the writer
        // (200 k atoms at 8 A without distances: 508 against 543 us with two)
        const int long_grid = (groups == RG_GROUPS_UNKNOWN && d2 == nullptr) ? std::min(grid, sm_count_cached() * 8) : grid;
        launch_chained(rg_pair_kernel<T>, long_grid, PAIR_THREADS, smem, stream, params_dev, ei64, shifts, d2,
                                                                                      (long long)E, glue, 0, nullptr);
    }
    DYNB_CUDA_OK(cudaGetLastError());
    return DYNB_OK;
}

template <typename T>
static int rg_halo_mark(const void* ws, const HaloArgs& ha, int64_t N, cudaStream_t stream)
{
    const unsigned char* w = rg_base(ws);
    const auto* params_dev = reinterpret_cast<const PairParams<T>*>(w + RG_PARAMS_OFFSET);
    // the numbers of records and runs are known on the device only: both passes stride, the first with a thread for every
    // record of a system with no more images than atoms
    launch_chained(rg_halo_owner_kernel<T>, (unsigned)((2 * N + 255) / 256), 256, 0, stream, params_dev, ha);
    launch_chained(rg_halo_runs_kernel<T>, sm_count_cached() * 8, 256, 0, stream, params_dev, ha);
    const int grid = sm_count_cached() * 4 * PAIR_GRID_WAVES;
    launch_chained(rg_halo_list_kernel<T>, sm_count_cached() * 8, 128, 0, stream, params_dev);
    if (ha.words == 1) launch_chained(rg_halo_kernel<T, false>, grid, PAIR_THREADS, 0, stream, params_dev, ha);
    else launch_chained(rg_halo_kernel<T, true>, grid, PAIR_THREADS, 0, stream, params_dev, ha);
    DYNB_CUDA_OK(cudaGetLastError());
    return DYNB_OK;
}

}  // namespace dynb

// ------------------------------------------------------------------------------------------
// C ABI
// ------------------------------------------------------------------------------------------
using namespace dynb;

extern "C" int dynb_rg_suggest_capacity(int64_t n_atoms, const void* cell_host, const uint8_t* pbc_host, double radius,
                                        int dtype, int64_t* src_capacity, int64_t* cell_capacity)
{
    if (n_atoms < 0 || src_capacity == nullptr || cell_capacity == nullptr) return fail_arg("bad arguments");
    if (dtype == DYNB_F32) return rg_suggest<float>(n_atoms, cell_host, pbc_host, radius, src_capacity, cell_capacity);
    if (dtype == DYNB_F64) return rg_suggest<double>(n_atoms, cell_host, pbc_host, radius, src_capacity, cell_capacity);
    return fail_arg("dtype must be DYNB_F32 or DYNB_F64");
}

extern "C" int dynb_rg_workspace_bytes(int64_t n_atoms, int64_t n_targets, int64_t src_capacity, int64_t cell_capacity,
                                       int dtype, int64_t* bytes)
{
    if (n_atoms < 0 || n_targets < 0 || src_capacity < 1 || cell_capacity < 1 || bytes == nullptr)
        return fail_arg("bad arguments");
    if (dtype != DYNB_F32 && dtype != DYNB_F64) return fail_arg("dtype must be DYNB_F32 or DYNB_F64");
    if (n_atoms >= (1ll << 31) || src_capacity >= (1ll << 31) || n_targets >= (1ll << 31) || cell_capacity >= (1ll << 31) - 8)
        return fail_arg("sizes must stay below 2^31");
    *bytes = rg_layout(n_atoms, n_targets, src_capacity, cell_capacity, dtype).total + RG_WS_ALIGN;
    return DYNB_OK;
}

static int rg_plan_any(const void* pos_dev, int dtype, int64_t n_atoms, const void* cell_host, const uint8_t* pbc_host, double radius,
                       const int64_t* target_indices_dev, int64_t n_targets, void* workspace_dev, int64_t workspace_bytes,
                       int64_t src_capacity, int64_t cell_capacity, int32_t* neighbor_counts_dev, dynb_rg_header* header_host,
                       bool bins_only, void* stream)
{
    if (n_atoms <= 0 || n_targets <= 0) return fail_arg("n_atoms and n_targets must be positive (handle empty input in the caller)");
    if (pos_dev == nullptr || workspace_dev == nullptr) return fail_arg("null device pointer");
    if (target_indices_dev == nullptr && n_targets != n_atoms) return fail_arg("n_targets must equal n_atoms without target_indices");
    if (src_capacity < 1 || cell_capacity < 1) return fail_arg("capacities must be positive");
    if (n_atoms >= (1ll << 31) || src_capacity >= (1ll << 31) || n_targets >= (1ll << 31) || cell_capacity >= (1ll << 31) - 8)
        return fail_arg("sizes must stay below 2^31");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (dtype == DYNB_F32)
        return rg_plan<float>(pos_dev, n_atoms, cell_host, pbc_host, radius, target_indices_dev, n_targets, workspace_dev,
                              workspace_bytes, src_capacity, cell_capacity, neighbor_counts_dev, header_host, bins_only, s);
    if (dtype == DYNB_F64)
        return rg_plan<double>(pos_dev, n_atoms, cell_host, pbc_host, radius, target_indices_dev, n_targets, workspace_dev,
                               workspace_bytes, src_capacity, cell_capacity, neighbor_counts_dev, header_host, bins_only, s);
    return fail_arg("dtype must be DYNB_F32 or DYNB_F64");
}

extern "C" int dynb_rg_plan(const void* pos_dev, int dtype, int64_t n_atoms, const void* cell_host,
                            const uint8_t* pbc_host, double radius, const int64_t* target_indices_dev,
                            int64_t n_targets, void* workspace_dev, int64_t workspace_bytes, int64_t src_capacity,
                            int64_t cell_capacity, int32_t* neighbor_counts_dev, dynb_rg_header* header_host,
                            void* stream)
{
    return rg_plan_any(pos_dev, dtype, n_atoms, cell_host, pbc_host, radius, target_indices_dev, n_targets, workspace_dev,
                       workspace_bytes, src_capacity, cell_capacity, neighbor_counts_dev, header_host, false, stream);
}

extern "C" int dynb_rg_bin(const void* pos_dev, int dtype, int64_t n_atoms, const void* cell_host, const uint8_t* pbc_host,
                           double radius, void* workspace_dev, int64_t workspace_bytes, int64_t src_capacity, int64_t cell_capacity,
                           dynb_rg_header* header_host, void* stream)
{
    return rg_plan_any(pos_dev, dtype, n_atoms, cell_host, pbc_host, radius, nullptr, n_atoms, workspace_dev, workspace_bytes,
                       src_capacity, cell_capacity, nullptr, header_host, true, stream);
}

static int rg_fill_any(const void* workspace_dev, int dtype, int64_t* edge_index_dev, float* shifts_dev, void* dist_sq_dev,
                       const GlueArgs* glue, int64_t* total_dev, int64_t E, int64_t groups, int64_t long_lists, void* stream)
{
    if (workspace_dev == nullptr) return fail_arg("null workspace");
    if (E < 0) return fail_arg("E must be non-negative");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    if (E == 0) {
        if (total_dev != nullptr) DYNB_CUDA_OK(cudaMemsetAsync(total_dev, 0, sizeof(int64_t), s));
        return DYNB_OK;
    }
    if (edge_index_dev == nullptr || shifts_dev == nullptr) return fail_arg("null output pointer");
    if (dtype == DYNB_F32) return rg_fill<float>(workspace_dev, edge_index_dev, shifts_dev, dist_sq_dev, E, glue, total_dev, groups, long_lists, s);
    if (dtype == DYNB_F64) return rg_fill<double>(workspace_dev, edge_index_dev, shifts_dev, dist_sq_dev, E, glue, total_dev, groups, long_lists, s);
    return fail_arg("dtype must be DYNB_F32 or DYNB_F64");
}

extern "C" int dynb_rg_fill(const void* workspace_dev, int dtype, int64_t* edge_index_dev, float* cell_shifts_dev,
                            void* dist_sq_dev, int64_t E, void* stream)
{
    return rg_fill_any(workspace_dev, dtype, edge_index_dev, cell_shifts_dev, dist_sq_dev, nullptr, nullptr, E, RG_GROUPS_UNKNOWN, 1, stream);
}

extern "C" int dynb_rg_fill_counted(const void* workspace_dev, int dtype, int64_t* edge_index_dev, float* cell_shifts_dev,
                                    void* dist_sq_dev, int64_t E, int long_lists, int64_t* total_dev, void* stream)
{
    return dynb_rg_fill_groups(workspace_dev, dtype, edge_index_dev, cell_shifts_dev, dist_sq_dev, E, RG_GROUPS_UNKNOWN, long_lists, total_dev, stream);
}

extern "C" int dynb_rg_fill_groups(const void* workspace_dev, int dtype, int64_t* edge_index_dev, float* cell_shifts_dev,
                                   void* dist_sq_dev, int64_t E, int64_t groups, int64_t long_lists, int64_t* total_dev, void* stream)
{
    return rg_fill_any(workspace_dev, dtype, edge_index_dev, cell_shifts_dev, dist_sq_dev, nullptr, total_dev, E, groups, long_lists, stream);
}

extern "C" int dynb_rg_fill_glue(const void* workspace_dev, int dtype, int64_t* edge_index_dev, float* unit_shifts_dev,
                                 float* cart_shifts_dev, const float* cell_host, int negate_shifts, const int64_t* id_map_dev,
                                 int64_t E, void* stream)
{
    if (negate_shifts != 0 && negate_shifts != 1) return fail_arg("negate_shifts must be 0 or 1");
    if (cart_shifts_dev != nullptr && cell_host == nullptr) return fail_arg("cell_host is required with cart_shifts_dev");
    GlueArgs g{};
    g.cart = cart_shifts_dev;
    g.id_map = reinterpret_cast<const long long*>(id_map_dev);
    g.negate = negate_shifts;
    for (int k = 0; k < 9; k++) g.c[k] = cell_host != nullptr ? cell_host[k] : 0.0f;
    return rg_fill_any(workspace_dev, dtype, edge_index_dev, unit_shifts_dev, nullptr, &g, nullptr, E, RG_GROUPS_UNKNOWN, 1, stream);
}

extern "C" int dynb_rg_halo_mark_rank(const void* workspace_dev, int dtype, const int64_t* owner_dev, int64_t n_atoms,
                                      int64_t world_size, int64_t rank, uint32_t* needed_dev, uint8_t* has_foreign_dev, uint32_t* bad_dev, void* stream)
{
    if (workspace_dev == nullptr || owner_dev == nullptr || needed_dev == nullptr || has_foreign_dev == nullptr)
        return fail_arg("null pointer");
    if (n_atoms <= 0 || world_size < 1 || world_size > 32000 || rank < -1 || rank >= world_size) return fail_arg("bad sizes");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    HaloArgs ha;
    ha.owner = reinterpret_cast<const long long*>(owner_dev);
    ha.needed = needed_dev;
    ha.has_foreign = has_foreign_dev;
    ha.bad = bad_dev;
    ha.words = (int)((world_size + 31) / 32);
    ha.rank = (int)rank;
    DYNB_CUDA_OK(clear_ranges(s, {needed_dev, n_atoms * ha.words * 4, 0}, {has_foreign_dev, n_atoms, 0}));
    if (dtype == DYNB_F32) return rg_halo_mark<float>(workspace_dev, ha, n_atoms, s);
    if (dtype == DYNB_F64) return rg_halo_mark<double>(workspace_dev, ha, n_atoms, s);
    return fail_arg("dtype must be DYNB_F32 or DYNB_F64");
}

extern "C" int dynb_rg_halo_mark(const void* workspace_dev, int dtype, const int64_t* owner_dev, int64_t n_atoms,
                                 int64_t world_size, uint32_t* needed_dev, uint8_t* has_foreign_dev, void* stream)
{
    return dynb_rg_halo_mark_rank(workspace_dev, dtype, owner_dev, n_atoms, world_size, -1, needed_dev, has_foreign_dev, nullptr, stream);
}
