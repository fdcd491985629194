// Build phase on the device: ordered sampling, the density estimator, the frame splat, S(E), and
// the screening (R), constraint (B) and Dirichlet (K) stencils with their Galerkin hierarchy.
//
// Reference correspondence (paths relative to the reference checkout):
//   sort by cell             OrderedSampler                      Include/OrderedSamples.inl:32-85
//   density splat            TreeEstimator ctor / addSamples     Include/GridSamples.inl:361-391,436-491,740-771
//   estimator queries        TreeEstimator::operator()/depth     Include/GridSamples.inl:774-896
//   frame splat              Reconstructor ctor                  ExteriorPoissonRecon/ExteriorPoisson.h:181-264
//   S(E)                     TreeSplatter::operator()(p)         Include/GridSamples.inl:600-651
//   R                        ScalarFunctions::deltaMass          Include/Hat.scalars.inl:977-1063
//   B, c                     ScalarFunctions::stiffness, ctor    Include/Hat.scalars.inl:1585-1690, SystemEnergy.h:447-462
//   K                        StiffnessStencil / FullIntegrationStencil  Include/Hat.scalars.inl:261-293,528-545
//   Galerkin                 SingleCycleCascadicSystemEnergy::restrict  Include/SystemEnergy.h:464-477
//
// The reference's trees (RegularTreeNode) are stored here as dense per-depth vertex grids: a node
// that the reference never creates never receives data, so its dense value is zero.  The only
// structural information the reference uses is which cells have children (the depth of the leaf
// containing a point); it is kept as one byte per cell and depth.
//
// Splats are deterministic gathers: samples are sorted by the Morton key of their cell, so the
// samples of any coarser cell are one contiguous range; every output vertex is reduced by one
// warp in a fixed order.
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <string>
#include <vector>

#include <cub/cub.cuh>

#include "epr_common.cuh"
#include "epr_context.h"

namespace epr {

namespace {

constexpr int kMaxDeg = 9;  // 2 * 4 + 1

// ---------------------------------------------------------------------------------------------
// small device helpers
// ---------------------------------------------------------------------------------------------
__device__ inline void bspline_eval(int deg, double x, double *v)
{
    // iterative form of the recursive evaluation of GridSamples.inl:50-65
    v[deg] = 1.;
    for (int k = 1; k <= deg; k++)
    {
        const double scale = 1. / k;
        int b = deg - k;
        v[b] = v[b + 1] * (1. - x) * scale;
        for (int i = 1; i < k; i++)
        {
            double x1 = (x - i + k), x2 = (-x + i + 1);
            v[b + i] = (v[b + i] * x1 + v[b + i + 1] * x2) * scale;
        }
        v[b + k] *= x * scale;
    }
}

template <int D>
__host__ __device__ inline int64_t morton(const int *E, int bits)
{
    int64_t k = 0;
    for (int b = bits - 1; b >= 0; b--)
        for (int d = 0; d < D; d++) k = (k << 1) | ((E[d] >> b) & 1);
    return k;
}

template <int D>
__host__ __device__ inline void demorton(int64_t k, int bits, int *E)
{
    for (int d = 0; d < D; d++) E[d] = 0;
    for (int b = 0; b < bits; b++)
        for (int d = D - 1; d >= 0; d--) { E[d] |= (int)(k & 1) << b; k >>= 1; }
}

// first index in sorted keys[0..n) with key >= v
__device__ inline int64_t lower_bound(const int64_t *keys, int64_t n, int64_t v)
{
    int64_t lo = 0, hi = n;
    while (lo < hi)
    {
        int64_t mid = (lo + hi) >> 1;
        if (keys[mid] < v) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// cell of p at resolution res as the reference's tree descent finds it (strict ">" at splits,
// Misha/RegularTree.inl:538-543): points on a face belong to the lower cell
__device__ inline int tree_cell(double p, int res)
{
    double s = p * res;
    int o = (int)floor(s);
    if ((double)o == s && o > 0) o--;
    return o;
}

__device__ inline double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// warp_sum of W values at once: each exchange halves the values a lane keeps, so that 13 values take 16
// additions instead of 65 (and a quarter of the shuffles); value w ends in the lanes l with
// l / (32 / sums_width(W)) = w.  Every value is added up over the lanes in warp_sum's own order.
__host__ __device__ constexpr int sums_width(int W) { return W <= 1 ? 1 : 2 * sums_width((W + 1) / 2); }
template <int W>
__device__ __forceinline__ double warp_sums(const double *value, int lane)
{
    constexpr int P = sums_width(W);
    static_assert(P <= 32, "at most one value per lane");
    double v[P];
#pragma unroll
    for (int k = 0; k < P; k++) v[k] = k < W ? value[k] : 0.;
    int keep = P;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
    {
        if (keep > 1)
        {
            keep /= 2;
            const bool upper = lane & o;
#pragma unroll
            for (int k = 0; k < P / 2; k++)
                if (k < keep)
                {
                    const double mine = upper ? v[k + keep] : v[k], theirs = upper ? v[k] : v[k + keep];
                    v[k] = mine + __shfl_xor_sync(0xffffffffu, theirs, o);
                }
        }
        else v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
    return v[0];
}

inline unsigned int nblocks(int64_t n, int t) { return (unsigned int)((n + t - 1) / t); }

// ---------------------------------------------------------------------------------------------
// ordered sampling
// ---------------------------------------------------------------------------------------------
template <int D>
__global__ void cell_keys_kernel(const double *pos, int64_t n, int depth, int64_t *keys, int *vals)
{
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    int r = 1 << depth;
    int E[D];
    for (int d = 0; d < D; d++)
    {
        int e = (int)floor(pos[i * D + d] * r);
        E[d] = e < 0 ? 0 : (e > r - 1 ? r - 1 : e);
    }
    keys[i] = morton<D>(E, depth);
    vals[i] = (int)i;
}

__global__ void cell_flags_kernel(const int64_t *keys, int64_t n, int *flags)
{
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    flags[i] = (i == 0 || keys[i] != keys[i - 1]) ? 1 : 0;
}

__global__ void cell_start_kernel(const int64_t *keys, const int *flags, const int *ids, int64_t n, int *cellStart,
                                  int64_t *cellKey)
{
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (flags[i]) { cellStart[ids[i]] = (int)i; cellKey[ids[i]] = keys[i]; }
    // ids is the exclusive scan of the flags: the last sample's cell is ids + flags - 1
    if (i == n - 1) cellStart[ids[i] + flags[i]] = (int)n;
}

template <int D>
__global__ void finest_map_kernel(const int64_t *cellKey, int64_t ncells, int depth, int *map)
{
    int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= ncells) return;
    int E[D];
    demorton<D>(cellKey[k], depth, E);
    int r = 1 << depth;
    int64_t e = 0;
    for (int d = 0; d < D; d++) e = e * r + E[d];
    map[e] = (int)k;
}

// merged sample of each occupied cell: mean position and (count, sum p, sum p p^T)
// (GridSamples.inl:381-388 with DensityAndNoiseInfo(p, 1), :74)
template <int D>
__global__ void merge_cells_kernel(const double *pos, const int *order, const int *cellStart, int64_t ncells,
                                   double *mean, double *datum)
{
    constexpr int W = 1 + D + D * D;
    int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= ncells) return;
    double p[D], dat[W];
    for (int d = 0; d < D; d++) p[d] = 0;
    for (int w = 0; w < W; w++) dat[w] = 0;
    for (int j = cellStart[k]; j < cellStart[k + 1]; j++)
    {
        const double *q = pos + (int64_t)order[j] * D;
        for (int d = 0; d < D; d++) p[d] += q[d];
        dat[0] += 1.;
        for (int d = 0; d < D; d++) dat[1 + d] += q[d];
        for (int a = 0; a < D; a++)
            for (int b = 0; b < D; b++) dat[1 + D + a * D + b] += q[a] * q[b];
    }
    double cnt = (double)(cellStart[k + 1] - cellStart[k]);
    for (int d = 0; d < D; d++) mean[k * D + d] = p[d] / cnt;
    for (int w = 0; w < W; w++) datum[k * W + w] = dat[w];
}

// ---------------------------------------------------------------------------------------------
// tree structure: refined[t][cell] = 1 when the depth-t cell has children (RegularTree.inl:728-845)
// ---------------------------------------------------------------------------------------------
template <int D>
__global__ void refine_kernel(const int64_t *cellKey, int64_t ncells, int depth, int t, int KR, const uint8_t *prevRefined,
                              uint8_t *refined)
{
    int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= ncells) return;
    int E[D];
    demorton<D>(cellKey[k], depth, E);
    int lo[D], hi[D], I[D];
    int side = 1 << t, pside = 1 << (t - 1);
    for (int d = 0; d < D; d++)
    {
        int ct = E[d] >> (depth - t);  // ancestor at tree depth t+1
        lo[d] = (ct - KR) >> 1;
        hi[d] = (ct + KR + 1) >> 1;
        I[d] = lo[d];
    }
    while (true)
    {
        bool ok = true;
        int64_t li = 0, pi = 0;
        for (int d = 0; d < D; d++)
        {
            if (I[d] < 0 || I[d] >= side) ok = false;
            li = li * side + I[d];
            pi = pi * pside + (I[d] >> 1);
        }
        if (ok && (t == 1 || prevRefined[pi])) refined[li] = 1;
        int d = D - 1;
        for (; d >= 0; d--) { if (++I[d] <= hi[d]) break; I[d] = lo[d]; }
        if (d < 0) break;
    }
}

// ---------------------------------------------------------------------------------------------
// splat gathers: one warp per vertex of tree depth t (resolution 2^(t-1))
// ---------------------------------------------------------------------------------------------
struct SplatArgs
{
    const int64_t *cellKey;
    const int *cellStart;
    int64_t ncells;
    int depth;  // finest depth
    int t;      // tree depth of the grid
    int KR;     // kernel radius (B-spline degree 2 KR + 1)
    const int *rlo = nullptr, *rhi = nullptr;  // occupied-cell range of every depth-t cell, by Morton code
};

// range of occupied cells inside the depth-t cell C
template <int D>
__device__ inline void cell_range(const SplatArgs &a, const int *C, int64_t &lo, int64_t &hi)
{
    if (a.rlo)
    {
        const int res = 1 << (a.t - 1);
        int64_t li = 0;
        for (int d = 0; d < D; d++) li = li * res + C[d];
        lo = a.rlo[li];
        hi = a.rhi[li];
        return;
    }
    int64_t m = morton<D>(C, a.t - 1);
    int s = a.depth + 1 - a.t;  // levels between depth-t cells and finest cells
    lo = lower_bound(a.cellKey, a.ncells, m << (D * s));
    hi = lower_bound(a.cellKey, a.ncells, (m + 1) << (D * s));
}

// Occupied-cell range of every depth-t cell: the occupied finest cells are sorted by Morton key, so
// the ones below a depth-t cell are contiguous; mark where each ancestor's run starts and ends.
// (stored by the row-major index of the depth-t cell)
template <int D>
__global__ void level_ranges_kernel(const int64_t *cellKey, int64_t ncells, int t, int shift, int *rlo, int *rhi)
{
    int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= ncells) return;
    int64_t anc = cellKey[k] >> shift;
    int C[D];
    demorton<D>(anc, t - 1, C);
    const int res = 1 << (t - 1);
    int64_t li = 0;
    for (int d = 0; d < D; d++) li = li * res + C[d];
    if (k == 0 || (cellKey[k - 1] >> shift) != anc) rlo[li] = (int)k;
    if (k == ncells - 1 || (cellKey[k + 1] >> shift) != anc) rhi[li] = (int)(k + 1);
}

// ---------------------------------------------------------------------------------------------
// Chunked gathers for the coarse tree levels.  There a vertex's window covers a large part of the
// domain, so one warp per vertex would walk hundreds of thousands of items.  Instead each vertex's
// item list (the concatenation, in window order, of the items of its window cells) is cut into
// chunks of kChunk items, one warp reduces each chunk into a partial sum, and a final pass adds a
// vertex's partials in chunk order: the result is still deterministic.
// ---------------------------------------------------------------------------------------------
constexpr int kChunk = 2048;

// Item range of one window cell: occupied-cell indices (merged density data) or sample positions
// in the sorted order (frame samples).
template <int D, bool Samples>
__device__ inline void item_range(const SplatArgs &a, const int *C, int &lo, int &hi)
{
    int64_t l, h;
    cell_range<D>(a, C, l, h);
    if (Samples) { lo = a.cellStart[l]; hi = a.cellStart[h]; }
    else { lo = (int)l; hi = (int)h; }
}

// (a level's vertices are counted in 32 bits: chunked_level scans them as ints)
template <int D>
__device__ inline void vertex_of(int64_t vi, int nv, int *v)
{
    uint32_t u = (uint32_t)vi;
    for (int d = D - 1; d >= 0; d--)
    {
        const uint32_t q = u / (uint32_t)nv;
        v[d] = (int)(u - q * (uint32_t)nv);
        u = q;
    }
}

template <int D>
__device__ inline bool window_next(int *C, const int *clo, const int *chi)
{
    int d = D - 1;
    for (; d >= 0; d--) { if (++C[d] <= chi[d]) return true; C[d] = clo[d]; }
    return false;
}

template <int D, bool Samples>
__global__ void vertex_chunks_kernel(SplatArgs a, int *nchunks)
{
    int res = 1 << (a.t - 1), nv = res + 1;
    int64_t NV = 1;
    for (int d = 0; d < D; d++) NV *= nv;
    int64_t vi = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (vi >= NV) return;
    int v[D], clo[D], chi[D], C[D];
    vertex_of<D>(vi, nv, v);
    for (int d = 0; d < D; d++) { clo[d] = max(0, v[d] - a.KR - 1); chi[d] = min(res - 1, v[d] + a.KR); C[d] = clo[d]; }
    int64_t count = 0;
    do
    {
        int lo, hi;
        item_range<D, Samples>(a, C, lo, hi);
        count += hi - lo;
    } while (window_next<D>(C, clo, chi));
    nchunks[vi] = (int)((count + kChunk - 1) / kChunk);
}

// Contribution of item `it` to vertex v through window cell C, added to acc.
// Density: a merged cell (mean position, summed (1, p, p p^T)) splatted with the degree 2 KR + 1
// B-spline weights of its mean and the estimator's depth weight (TreeSplatter::_addSample,
// GridSamples.inl:458-491; TreeEstimator ctor :749-760).  The window is centred on the depth-t
// ancestor of the item's cell while the weights come from floor(p res), as in the reference.
// The per-axis B-spline values of every item at the level are tabulated once (item_bspline_kernel)
// instead of once per (vertex, item) pair; the products keep the reference's order.
template <int D>
struct DensityItem
{
    static constexpr int W = 1 + D + D * D;
    const double *bs;  // per item: D x (deg + 1) B-spline values at this level
    const double *datum;
    double depthWeight;
    __device__ void operator()(const SplatArgs &a, int it, const int *v, const int *C, double *acc) const
    {
        const int nb = 2 * a.KR + 2;
        double wt = depthWeight;
        const double *b = bs + (int64_t)it * D * nb;
        for (int d = 0; d < D; d++) wt *= b[d * nb + v[d] - (C[d] - a.KR)];
        for (int w = 0; w < W; w++) acc[w] += wt * datum[(int64_t)it * W + w];
    }
};

// Frame sample: normalised frame times the sample's measure and 2^(2 depth), split between the two
// tree depths bracketing its estimated depth with weights 2^((d-1) D) (ExteriorPoisson.h:181-228,
// GridSamples.inl:436-456), B-spline weights of the sample position.  Per sorted sample: the
// level weight and B-spline values (skew_level_kernel) and the scaled frame (skew_frame_kernel).
template <int D>
struct SkewItem
{
    static constexpr int W = D * (D - 1) / 2;
    const double *bs;     // per sorted sample: D x (deg + 1) B-spline values at this level
    const double *lw;     // per sorted sample: level weight at this level
    const double *frame;  // per sorted sample: W scaled frame values
    __device__ void operator()(const SplatArgs &a, int j, const int *v, const int *C, double *acc) const
    {
        const double l = lw[j];
        if (l == 0) return;
        const int nb = 2 * a.KR + 2;
        double wt = l;
        const double *b = bs + (int64_t)j * D * nb;
        for (int d = 0; d < D; d++) wt *= b[d * nb + v[d] - (C[d] - a.KR)];
        for (int k = 0; k < W; k++) acc[k] += wt * frame[(int64_t)j * W + k];
    }
};

// per-axis B-spline values of n points (pts[idx[j]] or pts[j]) at the resolution of tree depth t
template <int D>
__global__ void item_bspline_kernel(const double *pts, const int *idx, int64_t n, int t, int deg, const double *lw, double *bs)
{
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= n) return;
    if (lw && lw[j] == 0) return;
    const int64_t s = idx ? idx[j] : j;
    const int res = 1 << (t - 1);
    for (int d = 0; d < D; d++)
    {
        double pr = pts[s * D + d] * res;
        int e = (int)floor(pr);
        bspline_eval(deg, pr - e, bs + (j * D + d) * (deg + 1));
    }
}

// level weight of every sorted frame sample at tree depth t
__global__ void skew_level_kernel(const double *sdepth, const int *order, int64_t n, int t, int depth, int D, double *lw)
{
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int maxT = depth + 1;
    double dd = sdepth[order[j]] + 1.;
    double w = 0;
    if (dd >= maxT) w = (t == maxT) ? (double)(1ull << (depth * D)) : 0.;
    else if (dd <= 1) w = (t == 1) ? 1. : 0.;
    else
    {
        int d1 = (int)floor(dd), d2 = d1 + 1;
        double f = dd - d1;
        if (t == d1) w = (1. - f) * (double)(1ull << ((d1 - 1) * D));
        else if (t == d2) w = f * (double)(1ull << ((d2 - 1) * D));
    }
    lw[j] = w;
}

// normalised frame times measure and 2^(2 depth), per sorted sample
template <int D>
__global__ void skew_frame_kernel(const double *skew, const double *measure, const int *order, int64_t n, int depth, double *frame)
{
    constexpr int W = D * (D - 1) / 2;
    const int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int s = order[j];
    const double *sk = skew + (int64_t)s * W;
    double nrm = 0;
    for (int k = 0; k < W; k++) nrm += 2 * sk[k] * sk[k];
    nrm = sqrt(nrm);
    double m = measure[s], sc = (double)(1ull << (depth * 2));
    for (int k = 0; k < W; k++) frame[j * W + k] = sk[k] / nrm * m * sc;
}

// the vertex of every chunk, kept in the chunk's first partial sum until its warp has read it (a search by every
// warp took 21 dependent loads at depth 8)
__global__ void chunk_owner_kernel(const int *chunkStart, int64_t NV, int W, double *partial)
{
    const int64_t vi = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (vi >= NV) return;
    for (int c = chunkStart[vi]; c < chunkStart[vi + 1]; c++) partial[(int64_t)c * W] = __longlong_as_double(vi);
}

// One warp per chunk.  With outliers most chunks hold a few items of a vertex, and what a chunk costs beyond them
// decides: its sums in 16 additions (warp_sums), its vertex looked up, 32-bit index arithmetic.  Depth 7, 250K
// samples with 10 % outliers, finest level: densities 3.65 to 1.64 ms, frames 1.49 to 0.92 ms.  The vertex's window cells are taken 32 at a time: each lane looks up one
// cell's item range, a warp scan places the cells' items end to end, and the warp then walks the
// part of those items that falls into the chunk 32 items at a time, every lane finding the cell of
// its item by a binary search over the scanned offsets (shuffles).  Lanes stay busy however the
// items spread over the cells, and every lane's order of accumulation is fixed by the item index.
template <int D, bool Samples, class Item>
__global__ void chunk_gather_kernel(SplatArgs a, Item item, const int *chunkStart, int64_t nchunks, double *partial)
{
    constexpr int W = Item::W;
    const unsigned full = 0xffffffffu;
    int64_t chunk = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    int lane = threadIdx.x & 31;
    if (chunk >= nchunks) return;  // whole warps
    const int64_t vi = __double_as_longlong(partial[chunk * W]);  // the chunk's vertex (chunk_owner_kernel)
    __syncwarp();
    const int64_t first = (chunk - chunkStart[vi]) * kChunk, last = first + kChunk;
    int res = 1 << (a.t - 1), nv = res + 1;
    int v[D], clo[D], wd[D];
    vertex_of<D>(vi, nv, v);
    int ncell = 1;
    for (int d = 0; d < D; d++)
    {
        clo[d] = max(0, v[d] - a.KR - 1);
        wd[d] = min(res - 1, v[d] + a.KR) - clo[d] + 1;
        ncell *= wd[d];
    }
    double acc[W];
    for (int w = 0; w < W; w++) acc[w] = 0;
    int64_t base = 0;  // items of the window cells before the current batch
    for (int kb = 0; kb < ncell && base < last; kb += 32)
    {
        // this lane's cell (window order: last axis fastest) and its items
        const int k = kb + lane;
        int C[D], ilo = 0, cnt = 0;
        {
            int t = k < ncell ? k : 0;
            for (int d = D - 1; d >= 0; d--) { C[d] = clo[d] + t % wd[d]; t /= wd[d]; }
        }
        if (k < ncell)
        {
            int ihi;
            item_range<D, Samples>(a, C, ilo, ihi);
            cnt = ihi - ilo;
        }
        int incl = cnt;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            int n = __shfl_up_sync(full, incl, o);
            if (lane >= o) incl += n;
        }
        const int excl = incl - cnt;
        const int total = __shfl_sync(full, incl, 31);
        const int64_t b0 = max(base, first), b1 = min(base + (int64_t)total, last);
        for (int64_t t0 = b0; t0 < b1; t0 += 32)
        {
            const int64_t t = t0 + lane;
            const int r = (int)(t - base);  // position among this batch's items
            int own = 0;
#pragma unroll
            for (int step = 16; step > 0; step >>= 1)
            {
                const int cand = own + step;
                const int e = __shfl_sync(full, excl, cand & 31);
                if (cand < 32 && e <= r) own = cand;
            }
            const int olo = __shfl_sync(full, ilo, own), oex = __shfl_sync(full, excl, own);
            int Co[D];
#pragma unroll
            for (int d = 0; d < D; d++) Co[d] = __shfl_sync(full, C[d], own);
            if (t < b1) item(a, olo + (r - oex), v, Co, acc);
        }
        base += total;
    }
    const double sum = warp_sums<W>(acc, lane);
    constexpr int per = 32 / sums_width(W);  // lanes that hold the same sum
    if (lane % per == 0 && lane / per < W) partial[chunk * W + lane / per] = sum;
}

template <int W>
__global__ void chunk_finish_kernel(const int *chunkStart, int64_t NV, const double *partial, double scale, double *grid)
{
    int64_t vi = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (vi >= NV) return;
    double acc[W];
    for (int w = 0; w < W; w++) acc[w] = 0;
    for (int c = chunkStart[vi]; c < chunkStart[vi + 1]; c++)
        for (int w = 0; w < W; w++) acc[w] += partial[(int64_t)c * W + w];
    for (int w = 0; w < W; w++) grid[vi * W + w] = acc[w] * scale;
}

// ---------------------------------------------------------------------------------------------
// estimator queries (GridSamples.inl:774-896)
// ---------------------------------------------------------------------------------------------
template <int D>
struct DensityGrids
{
    const double *g[12];
    int depth;
};

// Interpolated splat data at p from tree depth t; only the first NW of the W components (the
// sample count alone for the depth search), each summed exactly as in the full interpolation.
template <int D, int NW = 1 + D + D * D>
__device__ void density_interp(const DensityGrids<D> &G, int t, const double *p, double *out)
{
    constexpr int W = 1 + D + D * D;
    for (int w = 0; w < NW; w++) out[w] = 0;
    if (t < 1) return;  // the root carries no data
    int res = 1 << (t - 1), nv = res + 1;
    int e[D];
    double lv[D][2];
    for (int d = 0; d < D; d++)
    {
        double s = p[d] * res;
        int f = (int)floor(s);
        double x = s - f;
        lv[d][0] = 1. - x;
        lv[d][1] = x;
        e[d] = tree_cell(p[d], res);
    }
    const double *g = G.g[t - 1];
    for (int c = 0; c < (1 << D); c++)
    {
        double s = 1.;
        int64_t vi = 0;
        bool in = true;
        for (int d = 0; d < D; d++)
        {
            int b = (c >> (D - 1 - d)) & 1;
            int o = e[d] + b;
            if (o < 0 || o > res) in = false;
            s *= lv[d][b];
            vi = vi * nv + o;
        }
        if (!in) continue;
        for (int w = 0; w < NW; w++) out[w] += g[vi * W + w] * s;
    }
}

template <int D>
__device__ double samples_per_cell(const DensityGrids<D> &G, int t, const double *p)
{
    double count;
    density_interp<D, 1>(G, t, p, &count);
    return count * (1. / (double)(1u << ((t - 1) * (D - 2))));  // a power of two
}

template <int D>
__device__ double est_depth_raw(const DensityGrids<D> &G, int maxT, const double *p)
{
    const double tg = (double)(1 << (D - 2));
    int d1 = maxT, d2 = maxT + 1;
    // s1: samples per cell at depth d1 (computed by the search), s2 at d2 = d1 + 1 (the previous s1)
    double s1 = samples_per_cell<D>(G, d1, p), s2 = 0;
    bool have2 = false;
    while (d2 > 1 && s1 < tg)
    {
        d1--, d2--;
        s2 = s1;
        have2 = true;
        s1 = d1 >= 1 ? samples_per_cell<D>(G, d1, p) : 0;
    }
    if (d2 == 1 || d2 == maxT + 1)
    {
        int d = (d2 == 1) ? 1 : maxT;
        double spc = (d2 == 1) ? s2 : s1;
        return d + log(spc / tg) / log(2.);
    }
    if (!have2) s2 = samples_per_cell<D>(G, d2, p);
    if (!s2) return d1;
    return d1 + log(tg / s1) / log(s2 / s1);
}

// ascending eigenvalues of a symmetric D x D matrix (cyclic Jacobi, until what is left off the diagonal is below
// 1e-20 of the matrix: the covariances here are differences good to 1e-16 of it, and their eigenvalues enter as
// shares of the trace; every loop unrolled, so that the matrix stays in registers)
template <int D>
__device__ void sym_eigenvalues(double a[D][D], double *ev)
{
    for (int sweep = 0; sweep < 64; sweep++)
    {
        double off = 0, diag = 0;
#pragma unroll
        for (int i = 0; i < D; i++)
        {
            diag += a[i][i] * a[i][i];
#pragma unroll
            for (int j = i + 1; j < D; j++) off += a[i][j] * a[i][j];
        }
        if (!(off > 1e-40 * diag)) break;
#pragma unroll
        for (int p = 0; p < D; p++)
#pragma unroll
            for (int q = p + 1; q < D; q++)
            {
                if (a[p][q] == 0) continue;
                double theta = (a[q][q] - a[p][p]) / (2 * a[p][q]);
                double t = (theta >= 0 ? 1. : -1.) / (fabs(theta) + sqrt(theta * theta + 1));
                double c = 1 / sqrt(t * t + 1), s = t * c;
#pragma unroll
                for (int k = 0; k < D; k++)
                {
                    double akp = a[k][p], akq = a[k][q];
                    a[k][p] = c * akp - s * akq;
                    a[k][q] = s * akp + c * akq;
                }
#pragma unroll
                for (int k = 0; k < D; k++)
                {
                    double apk = a[p][k], aqk = a[q][k];
                    a[p][k] = c * apk - s * aqk;
                    a[q][k] = s * apk + c * aqk;
                }
            }
    }
#pragma unroll
    for (int i = 0; i < D; i++) ev[i] = a[i][i];
#pragma unroll
    for (int i = 1; i < D; i++)
#pragma unroll
        for (int j = i; j > 0; j--)
            if (ev[j - 1] > ev[j]) { double t = ev[j]; ev[j] = ev[j - 1]; ev[j - 1] = t; }
}

template <int D>
__global__ void estimator_kernel(DensityGrids<D> G, const double *pos, const int *order, int64_t n, double *measure, double *noise,
                                 double *sdepth)
{
    constexpr int W = 1 + D + D * D;
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    i = order[i];  // neighbours in space together: one depth search and one set of vertices for a warp
    double p[D];
    for (int d = 0; d < D; d++) p[d] = pos[i * D + d];
    int maxT = G.depth + 1;
    double dd = est_depth_raw<D>(G, maxT, p);
    double info[W];
    if (dd >= maxT) density_interp<D>(G, maxT, p, info);
    else if (dd < 0) density_interp<D>(G, 1, p, info);
    else
    {
        int d1 = (int)floor(dd), d2 = d1 + 1;
        double f = dd - d1, b[W];
        density_interp<D>(G, d1, p, info);
        density_interp<D>(G, d2, p, b);
        for (int w = 0; w < W; w++) info[w] = info[w] * (1. - f) + b[w] * f;
    }
    double wsum = info[0];
    measure[i] = 1. / wsum;
    double C[D][D];
    for (int a = 0; a < D; a++)
        for (int b = 0; b < D; b++) C[a][b] = info[1 + D + a * D + b] / wsum - info[1 + a] / wsum * info[1 + b] / wsum;
    double ev[D];
    sym_eigenvalues<D>(C, ev);
    double sum = 0, low = 0;
    for (int d = 0; d < D; d++) { sum += ev[d]; if (d < 2) low += ev[d]; }
    noise[i] = (low * D) / (sum * 2);
    sdepth[i] = dd - 1.;  // depth(p) of the estimator: leaf of a sample is at the finest depth
}

// S(E) at element centres, summed over tree depths down to the leaf containing the centre
template <int D>
struct SkewGrids
{
    const double *g[12];
    const uint8_t *refined[12];
    int depth;
};

// FitBlade (ExteriorPoisson.h:411-438) of a packed skew matrix (entry (i, j), j < i, in (i, j)
// order; the matrix m(i, j) = p, m(j, i) = -p in the reference's (column, row) indexing,
// Hat.inl:45-52): the power iteration v2 = Next(v1), v1 <- -Next(v2) with
// Next(v) = normalised (m v - (v . m v) v), stopped when |v1 - v1'|^2 < 1e-10 or after 1000 steps
// (the command line's ProjectionIterations / ProjectionEpslion, ExteriorPoissonRecon.cpp:48-49);
// then a, b = v1, v2 scaled by |m|^(1/2) (Frobenius) and p(i, j) = (a_j b_i - a_i b_j) / 2.  The
// iteration starts from m's largest column (in m's image, never in its kernel; the reference starts
// from a random unit vector, which converges to the same blade).
template <int D>
__device__ void project_blade(double *p)
{
    double m[D][D];
    double sq = 0;
    for (int i = 0; i < D; i++) m[i][i] = 0;
    for (int i = 0, idx = 0; i < D; i++)
        for (int j = 0; j < i; j++, idx++)
        {
            // the reference's SquareMatrix is indexed (column, row) and S() * v sums over columns:
            // as a row-major matrix, row j column i holds p and row i column j holds -p
            m[j][i] = p[idx];
            m[i][j] = -p[idx];
            sq += 2 * p[idx] * p[idx];
        }
    if (sq == 0) return;
    auto next = [&](const double *v, double *out) {
        double w[D], dot = 0, n2 = 0;
        for (int i = 0; i < D; i++)
        {
            w[i] = 0;
            for (int j = 0; j < D; j++) w[i] += m[i][j] * v[j];
        }
        for (int i = 0; i < D; i++) dot += v[i] * w[i];
        for (int i = 0; i < D; i++) { w[i] -= dot * v[i]; n2 += w[i] * w[i]; }
        const double n = sqrt(n2);
        for (int i = 0; i < D; i++) out[i] = w[i] / n;
    };
    double v1[D], v2[D];
    int best = 0;
    double bn = -1;
    for (int k = 0; k < D; k++)
    {
        double n2 = 0;
        for (int i = 0; i < D; i++) n2 += m[i][k] * m[i][k];
        if (n2 > bn) { bn = n2; best = k; }
    }
    for (int i = 0; i < D; i++) { v1[i] = m[i][best] / sqrt(bn); v2[i] = 0; }
    for (int s = 0; s < 1000; s++)
    {
        double nv1[D];
        next(v1, v2);
        next(v2, nv1);
        double d2 = 0;
        for (int i = 0; i < D; i++) { nv1[i] = -nv1[i]; d2 += (v1[i] - nv1[i]) * (v1[i] - nv1[i]); }
        if (d2 < 1e-10) break;
        for (int i = 0; i < D; i++) v1[i] = nv1[i];
    }
    const double scale = sqrt(sqrt(sq));
    for (int i = 0, idx = 0; i < D; i++)
        for (int j = 0; j < i; j++, idx++) p[idx] = ((v1[j] * scale) * (v2[i] * scale) - (v1[i] * scale) * (v2[j] * scale)) / 2.;
}

// sum[v] = own[v] + the prolongation of the coarser level's sums: the vertex values accumulated over the tree
// depths, of which element_frame_kernel reads one depth (reading all nine of a depth-8 tree took 10.7 ms)
template <int D>
__global__ void accumulate_frames_kernel(int level, const double *own, const double *coarse, double *sum)
{
    constexpr int K = D * (D - 1) / 2;
    Grid<D> g(level), gc(level - 1);
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= g.N) return;
    int I[D];
    g.node(i, I);
    double acc[K];
#pragma unroll
    for (int k = 0; k < K; k++) acc[k] = 0;
    for (int c = 0; c < (1 << D); c++)
    {
        int J[D];
        bool use = true;
        double w = 1.;
#pragma unroll
        for (int d = 0; d < D; d++)
        {
            const int b = (c >> d) & 1;
            if (I[d] & 1) { J[d] = (I[d] >> 1) + b; w *= 0.5; }
            else { J[d] = I[d] >> 1; use = use && !b; }
        }
        if (!use) continue;
        const double *v = coarse + gc.node(J) * K;
#pragma unroll
        for (int k = 0; k < K; k++) acc[k] += w * v[k];
    }
#pragma unroll
    for (int k = 0; k < K; k++) sum[i * K + k] = own[i * K + k] + acc[k];
}

template <int D>
__global__ void element_frame_kernel(SkewGrids<D> G, double *S, int *leaf, int project)
{
    constexpr int K = D * (D - 1) / 2;
    int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const Grid<D> grid(G.depth);
    if (e >= grid.NE) return;
    int E[D];
    grid.elem(e, E);
    // the element centre (E + 1/2) / r lies inside a cell of every depth (its coordinate there is an odd
    // multiple of a power of two), so the cells are E's leading bits and its place in them the others
    int L = 1;
    while (L <= G.depth)
    {
        int side = 1 << L;
        int64_t li = 0;
        for (int d = 0; d < D; d++) li = li * side + (E[d] >> (G.depth + 1 - L));
        if (!G.refined[L][li]) break;
        L++;
    }
    // the sum over the tree depths 1..L of the splats' multilinear interpolants, which on a depth-L cell is
    // the interpolant of their accumulated vertex values
    double acc[K];
    for (int k = 0; k < K; k++) acc[k] = 0;
    {
        const int res = 1 << (L - 1), nv = res + 1, below = G.depth + 1 - L;
        const double unit = 1. / (double)(1 << below);
        int c[D];
        double lv[D][2];
        for (int d = 0; d < D; d++)
        {
            const double x = ((E[d] & ((1 << below) - 1)) + 0.5) * unit;
            lv[d][0] = 1. - x;
            lv[d][1] = x;
            c[d] = E[d] >> below;
        }
        const double *g = G.g[L - 1];
        for (int cc = 0; cc < (1 << D); cc++)
        {
            double w = 1.;
            int64_t vi = 0;
            for (int d = 0; d < D; d++)
            {
                int b = (cc >> (D - 1 - d)) & 1;
                w *= lv[d][b];
                vi = vi * nv + (c[d] + b);
            }
            for (int k = 0; k < K; k++) acc[k] += g[vi * K + k] * w;
        }
    }
    if (project) project_blade<D>(acc);
    for (int k = 0; k < K; k++) S[e * K + k] = acc[k];
    leaf[e] = L;
}

// ---------------------------------------------------------------------------------------------
// deterministic sums
// ---------------------------------------------------------------------------------------------
__global__ void sum_kernel(const double *v, int64_t n, int stride, int comps, double *partial)
{
    __shared__ double sh[32];
    double acc = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        for (int k = 0; k < comps; k++) { double x = v[i * stride + k]; acc += (comps == 1) ? x : 2 * x * x; }
    acc = warp_sum(acc);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) sh[w] = acc;
    __syncthreads();
    if (w == 0)
    {
        double t = lane < (int)(blockDim.x >> 5) ? sh[lane] : 0.;
        t = warp_sum(t);
        if (lane == 0) partial[blockIdx.x] = t;
    }
}
__global__ void sum_finish_kernel(const double *partial, int nb, double *out)
{
    double s = 0;
    for (int b = threadIdx.x; b < nb; b += 32) s += partial[b];
    s = warp_sum(s);
    if (threadIdx.x == 0) out[0] = s;
}

// ---------------------------------------------------------------------------------------------
// stencils
// ---------------------------------------------------------------------------------------------
__host__ __device__ inline double mass1(int a, int b) { return a == b ? 1. / 3. : 1. / 6.; }
__host__ __device__ inline double stiff1(int a, int b) { return a == b ? 1. : -1.; }

// R = sWeight * mean(measure) * sum_samples w phi_a phi_b.  First per occupied cell, a warp each: the sums
// over the cell's samples (in their order) of w phi_a phi_b for every pair of corners a <= b; 32 samples at
// a time put their weighted and plain hat values in shared memory, then every lane sums its pairs.  A
// sample's exponential and hats are formed once (a thread per node and its eight cells formed them eight
// times, in a loop as long as the densest cell: 6.9 ms at depth 7 with 200,000 samples).
template <int D>
struct CellPairs
{
    static constexpr int C = 1 << D, N = C * (C + 1) / 2;
    static __host__ __device__ constexpr int index(int a, int b) { return a <= b ? a * C - a * (a - 1) / 2 + (b - a) : index(b, a); }
};
template <int D>
__global__ void __launch_bounds__(128) cell_mass_kernel(const double *pos, const double *noise, const int *order, const int *cellStart,
                                                         const int64_t *cellKey, int64_t ncells, int depth, double nSigma, double *mass)
{
    using CP = CellPairs<D>;
    constexpr int C = CP::C, NP = (CP::N + 31) / 32;
    __shared__ double hats[4][32][C + 1];  // the last value of a row: the sample's weight
    const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t k = blockIdx.x * (int64_t)4 + wp;
    if (k >= ncells) return;  // whole warps
    const int r = 1 << depth;
    int E[D];
    demorton<D>(cellKey[k], depth, E);
    int pa[NP], pb[NP];
    double acc[NP];
#pragma unroll
    for (int n = 0; n < NP; n++)
    {
        int p = lane + 32 * n, a = 0;
        while (a < C - 1 && p >= C - a) { p -= C - a; a++; }
        pa[n] = a;
        pb[n] = min(a + p, C - 1);
        acc[n] = 0;
    }
    const int first = cellStart[k], last = cellStart[k + 1];
    for (int j0 = first; j0 < last; j0 += 32)
    {
        const int j = j0 + lane;
        if (j < last)
        {
            const int s = order[j];
            const double nz = noise[s];
            double lv[D][2];
#pragma unroll
            for (int d = 0; d < D; d++) { const double x = pos[(int64_t)s * D + d] * r - E[d]; lv[d][0] = 1. - x; lv[d][1] = x; }
#pragma unroll
            for (int c = 0; c < C; c++)
            {
                double h = 1.;
#pragma unroll
                for (int d = 0; d < D; d++) h *= lv[d][(c >> (D - 1 - d)) & 1];
                hats[wp][lane][c] = h;
            }
            hats[wp][lane][C] = exp(-nz * nz / (2. * nSigma * nSigma));
        }
        __syncwarp();
        const int cnt = min(32, last - j0);
        for (int t = 0; t < cnt; t++)
#pragma unroll
            for (int n = 0; n < NP; n++) acc[n] += hats[wp][t][pa[n]] * hats[wp][t][pb[n]] * hats[wp][t][C];
        __syncwarp();
    }
#pragma unroll
    for (int n = 0; n < NP; n++)
        if (lane + 32 * n < CP::N) mass[k * CP::N + lane + 32 * n] = acc[n];
}
// ... then gathered per column node from its cells
template <int D>
__global__ void screening_kernel(const double *mass, const int *cellOfFinest, int depth, const double *scaleDev, double *A)
{
    using CP = CellPairs<D>;
    constexpr int S = Dims<D>::S;
    Grid<D> g(depth);
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= g.N) return;
    int I[D];
    g.node(i, I);
    double acc[S];
#pragma unroll
    for (int o = 0; o < S; o++) acc[o] = 0;
    bool any = false;
#pragma unroll
    for (int a = 0; a < (1 << D); a++)
    {
        int E[D];
        bool ok = true;
#pragma unroll
        for (int d = 0; d < D; d++) { E[d] = I[d] - ((a >> (D - 1 - d)) & 1); if (E[d] < 0 || E[d] >= g.r) ok = false; }
        if (!ok) continue;
        const int k = cellOfFinest[g.elem(E)];
        if (k < 0) continue;
        any = true;
        const double *m = mass + (int64_t)k * CP::N;
#pragma unroll
        for (int b = 0; b < (1 << D); b++)
        {
            int o = 0;
#pragma unroll
            for (int d = 0; d < D; d++) o = o * 3 + (((b >> (D - 1 - d)) & 1) - ((a >> (D - 1 - d)) & 1) + 1);
            acc[o] += m[CP::index(a, b)];
        }
    }
    if (!any) return;
    const double sc = *scaleDev;
#pragma unroll
    for (int o = 0; o < S; o++) A[(int64_t)o * g.N + i] = acc[o] * sc;
}

// B(f2, f1) = sum_E sum_{a != b} S_E(b, a) int_E d_a phi_f1 d_b phi_f2 (column f1)
// (elements whose frame is zero contribute nothing and are skipped; the element and corner loops
// are unrolled so that the 3^D accumulators stay in registers).  S_E is skew, so an axis pair enters with
// (d_x phi_a d_y phi_b - d_y phi_a d_x phi_b): of the corner signs' products, +-1/4 each, the difference is 0 or
// +-1/2, and the mass factors of the other axes are constants.  A multiply-add per pair that is left, 12 an
// element and node in 3D, instead of 24 products of three factors each: 12.3 to 3.5 ms at depth 8 with 10 %
// outliers.
template <int D>
__global__ void __launch_bounds__(128) constraint_kernel(const double *Sel, int depth, double *B)
{
    constexpr int S = Dims<D>::S, K = Dims<D>::K;
    Grid<D> g(depth);
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= g.N) return;
    int I[D];
    g.node(i, I);
    double acc[S];
#pragma unroll
    for (int o = 0; o < S; o++) acc[o] = 0;
    double half = 0.5;  // times the element's side to the power D - 2, exact
    for (int d = 0; d < D - 2; d++) half /= g.r;
#pragma unroll
    for (int a = 0; a < (1 << D); a++)
    {
        int E[D];
        bool ok = true;
#pragma unroll
        for (int d = 0; d < D; d++) { E[d] = I[d] - ((a >> (D - 1 - d)) & 1); if (E[d] < 0 || E[d] >= g.r) ok = false; }
        if (!ok) continue;
        double s[K];
        bool zero = true;
#pragma unroll
        for (int k = 0; k < K; k++)
        {
            s[k] = Sel[g.elem(E) * K + k];
            zero = zero && s[k] == 0;
        }
        if (zero) continue;
#pragma unroll
        for (int k = 0; k < K; k++) s[k] *= half;
#pragma unroll
        for (int b = 0; b < (1 << D); b++)
        {
            int o = 0;
#pragma unroll
            for (int d = 0; d < D; d++) o = o * 3 + (((b >> (D - 1 - d)) & 1) - ((a >> (D - 1 - d)) & 1) + 1);
#pragma unroll
            for (int y = 1; y < D; y++)
#pragma unroll
                for (int x = 0; x < y; x++)
                {
                    const int ax = (a >> (D - 1 - x)) & 1, ay = (a >> (D - 1 - y)) & 1, bx = (b >> (D - 1 - x)) & 1, by = (b >> (D - 1 - y)) & 1;
                    const int sign = ((ax == by ? 1 : -1) - (ay == bx ? 1 : -1)) / 2;
                    if (sign == 0) continue;
                    double m = sign;
#pragma unroll
                    for (int d = 0; d < D; d++)
                        if (d != x && d != y) m *= mass1((a >> (D - 1 - d)) & 1, (b >> (D - 1 - d)) & 1);
                    acc[o] += m * s[y * (y - 1) / 2 + x];
                }
        }
    }
#pragma unroll
    for (int o = 0; o < S; o++) B[(int64_t)o * g.N + i] = acc[o];
}

// dst += w K with K the Dirichlet stiffness of the level.  At resolution 1 the reference's
// full-integration stencil table holds only node 0's row (Hat.scalars.inl:261-293: the interior
// case maps to index res/2 = 0 and the upper boundary case is never filled).
template <int D>
__global__ void dirichlet_kernel(int level, double w, double *dst)
{
    constexpr int S = Dims<D>::S;
    Grid<D> g(level);
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= g.N) return;
    if (g.r == 1 && i != 0) return;
    int I[D];
    g.node(i, I);
    const double h = 1. / g.r;
    // The elements shared by nodes I and J form a tensor product of per-axis sets, so
    // int grad phi_I . grad phi_J = sum_k prod_d (k == d ? s_d : m_d) with the per-axis sums of the
    // 1-D stiffness (s_d) and mass (m_d) entries over the shared 1-D elements.
    double sd[D][3], md[D][3];
    for (int d = 0; d < D; d++)
        for (int o = -1; o <= 1; o++)
        {
            int J = I[d] + o;
            double sv = 0, mv = 0;
            if (J >= 0 && J <= g.r)
            {
                int lo = max(max(I[d], J) - 1, 0), hi = min(min(I[d], J), g.r - 1);
                for (int e = lo; e <= hi; e++)
                {
                    int a = I[d] - e, b = J - e;
                    sv += stiff1(a, b) / h;
                    mv += mass1(a, b) * h;
                }
            }
            sd[d][o + 1] = sv;
            md[d][o + 1] = mv;
        }
    for (int o = 0; o < S; o++)
    {
        int off[D];
        stencil_offset<D>(o, off);
        bool ok = true;
        for (int d = 0; d < D; d++)
        {
            int J = I[d] + off[d];
            if (J < 0 || J > g.r) ok = false;
        }
        if (!ok) continue;
        double sum = 0;
        for (int k = 0; k < D; k++)
        {
            double v = 1.;
            for (int d = 0; d < D; d++) v *= (d == k) ? sd[d][off[d] + 1] : md[d][off[d] + 1];
            sum += v;
        }
        dst[(int64_t)o * g.N + i] += w * sum;
    }
}

// Galerkin coarsening P^T M P of a column stencil along one axis (P is a tensor product, so the axes follow
// each other; offsets along the other axes stay what they are).  One thread per node of the coarsened
// grid and offset along the other axes: the 9 entries of the up to three fine nodes 2J + g along the axis,
// weights 1 and 1/2, three entries out.  Memory-bound, and entries far from the samples are zero: a warp
// whose entries all are skips the arithmetic.  13 products per thread and axis, against 27 x 27 x 3 per
// coarse node for all axes at once (depth 8: two stencils 35 ms; on the small levels one thread's chain of
// dependent FP64 sums took 190 us a level).
// inner: nodes after the axis, nin / nout: nodes along it, digit: 3^(axes after it)
__global__ void __launch_bounds__(256) galerkin_axis_kernel(const double *__restrict__ in, double *__restrict__ out, uint32_t totalIn, uint32_t totalOut,
                                                             uint32_t inner, uint32_t nin, uint32_t nout, int digit)
{
    const uint32_t j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= totalOut) return;  // the last block's tail; the rest of the warp votes with the active mask
    const int other = blockIdx.y, hi = other / digit, lo = other - hi * digit;
    const uint32_t t = j / inner, k = j - t * inner, outer = t / nout, J = t - outer * nout;
    const uint32_t at = (outer * nin + 2 * J) * inner + k;
    double v[3][3];  // [fine node g + 1][offset f + 1]
    bool any = false;
#pragma unroll
    for (int g = 0; g < 3; g++)
    {
        const bool ok = g == 1 || (g == 0 ? J > 0 : J + 1 < nout);
#pragma unroll
        for (int f = 0; f < 3; f++)
        {
            const int64_t o = (int64_t)(hi * 3 + f) * digit + lo;
            v[g][f] = ok ? __ldcs(in + o * totalIn + (uint32_t)(at + (g - 1) * (int)inner)) : 0.;
            any = any || v[g][f] != 0.;
        }
    }
    double r[3] = {0., 0., 0.};
    if (__any_sync(__activemask(), any))
    {
        // row weight (1/2 for the outer nodes) times the parent weights of node g + f
        r[0] = 0.5 * v[0][0] + 0.25 * v[0][1] + 0.5 * v[1][0];
        r[1] = 0.25 * v[0][1] + 0.5 * v[0][2] + 0.5 * v[1][0] + v[1][1] + 0.5 * v[1][2] + 0.5 * v[2][0] + 0.25 * v[2][1];
        r[2] = 0.5 * v[1][2] + 0.25 * v[2][1] + 0.5 * v[2][2];
    }
#pragma unroll
    for (int f = 0; f < 3; f++) out[((int64_t)(hi * 3 + f) * digit + lo) * totalOut + j] = r[f];
}

// 3D, resolution >= 2: an entry depends on its offset and, per axis, on whether the node is on the lower
// boundary, inside or on the upper one: 27 classes x 27 offsets, tabulated once per block with
// dirichlet_kernel's own sums (the factors of one axis first, 9 of each kind).
__device__ __forceinline__ void dirichlet_table(int r, double w, double (*table)[27])
{
    constexpr int S = 27;
    __shared__ double stiff[3][3], mass[3][3];
    __shared__ bool inside[3][3];
    const double h = 1. / r;
    if (threadIdx.x < 9)
    {
        const int cd = threadIdx.x / 3, off = threadIdx.x % 3 - 1, I = cd == 0 ? 0 : cd == 2 ? r : 1, J = I + off;
        double sv = 0, mv = 0;
        const int lo = max(max(I, J) - 1, 0), hi = min(min(I, J), r - 1);
        for (int e = lo; e <= hi; e++)
        {
            sv += stiff1(I - e, J - e) / h;
            mv += mass1(I - e, J - e) * h;
        }
        stiff[cd][off + 1] = sv;
        mass[cd][off + 1] = mv;
        inside[cd][off + 1] = J >= 0 && J <= r;
    }
    __syncthreads();
    for (int k = threadIdx.x; k < 27 * S; k += blockDim.x)
    {
        const int cls = k / S, o = k - cls * S;
        const int cd[3] = {cls / 9, (cls / 3) % 3, cls % 3}, od[3] = {o / 9, (o / 3) % 3, o % 3};
        double sum = 0;
#pragma unroll
        for (int q = 0; q < 3; q++)
        {
            double v = 1.;
#pragma unroll
            for (int d = 0; d < 3; d++) v *= d == q ? stiff[cd[d]][od[d]] : mass[cd[d]][od[d]];
            sum += v;
        }
        table[cls][o] = inside[cd[0]][od[0]] && inside[cd[1]][od[1]] && inside[cd[2]][od[2]] ? w * sum : 0.;
    }
    __syncthreads();
}
__device__ __forceinline__ int boundary_class(const int *I, int r)
{
    int cls = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) cls = cls * 3 + (I[d] == 0 ? 0 : I[d] == r ? 2 : 1);
    return cls;
}
// dst += w K, one addition an entry, bound by the two passes over the stencil
__global__ void __launch_bounds__(256) dirichlet3_kernel(int level, double w, double *dst)
{
    __shared__ double table[27][27];
    Grid<3> g(level);
    dirichlet_table(g.r, w, table);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < g.N; i += (int64_t)gridDim.x * blockDim.x)
    {
        int I[3];
        g.node(i, I);
        const int cls = boundary_class(I, g.r);
        double a[27];  // every load before the first store: the compiler cannot know that they do not meet
#pragma unroll
        for (int o = 0; o < 27; o++) a[o] = dst[(int64_t)o * g.N + i];
#pragma unroll
        for (int o = 0; o < 27; o++) dst[(int64_t)o * g.N + i] = a[o] + table[cls][o];
    }
}
// (float)v on the integer pipe: a conversion instruction takes the FP64 pipe's time (64 cycles a warp, against
// some 20 for these), beside a pass over the stencils that the addition above already keeps it busy in.  Round to nearest even by adding half a unit of the
// 29 bits dropped (less one where the kept part is even); results outside float's normal range are converted
// by the instruction.
__device__ __forceinline__ float round_to_float(double v)
{
    const unsigned long long b = (unsigned long long)__double_as_longlong(v), mag = b & 0x7fffffffffffffffull;
    const unsigned int exponent = (unsigned int)(mag >> 52);
    if (mag != 0 && exponent - 897u >= 253u) return (float)v;
    const unsigned long long r = mag + (0x0fffffffull + ((mag >> 29) & 1));
    const unsigned int f = mag == 0 ? 0u : (unsigned int)(r >> 29) - (896u << 23);
    return __uint_as_float(f | ((unsigned int)(b >> 32) & 0x80000000u));
}
template <typename Real>
__device__ __forceinline__ Real rounded(double v)
{
    if constexpr (sizeof(Real) == 4) return round_to_float(v);
    else return v;
}
// A += w K and both stencils into the pair layout, in one pass: a thread per 16-byte vector of a lane of a node,
// the nodes in the natural order and grid.y over a lane's vectors.  No entry is in two vectors, so nothing is
// read twice, and a block follows only a dozen streams through memory; all 27 entries in one thread, 80 streams,
// came to 2.6 TB/s.  Bound by its traffic, 872 bytes a node in float: depth 8 in 3.95 ms (3.7 TB/s),
// against 2.3 ms for the addition and 4.4 ms for a conversion after it that walked each colour's nodes apart.
template <typename Real>
__global__ void __launch_bounds__(256) pair_system_kernel(int level, double w, double *A, const double *B, Real *out)
{
    using PL = PairLayout<Real>;
    constexpr int W = PL::W;
    __shared__ double table[27][27];
    __shared__ uint32_t before[8];  // nodes of the earlier colours
    const Grid<3> g(level);
    const uint32_t half[2] = {(uint32_t)g.r / 2 + 1, ((uint32_t)g.r + 1) / 2};  // nodes of a parity along an axis
    if (threadIdx.x < 8)
    {
        uint32_t n = 0;
        for (int c = 0; c < threadIdx.x; c++) n += half[c & 1] * half[(c >> 1) & 1] * half[(c >> 2) & 1];
        before[threadIdx.x] = n;
    }
    if (w != 0) dirichlet_table(g.r, w, table);
    else __syncthreads();
    const int s = (int)(threadIdx.x & 1), vec = (int)blockIdx.y;
    int off[W], mat[W];
#pragma unroll
    for (int u = 0; u < W; u++) PL::entry(s, vec * W + u, off[u], mat[u]);
    const int64_t step = (int64_t)gridDim.x * (blockDim.x / 2);
    const uint32_t n1 = (uint32_t)g.r + 1;
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 1; i < g.N; i += step)
    {
        double v[W];
#pragma unroll
        for (int u = 0; u < W; u++) v[u] = off[u] < 0 ? 0. : (mat[u] ? B : A)[off[u] * g.N + i];
        // a level has fewer than 2^32 nodes
        const uint32_t row = (uint32_t)i / n1;
        const int I[3] = {(int)(row / n1), (int)(row % n1), (int)((uint32_t)i - row * n1)};
        if (w != 0)
        {
            const double *add = table[boundary_class(I, g.r)];
#pragma unroll
            for (int u = 0; u < W; u++)
                if (off[u] >= 0 && mat[u] == 0)
                {
                    v[u] += add[off[u]];
                    A[off[u] * g.N + i] = v[u];
                }
        }
        Real r[W];
#pragma unroll
        for (int u = 0; u < W; u++)
        {
            // zeros where the neighbour is off the grid
            const int J0 = I[0] + off[u] / 9 - 1, J1 = I[1] + (off[u] / 3) % 3 - 1, J2 = I[2] + off[u] % 3 - 1;
            const bool in = off[u] >= 0 && (uint32_t)J0 < n1 && (uint32_t)J1 < n1 && (uint32_t)J2 < n1;
            r[u] = in ? rounded<Real>(v[u]) : (Real)0;
        }
        const uint32_t h0 = half[I[0] & 1], h1 = half[I[1] & 1], h2 = half[I[2] & 1], n = h0 * h1 * h2;
        const uint32_t j = ((uint32_t)(I[0] >> 1) * h1 + (I[1] >> 1)) * h2 + (I[2] >> 1);
        const int colour = (I[0] & 1) | (I[1] & 1) << 1 | (I[2] & 1) << 2;
        typename PL::Vec *dst = reinterpret_cast<typename PL::Vec *>(out + (int64_t)before[colour] * PL::kNode) + 2 * ((int64_t)n * vec + j) + s;
        if constexpr (W == 4) *dst = make_float4(r[0], r[1], r[2], r[3]);
        else *dst = make_double2(r[0], r[1]);
    }
}

__global__ void scale_by_kernel(double *v, const double *num, double mult, int64_t den)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) v[0] = num[0] * mult / (double)den;
}

template <typename T>
bool dalloc(Context &c, T **p, size_t count, const char *what)
{
    return c.alloc((void **)p, sizeof(T) * count, what);
}

// deterministic device sum of n values (comps==1) or of the Frobenius norms 2 sum v^2 of
// n packed K-vectors (comps==K); result left in *out (device)
bool device_sum(Context &c, const double *v, int64_t n, int comps, double *out)
{
    const int nb = 1024;
    double *partial = nullptr;
    if (!dalloc(c, &partial, nb, "alloc partial")) return false;
    sum_kernel<<<nb, 256, 0, c.stream>>>(v, n, comps, comps, partial);
    sum_finish_kernel<<<1, 32, 0, c.stream>>>(partial, nb, out);
    c.release(partial);
    return c.launch_ok("sum");
}

// Chunked gather of one tree level into grid (NV x W); returns false on a CUDA error.
template <int D, bool Samples, class Item>
bool chunked_level(Context &c, const SplatArgs &a, const Item &item, double scale, double *grid)
{
    constexpr int W = Item::W;
    cudaStream_t s = c.stream;
    int nv = (1 << (a.t - 1)) + 1;
    int64_t NV = 1;
    for (int d = 0; d < D; d++) NV *= nv;
    int *nch = nullptr, *start = nullptr;
    if (!dalloc(c, &nch, NV + 1, "chunks") || !dalloc(c, &start, NV + 1, "chunks")) return false;
    cudaMemsetAsync(nch + NV, 0, sizeof(int), s);
    vertex_chunks_kernel<D, Samples><<<nblocks(NV, 128), 128, 0, s>>>(a, nch);
    {
        size_t tmpBytes = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, tmpBytes, nch, start, (int)(NV + 1), s);
        void *tmp = nullptr;
        if (!c.alloc(&tmp, tmpBytes, "scan tmp")) return false;
        cub::DeviceScan::ExclusiveSum(tmp, tmpBytes, nch, start, (int)(NV + 1), s);
        c.release(tmp);
    }
    int total = 0;
    if (!c.cuda_ok(cudaMemcpyAsync(&total, start + NV, sizeof(int), cudaMemcpyDeviceToHost, s), "copy") ||
        !c.cuda_ok(cudaStreamSynchronize(s), "sync"))
        return false;
    double *partial = nullptr;
    if (total > 0)
    {
        if (!dalloc(c, &partial, (size_t)total * W, "partials")) return false;
        chunk_owner_kernel<<<nblocks(NV, 256), 256, 0, s>>>(start, NV, W, partial);
        chunk_gather_kernel<D, Samples, Item><<<nblocks((int64_t)total * 32, 256), 256, 0, s>>>(a, item, start, total, partial);
    }
    chunk_finish_kernel<W><<<nblocks(NV, 128), 128, 0, s>>>(start, NV, partial, scale, grid);
    c.release(partial);
    c.release(nch);
    c.release(start);
    return c.launch_ok("chunked gather");
}

template <int D>
bool build_impl(Context &c, Setup &st)
{
    constexpr int K = Dims<D>::K;
    constexpr int W = 1 + D + D * D;
    const int depth = c.depth;
    const int64_t n = (int64_t)st.n;
    cudaStream_t s = c.stream;
    st.release_built(c);
    cudaEventRecord(c.ev0, s);

    // ---- ordered sampling: Morton keys of the finest cells, stable radix sort ----
    int64_t *keys = nullptr, *keysSorted = nullptr;
    int *vals = nullptr, *flags = nullptr, *ids = nullptr;
    if (!dalloc(c, &keys, n, "keys") || !dalloc(c, &keysSorted, n, "keys") || !dalloc(c, &vals, n, "vals") ||
        !dalloc(c, &st.order, n, "order") || !dalloc(c, &flags, n, "flags") || !dalloc(c, &ids, n, "ids"))
        return false;
    cell_keys_kernel<D><<<nblocks(n, 256), 256, 0, s>>>(st.pos, n, depth, keys, vals);
    {
        size_t tmpBytes = 0;
        cub::DeviceRadixSort::SortPairs(nullptr, tmpBytes, keys, keysSorted, vals, st.order, (int)n, 0, D * depth, s);
        void *tmp = nullptr;
        if (!c.alloc(&tmp, tmpBytes, "sort tmp")) return false;
        cub::DeviceRadixSort::SortPairs(tmp, tmpBytes, keys, keysSorted, vals, st.order, (int)n, 0, D * depth, s);
        c.release(tmp);
    }
    cell_flags_kernel<<<nblocks(n, 256), 256, 0, s>>>(keysSorted, n, flags);
    {
        size_t tmpBytes = 0;
        cub::DeviceScan::ExclusiveSum(nullptr, tmpBytes, flags, ids, (int)n, s);
        void *tmp = nullptr;
        if (!c.alloc(&tmp, tmpBytes, "scan tmp")) return false;
        cub::DeviceScan::ExclusiveSum(tmp, tmpBytes, flags, ids, (int)n, s);
        c.release(tmp);
    }
    int lastId = 0, lastFlag = 0;
    if (!c.cuda_ok(cudaMemcpyAsync(&lastId, ids + n - 1, sizeof(int), cudaMemcpyDeviceToHost, s), "copy") ||
        !c.cuda_ok(cudaMemcpyAsync(&lastFlag, flags + n - 1, sizeof(int), cudaMemcpyDeviceToHost, s), "copy") ||
        !c.cuda_ok(cudaStreamSynchronize(s), "sync"))
        return false;
    st.ncells = lastId + lastFlag;
    const int64_t nc = st.ncells;
    if (!dalloc(c, &st.cellStart, nc + 1, "cellStart") || !dalloc(c, &st.cellKey, nc, "cellKey")) return false;
    cell_start_kernel<<<nblocks(n, 256), 256, 0, s>>>(keysSorted, flags, ids, n, st.cellStart, st.cellKey);
    c.release(keys); c.release(keysSorted); c.release(vals); c.release(flags); c.release(ids);
    {
        int first = -1, last = -1;
        if (!c.cuda_ok(cudaMemcpyAsync(&first, st.cellStart, sizeof(int), cudaMemcpyDeviceToHost, s), "copy") ||
            !c.cuda_ok(cudaMemcpyAsync(&last, st.cellStart + nc, sizeof(int), cudaMemcpyDeviceToHost, s), "copy") ||
            !c.cuda_ok(cudaStreamSynchronize(s), "sync"))
            return false;
        if (first != 0 || last != (int)n)
        {
            c.fail(EPR_ERR_STATE, "ordered sampling produced inconsistent cell ranges (%d, %d, %lld)", first, last, (long long)n);
            return false;
        }
    }
    Grid<D> gfine(depth);
    if (!dalloc(c, &st.cellOfFinest, gfine.NE, "cell map")) return false;
    cudaMemsetAsync(st.cellOfFinest, 0xff, sizeof(int) * gfine.NE, s);
    finest_map_kernel<D><<<nblocks(nc, 256), 256, 0, s>>>(st.cellKey, nc, depth, st.cellOfFinest);
    if (!c.launch_ok("ordered sampling")) return false;

    // ---- tree structure of both trees ----
    auto buildRefined = [&](std::vector<uint8_t *> &ref, int KR) -> bool {
        ref.assign(depth + 2, nullptr);
        for (int t = 1; t <= depth; t++)
        {
            int64_t cells = 1;
            for (int d = 0; d < D; d++) cells *= (int64_t)1 << t;
            if (!dalloc(c, &ref[t], cells, "refined")) return false;
            cudaMemsetAsync(ref[t], 0, cells, s);
            refine_kernel<D><<<nblocks(nc, 256), 256, 0, s>>>(st.cellKey, nc, depth, t, KR, t > 1 ? ref[t - 1] : nullptr, ref[t]);
        }
        return c.launch_ok("refine");
    };
    if (!buildRefined(st.refinedD, c.P.d_radius)) return false;
    if (!buildRefined(st.refinedS, c.P.t_radius)) return false;

    // ---- occupied-cell ranges of every depth-t cell (shared by both trees) ----
    std::vector<int *> rlo(depth + 2, nullptr), rhi(depth + 2, nullptr);
    for (int t = 1; t <= depth + 1; t++)
    {
        int64_t cells = (int64_t)1 << (D * (t - 1));
        if (!dalloc(c, &rlo[t], cells, "ranges") || !dalloc(c, &rhi[t], cells, "ranges")) return false;
        cudaMemsetAsync(rlo[t], 0, sizeof(int) * cells, s);
        cudaMemsetAsync(rhi[t], 0, sizeof(int) * cells, s);
        level_ranges_kernel<D><<<nblocks(nc, 256), 256, 0, s>>>(st.cellKey, nc, t, D * (depth + 1 - t), rlo[t], rhi[t]);
    }
    if (!c.launch_ok("level ranges")) return false;

    // ---- density splat of the merged cells ----
    double *mean = nullptr, *datum = nullptr;
    if (!dalloc(c, &mean, nc * D, "mean") || !dalloc(c, &datum, nc * W, "datum")) return false;
    merge_cells_kernel<D><<<nblocks(nc, 128), 128, 0, s>>>(st.pos, st.order, st.cellStart, nc, mean, datum);
    st.density.assign(depth + 1, nullptr);
    {
        int KR = c.P.d_radius;
        std::vector<double> bsv(2 * KR + 2);
        {
            // B-spline value at 1/2 of the centre piece (GridSamples.inl:753-756), on the host
            int deg = 2 * KR + 1;
            std::vector<double> v(deg + 1);
            v[deg] = 1.;
            for (int k = 1; k <= deg; k++)
            {
                const double scale = 1. / k;
                int b = deg - k;
                v[b] = v[b + 1] * (1. - 0.5) * scale;
                for (int i = 1; i < k; i++) v[b + i] = (v[b + i] * (0.5 - i + k) + v[b + i + 1] * (-0.5 + i + 1)) * scale;
                v[b + k] *= 0.5 * scale;
            }
            bsv = v;
        }
        double scale = std::pow(1. / bsv[KR + 1], 2);
        double *bs = nullptr;
        if (!dalloc(c, &bs, (size_t)nc * D * (2 * KR + 2), "bspline table")) return false;
        for (int t = 1; t <= depth + 1; t++)
        {
            Grid<D> gl(t - 1);
            if (!dalloc(c, &st.density[t - 1], gl.N * W, "density")) return false;
            SplatArgs a{st.cellKey, st.cellStart, nc, depth, t, KR, rlo[t], rhi[t]};
            double dw = scale / std::pow(std::pow(0.5, t - 1), D - 2);
            item_bspline_kernel<D><<<nblocks(nc, 256), 256, 0, s>>>(mean, nullptr, nc, t, 2 * KR + 1, nullptr, bs);
            DensityItem<D> item{bs, datum, dw};
            if (!chunked_level<D, false>(c, a, item, 1.0, st.density[t - 1])) return false;
        }
        c.release(bs);
    }
    c.release(mean); c.release(datum);
    if (!c.launch_ok("density splat")) return false;

    // ---- estimator queries per sample ----
    if (!dalloc(c, &st.measure, n, "measure") || !dalloc(c, &st.noise, n, "noise") || !dalloc(c, &st.sdepth, n, "depth")) return false;
    {
        DensityGrids<D> G;
        for (int l = 0; l <= depth; l++) G.g[l] = st.density[l];
        G.depth = depth;
        estimator_kernel<D><<<nblocks(n, 128), 128, 0, s>>>(G, st.pos, st.order, n, st.measure, st.noise, st.sdepth);
    }
    if (!c.launch_ok("estimator")) return false;

    // ---- frame splat ----
    st.skewGrid.assign(depth + 1, nullptr);
    {
        const int TR = c.P.t_radius;
        double *bs = nullptr, *lw = nullptr, *frame = nullptr;
        if (!dalloc(c, &bs, (size_t)n * D * (2 * TR + 2), "bspline table") || !dalloc(c, &lw, n, "level weights") ||
            !dalloc(c, &frame, (size_t)n * K, "frames"))
            return false;
        skew_frame_kernel<D><<<nblocks(n, 256), 256, 0, s>>>(st.skew, st.measure, st.order, n, depth, frame);
        for (int t = 1; t <= depth + 1; t++)
        {
            Grid<D> gl(t - 1);
            if (!dalloc(c, &st.skewGrid[t - 1], gl.N * K, "skew grid")) return false;
            SplatArgs a{st.cellKey, st.cellStart, nc, depth, t, TR, rlo[t], rhi[t]};
            skew_level_kernel<<<nblocks(n, 256), 256, 0, s>>>(st.sdepth, st.order, n, t, depth, D, lw);
            item_bspline_kernel<D><<<nblocks(n, 256), 256, 0, s>>>(st.pos, st.order, n, t, 2 * TR + 1, lw, bs);
            SkewItem<D> item{bs, lw, frame};
            if (!chunked_level<D, true>(c, a, item, std::pow(std::pow(0.5, depth), 1.5 * 2), st.skewGrid[t - 1])) return false;
        }
        c.release(bs); c.release(lw); c.release(frame);
    }
    if (!c.launch_ok("frame splat")) return false;

    for (int t = 1; t <= depth + 1; t++) { c.release(rlo[t]); c.release(rhi[t]); }

    // ---- S(E), leaf depths, c ----
    if (!dalloc(c, &st.S, gfine.NE * K, "S") || !dalloc(c, &st.leaf, gfine.NE, "leaf")) return false;
    {
        SkewGrids<D> G;
        G.g[0] = st.skewGrid[0];
        // the sums in the finest B, which is written in full below; what was built before ends here
        c.have_system = false;
        double *sums = c.levels[depth].B64;
        for (int l = 1; l <= depth; l++)
        {
            Grid<D> gl(l);
            accumulate_frames_kernel<D><<<nblocks(gl.N, 256), 256, 0, s>>>(l, st.skewGrid[l], G.g[l - 1], sums);
            G.g[l] = sums;
            sums += gl.N * K;
        }
        for (int t = 0; t <= depth + 1 && t < 12; t++) G.refined[t] = st.refinedS[t];
        G.depth = depth;
        element_frame_kernel<D><<<nblocks(gfine.NE, 128), 128, 0, s>>>(G, st.S, st.leaf, c.P.project);
    }
    // the adaptive indexer: its tables, and the frame field restricted to its elements for c and B
    const double *Sfit = st.S;
    double *Smasked = nullptr;
    if (c.P.adaptive_radius >= 0)
    {
        if (!build_adaptive(c, st.cellOfFinest) || !masked_frames(c, st.S, gfine.NE, K, &Smasked)) return false;
        Sfit = Smasked;
    }
    else c.release_adaptive();
    double *dsum = nullptr;
    if (!dalloc(c, &dsum, 4, "sums")) return false;
    if (!device_sum(c, Sfit, gfine.NE, K, dsum)) return false;
    double csum = 0;
    if (!c.cuda_ok(cudaMemcpyAsync(&csum, dsum, sizeof(double), cudaMemcpyDeviceToHost, s), "copy") ||
        !c.cuda_ok(cudaStreamSynchronize(s), "sync"))
        return false;
    c.c = csum / (double)gfine.NE;

    // ---- finest stencils: R (into A64), B ----
    Level &Lf = c.levels[depth];
    const int S = Dims<D>::S;
    cudaMemsetAsync(Lf.A64, 0, sizeof(double) * S * Lf.N, s);
    if (c.P.s_weight > 0)
    {
        if (!device_sum(c, st.measure, n, 1, dsum + 1)) return false;
        scale_by_kernel<<<1, 32, 0, s>>>(dsum + 2, dsum + 1, c.P.s_weight, n);
        // in the finest B too, where it holds them (fewer occupied cells than 0.75 (0.59 in 4D) times the nodes)
        double *own = nullptr, *mass = Lf.B64;
        if (nc * CellPairs<D>::N > S * Lf.N)
        {
            if (!dalloc(c, &own, (size_t)nc * CellPairs<D>::N, "cell masses")) return false;
            mass = own;
        }
        cell_mass_kernel<D><<<nblocks(nc, 4), 128, 0, s>>>(st.pos, st.noise, st.order, st.cellStart, st.cellKey, nc, depth, c.P.n_sigma, mass);
        screening_kernel<D><<<nblocks(Lf.N, 128), 128, 0, s>>>(mass, st.cellOfFinest, depth, dsum + 2, Lf.A64);
        c.release(own);
    }
    constraint_kernel<D><<<nblocks(Lf.N, 128), 128, 0, s>>>(Sfit, depth, Lf.B64);
    c.release(Smasked);
    if (!c.launch_ok("finest stencils")) return false;

    // ---- Galerkin hierarchy of R and B, then A = R + dWeight K on every level ----
    {
        // scratch: the finest level's colour blocks, which are written below, where it has any
        for (int l = 0; l <= depth; l++)
            if (!c.ensure_blocks(l)) return false;
        const size_t need = galerkin_scratch<D>(depth);
        double *own = nullptr, *scratch = (double *)Lf.Acb;
        if (c.block_bytes(depth) < need * sizeof(double))
        {
            if (!dalloc(c, &own, need, "galerkin scratch")) return false;
            scratch = own;
        }
        else Lf.synced = false;
        for (int l = depth; l > 0; l--)
        {
            launch_galerkin<D>(l, c.levels[l].A64, c.levels[l - 1].A64, scratch, s);
            launch_galerkin<D>(l, c.levels[l].B64, c.levels[l - 1].B64, scratch, s);
        }
        c.release(own);
    }
    if (!c.launch_ok("galerkin")) return false;
    for (int l = 0; l <= depth; l++)
    {
        if (D == 3 && pair_level<3>(l))
        {
            if (!pair_system(c, l, c.P.d_weight)) return false;
            continue;
        }
        if (!add_dirichlet(c, l)) return false;
        if (!c.sync_system32(l)) return false;
    }
    c.release(dsum);
    cudaEventRecord(c.ev1, s);
    if (!c.cuda_ok(cudaStreamSynchronize(s), "build sync")) return false;
    float ms = 0;
    cudaEventElapsedTime(&ms, c.ev0, c.ev1);
    c.stats.build_ms = ms;
    c.have_system = true;
    return true;
}

}  // namespace

bool add_dirichlet_to(Context &c, int level, double *dst, double w)
{
    int64_t N = c.levels[level].N;
    if (c.dim == 3 && level > 0) dirichlet3_kernel<<<std::min(nblocks(N, 256), 2u * 152u), 256, 0, c.stream>>>(level, w, dst);
    else if (c.dim == 3) dirichlet_kernel<3><<<nblocks(N, 128), 128, 0, c.stream>>>(level, w, dst);
    else dirichlet_kernel<4><<<nblocks(N, 128), 128, 0, c.stream>>>(level, w, dst);
    return c.launch_ok("dirichlet");
}

bool pair_system(Context &c, int level, double w)
{
    Level &L = c.levels[level];
    const unsigned int blocks = std::min(nblocks(2 * L.N, 256), 8u * 152u);
    if (c.lvl32(level))
        pair_system_kernel<float><<<dim3(blocks, PairLayout<float>::G), 256, 0, c.stream>>>(level, w, L.A64, L.B64, (float *)L.Acb);
    else
        pair_system_kernel<double><<<dim3(blocks, PairLayout<double>::G), 256, 0, c.stream>>>(level, w, L.A64, L.B64, (double *)L.Acb);
    return L.synced = c.launch_ok("pair layout");
}

bool add_dirichlet(Context &c, int level) { return add_dirichlet_to(c, level, c.levels[level].A64, c.P.d_weight); }

bool Setup::set_samples(Context &c, size_t n_, const double *pos_, const double *skew_)
{
    release(c);
    n = n_;
    size_t K = (size_t)(c.dim * (c.dim - 1) / 2);
    if (!dalloc(c, &pos, n * c.dim, "pos") || !dalloc(c, &skew, n * K, "skew")) return false;
    return c.cuda_ok(cudaMemcpyAsync(pos, pos_, sizeof(double) * n * c.dim, cudaMemcpyHostToDevice, c.stream), "upload pos") &&
           c.cuda_ok(cudaMemcpyAsync(skew, skew_, sizeof(double) * n * K, cudaMemcpyHostToDevice, c.stream), "upload skew") &&
           c.cuda_ok(cudaStreamSynchronize(c.stream), "sync");
}

bool Setup::build(Context &c)
{
    if (c.dim == 3) return build_impl<3>(c, *this);
    return build_impl<4>(c, *this);
}

bool Setup::get(Context &c, const std::string &name, double *out, size_t cap, size_t *count)
{
    auto copy_d = [&](const double *src, size_t num) -> bool {
        if (count) *count = num;
        if (!out) return true;
        if (!src) { c.fail(EPR_ERR_STATE, "'%s' is not available before epr_build", name.c_str()); return false; }
        if (cap < num) { c.fail(EPR_ERR_ARG, "output too small (%zu < %zu)", cap, num); return false; }
        populate(out, sizeof(double) * num);
        return c.cuda_ok(cudaMemcpyAsync(out, src, sizeof(double) * num, cudaMemcpyDeviceToHost, c.stream), "copy") &&
               c.cuda_ok(cudaStreamSynchronize(c.stream), "sync");
    };
    size_t K = (size_t)(c.dim * (c.dim - 1) / 2);
    int64_t NE = 1;
    for (int d = 0; d < c.dim; d++) NE *= (int64_t)1 << c.depth;
    if (name == "measure") return copy_d(measure, n);
    if (name == "noise") return copy_d(noise, n);
    if (name == "depth") return copy_d(sdepth, n);
    if (name == "S") return copy_d(S, (size_t)NE * K);
    if (name == "leaf_depth")
    {
        if (count) *count = (size_t)NE;
        if (!out) return true;
        if (!leaf) { c.fail(EPR_ERR_STATE, "not built"); return false; }
        if (cap < (size_t)NE) { c.fail(EPR_ERR_ARG, "output too small"); return false; }
        std::vector<int> h(NE);
        if (!c.cuda_ok(cudaMemcpyAsync(h.data(), leaf, sizeof(int) * NE, cudaMemcpyDeviceToHost, c.stream), "copy") ||
            !c.cuda_ok(cudaStreamSynchronize(c.stream), "sync"))
            return false;
        for (int64_t e = 0; e < NE; e++) out[e] = h[e];
        return true;
    }
    if (name == "ncells")
    {
        if (count) *count = 1;
        if (out && cap >= 1) out[0] = (double)ncells;
        return true;
    }
    c.fail(EPR_ERR_ARG, "unknown array '%s'", name.c_str());
    return false;
}

// Galerkin coarsening of any column stencil (also for the linear multigrid of epr_mg.cu)
template <int D>
size_t galerkin_scratch(int fineLevel)
{
    // the grids with one and two axes coarsened
    size_t n = (size_t)((1 << fineLevel) + 1), c = (size_t)((1 << (fineLevel - 1)) + 1), first = c, second = c * c;
    for (int d = 1; d < D; d++) first *= n;
    for (int d = 2; d < D; d++) second *= n;
    return (size_t)Dims<D>::S * (first + second);
}
template <int D>
void launch_galerkin(int fineLevel, const double *Mf, double *Mc, double *scratch, cudaStream_t s)
{
    uint32_t ext[D];
    for (int d = 0; d < D; d++) ext[d] = (1u << fineLevel) + 1;
    auto total = [&]() { uint32_t t = 1; for (int d = 0; d < D; d++) t *= ext[d]; return t; };
    const double *in = Mf;
    double *buf[2] = {scratch, nullptr};
    uint32_t inner = 1;
    int digit = 1;
    for (int d = D - 1; d >= 0; d--)
    {
        const uint32_t nin = ext[d], totalIn = total();
        ext[d] = (nin - 1) / 2 + 1;
        const uint32_t totalOut = total();
        if (d == D - 1) buf[1] = scratch + (size_t)Dims<D>::S * totalOut;
        double *out = d == 0 ? Mc : buf[(D - 1 - d) & 1];
        galerkin_axis_kernel<<<dim3(nblocks(totalOut, 256), Dims<D>::S / 3), 256, 0, s>>>(in, out, totalIn, totalOut, inner, nin, ext[d], digit);
        in = out;
        inner *= ext[d];
        digit *= 3;
    }
}
template size_t galerkin_scratch<3>(int);
template size_t galerkin_scratch<4>(int);
template void launch_galerkin<3>(int, const double *, double *, double *, cudaStream_t);
template void launch_galerkin<4>(int, const double *, double *, double *, cudaStream_t);

// the products of a build (everything but the samples), so that a context can be built again
void Setup::release_built(Context &c)
{
    c.release(order); c.release(cellKey); c.release(cellStart); c.release(cellOfFinest);
    c.release(measure); c.release(noise); c.release(sdepth); c.release(S); c.release(leaf);
    for (double *p : density) c.release(p);
    for (double *p : skewGrid) c.release(p);
    for (uint8_t *p : refinedD) c.release(p);
    for (uint8_t *p : refinedS) c.release(p);
    density.clear(); skewGrid.clear(); refinedD.clear(); refinedS.clear();
    measure = noise = sdepth = S = nullptr;
    order = cellStart = cellOfFinest = leaf = nullptr;
    cellKey = nullptr;
    ncells = 0;
}

void Setup::release(Context &c)
{
    release_built(c);
    c.release(pos); c.release(skew);
    pos = skew = nullptr;
    n = 0;
}

}  // namespace epr
