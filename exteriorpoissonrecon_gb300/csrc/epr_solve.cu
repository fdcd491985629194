// Solve-path kernels: energy, quadratic fit, paired Gauss-Seidel colour sweep, Gauss-Newton
// matvec, prolongation / restriction.  Templated on the dimension (3, 4) and the arithmetic type
// (double for the parity path, float for the fast path).
//
// Reference correspondence:
//   energy        SingleCycleCascadicSystemEnergy::energies          SystemEnergy.h:486-497
//   node fit      SingleCycleCascadicSystemEnergy::quadraticFit      SystemEnergy.h:542-643
//   GS colour     PairedGaussSeidelSolve (one parity colour)         ExteriorPoissonSolvers.h:156-196
//   prolongation  ScalarFunctions::prolongation                      Hat.scalars.inl:1747-1779
//   restriction   its transpose (the Galerkin restriction of MG.h:120-127)
#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <type_traits>

#include "epr_common.cuh"
#include "epr_element.cuh"
#include "epr_kernels.h"
#include "epr_step.cuh"

namespace epr {

namespace {

constexpr int kThreads = 128;

// r^(4-D)/2: scale from reference-element sums to physical integrals
template <int D, typename Real>
__device__ __forceinline__ Real wedge_scale(int r)
{
    return (D == 3 ? (Real)r : (Real)1) * (Real)0.5;
}

// entry k of a level's stencils (A, B) in the level's arithmetic
template <typename Real>
__device__ __forceinline__ Real stencil_a(const LevelPtrs<Real> &L, int64_t k) { return L.A ? L.A[k] : (Real)L.A64[k]; }
template <typename Real>
__device__ __forceinline__ Real stencil_b(const LevelPtrs<Real> &L, int64_t k) { return L.B ? L.B[k] : (Real)L.B64[k]; }

template <int D>
struct NodeCtx
{
    int I[D];
    int64_t stride[D];
};

// Wedge part of the quadratic model of node i, elements in canonical orientation.
template <int D, typename Real>
__device__ __forceinline__ void node_wedge_fit(const Grid<D> &g, const NodeCtx<D> &nc, int64_t i, const Real *xy, Real *h)
{
    FitSums<D, Real> sums;
    sums.clear();
    const Real2<Real> own = ld2(xy, i);
#pragma unroll 1
    for (int A = 0; A < (1 << D); A++)
    {
        bool ok = true;
        int64_t sd[D];
#pragma unroll
        for (int d = 0; d < D; d++)
        {
            const int e = nc.I[d] - cbit<D>(A, d);
            ok = ok && e >= 0 && e < g.r;
            sd[d] = cbit<D>(A, d) ? -nc.stride[d] : nc.stride[d];
        }
        if (!ok) continue;
        Real2<Real> df[1 << D];
        df[0] = own;
#pragma unroll
        for (int cc = 1; cc < (1 << D); cc++)
        {
            int64_t j = i;
#pragma unroll
            for (int d = 0; d < D; d++)
                if (cbit<D>(cc, d)) j += sd[d];
            df[cc] = Ops<Real>::sub(ld2(xy, j), own);
        }
        element_fit_sums<Real>(df, sums);
    }
    sums.add_to(h);
}

// Quadratic model of E(x + s e_i, y + t e_i): q = (Q20, Q02, Q11, Q10, Q01)
template <int D, typename Real>
__device__ __forceinline__ void node_fit(const LevelPtrs<Real> &L, const Grid<D> &g, const NodeCtx<D> &nc, int64_t i,
                                         const Real *xy, Real *q)
{
    Real h[5] = {0, 0, 0, 0, 0};
    node_wedge_fit<D, Real>(g, nc, i, xy, h);
    const Real sc = wedge_scale<D, Real>(g.r);
    q[0] = h[0] * sc;
    q[1] = h[1] * sc;
    q[2] = (Real)2 * h[2] * sc;
    q[3] = (Real)2 * h[3] * sc;
    q[4] = (Real)2 * h[4] * sc;
    // screening + Dirichlet (A column) and frame constraint (B column, without its diagonal)
    constexpr int S = Dims<D>::S;
    Real ax = 0, ay = 0, bx = 0, by = 0, acen = 0;
#pragma unroll 3
    for (int o = 0; o < S; o++)
    {
        int off[D];
        stencil_offset<D>(o, off);
        bool ok = true;
        int64_t j = i;
#pragma unroll
        for (int d = 0; d < D; d++)
        {
            int t = nc.I[d] + off[d];
            ok = ok && (t >= 0) && (t <= g.r);
            j += (int64_t)off[d] * nc.stride[d];
        }
        if (!ok) continue;
        Real a = stencil_a(L, (int64_t)o * L.N + i);
        Real b = stencil_b(L, (int64_t)o * L.N + i);
        Real2<Real> v = ld2(xy, j);
        ax += a * v.x;
        ay += a * v.y;
        if (o == Dims<D>::CENTER) acen = a;
        else { bx += b * v.x; by += b * v.y; }
    }
    q[0] += acen;
    q[1] += acen;
    q[3] += (Real)2 * ax - (Real)2 * by;
    q[4] += (Real)2 * ay + (Real)2 * bx;
}

template <int D>
__device__ __forceinline__ void make_ctx(const Grid<D> &g, int64_t i, NodeCtx<D> &nc)
{
    g.node(i, nc.I);
#pragma unroll
    for (int d = 0; d < D; d++) nc.stride[d] = g.stride(d);
}

// ---------------------------------------------------------------------------------------------
// deterministic block reduction of up to 3 doubles
// ---------------------------------------------------------------------------------------------
__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

template <int NV>
__device__ __forceinline__ void block_sum_store(double *v, double *dst)
{
    __shared__ double sh[NV][32];
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int k = 0; k < NV; k++)
    {
        double t = warp_sum(v[k]);
        if (lane == 0) sh[k][w] = t;
    }
    __syncthreads();
    if (w == 0)
    {
        int nw = (blockDim.x + 31) >> 5;
#pragma unroll
        for (int k = 0; k < NV; k++)
        {
            double t = lane < nw ? sh[k][lane] : 0.0;
            t = warp_sum(t);
            if (lane == 0) dst[k] = t;
        }
    }
}

// Natural: the level keeps its stencils in Real, so that no load asks (12 to 14 % of the float kernel)
template <int D, typename Real, bool Natural>
__global__ void __launch_bounds__(kThreads) energy_kernel(LevelPtrs<Real> L, const Real *xy, double *partial)
{
    Grid<D> g(L.level);
    double acc[3] = {0, 0, 0};
    const int64_t total = g.N > g.NE ? g.N : g.NE;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x)
    {
        if (t < g.NE)
        {
            int E[D];
            g.elem(t, E);
            Real2<Real> f[1 << D];
            int64_t base = 0;
#pragma unroll
            for (int d = 0; d < D; d++) base = base * (g.r + 1) + E[d];
#pragma unroll
            for (int c = 0; c < (1 << D); c++)
            {
                int64_t j = base;
#pragma unroll
                for (int d = 0; d < D; d++) j += cbit<D>(c, d) * g.stride(d);
                f[c] = ld2(xy, j);
            }
            acc[0] += (double)element_wedge<D, Real>(f);
        }
        if (t < g.N)
        {
            NodeCtx<D> nc;
            make_ctx<D>(g, t, nc);
            Real2<Real> me = ld2(xy, t);
            double by = 0, ax = 0, ay = 0;
            constexpr int S = Dims<D>::S;
            for (int o = 0; o < S; o++)
            {
                int off[D];
                stencil_offset<D>(o, off);
                bool ok = true;
                int64_t j = t;
#pragma unroll
                for (int d = 0; d < D; d++)
                {
                    int q = nc.I[d] + off[d];
                    ok = ok && (q >= 0) && (q <= g.r);
                    j += (int64_t)off[d] * nc.stride[d];
                }
                if (!ok) continue;
                Real2<Real> v = ld2(xy, j);
                const int64_t k = (int64_t)o * L.N + t;
                const double a = (double)(Natural ? L.A[k] : (Real)L.A64[k]), b = (double)(Natural ? L.B[k] : (Real)L.B64[k]);
                by += b * (double)v.y;
                ax += a * (double)v.x;
                ay += a * (double)v.y;
            }
            acc[1] += (double)me.x * by;
            acc[2] += (double)me.x * ax + (double)me.y * ay;
        }
    }
    block_sum_store<3>(acc, partial + 4 * blockIdx.x);
}

__global__ void finish_kernel(const double *partial, int nblocks, int nv, double *out, double scale0)
{
    // one warp per value, fixed order
    int v = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (v >= nv) return;
    double s = 0;
    for (int b = lane; b < nblocks; b += 32) s += partial[4 * b + v];
    s = warp_sum(s);
    if (lane == 0) out[v] = (v == 0) ? s * scale0 : s;
}

template <int D, typename Real>
__global__ void __launch_bounds__(kThreads) quadfit_kernel(LevelPtrs<Real> L, const Real *xy, double *out)
{
    Grid<D> g(L.level);
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= g.N) return;
    NodeCtx<D> nc;
    make_ctx<D>(g, i, nc);
    Real q[5];
    node_fit<D, Real>(L, g, nc, i, xy, q);
#pragma unroll
    for (int k = 0; k < 5; k++) out[i * 5 + k] = (double)q[k];
}

// sum over the nodes of |dE/dx_i|^2 + |dE/dy_i|^2 (the linear coefficients of the node fits)
template <int D, typename Real>
__global__ void __launch_bounds__(kThreads) grad_norm_kernel(LevelPtrs<Real> L, const Real *xy, double *partial)
{
    Grid<D> g(L.level);
    double acc[1] = {0};
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < g.N; i += (int64_t)gridDim.x * blockDim.x)
    {
        NodeCtx<D> nc;
        make_ctx<D>(g, i, nc);
        Real q[5];
        node_fit<D, Real>(L, g, nc, i, xy, q);
        acc[0] += (double)q[3] * (double)q[3] + (double)q[4] * (double)q[4];
    }
    block_sum_store<1>(acc, partial + 4 * blockIdx.x);
}

// Lane-parallel variant: a group of 2^D consecutive lanes updates one node, lane A integrating the
// node's element A (canonical orientation) and a share of its stencil column; the group reduces
// with shuffles in a fixed order and its first lane writes the update.
template <int D>
__device__ __forceinline__ float group_sum(float v)
{
#pragma unroll
    for (int o = (1 << D) / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, 1 << D);
    return v;
}
template <int D>
__device__ __forceinline__ double group_sum(double v)
{
#pragma unroll
    for (int o = (1 << D) / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, 1 << D);
    return v;
}
// The float kernels fit a sheared pair: (x, y - a x), or (x - b y, y) where y varies more than x, with one
// factor of at most 1 per node, from the products of the differences along the axes.  W is the same for
// the sheared pair, and with the step (s + b t, t + a s) the model's Hessian keeps its determinant, so any
// factor gives the same update in exact arithmetic.  Where the fields' gradients at the node are nearly
// parallel, |U|^2, |V|^2 and <U, V> of the plain pair agree to most of float's digits in the determinant and
// their rounding becomes the update's largest error; the sheared field's term is small instead.  (Eight
// random systems on level 6, one sweep against 64 bits, relative L2: up to 1e-5 with the plain pair, up to
// 5e-7 with the shear.)  Double (1e-14 off there) and double-float relax the plain pair.
template <typename Real>
constexpr bool shears() { return std::is_same<Real, float>::value; }

template <typename Real>
struct Shear
{
    Real a, b;  // one of them 0
};
__device__ __forceinline__ Shear<float> shear_of(float sxy, float sxx, float syy)
{
    const bool y = sxx >= syy;
    float f = __fdividef(sxy, y ? sxx : syy);
    f = fabsf(f) <= 2.f ? f : 0.f;  // also where the ratio is not finite
    return Shear<float>{y ? f : 0.f, y ? 0.f : f};
}
template <typename Real>
__device__ __forceinline__ Real2<Real> sheared(const Shear<Real> &sh, const Real2<Real> &v)
{
    return Real2<Real>{Ops<Real>::fma(-sh.b, v.y, v.x), Ops<Real>::fma(-sh.a, v.x, v.y)};
}

// q = (Q20, Q02, Q11, Q10, Q01) of the (sheared) pair from a node's wedge sums and its stencil columns:
// av = sum A_j (x, y)_j, bv = sum B_j (x, y)_j without the centre, acen the centre of A.  Linear in all
// of them, so lanes that share a node add their parts of q.
template <int D, typename Real>
__device__ __forceinline__ void fit_to_model(const FitSums<D, Real> &sums, Real sc, const Real2<Real> &av, const Real2<Real> &bv,
                                             Real acen, const Shear<Real> &sh, Real *q)
{
    using O = Ops<Real>;
    Real h[5] = {(Real)0, (Real)0, (Real)0, (Real)0, (Real)0};
    sums.add_to(h);
    const Real sc2 = O::add(sc, sc);
    const Real gx = O::mul((Real)2, O::sub(av.x, bv.y)), gy = O::mul((Real)2, O::add(av.y, bv.x));
    if constexpr (shears<Real>())
    {
        const Real aa = O::mul(sh.a, acen), ab = O::mul(sh.b, acen);
        q[0] = O::fma(h[0], sc, O::fma(sh.a, aa, acen));
        q[1] = O::fma(h[1], sc, O::fma(sh.b, ab, acen));
        q[2] = O::fma(h[2], sc2, O::mul((Real)2, O::add(aa, ab)));
        q[3] = O::fma(h[3], sc2, O::fma(sh.a, gy, gx));
        q[4] = O::fma(h[4], sc2, O::fma(sh.b, gx, gy));
    }
    else
    {
        q[0] = O::fma(h[0], sc, acen);
        q[1] = O::fma(h[1], sc, acen);
        q[2] = O::mul(h[2], sc2);
        q[3] = O::fma(h[3], sc2, gx);
        q[4] = O::fma(h[4], sc2, gy);
    }
}

// the step of node i from its whole model, by one thread
template <typename Real>
__device__ __forceinline__ void apply_step(const LevelPtrs<Real> &L, Real *xy, int64_t i, const Real *q, const Shear<Real> &sh, int separate,
                                           unsigned int *err)
{
    Real p0, p1;
    if (relaxed(L, i) && node_step<Real>(q, separate, p0, p1))
    {
        if constexpr (shears<Real>())
        {
            const Real s = p0;
            p0 = Ops<Real>::fma(sh.b, p1, p0);
            p1 = Ops<Real>::fma(sh.a, s, p1);
        }
        Real2<Real> v = ld2(xy, i);
        v.x += p0;
        v.y += p1;
        if (!finite_value<Real>(v.x) || !finite_value<Real>(v.y)) atomicOr(err, (unsigned int)ERR_NONFINITE);
        reinterpret_cast<Real2<Real> *>(xy)[i] = v;
    }
}

// Lane A's part of the update of the node at I: the fit of the node's element A and the stencil
// offsets that lane owns.  An offset's neighbour is a corner of every element on its side, and the
// lane owns it whose element lies on the lower-numbered existing side of every axis the offset does
// not move along; so each neighbour is one of the corners already in the lane's registers.
// Ac, Bc (optional): the colour's block of the colour-blocked stencils, the node being the colour's
// jc-th of nc; otherwise the natural stencils L.A, L.B are read.
// Chained: the caller is a colour's kernel, which may start before the colour ahead of it is done.
template <int D, typename Real, bool Chained = false>
__device__ __forceinline__ void gs_update_lanes_at(const LevelPtrs<Real> &L, Real *xy, const Grid<D> &g, const int *I, bool active,
                                                   int A, unsigned int *err, int separate = 0, const Real *Ac = nullptr,
                                                   const Real *Bc = nullptr, int64_t jc = 0, int64_t nc = 0)
{
    using O = Ops<Real>;
    using V = Real2<Real>;
    constexpr int C = 1 << D;
    int64_t i = 0;
    Real q[5] = {(Real)0, (Real)0, (Real)0, (Real)0, (Real)0};
    V f[C], av = {(Real)0, (Real)0}, bv = {(Real)0, (Real)0};
    Real ca[C], cb[C];
    Real acen = (Real)0, sxy = (Real)0, sxx = (Real)0, syy = (Real)0;
    Shear<Real> sh = {(Real)0, (Real)0};
    // node indices in 32 bits (every supported grid has < 2^32 nodes); signed strides of the
    // element mirrored so that the node is its corner 0
    int jj[C], other = 0;
    uint32_t iu = 0;
    bool ok = active;
    if (active)
    {
        int st[D], sd[D];
        st[D - 1] = 1;
#pragma unroll
        for (int d = D - 2; d >= 0; d--) st[d] = st[d + 1] * (g.r + 1);
        int first = 0;  // the lower-numbered existing side of every axis, as corner bits
#pragma unroll
        for (int d = 0; d < D; d++)
        {
            iu += (uint32_t)I[d] * (uint32_t)st[d];
            sd[d] = cbit<D>(A, d) ? -st[d] : st[d];
            const int e = I[d] - cbit<D>(A, d);
            ok = ok && e >= 0 && e < g.r;
            if (I[d] >= g.r) first |= 1 << (D - 1 - d);
        }
        i = iu;
        other = A ^ first;
        if (ok)
        {
#pragma unroll
            for (int cc = 0; cc < C; cc++)
            {
                jj[cc] = (int)iu;
#pragma unroll
                for (int d = 0; d < D; d++)
                    if (cbit<D>(cc, d)) jj[cc] += sd[d];
            }
            const int64_t step = Ac ? nc : L.N;
            const Real *pA = (Ac ? Ac + jc : L.A + i) + (int64_t)Dims<D>::CENTER * step;
            const Real *pB = (Ac ? Bc + jc : L.B + i) + (int64_t)Dims<D>::CENTER * step;
            int64_t so[D];
#pragma unroll
            for (int d = 0; d < D; d++) so[d] = cbit<D>(A, d) ? -(int64_t)ipow(3, D - 1 - d) * step : (int64_t)ipow(3, D - 1 - d) * step;
#pragma unroll
            for (int cc = 0; cc < C; cc++)
            {
                ca[cc] = cb[cc] = (Real)0;
                if ((other & ~cc & (C - 1)) == 0)
                {
                    int64_t o = 0;
#pragma unroll
                    for (int d = 0; d < D; d++)
                        if (cbit<D>(cc, d)) o += so[d];
                    ca[cc] = pA[o];
                    if (cc) cb[cc] = pB[o];
                }
            }
        }
    }
    // every lane, also one without an element: it may hold the node and write it
    if constexpr (Chained) await_previous();
    if (ok)
    {
#pragma unroll
        for (int cc = 0; cc < C; cc++) f[cc] = ld2(xy, (int64_t)(uint32_t)jj[cc]);
        acen = ca[0];
#pragma unroll
        for (int cc = 0; cc < C; cc++)
            if ((other & ~cc & (C - 1)) == 0)
            {
                av = O::fma(ca[cc], f[cc], av);
                if (cc) bv = O::fma(cb[cc], f[cc], bv);
            }
#pragma unroll
        for (int cc = 1; cc < C; cc++) f[cc] = O::sub(f[cc], f[0]);
        if constexpr (shears<Real>())
#pragma unroll
            for (int d = 0; d < D; d++)
            {
                sxy = O::fma(f[1 << d].x, f[1 << d].y, sxy);
                sxx = O::fma(f[1 << d].x, f[1 << d].x, sxx);
                syy = O::fma(f[1 << d].y, f[1 << d].y, syy);
            }
    }
    if constexpr (shears<Real>())
        if (!separate) sh = shear_of(group_sum<D>(sxy), group_sum<D>(sxx), group_sum<D>(syy));
    if (ok)
    {
        if constexpr (shears<Real>())
#pragma unroll
            for (int cc = 1; cc < C; cc++) f[cc] = sheared<Real>(sh, f[cc]);
        FitSums<D, Real> sums;
        sums.clear();
        element_fit_sums<Real>(f, sums);
        fit_to_model<D, Real>(sums, wedge_scale<D, Real>(g.r), av, bv, acen, sh, q);
    }
#pragma unroll
    for (int k = 0; k < 5; k++) q[k] = group_sum<D>(q[k]);
    if (!active || A != 0) return;
    apply_step<Real>(L, xy, i, q, sh, separate, err);
}

// Two lanes per node (large 3D levels): issue slots and the FMA pipe set the pace (a node's 2 x 800
// instructions against 287 bytes).  One depth-8 colour, float: 177 us where the colours follow each other as a solve runs them (0.52 of the measured
// copy bandwidth on 617 MB), 183 us launched by itself, against 600 us for a lane per element on a 12-point Gauss rule and 402 us for a lane
// per element on the rule used now (both by themselves; 171 us without the float kernels' shear); double at depth 7: 1.06 ms against 3.5 ms, the FP64 pipe busy.  Lane s takes the four
// elements on side s of axis 0 with the 18 grid points of its own and the node's plane in registers,
// the stencil columns of its plane, and of the node's plane the A column (lane 0) or the B column
// (lane 1), which the pair layout keeps as one run of 16-byte vectors per lane (PairLayout); one
// exchange joins the two.  (Scalar stencil loads instead of the vectors: 281 us.)  Against a lane per element a node's neighbourhood is read twice instead of
// eight times and its model summed in one shuffle round of five values instead of three.
// stencils: the colour's block of the pair layout, the node being its jc-th of nc.
template <typename Real>
__device__ __forceinline__ void gs_update_pair3(const LevelPtrs<Real> &L, Real *xy, const Grid<3> &g, const int *I, bool active, int s,
                                                unsigned int *err, int separate, const Real *stencils, int64_t jc, int64_t nc)
{
    using O = Ops<Real>;
    using V = Real2<Real>;
    using PL = PairLayout<Real>;
    int64_t i = 0;
    Real q[5] = {(Real)0, (Real)0, (Real)0, (Real)0, (Real)0};
    const V zero = {(Real)0, (Real)0};
    V P[9], Q[9], av = zero, bv = zero;
    Real acen = (Real)0, sxy = (Real)0, sxx = (Real)0, syy = (Real)0;
    Shear<Real> sh = {(Real)0, (Real)0};
    const bool lo1 = I[1] > 0, hi1 = I[1] < g.r, lo2 = I[2] > 0, hi2 = I[2] < g.r;
    const bool side = active && (s ? I[0] > 0 : I[0] < g.r);
    if (active)
    {
        const int st1 = g.r + 1, st0 = st1 * st1;
        const uint32_t iu = (uint32_t)I[0] * (uint32_t)st0 + (uint32_t)I[1] * (uint32_t)st1 + (uint32_t)I[2];
        i = iu;
        const V *own = reinterpret_cast<const V *>(xy) + iu;
        const V *far = own + (s ? -st0 : st0);
        typename PL::Vec cv[PL::G];
        const typename PL::Vec *pc = reinterpret_cast<const typename PL::Vec *>(stencils) + 2 * jc + s;
#pragma unroll
        for (int v = 0; v < PL::G; v++) cv[v] = stream_load(pc + 2 * v * nc);
        await_previous();
        if (side && lo1 && hi1 && lo2 && hi2)
        {
#pragma unroll
            for (int k = 0; k < 9; k++)
            {
                const int o = (k / 3 - 1) * st1 + k % 3 - 1;
                P[k] = own[o];
                Q[k] = far[o];
            }
        }
        else
        {
#pragma unroll
            for (int k = 0; k < 9; k++)
            {
                const int o1 = k / 3 - 1, o2 = k % 3 - 1, o = o1 * st1 + o2;
                const bool in = (o1 < 0 ? lo1 : o1 > 0 ? hi1 : true) && (o2 < 0 ? lo2 : o2 > 0 ? hi2 : true);
                P[k] = zero;
                Q[k] = zero;
                if (in) P[k] = own[o];
                if (in && side) Q[k] = far[o];
            }
        }
        // one partial sum per row of a plane: the columns cancel to a small gradient
        V ev = zero;
#pragma unroll
        for (int o1 = 0; o1 < 3; o1++)
        {
            V ar = zero, br = zero, cr = zero;
#pragma unroll
            for (int o2 = 0; o2 < 3; o2++)
            {
                const int k = 3 * o1 + o2;
                ar = O::fma(PL::at(cv, k), Q[k], ar);
                br = O::fma(PL::at(cv, 9 + k), Q[k], br);
                cr = O::fma(PL::at(cv, 18 + k), P[k], cr);
            }
            ev = O::add(ev, cr);
            av = O::add(av, ar);
            bv = O::add(bv, br);
        }
        if (s) bv = O::add(bv, ev);
        else
        {
            av = O::add(av, ev);
            acen = PL::at(cv, 18 + 4);
        }
        const V mid = P[4];
#pragma unroll
        for (int k = 0; k < 9; k++)
        {
            if (k != 4) P[k] = O::sub(P[k], mid);
            Q[k] = O::sub(Q[k], mid);
        }
        if constexpr (shears<Real>())
        {
            const V d1 = hi1 ? P[7] : P[1], d2 = hi2 ? P[5] : P[3];
            sxy = O::fma(d1.x, d1.y, O::mul(d2.x, d2.y));
            sxx = O::fma(d1.x, d1.x, O::mul(d2.x, d2.x));
            syy = O::fma(d1.y, d1.y, O::mul(d2.y, d2.y));
            if (side)
            {
                sxy = O::fma(Q[4].x, Q[4].y, sxy);
                sxx = O::fma(Q[4].x, Q[4].x, sxx);
                syy = O::fma(Q[4].y, Q[4].y, syy);
            }
        }
    }
    if (!active) await_previous();  // every thread waits
    if constexpr (shears<Real>())
        if (!separate)
        {
            sxy = O::add(sxy, __shfl_xor_sync(0xffffffffu, sxy, 1));
            sxx = O::add(sxx, __shfl_xor_sync(0xffffffffu, sxx, 1));
            syy = O::add(syy, __shfl_xor_sync(0xffffffffu, syy, 1));
            sh = shear_of(sxy, sxx, syy);
        }
    if (active)
    {
        if constexpr (shears<Real>())
#pragma unroll
            for (int k = 0; k < 9; k++)
            {
                if (k != 4) P[k] = sheared<Real>(sh, P[k]);
                Q[k] = sheared<Real>(sh, Q[k]);
            }
        FitSums<3, Real> sums;
        sums.clear();
        if (side)
#pragma unroll
            for (int e = 0; e < 4; e++)
            {
                const int a1 = e >> 1, a2 = e & 1;  // the element lies on the lower side of axis 1, 2
                if (!((a1 ? lo1 : hi1) && (a2 ? lo2 : hi2))) continue;
                V d[8];
#pragma unroll
                for (int c = 0; c < 8; c++)
                {
                    const int k = 3 * (1 + (((c >> 1) & 1) ? (a1 ? -1 : 1) : 0)) + 1 + ((c & 1) ? (a2 ? -1 : 1) : 0);
                    d[c] = (c & 4) ? Q[k] : P[k];
                }
                element_fit_sums<Real>(d, sums);
            }
        fit_to_model<3, Real>(sums, wedge_scale<3, Real>(g.r), av, bv, acen, sh, q);
    }
    if constexpr (sizeof(Real) == 8) next_may_start();
#pragma unroll
    for (int k = 0; k < 5; k++) q[k] = O::add(q[k], __shfl_xor_sync(0xffffffffu, q[k], 1));
    if (!active || s) return;
    apply_step<Real>(L, xy, i, q, sh, separate, err);
}

// Whether a level's colours start ahead of the end of the colour before (launch_colour).  Depth 8, all sweeps
// of a level, chained against not: float levels 4, 5, 6: 2.5, 1.5, 1.8 ms against 4.0, 2.3, 2.0, and 0.6 ms less
// each of levels 7 and 8; double level 3: 10.7 against 13.0, level 6: 49.1 against 49.8.  The blocks that start
// early are placed where the colour before leaves room, so they are spread unevenly: of no account where
// latency counts, but where a few blocks per SM keep the FP64 pipe busy the kernel waits for the fullest SM.  So
// in double a block lets the next colour start only when its own FP64 work is done (level 4: 12.2 ms; at its
// start: 37.5; unchained: 12.4), and a lane per element in double (level 5: 18.0 ms; chained: 21.0) is not chained.
template <typename Real, bool Pair>
__host__ __device__ constexpr bool chains_colours() { return sizeof(Real) == 4 || Pair; }

// lanes per node of the colour kernels of the large levels
template <int D, bool Pair>
__host__ __device__ constexpr int lanes_per_node() { return Pair ? 2 : 1 << D; }

// Resident blocks of 128 threads asked of the compiler.  Float pairs: 5 blocks (95 registers) 171 us a
// depth-8 colour (before the shear), 4 blocks 178, 6 blocks 174; float lanes in 4D: 5 blocks 80 us a depth-5 colour, 2
// blocks 137, 6 blocks 80.  Double is bound by the FP64 pipe at any occupancy.
template <int D, typename Real, bool Pair>
constexpr int lanes_min_blocks()
{
    if (sizeof(Real) == 8) return 2;
    return D == 3 ? (Pair ? 5 : 6) : 5;
}

template <int D, typename Real, bool Pair>
__device__ __forceinline__ void gs_node_lanes(const LevelPtrs<Real> &L, const Grid<D> &g, const int *I, bool active, int lane, unsigned int *err,
                                              int separate, const Colour<D> &col, int64_t cbBase, int64_t jc)
{
    if constexpr (sizeof(Real) == 4) next_may_start();
    if constexpr (Pair)
    {
        // a colour's block starts after 27 values per node of the colours before it
        gs_update_pair3<Real>(L, L.xy, g, I, active, lane, err, separate, L.Acb + cbBase / 27 * PairLayout<Real>::kNode, jc, col.n);
        return;
    }
    const Real *Ac = L.Acb ? L.Acb + cbBase : nullptr, *Bc = L.Bcb ? L.Bcb + cbBase : nullptr;
    if constexpr (!Pair) gs_update_lanes_at<D, Real, true>(L, L.xy, g, I, active, lane, err, separate, Ac, Bc, jc, col.n);
}

// One colour, groups of lanes along the colour's nodes of the last two axes: grid.x = blocks of
// TPB / lanes nodes over the cnt[D-2] x cnt[D-1] nodes of a plane (flat, so that only a plane's last
// block is partly empty), by = the leading axes' node.
template <int D, typename Real, bool Pair, int TPB>
__device__ __forceinline__ void gs_lanes_body(const LevelPtrs<Real> &L, const Colour<D> &col, int64_t cbBase, unsigned int *err,
                                              int separate, int bx, int by)
{
    constexpr int LPN = lanes_per_node<D, Pair>(), NPB = TPB / LPN;
    Grid<D> g(L.level);
    const uint32_t plane = (uint32_t)(col.cnt[D - 2] * col.cnt[D - 1]), c1 = (uint32_t)col.cnt[D - 1];
    const uint32_t p = (uint32_t)bx * NPB + threadIdx.x / LPN;
    int I[D];
    const uint32_t j1 = p / c1;
    I[D - 1] = 2 * (int)(p - j1 * c1) + col.par[D - 1];
    I[D - 2] = 2 * (int)j1 + col.par[D - 2];
    if constexpr (D == 3) I[0] = 2 * by + col.par[0];
    else
    {
        I[1] = 2 * (by % col.cnt[1]) + col.par[1];
        I[0] = 2 * (by / col.cnt[1]) + col.par[0];
    }
    gs_node_lanes<D, Real, Pair>(L, g, I, p < plane, threadIdx.x % LPN, err, separate, col, cbBase, (int64_t)by * plane + p);
}

template <int D, typename Real, bool Pair>
__global__ void __launch_bounds__(kThreads, lanes_min_blocks<D, Real, Pair>())
    gs_colour_lanes_kernel(LevelPtrs<Real> L, Colour<D> col, int64_t cbBase, unsigned int *err, int separate)
{
    gs_lanes_body<D, Real, Pair, kThreads>(L, col, cbBase, err, separate, blockIdx.x, blockIdx.y);
}

// One colour of an adaptive level: the colour's active nodes from its list (colour-local indices),
// each node's update computed the same way
template <int D, typename Real, bool Pair>
__global__ void __launch_bounds__(kThreads, lanes_min_blocks<D, Real, Pair>())
    gs_colour_lanes_list_kernel(LevelPtrs<Real> L, Colour<D> col, int64_t cbBase, const int *list, int count, unsigned int *err,
                                int separate)
{
    constexpr int LPN = lanes_per_node<D, Pair>(), NPB = kThreads / LPN;
    Grid<D> g(L.level);
    const int k = blockIdx.x * NPB + threadIdx.x / LPN;
    const bool active = k < count;
    const int64_t jc = active ? list[k] : 0;
    int I[D];
    col.node(jc, I);
    gs_node_lanes<D, Real, Pair>(L, g, I, active, threadIdx.x % LPN, err, separate, col, cbBase, jc);
}

// the same colour of every reconstruction of a lockstep batch (3D): block = TPB threads, grid.y =
// reconstruction x the colour's count on axis 0
template <typename Real, int TPB, bool Pair>
__global__ void __launch_bounds__(TPB, lanes_min_blocks<3, Real, Pair>() * kThreads / TPB)
    gs_colour_lanes_batch_kernel(const BatchJob<Real> *jobs, Colour<3> col, int64_t cbBase)
{
    const int m = blockIdx.y / col.cnt[0], by = blockIdx.y - m * col.cnt[0];
    const BatchJob<Real> &b = jobs[m];
    gs_lanes_body<3, Real, Pair, TPB>(b.L, col, cbBase, b.err, b.separate, blockIdx.x, by);
}

// All sweeps of a small 4D level in float (16 and 81 nodes) in one thread block: the colours follow each other
// behind a block barrier, which also makes each colour's writes visible to the next.  The level's
// coefficients, and its stencils when they fit, live in shared memory for the whole schedule.
template <int D, typename Real, bool SmemStencil>
__global__ void __launch_bounds__(256) gs_level_kernel(LevelPtrs<Real> L, int iters, unsigned int *err, int separate)
{
    Grid<D> g(L.level);
    constexpr int S = Dims<D>::S;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    Real *xy = reinterpret_cast<Real *>(smem_raw);
    for (int64_t k = threadIdx.x; k < 2 * g.N; k += blockDim.x) xy[k] = L.xy[k];
    LevelPtrs<Real> Ls = L;
    if constexpr (SmemStencil)
    {
        Real *A = xy + 2 * g.N, *B = A + S * g.N;
        for (int64_t k = threadIdx.x; k < S * g.N; k += blockDim.x) { A[k] = L.A[k]; B[k] = L.B[k]; }
        Ls.A = A;
        Ls.B = B;
    }
    __syncthreads();
    for (int it = 0; it < iters; it++)
        for (int c = 0; c < (1 << D); c++)
        {
            Colour<D> col(g, c);
            const int per = blockDim.x >> D;  // nodes per pass of the block
            const int A = threadIdx.x & ((1 << D) - 1);
            for (int64_t j0 = 0; j0 < col.n; j0 += per)
            {
                int64_t j = j0 + (threadIdx.x >> D);
                bool active = j < col.n;
                int I[D];
                if (active) col.node(j, I);
                else
                    for (int d = 0; d < D; d++) I[d] = 0;
                gs_update_lanes_at<D, Real>(Ls, xy, g, I, active, A, err, separate);
            }
            __syncthreads();
        }
    for (int64_t k = threadIdx.x; k < 2 * g.N; k += blockDim.x) L.xy[k] = xy[k];
}

template <int D, typename Real>
__global__ void __launch_bounds__(kThreads) gn_matvec_kernel(LevelPtrs<Real> L, const Real *xy, const Real *dxy, Real *out)
{
    Grid<D> g(L.level);
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= g.N) return;
    NodeCtx<D> nc;
    make_ctx<D>(g, i, nc);
    Real2<Real> acc = {(Real)0, (Real)0};
    const Real2<Real> own = ld2(xy, i), down = ld2(dxy, i);
#pragma unroll 1
    for (int A = 0; A < (1 << D); A++)
    {
        bool ok = true;
        int64_t sd[D];
#pragma unroll
        for (int d = 0; d < D; d++)
        {
            const int e = nc.I[d] - cbit<D>(A, d);
            ok = ok && e >= 0 && e < g.r;
            sd[d] = cbit<D>(A, d) ? -nc.stride[d] : nc.stride[d];
        }
        if (!ok) continue;
        Real2<Real> df[1 << D], dd[1 << D];
        df[0] = own;
        dd[0] = down;
#pragma unroll
        for (int cc = 1; cc < (1 << D); cc++)
        {
            int64_t j = i;
#pragma unroll
            for (int d = 0; d < D; d++)
                if (cbit<D>(cc, d)) j += sd[d];
            df[cc] = Ops<Real>::sub(ld2(xy, j), own);
            dd[cc] = Ops<Real>::sub(ld2(dxy, j), down);
        }
        element_gn<Real>(df, dd, acc);
    }
    const Real sc = wedge_scale<D, Real>(g.r) * (Real)(D == 3 ? 1.0 / 256.0 : 1.0 / 4096.0);
    Real ox = -acc.y * sc, oy = acc.x * sc;
    constexpr int S = Dims<D>::S;
    for (int o = 0; o < S; o++)
    {
        int off[D];
        stencil_offset<D>(o, off);
        bool ok = true;
        int64_t j = i;
#pragma unroll
        for (int d = 0; d < D; d++)
        {
            int t = nc.I[d] + off[d];
            ok = ok && (t >= 0) && (t <= g.r);
            j += (int64_t)off[d] * nc.stride[d];
        }
        if (!ok) continue;
        Real a = stencil_a(L, (int64_t)o * L.N + i);
        Real2<Real> v = ld2(dxy, j);
        ox += a * v.x;
        oy += a * v.y;
    }
    reinterpret_cast<Real2<Real> *>(out)[i] = Real2<Real>{ox, oy};
}

// the multilinear interpolant of the coarse pairs at fine node i
template <int D, typename Real>
__device__ __forceinline__ Real2<Real> prolonged(const Grid<D> &gc, const Grid<D> &gf, const Real *coarse, int64_t i)
{
    int F[D];
    gf.node(i, F);
    Real sx = 0, sy = 0;
#pragma unroll
    for (int c = 0; c < (1 << D); c++)
    {
        bool use = true;
        Real w = 1;
        int I[D];
#pragma unroll
        for (int d = 0; d < D; d++)
        {
            int b = (c >> d) & 1;
            if (F[d] & 1) { I[d] = (F[d] >> 1) + b; w *= (Real)0.5; }
            else { I[d] = F[d] >> 1; if (b) use = false; }
        }
        if (!use) continue;
        Real2<Real> v = ld2(coarse, gc.node(I));
        sx += w * v.x;
        sy += w * v.y;
    }
    return Real2<Real>{sx, sy};
}
template <int D, typename Real>
__device__ __forceinline__ void prolong_at(int coarseLevel, const Real *coarse, Real *fine, int add, int64_t i,
                                           const uint8_t *fineStatus = nullptr)
{
    Grid<D> gc(coarseLevel), gf(coarseLevel + 1);
    if (i >= gf.N) return;
    // the adaptive prolongation reaches indexed fine functions only (ffChildNeighbors,
    // Hat.scalars.inl:1747-1779); the others stay zero
    if (fineStatus && fineStatus[i] == 0)
    {
        if (!add) reinterpret_cast<Real2<Real> *>(fine)[i] = Real2<Real>{(Real)0, (Real)0};
        return;
    }
    const Real2<Real> v = prolonged<D, Real>(gc, gf, coarse, i);
    Real2<Real> *o = reinterpret_cast<Real2<Real> *>(fine);
    if (add) { Real2<Real> cur = o[i]; o[i] = Real2<Real>{cur.x + v.x, cur.y + v.y}; }
    else o[i] = v;
}
// out = fine - P coarse (P coarse zero at fine nodes without a function): a level's hierarchical coefficients
template <int D>
__global__ void __launch_bounds__(256) hierarchical_kernel(int coarseLevel, const double *coarse, const double *fine, double *out,
                                                            const uint8_t *fineStatus)
{
    Grid<D> gc(coarseLevel), gf(coarseLevel + 1);
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= gf.N) return;
    double2 p = {0., 0.};
    if (!(fineStatus && fineStatus[i] == 0)) p = prolonged<D, double>(gc, gf, coarse, i);
    const double2 v = ld2(fine, i);
    reinterpret_cast<double2 *>(out)[i] = double2{v.x - p.x, v.y - p.y};
}
template <int D, typename Real>
__global__ void prolong_kernel(int coarseLevel, const Real *coarse, Real *fine, int add, const uint8_t *fineStatus)
{
    prolong_at<D, Real>(coarseLevel, coarse, fine, add, blockIdx.x * (int64_t)blockDim.x + threadIdx.x, fineStatus);
}
// grid.y = reconstruction of a lockstep batch
template <typename Real>
__global__ void prolong_add_batch_kernel(const XferJob *jobs, int coarseLevel)
{
    const XferJob &j = jobs[blockIdx.y];
    prolong_at<3, Real>(coarseLevel, (const Real *)j.src, (Real *)j.dst, 1, blockIdx.x * (int64_t)blockDim.x + threadIdx.x);
}
__global__ void f2d_batch_kernel(const XferJob *jobs, int64_t n)
{
    const XferJob &j = jobs[blockIdx.y];
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) ((double *)j.dst)[i] = (double)((const float *)j.src)[i];
}
__global__ void d2f_batch_kernel(const XferJob *jobs, int64_t n)
{
    const XferJob &j = jobs[blockIdx.y];
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) ((float *)j.dst)[i] = (float)((const double *)j.src)[i];
}

template <int D, typename Real>
__global__ void restrict_kernel(int coarseLevel, const Real *fine, Real *coarse)
{
    Grid<D> gc(coarseLevel), gf(coarseLevel + 1);
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= gc.N) return;
    int I[D];
    gc.node(i, I);
    Real sx = 0, sy = 0;
    constexpr int S = Dims<D>::S;
#pragma unroll 3
    for (int o = 0; o < S; o++)
    {
        int off[D], F[D];
        stencil_offset<D>(o, off);
        bool ok = true;
        Real w = 1;
#pragma unroll
        for (int d = 0; d < D; d++)
        {
            F[d] = 2 * I[d] + off[d];
            ok = ok && F[d] >= 0 && F[d] <= gf.r;
            if (off[d]) w *= (Real)0.5;
        }
        if (!ok) continue;
        Real2<Real> v = ld2(fine, gf.node(F));
        sx += w * v.x;
        sy += w * v.y;
    }
    reinterpret_cast<Real2<Real> *>(coarse)[i] = Real2<Real>{sx, sy};
}

template <typename Real>
__global__ void scale_kernel(Real *v, int64_t n, double s)
{
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) v[i] = (Real)((double)v[i] * s);
}
template <typename Real>
__global__ void axpy_kernel(Real *y, const Real *x, int64_t n, double a)
{
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) y[i] = (Real)((double)y[i] + a * (double)x[i]);
}
__global__ void d2f_kernel(const double *in, float *out, int64_t n)
{
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = (float)in[i];
}
__global__ void f2d_kernel(const float *in, double *out, int64_t n)
{
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) out[i] = (double)in[i];
}

inline unsigned int blocks_for(int64_t n, int t = kThreads) { return (unsigned int)((n + t - 1) / t); }

// the 4D float levels that relax in one block
constexpr int64_t kBlockMaxNodes4 = 81;
constexpr size_t kLevelSmemLimit = 200 * 1024;

}  // namespace

// ---------------------------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------------------------
template <int D, typename Real>
void launch_energy(const LevelPtrs<Real> &L, const Real *xy, const Reduce &red, cudaStream_t s)
{
    Grid<D> g(L.level);
    int64_t total = g.N > g.NE ? g.N : g.NE;
    int nb = (int)blocks_for(total);
    if (nb > Reduce::kMaxBlocks) nb = Reduce::kMaxBlocks;
    if (nb < 1) nb = 1;
    if (L.A) energy_kernel<D, Real, true><<<nb, kThreads, 0, s>>>(L, xy, red.partial);
    else energy_kernel<D, Real, false><<<nb, kThreads, 0, s>>>(L, xy, red.partial);
    double scale0 = (D == 3 ? (double)g.r : 1.0) * 0.5;
    finish_kernel<<<1, 96, 0, s>>>(red.partial, nb, 3, red.out, scale0);
}

template <int D, typename Real>
void launch_grad_norm(const LevelPtrs<Real> &L, const Real *xy, const Reduce &red, cudaStream_t s)
{
    Grid<D> g(L.level);
    int nb = (int)blocks_for(g.N);
    if (nb > Reduce::kMaxBlocks) nb = Reduce::kMaxBlocks;
    if (nb < 1) nb = 1;
    grad_norm_kernel<D, Real><<<nb, kThreads, 0, s>>>(L, xy, red.partial);
    finish_kernel<<<1, 32, 0, s>>>(red.partial, nb, 1, red.out, 1.0);
}

template <int D, typename Real>
void launch_quadfit(const LevelPtrs<Real> &L, const Real *xy, double *out, cudaStream_t s)
{
    Grid<D> g(L.level);
    quadfit_kernel<D, Real><<<blocks_for(g.N), kThreads, 0, s>>>(L, xy, out);
}

template <int D, typename Real>
bool launch_gs_colour(const LevelPtrs<Real> &L, int colour, unsigned int *err, cudaStream_t s, int separate, bool after)
{
    Grid<D> g(L.level);
    Colour<D> col(g, colour);
    if (col.n == 0) return false;
    if constexpr (D == 3)
        if (small_colour_level<Real>(L.level))
        {
            launch_small_colour<Real>(L, colour, err, s, separate, nullptr, after);
            return true;
        }
    if constexpr (D == 4 && std::is_same<Real, double>::value)
        if (small4_colour_level(L.level))
        {
            launch_small4_colour(L, colour, err, s, separate, after);
            return true;
        }
    const int64_t cb = colour_block_base<D>(g, colour);
    auto launch = [&](auto pair) {
        constexpr bool Pair = decltype(pair)::value;
        constexpr int NPB = kThreads / lanes_per_node<D, Pair>();
        const bool chained = after && chains_colours<Real, Pair>();
        if (L.alist)
        {
            // adaptive level: only the colour's active nodes
            const int count = L.aoff[colour + 1] - L.aoff[colour];
            if (count > 0)
                launch_colour(gs_colour_lanes_list_kernel<D, Real, Pair>, dim3(blocks_for(count, NPB)), 1, kThreads, 0, s, chained, L, col, cb,
                              L.alist + L.aoff[colour], count, err, separate);
            return count > 0;
        }
        dim3 grid(blocks_for((int64_t)col.cnt[D - 2] * col.cnt[D - 1], NPB), (unsigned)(D == 3 ? col.cnt[0] : col.cnt[0] * col.cnt[1]));
        launch_colour(gs_colour_lanes_kernel<D, Real, Pair>, grid, 1, kThreads, 0, s, chained, L, col, cb, err, separate);
        return true;
    };
    if constexpr (D == 3)
        if (pair_level<D>(L.level)) return launch(std::true_type{});
    return launch(std::false_type{});
}

cudaError_t prepare_gs_kernels(int *blocks3)
{
    if (const cudaError_t e = prepare_small_kernels(blocks3)) return e;
    return cudaFuncSetAttribute(gs_level_kernel<4, float, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLevelSmemLimit);
}

template <int D, typename Real>
int launch_gs_sweeps(const LevelPtrs<Real> &L, int iters, unsigned int *err, cudaStream_t s, int separate)
{
    Grid<D> g(L.level);
    if (iters <= 0) return 0;
    if constexpr (D == 3)
        if (small_level<Real>(L.level))
        {
            launch_small_level<Real>(L, iters, err, s, separate, nullptr);
            return 1;
        }
    if constexpr (D == 4 && std::is_same<Real, double>::value)
        if (launch_small4(L, iters, err, s, separate)) return 1;
    if constexpr (D == 4 && std::is_same<Real, float>::value)
        if (g.N <= kBlockMaxNodes4)
        {
            const int64_t colour0 = Colour<D>(g, 0).n;  // the colour of even nodes is the largest
            const size_t xyBytes = 2 * g.N * sizeof(Real), stBytes = 2 * (size_t)Dims<D>::S * g.N * sizeof(Real);
            // lanes per node: one pass per colour where the block allows it, whole warps
            const int threads = (int)std::min<int64_t>(256, ((colour0 << D) + 31) / 32 * 32);
            if (xyBytes + stBytes <= kLevelSmemLimit) gs_level_kernel<D, Real, true><<<1, threads, xyBytes + stBytes, s>>>(L, iters, err, separate);
            else gs_level_kernel<D, Real, false><<<1, threads, xyBytes, s>>>(L, iters, err, separate);
            return 1;
        }
    int n = 0;
    bool after = false;
    for (int it = 0; it < iters; it++)
        for (int c = 0; c < (1 << D); c++)
        {
            after = launch_gs_colour<D, Real>(L, c, err, s, separate, after) || after;
            n++;
        }
    return n;
}

// ---------------------------------------------------------------------------------------------
// double-float levels (3D levels 0-3 of the float solve's coarse band)
// ---------------------------------------------------------------------------------------------
// double coefficients -> pairs at the level's new exponent (the largest magnitude in [1, 2))
__device__ __forceinline__ void df_push_body(const double *in, df *out, int64_t n, int *kexp, int level)
{
    __shared__ double wmax[32];
    __shared__ int k;
    double m = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) m = fmax(m, fabs(in[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        double mm = 0.0;
        for (int w = 0; w < (int)((blockDim.x + 31) >> 5); w++) mm = fmax(mm, wmax[w]);
        k = mm > 0.0 ? ilogb(mm) : 0;
        kexp[level] = k;
    }
    __syncthreads();
    for (int64_t i = threadIdx.x; i < n; i += blockDim.x) out[i] = df(ldexp(in[i], -k));
}
__global__ void df_push_kernel(const double *in, df *out, int64_t n, int *kexp, int level) { df_push_body(in, out, n, kexp, level); }
__global__ void df_push_batch_kernel(const XferJob *jobs, int64_t n, int level)
{
    const XferJob &j = jobs[blockIdx.x];
    df_push_body((const double *)j.src, (df *)j.dst, n, j.kexp, level);
}
__global__ void df_pull_batch_kernel(const XferJob *jobs, int64_t n, int level)
{
    const XferJob &j = jobs[blockIdx.y];
    const int k = j.kexp[level];
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) ((double *)j.dst)[i] = ldexp((double)((const df *)j.src)[i], k);
}

__global__ void df_pull_kernel(const df *in, double *out, int64_t n, const int *kexp, int level)
{
    const int k = kexp[level];
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = ldexp((double)in[i], k);
}

__global__ void d2df_kernel(const double *in, df *out, int64_t n)
{
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) out[i] = df(in[i]);
}

void launch_df_push(const double *in, df *out, int64_t n, int *kexp, int level, cudaStream_t s)
{
    df_push_kernel<<<1, 256, 0, s>>>(in, out, n, kexp, level);
}
void launch_df_pull(const df *in, double *out, int64_t n, const int *kexp, int level, cudaStream_t s)
{
    df_pull_kernel<<<(unsigned)std::min<int64_t>(blocks_for(n, 256), 1024), 256, 0, s>>>(in, out, n, kexp, level);
}
void launch_d2df(const double *in, df *out, int64_t n, cudaStream_t s)
{
    if (n) d2df_kernel<<<(unsigned)std::min<int64_t>(blocks_for(n, 256), 1024), 256, 0, s>>>(in, out, n);
}

template <int D, typename Real>
void launch_gn_matvec(const LevelPtrs<Real> &L, const Real *xy, const Real *dxy, Real *out, cudaStream_t s)
{
    Grid<D> g(L.level);
    gn_matvec_kernel<D, Real><<<blocks_for(g.N), kThreads, 0, s>>>(L, xy, dxy, out);
}

template <int D, typename Real>
void launch_prolong(int coarseLevel, const Real *coarse, Real *fine, int add, cudaStream_t s, const uint8_t *fineStatus)
{
    Grid<D> gf(coarseLevel + 1);
    prolong_kernel<D, Real><<<blocks_for(gf.N, 256), 256, 0, s>>>(coarseLevel, coarse, fine, add, fineStatus);
}

template <int D>
void launch_hierarchical(int coarseLevel, const double *coarse, const double *fine, double *out, cudaStream_t s, const uint8_t *fineStatus)
{
    Grid<D> gf(coarseLevel + 1);
    hierarchical_kernel<D><<<blocks_for(gf.N, 256), 256, 0, s>>>(coarseLevel, coarse, fine, out, fineStatus);
}
template void launch_hierarchical<3>(int, const double *, const double *, double *, cudaStream_t, const uint8_t *);
template void launch_hierarchical<4>(int, const double *, const double *, double *, cudaStream_t, const uint8_t *);

template <int D, typename Real>
void launch_restrict(int coarseLevel, const Real *fine, Real *coarse, cudaStream_t s)
{
    Grid<D> gc(coarseLevel);
    restrict_kernel<D, Real><<<blocks_for(gc.N, 256), 256, 0, s>>>(coarseLevel, fine, coarse);
}

template <typename Real>
void launch_scale(Real *v, int64_t n, double sc, cudaStream_t st)
{
    if (n) scale_kernel<Real><<<blocks_for(n, 256), 256, 0, st>>>(v, n, sc);
}
template <typename Real>
void launch_axpy(Real *y, const Real *x, int64_t n, double a, cudaStream_t st)
{
    if (n) axpy_kernel<Real><<<blocks_for(n, 256), 256, 0, st>>>(y, x, n, a);
}
__global__ void split_pairs_kernel(const double *xy, double *x, double *y, int64_t n)
{
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) { double2 v = reinterpret_cast<const double2 *>(xy)[i]; x[i] = v.x; y[i] = v.y; }
}
__global__ void merge_pairs_kernel(const double *x, const double *y, double *xy, int64_t n)
{
    int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i < n) reinterpret_cast<double2 *>(xy)[i] = double2{x[i], y[i]};
}
void launch_split_pairs(const double *xy, double *x, double *y, int64_t n, cudaStream_t st)
{
    if (n) split_pairs_kernel<<<blocks_for(n, 256), 256, 0, st>>>(xy, x, y, n);
}
void launch_merge_pairs(const double *x, const double *y, double *xy, int64_t n, cudaStream_t st)
{
    if (n) merge_pairs_kernel<<<blocks_for(n, 256), 256, 0, st>>>(x, y, xy, n);
}
void launch_convert_d2f(const double *in, float *out, int64_t n, cudaStream_t st)
{
    if (n) d2f_kernel<<<blocks_for(n, 256), 256, 0, st>>>(in, out, n);
}
void launch_convert_f2d(const float *in, double *out, int64_t n, cudaStream_t st)
{
    if (n) f2d_kernel<<<blocks_for(n, 256), 256, 0, st>>>(in, out, n);
}

// ---------------------------------------------------------------------------------------------
// lockstep batches (3D)
// ---------------------------------------------------------------------------------------------
template <typename Real, int TPB, bool Pair>
static void launch_lanes_batch_as(const BatchJob<Real> *jobs, const Colour<3> &col, int64_t cb, int count, cudaStream_t s, bool after)
{
    constexpr int NPB = TPB / lanes_per_node<3, Pair>();
    // grid.y = reconstruction x axis-0 count, at most 65,535: chunks of reconstructions
    const int per = std::max(1, 65535 / col.cnt[0]);
    constexpr bool chained = chains_colours<Real, Pair>();
    for (int m0 = 0; m0 < count; m0 += per)
    {
        const int cnt = std::min(per, count - m0);
        dim3 grid(blocks_for((int64_t)col.cnt[1] * col.cnt[2], NPB), (unsigned)(cnt * col.cnt[0]));
        launch_colour(gs_colour_lanes_batch_kernel<Real, TPB, Pair>, grid, 1, TPB, 0, s, chained && (after || m0 > 0), jobs + m0, col, cb);
    }
}
template <typename Real, int TPB>
static void launch_lanes_batch(const BatchJob<Real> *jobs, int level, const Colour<3> &col, int64_t cb, int count,
                               cudaStream_t s, bool after)
{
    if (pair_level<3>(level)) launch_lanes_batch_as<Real, TPB, true>(jobs, col, cb, count, s, after);
    else launch_lanes_batch_as<Real, TPB, false>(jobs, col, cb, count, s, after);
}

template <typename Real>
bool launch_colour_batch(const BatchJob<Real> *jobs, int level, int colour, int count, int tile, cudaStream_t s, bool after)
{
    if (count <= 0) return false;
    Grid<3> g(level);
    Colour<3> col(g, colour);
    if (col.n == 0) return false;
    const int64_t cb = colour_block_base<3>(g, colour);
    if (small_colour_level<Real>(level))
    {
        launch_small_colour_batch<Real>(jobs, level, colour, count, s, after);
        return true;
    }
    if constexpr (std::is_same<Real, df>::value) return false;  // double-float levels are 3D levels <= 3
    else
    {
        if (tile == 0) launch_lanes_batch<Real, 64>(jobs, level, col, cb, count, s, after);
        else if (tile == 2) launch_lanes_batch<Real, 256>(jobs, level, col, cb, count, s, after);
        else launch_lanes_batch<Real, 128>(jobs, level, col, cb, count, s, after);
        return true;
    }
}

template <typename Real>
void launch_prolong_add_batch(const XferJob *jobs, int coarseLevel, int count, cudaStream_t s)
{
    if (count <= 0) return;
    Grid<3> gf(coarseLevel + 1);
    prolong_add_batch_kernel<Real><<<dim3(blocks_for(gf.N, 256), (unsigned)count), 256, 0, s>>>(jobs, coarseLevel);
}
void launch_f2d_batch(const XferJob *jobs, int64_t n, int count, cudaStream_t s)
{
    if (count > 0 && n) f2d_batch_kernel<<<dim3(blocks_for(n, 256), (unsigned)count), 256, 0, s>>>(jobs, n);
}
void launch_d2f_batch(const XferJob *jobs, int64_t n, int count, cudaStream_t s)
{
    if (count > 0 && n) d2f_batch_kernel<<<dim3(blocks_for(n, 256), (unsigned)count), 256, 0, s>>>(jobs, n);
}
void launch_df_pull_batch(const XferJob *jobs, int64_t n, int level, int count, cudaStream_t s)
{
    if (count > 0 && n) df_pull_batch_kernel<<<dim3(blocks_for(n, 256), (unsigned)count), 256, 0, s>>>(jobs, n, level);
}
void launch_df_push_batch(const XferJob *jobs, int64_t n, int level, int count, cudaStream_t s)
{
    if (count > 0 && n) df_push_batch_kernel<<<count, 256, 0, s>>>(jobs, n, level);
}

template bool launch_colour_batch<float>(const BatchJob<float> *, int, int, int, int, cudaStream_t, bool);
template bool launch_colour_batch<double>(const BatchJob<double> *, int, int, int, int, cudaStream_t, bool);
template bool launch_colour_batch<df>(const BatchJob<df> *, int, int, int, int, cudaStream_t, bool);
template void launch_prolong_add_batch<float>(const XferJob *, int, int, cudaStream_t);
template void launch_prolong_add_batch<double>(const XferJob *, int, int, cudaStream_t);

#define EPR_INSTANTIATE(D, R)                                                                          \
    template void launch_energy<D, R>(const LevelPtrs<R> &, const R *, const Reduce &, cudaStream_t);   \
    template void launch_quadfit<D, R>(const LevelPtrs<R> &, const R *, double *, cudaStream_t);        \
    template void launch_grad_norm<D, R>(const LevelPtrs<R> &, const R *, const Reduce &, cudaStream_t); \
    template bool launch_gs_colour<D, R>(const LevelPtrs<R> &, int, unsigned int *, cudaStream_t, int, bool); \
    template int launch_gs_sweeps<D, R>(const LevelPtrs<R> &, int, unsigned int *, cudaStream_t, int); \
    template void launch_gn_matvec<D, R>(const LevelPtrs<R> &, const R *, const R *, R *, cudaStream_t); \
    template void launch_prolong<D, R>(int, const R *, R *, int, cudaStream_t, const uint8_t *);                         \
    template void launch_restrict<D, R>(int, const R *, R *, cudaStream_t);

EPR_INSTANTIATE(3, double)
EPR_INSTANTIATE(3, float)
EPR_INSTANTIATE(4, double)
EPR_INSTANTIATE(4, float)
template void launch_scale<double>(double *, int64_t, double, cudaStream_t);
template void launch_scale<float>(float *, int64_t, double, cudaStream_t);
template void launch_axpy<double>(double *, const double *, int64_t, double, cudaStream_t);
template void launch_axpy<float>(float *, const float *, int64_t, double, cudaStream_t);

}  // namespace epr
