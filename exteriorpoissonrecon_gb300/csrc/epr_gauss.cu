// Paired Gauss-Seidel sweeps in float that a caller runs by itself (epr_gs), on the 2 x 2 x 3^(D-2)-point Gauss
// rule: levels of more than 729 nodes (gauss_level).
//
// A solve relaxes with the modal fit, whose last bits differ.  Over a whole solve that does not show (relative
// differences of 1e-7), but at nodes where the fields' gradients are nearly parallel one sweep divides by a
// determinant of the size of the Gauss rule's rounding error: of a field of 10^5 to 10^6 nodes a handful are good to
// two or three digits (in L2 up to 1e-5 off 64 bits; the modal fit with its shear 5e-7).  A program that drives single
// sweeps sees the two rules' difference there, so its sweeps keep the arithmetic, operation for operation, that their
// results have always had.  What it gives up is the fit's accuracy at those nodes and half its speed, and that
// such a program's own schedule of sweeps and prolongations ends where epr_solve ends to rounding only.
//
// Bound by instruction issue: a node's 2^D elements take 36 points each in 3D and 216 in 4D (a depth-8 colour
// 600 us, where the modal rule on two lanes per node takes 183 us).  Resident blocks of 128 threads asked of the
// compiler, a call with its copies, compared side by side: 4D level 5, two sweeps, 2 blocks (255 registers) 10.3 ms, 3
// blocks 8.75, 5 blocks 11.4 (spills); 3D level 6, four sweeps, 9 blocks 0.89 ms, 7 blocks 0.86, 6 blocks 0.89 (by
// themselves the chosen ones take 8.5 and 0.92 ms).  The colours are chained (launch_colour).
#include <algorithm>
#include <cmath>

#include "epr_common.cuh"
#include "epr_element.cuh"
#include "epr_kernels.h"
#include "epr_step.cuh"

namespace epr {

namespace {

// The five sums of a corner: with p = (x_P, y_P), q = (x_Q, y_Q) the P- and Q-derivatives at a point,
// T = phP q - phQ p = (V, -U) and W = y_P x_Q - x_P y_Q, (h1, h0) += (w T) * T, (h4, -h3) += (w T) * W, h2 += wU V.
struct GaussSums
{
    float2 hv = {0.f, 0.f}, hw = {0.f, 0.f};
    float h2 = 0.f;
};

__device__ __forceinline__ float2 splat2(float v) { return make_float2(v, v); }

// differences along the component's axis P (AisP) or Q, interpolated at the two points of the other
template <int D, int K, bool AisP>
__device__ __forceinline__ void differences(const float2 *f, float2 (&t)[2][1 << (D - 2)])
{
    using Cp = Component<D, K>;
    constexpr int NO = 1 << Cp::M;
    float2 dif[2][NO];
#pragma unroll
    for (int bB = 0; bB < 2; bB++)
#pragma unroll
        for (int bo = 0; bo < NO; bo++)
        {
            const int c1 = AisP ? Cp::corner(1, bB, bo) : Cp::corner(bB, 1, bo);
            const int c0 = AisP ? Cp::corner(0, bB, bo) : Cp::corner(bB, 0, bo);
            dif[bB][bo] = __ffma2_rn(f[c0], splat2(-1.f), f[c1]);
        }
#pragma unroll
    for (int g = 0; g < 2; g++)
#pragma unroll
        for (int bo = 0; bo < NO; bo++)
            t[g][bo] = __ffma2_rn(splat2(hat2<float>(1, g)), dif[1][bo], __fmul2_rn(splat2(hat2<float>(0, g)), dif[0][bo]));
}

// ... at point go of the three (nine) of the remaining axes
template <int M>
__device__ __forceinline__ float2 at_point(const float2 *t, int go)
{
    if constexpr (M == 1) return __ffma2_rn(splat2(hat3<float>(1, go)), t[1], __fmul2_rn(splat2(hat3<float>(0, go)), t[0]));
    else
    {
        const float2 a0 = splat2(hat3<float>(0, go / 3)), a1 = splat2(hat3<float>(1, go / 3));
        const float2 u0 = __ffma2_rn(a1, t[2], __fmul2_rn(a0, t[0])), u1 = __ffma2_rn(a1, t[3], __fmul2_rn(a0, t[1]));
        return __ffma2_rn(splat2(hat3<float>(1, go % 3)), u1, __fmul2_rn(splat2(hat3<float>(0, go % 3)), u0));
    }
}

template <int D, int K>
__device__ __forceinline__ void add_component(const float2 *c, GaussSums &acc)
{
    constexpr int M = Component<D, K>::M;
    float2 tP[2][1 << M], tQ[2][1 << M];
    differences<D, K, true>(c, tP);
    differences<D, K, false>(c, tQ);
#pragma unroll
    for (int go = 0; go < ipow(3, M); go++)
    {
        float lo;
        if constexpr (M == 1) lo = hat3<float>(0, go);
        else lo = hat3<float>(0, go / 3) * hat3<float>(0, go % 3);
        const float wo = (float)other_weight<M>(go);
        float2 Pg[2], Qg[2];
#pragma unroll
        for (int g = 0; g < 2; g++)
        {
            Pg[g] = at_point<M>(tP[g], go);
            Qg[g] = at_point<M>(tQ[g], go);
        }
#pragma unroll
        for (int gp = 0; gp < 2; gp++)
#pragma unroll
            for (int gq = 0; gq < 2; gq++)
            {
                const float w = (float)(Gauss::W2(gp) * Gauss::W2(gq)) * wo;
                const float phP = -hat2<float>(0, gq) * lo, phQ = -hat2<float>(0, gp) * lo;
                const float2 p = Pg[gq], q = Qg[gp];
                const float W = fmaf(p.y, q.x, -(p.x * q.y));
                const float2 T = __ffma2_rn(splat2(phP), q, __fmul2_rn(splat2(-phQ), p));
                const float2 wT = __fmul2_rn(splat2(w), T);
                acc.hv = __ffma2_rn(wT, T, acc.hv);
                acc.hw = __ffma2_rn(wT, splat2(W), acc.hw);
                acc.h2 = fmaf(-wT.y, T.x, acc.h2);
            }
    }
}

template <int D>
__device__ __forceinline__ float lanes_sum(float v)
{
#pragma unroll
    for (int o = (1 << D) / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o, 1 << D);
    return v;
}

// the paired or separate step, the determinant as written
__device__ __forceinline__ bool plain_step(const float *q, int separate, float &p0, float &p1)
{
    const float h00 = 2.f * q[0], h11 = 2.f * q[1], h01 = q[2];
    if (separate)
    {
        p0 = 0;
        p1 = 0;
        if ((double)h00 > 1e-20) p0 = -((h01 + h01) * p1 + q[3]) / (2.f * h00);
        if ((double)h11 > 1e-20) p1 = -((h01 + h01) * p0 + q[4]) / (2.f * h11);
        return true;
    }
    const float det = h00 * h11 - h01 * h01;
    if (!(fabs((double)det) > 1e-20)) return false;
    p0 = -(h11 * q[3] - h01 * q[4]) / det / 2.f;
    p1 = -(-h01 * q[3] + h00 * q[4]) / det / 2.f;
    return true;
}

constexpr int kGaussThreads = 128;

// One colour, 2^D lanes per node: lane A takes the node's element A, mirrored so that the node is its corner 0,
// and every 2^D-th entry of its stencil column.  list (optional): the colour's active nodes of an adaptive level.
// Stencils: the colour blocks, or on pair levels the pair layout (the same values).
template <int D>
__global__ void __launch_bounds__(kGaussThreads, D == 3 ? 7 : 3)
    gauss_colour_kernel(LevelPtrs<float> L, Colour<D> col, int64_t cbBase, const int *list, int64_t count, unsigned int *err, int separate)
{
    constexpr int C = 1 << D, S = Dims<D>::S;
    next_may_start();
    const Grid<D> g(L.level);
    const int A = threadIdx.x & (C - 1);
    const int64_t k = (int64_t)blockIdx.x * (kGaussThreads >> D) + (threadIdx.x >> D);
    const bool active = k < count;
    const int64_t jc = !active ? 0 : list ? list[k] : k;
    int I[D];
    col.node(jc, I);
    const bool pair = D == 3 && pair_level<D>(L.level);
    int64_t i = 0;
    float h[5] = {0, 0, 0, 0, 0};
    float ax = 0, ay = 0, bx = 0, by = 0, acen = 0;
    await_previous();
    if (active)
    {
        int st[D], sd[D];
        st[D - 1] = 1;
#pragma unroll
        for (int d = D - 2; d >= 0; d--) st[d] = st[d + 1] * (g.r + 1);
        uint32_t iu = 0;
        bool ok = true;
#pragma unroll
        for (int d = 0; d < D; d++)
        {
            iu += (uint32_t)I[d] * (uint32_t)st[d];
            sd[d] = cbit<D>(A, d) ? -st[d] : st[d];
            const int e = I[d] - cbit<D>(A, d);
            ok = ok && e >= 0 && e < g.r;
        }
        i = iu;
        if (ok)
        {
            float2 c[C];
#pragma unroll
            for (int cc = 0; cc < C; cc++)
            {
                int jj = (int)iu;
#pragma unroll
                for (int d = 0; d < D; d++)
                    if (cbit<D>(cc, d)) jj += sd[d];
                c[cc] = ld2(L.xy, (int64_t)(uint32_t)jj);
            }
            GaussSums acc;
            add_component<D, 0>(c, acc);
            add_component<D, 1>(c, acc);
            add_component<D, 2>(c, acc);
            if constexpr (D == 4)
            {
                add_component<D, 3>(c, acc);
                add_component<D, 4>(c, acc);
                add_component<D, 5>(c, acc);
            }
            h[0] += acc.hv.y;
            h[1] += acc.hv.x;
            h[2] += acc.h2;
            h[3] -= acc.hw.y;
            h[4] += acc.hw.x;
        }
        for (int o = A; o < S; o += C)
        {
            int off[D];
            stencil_offset<D>(o, off);
            bool in = true;
            int jj = (int)iu;
#pragma unroll
            for (int d = 0; d < D; d++)
            {
                const int t = I[d] + off[d];
                in = in && (t >= 0) && (t <= g.r);
                jj += off[d] * st[d];
            }
            if (!in) continue;
            float a, b;
            if (pair)
            {
                // PairLayout::entry: A and B of 0..8 with lane 1 and of 18..26 with lane 0, of 9..17 with lane 0 (A) and
                // 1 (B, but for the centre, which is not used)
                const float *at = L.Acb + cbBase / 27 * PairLayout<float>::kNode + 8 * jc;
                const bool mid = o >= 9 && o < 18;
                const int ea = mid ? o + 9 : o % 9, eb = mid ? ea : ea + 9, sa = o < 9 ? 4 : 0, sb = o < 18 ? 4 : 0;
                a = at[8 * col.n * (ea >> 2) + sa + (ea & 3)];
                b = at[8 * col.n * (eb >> 2) + sb + (eb & 3)];
            }
            else
            {
                a = L.Acb[cbBase + (int64_t)o * col.n + jc];
                b = L.Bcb[cbBase + (int64_t)o * col.n + jc];
            }
            const float2 v = ld2(L.xy, (int64_t)(uint32_t)jj);
            ax += a * v.x;
            ay += a * v.y;
            if (o == Dims<D>::CENTER) acen = a;
            else { bx += b * v.x; by += b * v.y; }
        }
    }
#pragma unroll
    for (int n = 0; n < 5; n++) h[n] = lanes_sum<D>(h[n]);
    ax = lanes_sum<D>(ax); ay = lanes_sum<D>(ay); bx = lanes_sum<D>(bx); by = lanes_sum<D>(by); acen = lanes_sum<D>(acen);
    if (!active || A != 0) return;
    const float sc = (D == 3 ? (float)g.r : 1.f) * 0.5f;
    float q[5], p0, p1;
    q[0] = h[0] * sc + acen;
    q[1] = h[1] * sc + acen;
    q[2] = 2.f * h[2] * sc;
    q[3] = 2.f * h[3] * sc + 2.f * ax - 2.f * by;
    q[4] = 2.f * h[4] * sc + 2.f * ay + 2.f * bx;
    if (relaxed(L, i) && plain_step(q, separate, p0, p1))
    {
        float2 v = ld2(L.xy, i);
        v.x += p0;
        v.y += p1;
        if (!isfinite(v.x) || !isfinite(v.y)) atomicOr(err, (unsigned int)ERR_NONFINITE);
        reinterpret_cast<float2 *>(L.xy)[i] = v;
    }
}

}  // namespace

template <int D>
int launch_gauss_sweeps(const LevelPtrs<float> &L, int iters, unsigned int *err, cudaStream_t s, int separate)
{
    const Grid<D> g(L.level);
    bool after = false;
    int n = 0;
    for (int it = 0; it < iters; it++)
        for (int c = 0; c < (1 << D); c++)
        {
            const Colour<D> col(g, c);
            const int64_t count = L.alist ? L.aoff[c + 1] - L.aoff[c] : col.n;
            n++;
            if (!count) continue;
            launch_colour(gauss_colour_kernel<D>, dim3((unsigned)((count + (kGaussThreads >> D) - 1) / (kGaussThreads >> D))), 1, kGaussThreads, 0, s,
                          after, L, col, colour_block_base<D>(g, c), L.alist ? L.alist + L.aoff[c] : nullptr, count, err, separate);
            after = true;
        }
    return n;
}
template int launch_gauss_sweeps<3>(const LevelPtrs<float> &, int, unsigned int *, cudaStream_t, int);
template int launch_gauss_sweeps<4>(const LevelPtrs<float> &, int, unsigned int *, cudaStream_t, int);

}  // namespace epr
