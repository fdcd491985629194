// Relaxation of the small levels.  3D levels 0-3 (8, 27, 125 and 729 nodes): all sweeps of a level in one launch,
// on one block (levels 0 and 1), a cluster of eight blocks (level 2) or of 16 (level 3; eight where the device
// holds no larger one), solo and for every member of a lockstep batch; in double levels 3 and 4 by one launch per
// colour.  4D levels 0-3 in double further down.
//
// What bounds them: nothing but the dependent chain of a colour phase, thousands of times (a depth-8
// schedule has 38,400 phases on these levels, of 1 to 125 nodes).  So the work of a phase is laid out for
// the shortest chain:
//  * Every element has exactly one corner in each parity colour, so a colour's (node, element) incidences
//    are the level's 8^L elements.  They are listed with the nodes of most elements first (8, 4, 2, 1: runs
//    that never straddle a multiple of 8), so consecutive runs of incidences go to the blocks of a cluster
//    in equal shares and a node's incidences always meet in one block: one cluster barrier a phase, after
//    the new values are written into every block's replica of the coefficients.
//  * An incidence is spread over 16 lanes: one per field, wedge component and Gauss-Jacobi point, with one
//    stencil offset each.  Lanes of the two points share the work of the element's two faces, lanes of the
//    two fields the minors, and the sums over lanes halve the values with the lanes, so that a lane's
//    chain is 37 operations.  In double that count is the time: an SM sub-partition takes some 64 cycles
//    for a warp's FP64 instruction however many of its lanes are active.
//  * Double-float runs on loosely normalised pairs: sums keep the error term of the leading parts but are
//    renormalised only before a product or where they are stored, so that a chain of sums costs one
//    addition's latency each instead of thirteen operations'.  The sums that cancel most are done in full: an
//    incidence's over its lanes, the two differences of the step, the update (FullSums).
// Float levels compute in double-float, loose throughout, and store float: the arithmetic is not what their phases
// wait for, and its error not what their result shows.
//
// Error of one and of eight sweeps in double-float against 80-bit arithmetic, as a ratio to the 12-point Gauss rule
// on fully normalised pairs (geometric means over 140 systems of each level 0-3: random ones and those of built
// curves at several stages of their relaxation; standard error 0.03): 1.00, 0.96, 0.93, 1.00 at 0.80, 0.63, 1.20,
// 2.61 us a phase of a built curve's system.  All sums loose, a node's incidences one after another: 1.28, 1.22, 1.07, 1.18
// at 0.72, 0.59, 1.17, 2.45 us; the node sums in full as well: 1.00, 0.97, 0.91, 0.96 at 0.80, 0.69, 1.25, 2.71 us; every
// sum and product in full: 0.95, 0.89, 0.88, 0.95 at 1.03, 0.83, 1.61, 3.58 us.
//
// Levels 0, 1, 2, 3 of a depth-8 schedule (20,480, 10,240, 5,120 and 2,560 phases): 16.5, 9.2, 6.1 and 6.7 ms
// in double-float and 48.8, 28.3, 15.6 and 10.7 ms in double.  With the incidence on 12 Gauss points of
// one warp, fully normalised pairs and a launch per colour from level 2 on they took 42, 34, 33.5 and
// 17.7 ms, and 92, 73, 58 and 29 ms.  Four lanes per incidence (a component each) were slower wherever
// tried (double 72, 71, 38 and 24 ms; double-float level 3 on eight SMs 7.5 ms).
//
// The integrals are those of epr_element.cuh (signed corner sums, minors, the two-point Gauss-Jacobi
// rule), per component and point: with u = q - p and e = 2 m - p - q a point's share of |U|^2, |V|^2 and
// <U, V> is 7/6 u u + 1/6 e e.
#include <algorithm>
#include <cstring>
#include <type_traits>

#include <cooperative_groups.h>

#include "epr_common.cuh"
#include "epr_element.cuh"
#include "epr_kernels.h"
#include "epr_step.cuh"

namespace epr {

namespace {

namespace cg = cooperative_groups;

// ---------------------------------------------------------------------------------------------
// loose arithmetic
// ---------------------------------------------------------------------------------------------
template <typename Real>
struct Loose
{
    static __device__ __forceinline__ Real add(Real a, Real b) { return Ops<Real>::add(a, b); }
    static __device__ __forceinline__ Real sub(Real a, Real b) { return Ops<Real>::sub(a, b); }
    static __device__ __forceinline__ Real mul(Real a, Real b) { return Ops<Real>::mul(a, b); }
    static __device__ __forceinline__ Real muladd(Real a, Real b, Real c) { return Ops<Real>::fma(a, b, c); }
    static __device__ __forceinline__ Real norm(Real a) { return a; }
    static __device__ __forceinline__ Real times2(Real a) { return Ops<Real>::add(a, a); }
};
// Sums: the leading parts' error term joins the trailing parts (absolute error 2^-48 of the operands); the
// trailing part may grow to a few units of the leading one's last place until norm().  Products of
// such pairs neglect the product of the trailing parts.
template <>
struct Loose<df>
{
    static __device__ __forceinline__ df add(df a, df b)
    {
        const df s = two_sum(a.hi, b.hi);
        return df(s.hi, __fadd_rn(__fadd_rn(a.lo, b.lo), s.lo));
    }
    static __device__ __forceinline__ df sub(df a, df b) { return add(a, -b); }
    static __device__ __forceinline__ df mul(df a, df b)
    {
        const float p = __fmul_rn(a.hi, b.hi);
        float e = __fmaf_rn(a.hi, b.hi, -p);
        e = __fmaf_rn(a.hi, b.lo, e);
        return df(p, __fmaf_rn(a.lo, b.hi, e));
    }
    static __device__ __forceinline__ df muladd(df a, df b, df c) { return add(mul(a, b), c); }
    static __device__ __forceinline__ df norm(df a) { return quick_two_sum(a.hi, a.lo); }
    static __device__ __forceinline__ df times2(df a) { return df(2.f * a.hi, 2.f * a.lo); }
};

// Sums with an error relative to the result
template <typename Real>
struct FullSums
{
    static __device__ __forceinline__ Real add(Real a, Real b) { return Ops<Real>::add(a, b); }
    static __device__ __forceinline__ Real muladd(Real a, Real b, Real c) { return add(Loose<Real>::mul(a, b), c); }
};
template <>
struct FullSums<double> : Loose<double>
{
};
// Those of float levels: loose.  A schedule drives their coefficients into float's denormal numbers (level 1 at
// depth 8 ends near 1e-40), where every product is rounded to a multiple of 1.4e-45.  So the step's numerator,
// entries of the Hessian (below 1 there) times the gradient, is formed `up` times as large, and its divisor brings
// it down again.  Level 1 at depth 8 against double, geometric mean of ten inputs: 4.8e-4 (by 4: 1.05e-3, as with
// the Gauss rule in float; unscaled 4.7e-3; by 4,096: 4.2e-4).
struct FloatSums : Loose<df>
{
    static constexpr float up = 16.f;
};
// the sums of a level stored as Store
template <typename Store>
using SmallSums = typename std::conditional<std::is_same<Store, float>::value, FloatSums, FullSums<Store>>::type;
template <typename Sum, typename Real>
__device__ __forceinline__ Real scaled_up(Real v)
{
    if constexpr (std::is_same<Sum, FloatSums>::value) return df(Sum::up * v.hi, Sum::up * v.lo);
    else return v;
}
template <typename Sum, typename Real>
__device__ __forceinline__ Real scaled_down(Real v)
{
    if constexpr (std::is_same<Sum, FloatSums>::value) return df(v.hi * (1.f / Sum::up), v.lo * (1.f / Sum::up));
    else return v;
}

// -1 / (2 d): in double-float from the float reciprocal of the leading part and one Newton correction from the
// remainder
__device__ __forceinline__ df minus_half_over(df d)
{
    const float r = __frcp_rn(d.hi), m = -0.5f * r;
    const float rem = __fmaf_rn(-m, d.lo, __fmaf_rn(-m, d.hi, -0.5f));
    return quick_two_sum(m, __fmul_rn(rem, r));
}
__device__ __forceinline__ double minus_half_over(double d) { return -0.5 / d; }

// Component w (0 x, 1 y) of a node's step from q0, q1 (the model's Q20, Q02), cross = -Q11 / 2 and half the
// gradient (g0, g1): -H^{-1} grad / 2, or the separate update; false where it is not applied
template <typename Real, typename Sum = Loose<Real>>
__device__ __forceinline__ bool small_step(Real q0, Real q1, Real cross, Real g0, Real g1, int w, int separate, Real &p)
{
    using L = Loose<Real>;
    if (separate)
    {
        const Real q[5] = {q0, q1, -L::times2(cross), L::times2(g0), L::times2(g1)};
        Real p0, p1;
        node_step_tiny<Real>(q, separate, p0, p1);
        p = w ? p1 : p0;
        return true;
    }
    // det H = 4 d
    const Real d = L::norm(Sum::muladd(q0, q1, -L::mul(cross, cross)));
    const Real a = w ? q0 : q1, ga = scaled_up<Sum>(w ? g1 : g0), gb = scaled_up<Sum>(w ? g0 : g1);
    const Real n = L::norm(Sum::muladd(a, ga, L::mul(cross, gb)));
    if (!exceeds<Real>(abs_value<Real>(d), 0.25e-20)) return false;
    p = L::norm(L::mul(n, scaled_down<Sum>(minus_half_over(d))));
    return true;
}

// ---------------------------------------------------------------------------------------------
// incidence tables
// ---------------------------------------------------------------------------------------------
// entry of incidence k of a colour: node (13 bits), corner of the element at the node (3 bits), the node's
// incidences where this is its first (4 bits, else 0)
constexpr int kSmallLevels = kSmallLevels3;
__host__ __device__ constexpr int small_base(int level) { return 8 * ((ipow(8, level) - 1) / 7); }
__device__ uint32_t g_incidences[small_base(kSmallLevels)];

void host_incidences(uint32_t *out)
{
    for (int level = 0; level < kSmallLevels; level++)
    {
        const Grid<3> g(level);
        const int n1 = g.r + 1, ni = ipow(8, level);
        for (int c = 0; c < 8; c++)
        {
            const Colour<3> col(g, c);
            uint32_t *dst = out + small_base(level) + c * ni;
            for (int want = 8; want > 0; want >>= 1)
                for (int64_t j = 0; j < col.n; j++)
                {
                    int I[3], cnt = 0, corner[8];
                    col.node(j, I);
                    for (int A = 0; A < 8; A++)
                    {
                        bool ok = true;
                        for (int d = 0; d < 3; d++) { const int e = I[d] - cbit<3>(A, d); ok = ok && e >= 0 && e < g.r; }
                        if (ok) corner[cnt++] = A;
                    }
                    if (cnt != want) continue;
                    const uint32_t node = (uint32_t)((I[0] * n1 + I[1]) * n1 + I[2]);
                    for (int k = 0; k < cnt; k++) *dst++ = node | (uint32_t)corner[k] << 13 | (uint32_t)(k == 0 ? cnt : 0) << 16;
                }
        }
    }
}

// ---------------------------------------------------------------------------------------------
// one incidence's share of the node's model
// ---------------------------------------------------------------------------------------------
// signed strides of the element mirrored so that the node is its corner 0
template <int N1>
__device__ __forceinline__ void mirrored_strides(int A, int *s)
{
    s[0] = (A & 4) ? -N1 * N1 : N1 * N1;
    s[1] = (A & 2) ? -N1 : N1;
    s[2] = (A & 1) ? -1 : 1;
}

// stencil entries of the offset that leads from the node at I along corner cc of its element A, when that
// element owns the offset (the lower-numbered existing side of the axes the offset does not move along),
// else 0; b without the centre
template <typename Real, typename Store>
__device__ __forceinline__ void owned_entry(const LevelPtrs<Store> &L, int N1, int node, int A, int cc, Real &a, Real &b)
{
    const int I[3] = {node / (N1 * N1), (node / N1) % N1, node % N1};
    int first = 0, o = 13;
    const int three[3] = {9, 3, 1};
#pragma unroll
    for (int d = 0; d < 3; d++)
    {
        if (I[d] == N1 - 1) first |= 4 >> d;
        if (cc & (4 >> d)) o += (A & (4 >> d)) ? -three[d] : three[d];
    }
    const bool own = ((A ^ first) & ~cc & 7) == 0;
    a = own ? widen<Real>(L.A[(int64_t)o * L.N + node]) : (Real)0;
    b = own && cc ? widen<Real>(L.B[(int64_t)o * L.N + node]) : (Real)0;
}

template <typename Real>
__device__ __forceinline__ Real jacobi_w(int k) { return k ? (Real)Jacobi::W(1) : (Real)Jacobi::W(0); }
// weights of a point's squares u u and e e
template <typename Real>
__device__ __forceinline__ Real square_weight(int k, int e)
{
    constexpr double w0 = Jacobi::W(0) * (1.0 + Jacobi::S(0)), w1 = Jacobi::W(1) * (1.0 + Jacobi::S(1));
    if (e) return k ? (Real)(w1 / 6.0) : (Real)(w0 / 6.0);
    return k ? (Real)(w1 * 7.0 / 6.0) : (Real)(w0 * 7.0 / 6.0);
}

// Sixteen lanes per incidence: lane r = (field f = r / 8, k = r % 8); k < 6: component k / 2 at point k % 2.
// The lane forms its own field's sums on face k % 2 of the component's third axis and takes the other face
// from its neighbour, and exchanges q, p, m with the lane of the other field.  Its values are
//   v0 the square part of the own field's diagonal (with the centre of A), v1 the linear part and B column,
//   v2 the A column, v3 the cross part, and over all lanes
//   Q20 = y.v0, Q02 = x.v0, -Q11 / 2 = x.v3 + y.v3, Q10 / 2 = y.v1 + x.v2, Q01 / 2 = x.v1 + y.v2.
// (The minors of the y lanes come out with the opposite sign, which is the sign -<W, U> needs.)
template <typename Real>
struct Lane16
{
    int ap, aq, ar;       // axes P, Q, R of the lane's component
    Real co, cx;          // weights of the own and the other face: 1 + s, 1 - s or the reverse
    Real w1, w2, wl;      // weights of the squares and the linear part, 0 on lanes without a component
    Real s1, s2, sl;      // ... scaled by the level's wedge factor
    __device__ __forceinline__ void init(int r)
    {
        const int k = r & 7, comp = k >> 1, t = k & 1;
        ap = comp == 0 ? 1 : 2;
        aq = comp >= 2 ? 1 : 0;
        ar = comp == 0 ? 2 : comp == 1 ? 1 : 0;
        const Real cp = t ? (Real)(1.0 + Jacobi::S(1)) : (Real)(1.0 + Jacobi::S(0));
        const Real cm = t ? (Real)(1.0 - Jacobi::S(1)) : (Real)(1.0 - Jacobi::S(0));
        co = t ? cm : cp;
        cx = t ? cp : cm;
        w1 = comp < 3 ? square_weight<Real>(t, 0) : (Real)0;
        w2 = comp < 3 ? square_weight<Real>(t, 1) : (Real)0;
        wl = comp < 3 ? jacobi_w<Real>(t) : (Real)0;
    }
    __device__ __forceinline__ void scale(Real sc)
    {
        s1 = sc * w1;
        s2 = sc * w2;
        sl = sc * wl;
    }
};

// the lane's sum over the incidence: value 2 (k / 4) + (k / 2) % 2 of its field
template <typename Real, typename Sum, int N1>
__device__ __forceinline__ Real incidence16(const Lane16<Real> &ln, const Real *xy, int node, int A, int r, bool wedge, Real a, Real b)
{
    using L = Loose<Real>;
    const int f = r >> 3, k = r & 7;
    int s[3];
    mirrored_strides<N1>(A, s);
    const Real *own = xy + 2 * node + f;
    Real v[4];
    {
        const Real nb = own[2 * ((k & 4 ? s[0] : 0) + (k & 2 ? s[1] : 0) + (k & 1 ? s[2] : 0))];
        v[0] = k == 0 ? a : (Real)0;
        v[1] = L::mul(f ? -b : b, nb);
        v[2] = L::mul(a, nb);
        v[3] = (Real)0;
    }
    if (wedge)
    {
        const int sP = 2 * (ln.ap == 1 ? s[1] : s[2]), sQ = 2 * (ln.aq == 0 ? s[0] : s[1]), sR = 2 * (ln.ar == 2 ? s[2] : ln.ar == 1 ? s[1] : s[0]);
        const Real *c = own + (k & 1 ? sR : 0);
        const Real c00 = c[0], c01 = c[sQ], c10 = c[sP], c11 = c[sP + sQ];
        const Real u0 = L::sub(c00, c01), u1 = L::sub(c10, c11);
        const Real fq = L::norm(L::add(u0, u1)), fm = L::norm(L::sub(u0, u1));
        const Real fp = L::norm(L::add(L::sub(c00, c10), L::sub(c01, c11)));
        const Real q = L::norm(L::muladd(ln.co, fq, L::mul(ln.cx, shfl_xor_any(fq, 1))));
        const Real p = L::norm(L::muladd(ln.co, fp, L::mul(ln.cx, shfl_xor_any(fp, 1))));
        const Real m = L::norm(L::muladd(ln.co, fm, L::mul(ln.cx, shfl_xor_any(fm, 1))));
        const Real q2 = shfl_xor_any(q, 8), p2 = shfl_xor_any(p, 8), m2 = shfl_xor_any(m, 8);
        const Real W1 = L::norm(L::muladd(q, p2, -L::mul(p, q2)));
        // x lanes form WP = [m, p], y lanes WQ = [q, m]
        const Real Wo = L::norm(L::muladd(f ? q : m, f ? m2 : p2, -L::mul(f ? m : p, f ? q2 : m2)));
        const Real Wt = -shfl_xor_any(Wo, 8);
        const Real WP = f ? Wt : Wo, WQ = f ? Wo : Wt;
        const Real a1 = L::norm(L::sub(q, m)), a2 = L::norm(L::sub(m, p));
        const Real u = L::norm(L::add(a1, a2)), e = L::norm(L::sub(a2, a1));
        const Real lin = L::norm(L::muladd((Real)(1.0 / 3.0), L::norm(L::muladd(a2, WP, L::mul(a1, WQ))), L::mul(u, W1)));
        const Real us = L::norm(L::mul(ln.s1, u)), es = L::norm(L::mul(ln.s2, e));
        const Real got = shfl_xor_any(f ? u : e, 8);
        v[0] = L::muladd(es, e, L::muladd(us, u, v[0]));
        v[1] = L::muladd(ln.sl, lin, v[1]);
        v[3] = L::mul(f ? es : us, got);
    }
    // sum over the field's eight lanes, the values halved with the lanes
    const bool h4 = (k & 4) != 0, h2 = (k & 2) != 0;
    const Real t0 = Sum::add(h4 ? v[2] : v[0], shfl_xor_any(h4 ? v[0] : v[2], 4));
    const Real t1 = Sum::add(h4 ? v[3] : v[1], shfl_xor_any(h4 ? v[1] : v[3], 4));
    Real t = Sum::add(h2 ? t1 : t0, shfl_xor_any(h2 ? t0 : t1, 2));
    t = Sum::add(t, shfl_xor_any(t, 1));
    return L::norm(t);
}

// The node's step by its 16 lanes, lane r the component r % 2; x[0..3] the x lanes' values, x[4..7] the y lanes'
template <typename Real, typename Sum>
__device__ __forceinline__ bool group_step(const Real *x, int r, int separate, Real &p)
{
    using L = Loose<Real>;
    const Real cross = L::norm(L::add(x[3], x[7])), g0 = L::norm(L::add(x[5], x[2])), g1 = L::norm(L::add(x[1], x[6]));
    return small_step<Real, Sum>(x[4], x[0], cross, g0, g1, r & 1, separate, p);
}
// the group's eight values from its lanes' sums (level 0: a single incidence)
template <typename Real>
__device__ __forceinline__ void values_of_incidence(Real t, Real *x)
{
#pragma unroll
    for (int n = 0; n < 8; n++) x[n] = shfl_group<16>(t, (n >> 2) * 8 + (n & 3) * 2);
}
// ... from the sums of the node's cnt incidences in shared memory: lane r adds every second incidence of
// value r % 8 in pairs, the halves meet by a shuffle
template <typename Real>
__device__ __forceinline__ void values_of_node(const Real *part, int slot, int cnt, int r, Real *x)
{
    using L = Loose<Real>;
    Real v[4];
#pragma unroll
    for (int n = 0; n < 4; n++)
    {
        const int k = 2 * n + (r >> 3);
        v[n] = k < cnt ? part[(slot + k) * 8 + (r & 7)] : (Real)0;
    }
    Real t = L::add(L::add(v[0], v[1]), L::add(v[2], v[3]));
    t = L::norm(L::add(t, shfl_xor_any(t, 8)));
#pragma unroll
    for (int n = 0; n < 8; n++) x[n] = shfl_group<16>(t, n);
}

// ---------------------------------------------------------------------------------------------
// all sweeps of a level in one block or cluster
// ---------------------------------------------------------------------------------------------
// the arithmetic of a level stored as Store
template <typename Store>
using SmallReal = typename std::conditional<std::is_same<Store, double>::value, double, df>::type;

// NB: blocks of a level
template <typename Store, int LEVEL, int NB = (LEVEL < 2 ? 1 : 8)>
struct SmallShape
{
    using Real = SmallReal<Store>;
    static constexpr int N1 = (1 << LEVEL) + 1, NN = N1 * N1 * N1, NI = ipow(8, LEVEL);
    static constexpr int NC = NB;
    static constexpr int IPB = NI / NC;  // incidences per block and colour
    static constexpr int kThreads = IPB * 16 < 32 ? 32 : IPB * 16;
    static constexpr size_t kBytes = sizeof(Real2<Real>) * ((NN + 1) / 2 * 2) + sizeof(Real) * (2 * 64 * IPB + IPB * 8) + sizeof(uint32_t) * 8 * IPB;
};

template <typename Store, int LEVEL, int NB>
__device__ __forceinline__ void small_body(const LevelPtrs<Store> &L, int iters, unsigned int *err, int separate, int *kexp)
{
    using SH = SmallShape<Store, LEVEL, NB>;
    using Real = typename SH::Real;
    using V = Real2<Real>;
    using LA = Loose<Real>;
    using Sum = SmallSums<Store>;
    constexpr int N1 = SH::N1, NN = SH::NN, IPB = SH::IPB, NC = SH::NC;
    constexpr bool kDF = std::is_same<Store, df>::value;
    extern __shared__ __align__(16) unsigned char small_smem[];
    V *xy = reinterpret_cast<V *>(small_smem);
    Real *As = reinterpret_cast<Real *>(xy + (NN + 1) / 2 * 2), *Bs = As + 64 * IPB, *part = Bs + 64 * IPB;
    uint32_t *tab = reinterpret_cast<uint32_t *>(part + IPB * 8);
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = NC > 1 ? (int)cluster.block_rank() : 0;
    auto level_sync = [&]() {
        if constexpr (NC > 1) cluster.sync();
        else __syncthreads();
    };
    for (int k = threadIdx.x; k < NN; k += blockDim.x)
    {
        const Real2<Store> v = reinterpret_cast<const Real2<Store> *>(L.xy)[k];
        xy[k] = V{widen<Real>(v.x), widen<Real>(v.y)};
    }
    for (int k = threadIdx.x; k < 8 * IPB; k += blockDim.x)
    {
        const int c = k / IPB, slot = k - c * IPB;
        const uint32_t e = g_incidences[small_base(LEVEL) + c * SH::NI + rank * IPB + slot];
        const int node = (int)(e & 8191u);
        tab[k] = e | (L.status == nullptr || L.status[node] == 2 ? 1u << 20 : 0u);
        for (int cc = 0; cc < 8; cc++) owned_entry<Real, Store>(L, N1, node, (int)(e >> 13) & 7, cc, As[8 * k + cc], Bs[8 * k + cc]);
    }
    const int slot = (int)threadIdx.x / 16, r = (int)threadIdx.x % 16;
    const bool live = slot < IPB;
    const int at = live ? slot : 0;  // level 0: the idle half of the warp shadows the incidence
    Lane16<Real> ln;
    ln.init(r);
    int ke = kDF && kexp ? kexp[LEVEL] : 0;
    bool wedge = true;
    auto set_scale = [&]() {
        // wedge sums -> physical integrals at the level's exponent; a factor that underflows to zero
        // (coefficients below 2^-75) makes every wedge term exactly zero, so they are not formed
        Real sc = (Real)(0.5 * (1 << LEVEL) / 256.0);
        if constexpr (kDF)
        {
            sc = ldexp_df(sc, 2 * ke);
            wedge = sc.hi != 0.f;
        }
        ln.scale(sc);
    };
    set_scale();
    level_sync();  // every replica ready before any remote write
    bool pending = false;  // a cluster barrier arrived at but not yet waited for
    for (int it = 0; it < iters; it++)
    {
#pragma unroll 1
        for (int c = 0; c < 8; c++)
        {
            const uint32_t e = tab[c * IPB + at];
            const int node = (int)(e & 8191u), A = (int)(e >> 13) & 7, cnt = live ? (int)(e >> 16) & 15 : 0;
            const int own = 8 * (c * IPB + at) + (r & 7);
            const Real old = reinterpret_cast<const Real *>(xy)[2 * node + (r & 1)];  // before the first shuffle
            const Real t = incidence16<Real, Sum, N1>(ln, reinterpret_cast<const Real *>(xy), node, A, r, wedge, As[own], Bs[own]);
            Real x[8];
            if constexpr (LEVEL == 0) values_of_incidence<Real>(t, x);
            else
            {
                if (!(r & 1)) part[slot * 8 + (r >> 3) * 4 + ((r & 7) >> 1)] = t;
                __syncthreads();
                values_of_node<Real>(part, slot, cnt, r, x);
            }
            if constexpr (NC > 1)
                if (pending)
                {
                    cluster.barrier_wait();
                    pending = false;
                }
            Real p;
            if (cnt && (e >> 20 & 1u) && group_step<Real, Sum>(x, r, separate, p))
            {
                const Real cur = LA::norm(Sum::add(old, p));
                if (r < 2 && !finite_value<Real>(cur)) atomicOr(err, (unsigned int)ERR_NONFINITE);
                // lane r writes component r % 2 into replicas r / 2, r / 2 + 8
#pragma unroll
                for (int n = r >> 1; n < NC; n += 8)
                {
                    V *to = xy;
                    if constexpr (NC > 1) to = cluster.map_shared_rank(xy, (unsigned)n);
                    reinterpret_cast<Real *>(to)[2 * node + (r & 1)] = cur;
                }
            }
            level_sync();  // every replica updated before the next colour reads it
        }
        if constexpr (kDF)
            if (kexp)
            {
                // keep the stored coefficients near 1: a new power-of-two exponent after every sweep; the
                // replicas hold the same values, so every block picks the same one.  No block writes into a
                // replica before its block has rescaled it: the barrier is waited for before the next write.
                const int shift = df_rescale_shift(reinterpret_cast<const df *>(xy), 2 * NN);
                if (shift)
                {
                    df *w = reinterpret_cast<df *>(xy);
                    for (int k = threadIdx.x; k < 2 * NN; k += blockDim.x) w[k] = ldexp_df(w[k], shift);
                    ke -= shift;
                    set_scale();
                    __syncthreads();
                }
                if constexpr (NC > 1)
                {
                    cluster.barrier_arrive();
                    pending = true;
                }
            }
    }
    if constexpr (NC > 1)
        if (pending) cluster.barrier_wait();
    if (rank == 0)
    {
        for (int k = threadIdx.x; k < NN; k += blockDim.x)
            reinterpret_cast<Real2<Store> *>(L.xy)[k] = Real2<Store>{narrow<Store>(xy[k].x), narrow<Store>(xy[k].y)};
        if (kDF && kexp && threadIdx.x == 0) kexp[LEVEL] = ke;
    }
    if constexpr (NC > 1) cluster.sync();  // no block leaves while another may still address its shared memory
}

template <typename Store, int LEVEL, int NB>
__global__ void __launch_bounds__(SmallShape<Store, LEVEL, NB>::kThreads)
    small_kernel(LevelPtrs<Store> L, int iters, unsigned int *err, int separate, int *kexp)
{
    small_body<Store, LEVEL, NB>(L, iters, err, separate, kexp);
}
// one block or cluster per reconstruction of a lockstep batch
template <typename Store, int LEVEL, int NB>
__global__ void __launch_bounds__(SmallShape<Store, LEVEL, NB>::kThreads) small_batch_kernel(const BatchJob<Store> *jobs)
{
    const BatchJob<Store> &b = jobs[blockIdx.x / NB];
    small_body<Store, LEVEL, NB>(b.L, b.iters, b.err, b.separate, b.kexp);
}

// ---------------------------------------------------------------------------------------------
// one colour per launch: blocks of eight incidences (whole nodes)
// ---------------------------------------------------------------------------------------------
template <typename Store, int LEVEL>
__device__ __forceinline__ void small_colour_body(const LevelPtrs<Store> &L, int colour, unsigned int *err, int separate, const int *kexp)
{
    using SH = SmallShape<Store, LEVEL>;
    using Real = SmallReal<Store>;
    using V = Real2<Real>;
    using LA = Loose<Real>;
    using Sum = SmallSums<Store>;
    constexpr int N1 = SH::N1, NI = SH::NI;
    __shared__ Real part[8 * 8];
    __shared__ V around[8][27];  // every incidence's node with its neighbours, widened
    const int slot = (int)threadIdx.x >> 4, r = (int)threadIdx.x & 15;
    const int k0 = (int)blockIdx.x * 8 + slot;
    const bool live = k0 < NI;
    const uint32_t e = g_incidences[small_base(LEVEL) + colour * NI + (live ? k0 : 0)];
    const int node = (int)(e & 8191u), A = (int)(e >> 13) & 7, cnt = live ? (int)(e >> 16) & 15 : 0;
    Lane16<Real> ln;
    ln.init(r);
    Real sc = (Real)(0.5 * (1 << LEVEL) / 256.0);
    if constexpr (std::is_same<Store, df>::value)
        if (kexp) sc = ldexp_df(sc, 2 * kexp[LEVEL]);
    ln.scale(sc);
    Real a, b;
    owned_entry<Real, Store>(L, N1, node, A, r & 7, a, b);
    const int I[3] = {node / (N1 * N1), (node / N1) % N1, node % N1};
    await_previous();
    for (int o = r; o < 27; o += 16)
    {
        const int J[3] = {I[0] + o / 9 - 1, I[1] + (o / 3) % 3 - 1, I[2] + o % 3 - 1};
        const bool in = J[0] >= 0 && J[0] < N1 && J[1] >= 0 && J[1] < N1 && J[2] >= 0 && J[2] < N1;
        const Real2<Store> v = in ? reinterpret_cast<const Real2<Store> *>(L.xy)[(J[0] * N1 + J[1]) * N1 + J[2]] : Real2<Store>{(Store)0, (Store)0};
        around[slot][o] = V{widen<Real>(v.x), widen<Real>(v.y)};
    }
    __syncwarp();
    const Real *mine = reinterpret_cast<const Real *>(around[slot]);
    const Real t = incidence16<Real, Sum, 3>(ln, mine, 13, A, r, true, a, b);
    next_may_start();
    if (!(r & 1)) part[slot * 8 + (r >> 3) * 4 + ((r & 7) >> 1)] = t;
    __syncthreads();
    Real x[8], p;
    values_of_node<Real>(part, slot, cnt, r, x);
    if (cnt && relaxed(L, node) && group_step<Real, Sum>(x, r, separate, p) && r < 2)
    {
        const Real cur = LA::norm(Sum::add(mine[26 + r], p));
        if (!finite_value<Real>(cur)) atomicOr(err, (unsigned int)ERR_NONFINITE);
        L.xy[2 * node + r] = narrow<Store>(cur);
    }
}

template <typename Store, int LEVEL>
__global__ void __launch_bounds__(128) small_colour_kernel(LevelPtrs<Store> L, int colour, unsigned int *err, int separate, const int *kexp)
{
    small_colour_body<Store, LEVEL>(L, colour, err, separate, kexp);
}
// grid.y = reconstruction of a lockstep batch
template <typename Store, int LEVEL>
__global__ void __launch_bounds__(128) small_colour_batch_kernel(const BatchJob<Store> *jobs, int colour)
{
    const BatchJob<Store> &b = jobs[blockIdx.y];
    small_colour_body<Store, LEVEL>(b.L, colour, b.err, b.separate, b.kexp);
}

// ---------------------------------------------------------------------------------------------
// 4D levels 0-3 in double: a warp per incidence, lane = (wedge component, Gauss-Jacobi point of the two
// other axes).  The four lanes of a component form one (P, Q) face each and combine them along R and S by two
// exchanges, so a lane's chain is some 85 FP64 instructions against 850 for a lane per element, with every
// SM sub-partition on an incidence of its own.  16 incidences (a node has up to 16) go to a cluster of four
// blocks of four warps and meet in the block of the node's first one.  Level 1, with 16 incidences a colour,
// runs all sweeps on one such cluster, level 0 on one warp; levels 2 and 3 take a launch per colour, and from
// level 4 on a lane per element fills the device.
// ---------------------------------------------------------------------------------------------
constexpr int kSmallLevels4 = 4;
__host__ __device__ constexpr int small_base4(int level) { return 16 * ((ipow(16, level) - 1) / 15); }
// entry: node (13 bits), corner of the element at the node (4 bits), the node's incidences on its first (5 bits)
__device__ uint32_t g_incidences4[small_base4(kSmallLevels4)];

void host_incidences4(uint32_t *out)
{
    for (int level = 0; level < kSmallLevels4; level++)
    {
        const Grid<4> g(level);
        for (int c = 0; c < 16; c++)
        {
            const Colour<4> col(g, c);
            uint32_t *dst = out + small_base4(level) + c * ipow(16, level);
            for (int want = 16; want > 0; want >>= 1)
                for (int64_t j = 0; j < col.n; j++)
                {
                    int I[4], cnt = 0, corner[16];
                    col.node(j, I);
                    for (int A = 0; A < 16; A++)
                    {
                        bool ok = true;
                        for (int d = 0; d < 4; d++) { const int e = I[d] - cbit<4>(A, d); ok = ok && e >= 0 && e < g.r; }
                        if (ok) corner[cnt++] = A;
                    }
                    if (cnt != want) continue;
                    const uint32_t node = (uint32_t)g.node(I);
                    for (int k = 0; k < cnt; k++) *dst++ = node | (uint32_t)corner[k] << 13 | (uint32_t)(k == 0 ? cnt : 0) << 17;
                }
        }
    }
}

// owned_entry in 4D
__device__ __forceinline__ void owned_entry4(const LevelPtrs<double> &L, int n1, int node, int A, int cc, double &a, double &b)
{
    int first = 0, o = 40, rest = node, three = 1;
#pragma unroll
    for (int d = 3; d >= 0; d--)
    {
        const int bit = 8 >> d, I = rest % n1;
        rest /= n1;
        if (I == n1 - 1) first |= bit;
        if (cc & bit) o += (A & bit) ? -three : three;
        three *= 3;
    }
    const bool own = ((A ^ first) & ~cc & 15) == 0;
    a = own ? L.A[(int64_t)o * L.N + node] : 0.;
    b = own && cc ? L.B[(int64_t)o * L.N + node] : 0.;
}

struct Lane4D
{
    int bp, bq, br, bs;       // corner bits of the component's axes P, Q and the others R, S
    double coR, cxR, coS, cxS;  // weights of the own and the other face along R and S
    double s1, s2, l1, l3;    // weights of the squares and the linear part (0 on idle lanes)
    __device__ __forceinline__ void init(int lane, double sc)
    {
        const int comp = lane >> 2, i = lane & 1, j = (lane >> 1) & 1;
        const int P = comp == 0 ? 1 : comp < 3 ? 2 : 3, Q = comp == 0 ? 0 : comp < 3 ? comp - 1 : comp < 6 ? comp - 3 : 2;
        int R = 0;
        while (R == P || R == Q) R++;
        const int S = 6 - P - Q - R;
        bp = 8 >> P;
        bq = 8 >> Q;
        br = 8 >> R;
        bs = 8 >> S;
        const double cp[2] = {1.0 + Jacobi::S(0), 1.0 + Jacobi::S(1)}, cm[2] = {1.0 - Jacobi::S(0), 1.0 - Jacobi::S(1)};
        coR = i ? cm[1] : cp[0];
        cxR = i ? cp[1] : cm[0];
        coS = j ? cm[1] : cp[0];
        cxS = j ? cp[1] : cm[0];
        const double w = comp < 6 ? (i ? Jacobi::W(1) : Jacobi::W(0)) * (j ? Jacobi::W(1) : Jacobi::W(0)) * sc : 0.;
        const double wv = w * (i ? cp[1] : cp[0]) * (j ? cp[1] : cp[0]);
        s1 = wv * (7.0 / 6.0);
        s2 = wv / 6.0;
        l1 = w;
        l3 = w / 3.0;
    }
};

// the incidence's sums on every lane: v = (Q20, Q02, -Q11 / 2, Q10 / 2, Q01 / 2); at(offset) reads the pair
// that many nodes from the node, (a, b) the lane's stencil entry (corner lane % 16 on lanes 0-15)
template <typename At>
__device__ __forceinline__ void incidence4d(const Lane4D &ln, const int *stride, int A, int lane, double a, double b, At at, double *v)
{
    using O = Ops<double>;
    using V = double2;
    auto step = [&](int bits) {  // node offset along the mirrored element's edges
        int o = 0;
#pragma unroll
        for (int d = 0; d < 4; d++)
            if (bits & (8 >> d)) o += (A & (8 >> d)) ? -stride[d] : stride[d];
        return o;
    };
    {
        const V n = at(step(lane & 15));
        v[0] = v[1] = lane == 0 ? a : 0.;
        v[2] = 0.;
        v[3] = O::fma(a, n.x, -O::mul(b, n.y));
        v[4] = O::fma(a, n.y, O::mul(b, n.x));
    }
    const int base = step((lane & 1 ? ln.br : 0) | (lane & 2 ? ln.bs : 0)), sp = step(ln.bp), sq = step(ln.bq);
    const V c00 = at(base), c01 = at(base + sq), c10 = at(base + sp), c11 = at(base + sp + sq);
    const V u0 = O::sub(c00, c01), u1 = O::sub(c10, c11);
    V q = O::add(u0, u1), m = O::sub(u0, u1), p = O::add(O::sub(c00, c10), O::sub(c01, c11));
    auto other = [](V x, int o) { return V{__shfl_xor_sync(0xffffffffu, x.x, o), __shfl_xor_sync(0xffffffffu, x.y, o)}; };
    auto combine = [&](V x, double co, double cx, int o) { return O::fma(co, x, O::scale(cx, other(x, o))); };
    q = combine(combine(q, ln.coR, ln.cxR, 1), ln.coS, ln.cxS, 2);
    p = combine(combine(p, ln.coR, ln.cxR, 1), ln.coS, ln.cxS, 2);
    m = combine(combine(m, ln.coR, ln.cxR, 1), ln.coS, ln.cxS, 2);
    const double W1 = O::mul(ln.l1, minor2<double>(q, p)), WP = O::mul(ln.l3, minor2<double>(m, p)), WQ = O::mul(ln.l3, minor2<double>(q, m));
    const V a1 = O::sub(q, m), a2 = O::sub(m, p), u = O::add(a1, a2), e = O::sub(a2, a1);
    v[4] = O::fma(u.x, W1, O::fma(a1.x, WQ, O::fma(a2.x, WP, v[4])));
    v[3] = O::fma(-u.y, W1, O::fma(-a1.y, WQ, O::fma(-a2.y, WP, v[3])));
    const V us = O::scale(ln.s1, u), es = O::scale(ln.s2, e);
    v[0] = O::fma(us.y, u.y, O::fma(es.y, e.y, v[0]));
    v[1] = O::fma(us.x, u.x, O::fma(es.x, e.x, v[1]));
    v[2] = O::fma(us.x, u.y, O::mul(es.x, e.y));
    // four values halved with the lanes (lane's value: 2 (lane / 16) + (lane / 8) % 2), the fifth on every lane
    const bool h16 = (lane & 16) != 0, h8 = (lane & 8) != 0;
    double k0 = O::add(h16 ? v[2] : v[0], __shfl_xor_sync(0xffffffffu, h16 ? v[0] : v[2], 16));
    const double k1 = O::add(h16 ? v[3] : v[1], __shfl_xor_sync(0xffffffffu, h16 ? v[1] : v[3], 16));
    k0 = O::add(h8 ? k1 : k0, __shfl_xor_sync(0xffffffffu, h8 ? k0 : k1, 8));
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) k0 = O::add(k0, __shfl_xor_sync(0xffffffffu, k0, o));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[4] = O::add(v[4], __shfl_xor_sync(0xffffffffu, v[4], o));
#pragma unroll
    for (int n = 0; n < 4; n++) v[n] = __shfl_sync(0xffffffffu, k0, 8 * n);
}

// the node's values from its cnt incidences' parts: lane adds every fourth one of value lane % 8
__device__ __forceinline__ void values_of_node4(const double *part, int cnt, int lane, double *x)
{
    const int n = lane & 7;
    double t = 0.;
    if (n < 5)
        for (int k = lane >> 3; k < cnt; k += 4) t = __dadd_rn(t, part[k * 5 + n]);
    t = __dadd_rn(t, __shfl_xor_sync(0xffffffffu, t, 8));
    t = __dadd_rn(t, __shfl_xor_sync(0xffffffffu, t, 16));
#pragma unroll
    for (int k = 0; k < 5; k++) x[k] = __shfl_sync(0xffffffffu, t, k);
}

// all sweeps of level 0 (one warp) or 1 (a cluster of four blocks of four warps)
template <int LEVEL>
__global__ void __launch_bounds__(LEVEL == 0 ? 32 : 128) small4_kernel(LevelPtrs<double> L, int iters, unsigned int *err, int separate)
{
    constexpr int N1 = (1 << LEVEL) + 1, NN = N1 * N1 * N1 * N1, NI = ipow(16, LEVEL), NC = LEVEL == 0 ? 1 : 4, IPB = NI / NC;
    __shared__ double2 xy[NN];
    __shared__ double As[16][IPB][16], Bs[16][IPB][16];
    __shared__ double part[16][5];
    __shared__ uint32_t tab[16][IPB];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = NC > 1 ? (int)cluster.block_rank() : 0;
    auto level_sync = [&]() {
        if constexpr (NC > 1) cluster.sync();
        else __syncwarp();
    };
    for (int k = threadIdx.x; k < NN; k += blockDim.x) xy[k] = ld2(L.xy, k);
    for (int k = threadIdx.x; k < 16 * IPB * 16; k += blockDim.x)
    {
        const int c = k / (16 * IPB), slot = (k >> 4) % IPB, cc = k & 15;
        const uint32_t e = g_incidences4[small_base4(LEVEL) + c * NI + rank * IPB + slot];
        const int node = (int)(e & 8191u);
        owned_entry4(L, N1, node, (int)(e >> 13) & 15, cc, As[c][slot][cc], Bs[c][slot][cc]);
        if (cc == 0)
        {
            // the block of the node's first incidence, where its incidences meet
            const uint32_t *all = g_incidences4 + small_base4(LEVEL) + c * NI;
            int own = rank * IPB + slot;
            while ((all[own] >> 17 & 31u) == 0) own--;
            tab[c][slot] = e | (relaxed(L, node) ? 1u << 22 : 0u) | (uint32_t)(own / IPB) << 23;
        }
    }
    const int slot = (int)threadIdx.x >> 5, lane = (int)threadIdx.x & 31, global = rank * IPB + slot;
    const int stride[4] = {N1 * N1 * N1, N1 * N1, N1, 1};
    Lane4D ln;
    ln.init(lane, 0.5 / 4096.0);
    if constexpr (NC == 1) __syncthreads();
    else cluster.sync();  // every replica ready before any remote write
    for (int it = 0; it < iters; it++)
    {
#pragma unroll 1
        for (int c = 0; c < 16; c++)
        {
            const uint32_t e = tab[c][slot];
            const int node = (int)(e & 8191u), A = (int)(e >> 13) & 15, cnt = (int)(e >> 17) & 31;
            const double a = lane < 16 ? As[c][slot][lane & 15] : 0., b = lane < 16 ? Bs[c][slot][lane & 15] : 0.;
            const double old = reinterpret_cast<const double *>(xy)[2 * node + (lane & 1)];  // before the first shuffle
            double v[5];
            incidence4d(ln, stride, A, lane, a, b, [&](int o) { return xy[node + o]; }, v);
            if constexpr (NC > 1)
            {
                if (lane < 5)
                    cluster.map_shared_rank(&part[0][0], e >> 23 & 3u)[global * 5 + lane] =
                        lane == 0 ? v[0] : lane == 1 ? v[1] : lane == 2 ? v[2] : lane == 3 ? v[3] : v[4];
                cluster.sync();
            }
            double x[5];
            if constexpr (NC > 1) values_of_node4(part[global], cnt, lane, x);
            else
#pragma unroll
                for (int k = 0; k < 5; k++) x[k] = v[k];
            double p;
            if (cnt && (e >> 22 & 1u) && small_step<double>(x[0], x[1], x[2], x[3], x[4], lane & 1, separate, p))
            {
                const double cur = __dadd_rn(old, p);
                if (lane < 2 && !isfinite(cur)) atomicOr(err, (unsigned int)ERR_NONFINITE);
                // lane writes component lane % 2 into replica lane / 2
                if (lane < 2 * NC)
                {
                    double2 *to = xy;
                    if constexpr (NC > 1) to = cluster.map_shared_rank(xy, (unsigned)(lane >> 1));
                    reinterpret_cast<double *>(to)[2 * node + (lane & 1)] = cur;
                }
            }
            level_sync();  // every replica updated before the next colour reads it
        }
    }
    if (rank == 0)
        for (int k = threadIdx.x; k < NN; k += blockDim.x) reinterpret_cast<double2 *>(L.xy)[k] = xy[k];
    if constexpr (NC > 1) cluster.sync();  // no block leaves while another may still address its shared memory
}

// one colour of level 2 or 3: clusters of four blocks of four warps, 16 incidences each
template <int LEVEL>
__global__ void __launch_bounds__(128) small4_colour_kernel(LevelPtrs<double> L, int colour, unsigned int *err, int separate)
{
    constexpr int N1 = (1 << LEVEL) + 1, NI = ipow(16, LEVEL);
    __shared__ double part[16][5];
    cg::cluster_group cluster = cg::this_cluster();
    const int rank = (int)cluster.block_rank(), lane = (int)threadIdx.x & 31;
    const int slot = rank * 4 + ((int)threadIdx.x >> 5), first = ((int)blockIdx.x >> 2) * 16;  // of the cluster's 16 incidences
    const uint32_t *tab = g_incidences4 + small_base4(LEVEL) + colour * NI + first;
    const uint32_t e = tab[slot];
    const int node = (int)(e & 8191u), A = (int)(e >> 13) & 15, cnt = (int)(e >> 17) & 31;
    const int stride[4] = {N1 * N1 * N1, N1 * N1, N1, 1};
    Lane4D ln;
    ln.init(lane, 0.5 / 4096.0);
    double a = 0., b = 0., v[5];
    if (lane < 16) owned_entry4(L, N1, node, A, lane, a, b);
    await_previous();
    incidence4d(ln, stride, A, lane, a, b, [&](int o) { return ld2(L.xy, node + o); }, v);
    next_may_start();
    int own = slot;
    while ((tab[own] >> 17 & 31u) == 0) own--;
    cluster.sync();  // the cluster's blocks have started
    if (lane < 5)
        cluster.map_shared_rank(&part[0][0], (unsigned)(own >> 2))[slot * 5 + lane] =
            lane == 0 ? v[0] : lane == 1 ? v[1] : lane == 2 ? v[2] : lane == 3 ? v[3] : v[4];
    cluster.sync();
    double x[5], p;
    values_of_node4(part[slot], cnt, lane, x);
    if (cnt && relaxed(L, node) && lane < 2 && small_step<double>(x[0], x[1], x[2], x[3], x[4], lane, separate, p))
    {
        const double cur = __dadd_rn(L.xy[2 * (int64_t)node + lane], p);
        if (!isfinite(cur)) atomicOr(err, (unsigned int)ERR_NONFINITE);
        L.xy[2 * (int64_t)node + lane] = cur;
    }
}

template <typename F>
void with_level(int level, F &&f)
{
    if (level == 0) f(std::integral_constant<int, 0>{});
    else if (level == 1) f(std::integral_constant<int, 1>{});
    else if (level == 2) f(std::integral_constant<int, 2>{});
    else if (level == 3) f(std::integral_constant<int, 3>{});
    else f(std::integral_constant<int, 4>{});
}

// f(level, blocks) as constants for a small level.  Level 3 runs on a cluster of `blocks3` blocks, 16 or 8: 16 where
// the device can hold such a cluster (512 incidences of about 600 instructions: issue-bound, 2.7 us a colour phase
// against 4.3 on 8 blocks).  The node sums run in one order whatever the cluster size, so the results are the same
// bits.
template <typename Store, typename F>
void with_shape(int level, int blocks3, F &&f)
{
    with_level(level, [&](auto lv) {
        constexpr int LEVEL = decltype(lv)::value;
        if constexpr (small_level<Store>(LEVEL))
        {
            if constexpr (LEVEL == 3)
                if (blocks3 == 16) return f(lv, std::integral_constant<int, 16>{});
            f(lv, std::integral_constant<int, (LEVEL < 2 ? 1 : 8)>{});
        }
    });
}

template <typename Store>
cudaError_t prepare_store(int blocks3)
{
    cudaError_t err = cudaSuccess;
    auto set = [&](const void *k, cudaFuncAttribute a, int v) {
        if (err == cudaSuccess) err = cudaFuncSetAttribute(k, a, v);
    };
    auto shape = [&](int l, int blocks) {
        with_shape<Store>(l, blocks, [&](auto lv, auto nb) {
            constexpr int LEVEL = decltype(lv)::value, NB = decltype(nb)::value;
            const int bytes = (int)SmallShape<Store, LEVEL, NB>::kBytes;
            for (const void *k : {(const void *)small_kernel<Store, LEVEL, NB>, (const void *)small_batch_kernel<Store, LEVEL, NB>})
            {
                set(k, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
                if (NB > 8) set(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
            }
        });
    };
    for (int l = 0; l < kSmallLevels; l++) shape(l, 8);
    if (blocks3 == 16) shape(3, 16);
    return err;
}

bool holds_16_blocks()
{
    using SH = SmallShape<df, 3, 16>;
    const void *k = (const void *)small_kernel<df, 3, 16>;
    bool ok = cudaFuncSetAttribute(k, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
              cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SH::kBytes) == cudaSuccess;
    int clusters = 0;
    if (ok)
    {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(16, 1, 1);
        cfg.blockDim = dim3(SH::kThreads, 1, 1);
        cfg.dynamicSmemBytes = SH::kBytes;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 16;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        if (cudaOccupancyMaxActiveClusters(&clusters, k, &cfg) != cudaSuccess) clusters = 0;
    }
    cudaGetLastError();  // an unsupported query leaves no error behind
    return clusters >= 1;
}

}  // namespace

cudaError_t prepare_small_kernels(int *blocks3)
{
    static uint32_t host[small_base(kSmallLevels)];
    host_incidences(host);
    static uint32_t host4[small_base4(kSmallLevels4)];
    host_incidences4(host4);
    *blocks3 = holds_16_blocks() ? 16 : 8;
    cudaError_t e = cudaMemcpyToSymbol(g_incidences, host, sizeof(host));
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_incidences4, host4, sizeof(host4));
    if (e == cudaSuccess) e = prepare_store<float>(*blocks3);
    if (e == cudaSuccess) e = prepare_store<double>(*blocks3);
    if (e == cudaSuccess) e = prepare_store<df>(*blocks3);
    if (e != cudaSuccess) cudaGetLastError();  // reported by the caller
    return e;
}

template <typename Store>
void launch_small_level(const LevelPtrs<Store> &L, int iters, unsigned int *err, cudaStream_t s, int separate, int *kexp)
{
    with_shape<Store>(L.level, L.blocks3, [&](auto lv, auto nb) {
        constexpr int LEVEL = decltype(lv)::value, NB = decltype(nb)::value;
        using SH = SmallShape<Store, LEVEL, NB>;
        launch_colour(small_kernel<Store, LEVEL, NB>, dim3(NB), NB, SH::kThreads, SH::kBytes, s, false, L, iters, err, separate, kexp);
    });
}

template <typename Store>
void launch_small_level_batch(const BatchJob<Store> *jobs, int level, int count, int blocks3, cudaStream_t s)
{
    if (count <= 0) return;
    with_shape<Store>(level, blocks3, [&](auto lv, auto nb) {
        constexpr int LEVEL = decltype(lv)::value, NB = decltype(nb)::value;
        using SH = SmallShape<Store, LEVEL, NB>;
        launch_colour(small_batch_kernel<Store, LEVEL, NB>, dim3(NB * count), NB, SH::kThreads, SH::kBytes, s, false, jobs);
    });
}

template <typename Store>
void launch_small_colour(const LevelPtrs<Store> &L, int colour, unsigned int *err, cudaStream_t s, int separate, const int *kexp, bool after)
{
    with_level(L.level, [&](auto lv) {
        constexpr int LEVEL = decltype(lv)::value;
        if constexpr (LEVEL < 4 || std::is_same<Store, double>::value)
            launch_colour(small_colour_kernel<Store, LEVEL>, dim3((ipow(8, LEVEL) + 7) / 8), 1, 128, 0, s, after, L, colour, err, separate, kexp);
    });
}

template <typename Store>
void launch_small_colour_batch(const BatchJob<Store> *jobs, int level, int colour, int count, cudaStream_t s, bool after)
{
    for (int m0 = 0; m0 < count; m0 += 65535)
        with_level(level, [&](auto lv) {
            constexpr int LEVEL = decltype(lv)::value;
            if constexpr (LEVEL < 4 || std::is_same<Store, double>::value)
                launch_colour(small_colour_batch_kernel<Store, LEVEL>, dim3((ipow(8, LEVEL) + 7) / 8, (unsigned)std::min(65535, count - m0)), 1, 128,
                              0, s, after || m0 > 0, jobs + m0, colour);
        });
}

bool launch_small4(const LevelPtrs<double> &L, int iters, unsigned int *err, cudaStream_t s, int separate)
{
    if (L.level == 0) launch_colour(small4_kernel<0>, dim3(1), 1, 32, 0, s, false, L, iters, err, separate);
    else if (L.level == 1) launch_colour(small4_kernel<1>, dim3(4), 4, 128, 0, s, false, L, iters, err, separate);
    else return false;
    return true;
}
void launch_small4_colour(const LevelPtrs<double> &L, int colour, unsigned int *err, cudaStream_t s, int separate, bool after)
{
    if (L.level == 2) launch_colour(small4_colour_kernel<2>, dim3(64), 4, 128, 0, s, after, L, colour, err, separate);
    else launch_colour(small4_colour_kernel<3>, dim3(1024), 4, 128, 0, s, after, L, colour, err, separate);
}

#define EPR_SMALL(T)                                                                                              \
    template void launch_small_level<T>(const LevelPtrs<T> &, int, unsigned int *, cudaStream_t, int, int *);      \
    template void launch_small_level_batch<T>(const BatchJob<T> *, int, int, int, cudaStream_t);                      \
    template void launch_small_colour<T>(const LevelPtrs<T> &, int, unsigned int *, cudaStream_t, int, const int *, bool); \
    template void launch_small_colour_batch<T>(const BatchJob<T> *, int, int, int, cudaStream_t, bool);
EPR_SMALL(float)
EPR_SMALL(double)
EPR_SMALL(df)

}  // namespace epr
