// Exact element integrals of the quartic "wedge" term of the energy.
//
// On one element the fields x, y are multilinear; the 2-form
//     W(x,y)_{PQ} = (d_P y d_Q x - d_P x d_Q y) / 2         (P > Q)
// is the reference's alternating product grad x ^ grad y (Include/Hat.inl:32-37, 243-248:
// packed entry (i,j), i > j, of (v1 v2^T - v2 v1^T)/2 with v1 = grad x, v2 = grad y), and the
// fitting energy integrates its Frobenius norm (Hat.inl:358-370: the packed inner product counts
// every off-diagonal entry twice).  The reference evaluates these integrals through precomputed
// per-node stencils of 1,358 (3D) / 22,952 (4D) coefficients (Hat.products.inl:32-107).  Here
// they are integrated per element and per component, exactly, in one of two ways:
//   * the node fits of a solve's relaxation, the 3D energy and the Gauss-Newton product on signed sums of the corner
//     differences and their minors (below, "Quadratic-fit integrals");
//   * the 4D energy, the alternating system, the bi-quadratic fit (epr_mg.cu) and a caller's own float sweeps
//     (epr_gauss.cu) on a Gauss rule: component (P,Q) of W is linear in xi_P and xi_Q and quadratic in the other
//     coordinates, so the product of two such components takes 2 x 2 x 3^(D-2) points (12 in 3D, 36 in 4D), with
//     gradients by sum factorisation (corner differences along one axis, then 1-D interpolation axis by axis).
//
// All routines work in reference-element units; integrals over the physical element (side 1/r)
// are the returned sums times r^(4-D)/2, which the callers apply (a power of two: exact).
#pragma once
#include <type_traits>

#include "epr_common.cuh"
#include "epr_df.cuh"

namespace epr {

template <int D>
__host__ __device__ constexpr int cbit(int c, int d) { return (c >> (D - 1 - d)) & 1; }

// The two axes (P > Q) of packed component k, in the reference's packing order
// (k = P(P-1)/2 + Q, Hat.inl:32-37), and the remaining axes in increasing order.
template <int D, int K>
struct Component
{
    static constexpr int P = (K == 0) ? 1 : (K <= 2) ? 2 : (K <= 5) ? 3 : -1;
    static constexpr int Q = K - P * (P - 1) / 2;
    static constexpr int M = D - 2;
    // the m-th axis that is neither P nor Q (Q < P): branch-free, so that with m a constant after
    // unrolling every corner index below folds to a constant and the corner arrays the callers
    // index stay in registers
    static constexpr int other(int m)
    {
        const int a = m + (m >= Q ? 1 : 0);
        return a + (a >= P ? 1 : 0);
    }
    // corner index with the given bits on P, Q and the others (others: bit (M-1-m) of bo <-> axis other(m))
    static constexpr int corner(int bP, int bQ, int bo)
    {
        int c = bP << (D - 1 - P) | bQ << (D - 1 - Q);
        for (int m = 0; m < M; m++) c |= ((bo >> (M - 1 - m)) & 1) << (D - 1 - other(m));
        return c;
    }
};

// 1-D hat pieces at Gauss points
template <typename Real>
__device__ __forceinline__ Real hat2(int b, int g) { return b ? (Real)Gauss::X2(g) : (Real)(1.0 - Gauss::X2(g)); }
template <typename Real>
__device__ __forceinline__ Real hat3(int b, int g) { return b ? (Real)Gauss::X3(g) : (Real)(1.0 - Gauss::X3(g)); }
template <typename Real>
__host__ __device__ constexpr Real hat3c(int b, int g) { return b ? Real(Gauss::X3(g)) : Real(1.0 - Gauss::X3(g)); }

// Derivative of a multilinear corner field along axis A (the "derived" axis), tabulated at
// 2 Gauss points of axis B (the partner axis of the component) and 3 Gauss points of each other
// axis.  out[g * 3^M + go] with go enumerating the others (first other slowest).
template <int D, int K, bool AisP, typename Real>
__device__ __forceinline__ void derivative_table(const Real *f, Real *out)
{
    using Cp = Component<D, K>;
    constexpr int M = Cp::M;
    constexpr int NO = 1 << M;      // other-axis corners
    constexpr int NG = ipow(3, M);  // other-axis Gauss points
    // difference along A, indexed [bB][bo]
    Real dif[2][NO];
#pragma unroll
    for (int bB = 0; bB < 2; bB++)
#pragma unroll
        for (int bo = 0; bo < NO; bo++)
        {
            int c1 = AisP ? Cp::corner(1, bB, bo) : Cp::corner(bB, 1, bo);
            int c0 = AisP ? Cp::corner(0, bB, bo) : Cp::corner(bB, 0, bo);
            dif[bB][bo] = f[c1] - f[c0];
        }
    // interpolate along B at the 2-point rule
    Real t[2][NO];
#pragma unroll
    for (int g = 0; g < 2; g++)
#pragma unroll
        for (int bo = 0; bo < NO; bo++) t[g][bo] = hat2<Real>(0, g) * dif[0][bo] + hat2<Real>(1, g) * dif[1][bo];
    // interpolate along the others at the 3-point rule
    if constexpr (M == 1)
    {
#pragma unroll
        for (int g = 0; g < 2; g++)
#pragma unroll
            for (int go = 0; go < 3; go++) out[g * NG + go] = hat3<Real>(0, go) * t[g][0] + hat3<Real>(1, go) * t[g][1];
    }
    else
    {
#pragma unroll
        for (int g = 0; g < 2; g++)
#pragma unroll
            for (int g0 = 0; g0 < 3; g0++)
            {
                Real u0 = hat3<Real>(0, g0) * t[g][0] + hat3<Real>(1, g0) * t[g][2];  // bo = b0*2 + b1
                Real u1 = hat3<Real>(0, g0) * t[g][1] + hat3<Real>(1, g0) * t[g][3];
#pragma unroll
                for (int g1 = 0; g1 < 3; g1++) out[g * NG + g0 * 3 + g1] = hat3<Real>(0, g1) * u0 + hat3<Real>(1, g1) * u1;
            }
    }
}

template <int M>
__device__ __forceinline__ double other_weight(int go)
{
    if constexpr (M == 1) return Gauss::W3(go);
    else return Gauss::W3(go / 3) * Gauss::W3(go % 3);
}

// ---------------------------------------------------------------------------------------------
// sum over the Gauss points of |W|^2 (reference units), one component
// ---------------------------------------------------------------------------------------------
template <int D, int K, typename Real>
__device__ __forceinline__ Real component_wedge(const Real *x, const Real *y)
{
    constexpr int NG = ipow(3, D - 2);
    Real xP[2 * NG], xQ[2 * NG], yP[2 * NG], yQ[2 * NG];
    derivative_table<D, K, true>(x, xP);
    derivative_table<D, K, false>(x, xQ);
    derivative_table<D, K, true>(y, yP);
    derivative_table<D, K, false>(y, yQ);
    Real s = 0;
#pragma unroll
    for (int gp = 0; gp < 2; gp++)
#pragma unroll
        for (int gq = 0; gq < 2; gq++)
#pragma unroll
            for (int go = 0; go < NG; go++)
            {
                Real w = (Real)(Gauss::W2(gp) * Gauss::W2(gq) * other_weight<D - 2>(go));
                Real W = yP[gq * NG + go] * xQ[gp * NG + go] - xP[gq * NG + go] * yQ[gp * NG + go];
                s += w * W * W;
            }
    return s;
}

// ---------------------------------------------------------------------------------------------
// Quadratic-fit integrals of corner 0 (every node's elements are taken in the canonical
// orientation, mirrored so that the node is their corner 0: mirroring along axis d flips the sign
// of every d-derivative, and each component of W, U and V carries exactly one derivative along each
// of its two axes, so the products below keep their sign).
//
// On the reference element with t = 2 xi - 1 a field is f = sum_a m_a t^a over subsets a of the
// axes.  With the corner differences d_c = f_c - f_0 and the signed sums
//     D_a = sum_c d_c prod_{d in a} (1 - 2 c_d) = (-1)^|a| 2^D m_a      (D_a = 1 for phi_0),
// the component (P, Q) of W(x, y) is, up to the sign (-1)^|g| of each monomial t^g and a constant,
//     W = sum_{b with Q, a with P} [D_b, D_a] t^(a+b-P-Q),    [u, v] = u_x v_y - u_y v_x,
// and U, V (x or y replaced by phi_0) have D_b - D_a in the place of the minor.  So along P and Q
// only the monomials 1, t_P, t_Q survive (weights 1, 1/3, 1/3; the t_P t_Q minors cancel), and
// along every other axis U and V carry phi_0's factor (1 + s), s = -t, which all five integrals
// share: they are exact on the two-point Gauss-Jacobi rule of the weight 1 + s, where the three
// minors are those of q = D_Q + s D_QR, p = D_P + s D_PR, m = D_PQ + s D_PQR (bilinear in (s_R, s_S)
// in 4D).  In 3D the sums |U|^2, |V|^2, <U,V> need no points at all: they are one quadratic form of
// the seven D_a, diagonal in the sums and differences that permuting the axes leaves apart.
//
// Per element and node this takes about 230 multiplies and adds in 3D and 1,200 in 4D (the
// 2 x 2 x 3^(D-2)-point Gauss rule on derivative tables took 750 and 6,000); in float the (x, y)
// pairs travel on the two-wide FP32 instructions.  The corner differences are formed first, so the
// rounding is relative to the variation over the element and not to the fields' offset.
// ---------------------------------------------------------------------------------------------
template <typename Real>
struct Ops
{
    using V = Real2<Real>;
    static __device__ __forceinline__ Real add(Real a, Real b) { return a + b; }
    static __device__ __forceinline__ Real sub(Real a, Real b) { return a - b; }
    static __device__ __forceinline__ Real mul(Real a, Real b) { return a * b; }
    static __device__ __forceinline__ Real fma(Real a, Real b, Real c) { return a * b + c; }
    static __device__ __forceinline__ V add(V a, V b) { return V{a.x + b.x, a.y + b.y}; }
    static __device__ __forceinline__ V sub(V a, V b) { return V{a.x - b.x, a.y - b.y}; }
    static __device__ __forceinline__ V scale(Real s, V a) { return V{s * a.x, s * a.y}; }
    static __device__ __forceinline__ V mul(V a, V b) { return V{a.x * b.x, a.y * b.y}; }
    static __device__ __forceinline__ V fma(V a, V b, V c) { return V{a.x * b.x + c.x, a.y * b.y + c.y}; }
    static __device__ __forceinline__ V fma(Real s, V b, V c) { return V{s * b.x + c.x, s * b.y + c.y}; }
};
// every rounding explicit, so that each kernel that inlines the fit computes the same bits
template <>
struct Ops<double>
{
    using V = double2;
    static __device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
    static __device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
    static __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
    static __device__ __forceinline__ double fma(double a, double b, double c) { return __fma_rn(a, b, c); }
    static __device__ __forceinline__ V add(V a, V b) { return V{add(a.x, b.x), add(a.y, b.y)}; }
    static __device__ __forceinline__ V sub(V a, V b) { return V{sub(a.x, b.x), sub(a.y, b.y)}; }
    static __device__ __forceinline__ V scale(double s, V a) { return V{mul(s, a.x), mul(s, a.y)}; }
    static __device__ __forceinline__ V mul(V a, V b) { return V{mul(a.x, b.x), mul(a.y, b.y)}; }
    static __device__ __forceinline__ V fma(V a, V b, V c) { return V{fma(a.x, b.x, c.x), fma(a.y, b.y, c.y)}; }
    static __device__ __forceinline__ V fma(double s, V b, V c) { return V{fma(s, b.x, c.x), fma(s, b.y, c.y)}; }
};
template <>
struct Ops<float>
{
    using V = float2;
    static __device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
    static __device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }
    static __device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
    static __device__ __forceinline__ float fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
    static __device__ __forceinline__ V add(V a, V b) { return __fadd2_rn(a, b); }
    static __device__ __forceinline__ V sub(V a, V b) { return __fadd2_rn(a, make_float2(-b.x, -b.y)); }
    static __device__ __forceinline__ V mul(V a, V b) { return __fmul2_rn(a, b); }
    static __device__ __forceinline__ V fma(V a, V b, V c) { return __ffma2_rn(a, b, c); }
    static __device__ __forceinline__ V scale(float s, V a) { return __fmul2_rn(make_float2(s, s), a); }
    static __device__ __forceinline__ V fma(float s, V b, V c) { return __ffma2_rn(make_float2(s, s), b, c); }
};

// minor [u, v] = u_x v_y - u_y v_x
template <typename Real>
__device__ __forceinline__ Real minor2(const Real2<Real> &u, const Real2<Real> &v)
{
    using O = Ops<Real>;
    return O::fma(u.x, v.y, -O::mul(u.y, v.x));
}

// The two-point Gauss-Jacobi rule of the weight 1 + s on [-1, 1] (mean value): s = 1/5 -+ sqrt(6)/5.
// Exact for cubics; its first moments are 1, 1/3, 1/3, 1/5.
struct Jacobi
{
    __host__ __device__ static constexpr double S(int k) { return k == 0 ? -0.28989794855663561964 : 0.68989794855663561964; }
    __host__ __device__ static constexpr double W(int k) { return k == 0 ? 0.36391723651204561 : 0.63608276348795439; }
};

// Sums of the fit over a node's elements, unscaled: hv = (|V|^2, |U|^2), h2 = -<U, V>, and the
// parts of (<V, W>, -<U, W>) per weight of the Jacobi points (a, and m with a further 1/3).
template <int D, typename Real>
struct FitSums
{
    static constexpr int NW = D == 3 ? 2 : 3;  // distinct point weights
    Real2<Real> hv, a[NW], m[NW];
    Real h2;
    __device__ __forceinline__ void clear()
    {
        hv = Real2<Real>{(Real)0, (Real)0};
        h2 = (Real)0;
#pragma unroll
        for (int k = 0; k < NW; k++) a[k] = m[k] = Real2<Real>{(Real)0, (Real)0};
    }
    // h += (|U|^2, |V|^2, <U,V>, <W,U>, <W,V>) in reference units
    __device__ __forceinline__ void add_to(Real *h) const
    {
        using O = Ops<Real>;
        constexpr double kq = D == 3 ? 11.0 / 6.0 / 192.0 : 1.0 / 4096.0, kl = D == 3 ? 1.0 / 256.0 : 1.0 / 4096.0;
        constexpr double w[3] = {D == 3 ? Jacobi::W(0) : Jacobi::W(0) * Jacobi::W(0),
                                 D == 3 ? Jacobi::W(1) : Jacobi::W(0) * Jacobi::W(1), Jacobi::W(1) * Jacobi::W(1)};
        Real2<Real> hw = {(Real)0, (Real)0};
#pragma unroll
        for (int k = 0; k < NW; k++) hw = O::fma((Real)(w[k] * kl), O::fma((Real)(1.0 / 3.0), m[k], a[k]), hw);
        h[0] = O::fma((Real)kq, hv.y, h[0]);
        h[1] = O::fma((Real)kq, hv.x, h[1]);
        h[2] = O::fma((Real)-kq, h2, h[2]);
        h[3] = O::sub(h[3], hw.y);
        h[4] = O::add(h[4], hw.x);
    }
};

// s.a[k] += q (W1 + WQ/3) - p (W1 + WP/3), s.m[k] += m (WP - WQ): one point of <T, W> (T = (V, -U))
// with T1 = q - p, TP = m - p, TQ = q - m and the minors W1 = [q, p], WP = [m, p], WQ = [q, m]
template <int D, typename Real>
__device__ __forceinline__ void fit_point(FitSums<D, Real> &s, int k, const Real2<Real> &q, const Real2<Real> &p, const Real2<Real> &m)
{
    using O = Ops<Real>;
    const Real third = (Real)(1.0 / 3.0);
    const Real W1 = minor2<Real>(q, p), WP = minor2<Real>(m, p), WQ = minor2<Real>(q, m);
    s.a[k] = O::fma(O::fma(third, WQ, W1), q, s.a[k]);
    s.a[k] = O::fma(-O::fma(third, WP, W1), p, s.a[k]);
    s.m[k] = O::fma(O::sub(WP, WQ), m, s.m[k]);
}

// one square of the quadratic forms: hv += w z^2, h2 += w z_x z_y
template <int D, typename Real>
__device__ __forceinline__ void fit_square(FitSums<D, Real> &s, double w, const Real2<Real> &z)
{
    using O = Ops<Real>;
    const Real2<Real> wz = w == 1.0 ? z : O::scale((Real)w, z);
    s.hv = O::fma(wz, z, s.hv);
    s.h2 = O::fma(wz.x, z.y, s.h2);
}

// The signed sums of the corner differences d[c] = f_c - f_0 (d[0] unused), one axis at a time (corner
// bits: axis 0 = 4, axis 1 = 2, axis 2 = 1): D_i, E_i = D of the two other axes, Fn = - D_012
template <typename Real>
__device__ __forceinline__ void signed_sums(const Real2<Real> (&d)[8], Real2<Real> (&Dm)[3], Real2<Real> (&E)[3], Real2<Real> &Fn)
{
    using O = Ops<Real>;
    using V = Real2<Real>;
    const V s01 = O::add(d[2], d[3]), t01 = O::sub(d[2], d[3]);
    const V s10 = O::add(d[4], d[5]), t10 = O::sub(d[4], d[5]);
    const V s11 = O::add(d[6], d[7]), t11 = O::sub(d[6], d[7]);
    const V ss0 = O::add(d[1], s01), st0 = O::sub(d[1], s01);
    const V ss1 = O::add(s10, s11), st1 = O::sub(s10, s11);
    const V ts0 = O::sub(t01, d[1]), tt0 = O::add(d[1], t01);  // tt0 with the opposite sign
    const V ts1 = O::add(t10, t11), tt1 = O::sub(t10, t11);
    Dm[0] = O::sub(ss0, ss1);
    Dm[1] = O::add(st0, st1);
    Dm[2] = O::add(ts0, ts1);
    E[2] = O::sub(st0, st1);
    E[1] = O::sub(ts0, ts1);
    E[0] = O::sub(tt1, tt0);
    Fn = O::add(tt0, tt1);
}
template <typename Real>
__device__ __forceinline__ void signed_sums(const Real2<Real> (&d)[16], Real2<Real> (&D)[16])
{
    using O = Ops<Real>;
    using V = Real2<Real>;
    D[0] = V{(Real)0, (Real)0};
#pragma unroll
    for (int c = 1; c < 16; c++) D[c] = d[c];
#pragma unroll
    for (int b = 1; b < 16; b <<= 1)
#pragma unroll
        for (int c = 0; c < 16; c++)
            if (!(c & b))
            {
                const V u = D[c], v = D[c | b];
                D[c] = (c == 0 && b == 1) ? v : O::add(u, v);
                D[c | b] = (c == 0 && b == 1) ? V{-v.x, -v.y} : O::sub(u, v);
            }
}

// the fit sums of corner 0
template <typename Real>
__device__ __forceinline__ void element_fit_sums(const Real2<Real> (&d)[8], FitSums<3, Real> &s)
{
    using O = Ops<Real>;
    using V = Real2<Real>;
    V Dm[3], E[3], Fn;
    signed_sums<Real>(d, Dm, E, Fn);
    // |U|^2, |V|^2, <U,V>: squares of the axis-symmetric and the two axis-antisymmetric combinations
    {
        constexpr double kappa = 4.0 / 11.0;
        constexpr double rho = 0.25 + 1.0 / 72.0 + 0.525 + 1.0 / 30.0 - 11.0 / 9.0 * kappa * kappa;
        const V d01 = O::add(Dm[0], Dm[1]), e01 = O::add(E[0], E[1]);
        const V pE = O::sub(E[0], E[1]), qE = O::fma((Real)-2.0, E[2], e01);
        const V sD = O::add(d01, Dm[2]), sE = O::add(e01, E[2]);
        fit_square<3, Real>(s, 1.0, O::fma((Real)-kappa, pE, O::sub(Dm[0], Dm[1])));
        fit_square<3, Real>(s, 1.0 / 3.0, O::fma((Real)-kappa, qE, O::fma((Real)-2.0, Dm[2], d01)));
        fit_square<3, Real>(s, rho * 9.0 / 11.0, pE);
        fit_square<3, Real>(s, rho * 3.0 / 11.0, qE);
        fit_square<3, Real>(s, 4.0 / 33.0, O::fma((Real)1.5, Fn, O::fma((Real)-0.5, sE, sD)));
        fit_square<3, Real>(s, 1.0 / 55.0, O::fma((Real)3.0, Fn, sE));
    }
    // <V,W>, -<U,W> at the two points of the axis that is neither P nor Q
#pragma unroll
    for (int k = 0; k < 2; k++)
    {
        const Real t = (Real)Jacobi::S(k);
#pragma unroll
        for (int P = 1; P < 3; P++)
#pragma unroll
            for (int Q = 0; Q < P; Q++)
                fit_point<3, Real>(s, k, O::fma(t, E[P], Dm[Q]), O::fma(t, E[Q], Dm[P]), O::fma(-t, Fn, E[3 - P - Q]));
    }
}

template <typename Real>
__device__ __forceinline__ void element_fit_sums(const Real2<Real> (&d)[16], FitSums<4, Real> &s)
{
    using O = Ops<Real>;
    using V = Real2<Real>;
    V D[16];
    signed_sums<Real>(d, D);
#pragma unroll
    for (int P = 1; P < 4; P++)
#pragma unroll
        for (int Q = 0; Q < P; Q++)
        {
            constexpr int ax[4] = {8, 4, 2, 1};
            const int R = Q > 0 ? 0 : (P > 1 ? 1 : 2), S = 6 - P - Q - R;
            const int p = ax[P], q = ax[Q], r = ax[R], t = ax[S];
#pragma unroll
            for (int i = 0; i < 2; i++)
            {
                const Real si = (Real)Jacobi::S(i);
                const V q0 = O::fma(si, D[q | r], D[q]), q1 = O::fma(si, D[q | r | t], D[q | t]);
                const V p0 = O::fma(si, D[p | r], D[p]), p1 = O::fma(si, D[p | r | t], D[p | t]);
                const V m0 = O::fma(si, D[p | q | r], D[p | q]), m1 = O::fma(si, D[p | q | r | t], D[p | q | t]);
#pragma unroll
                for (int j = 0; j < 2; j++)
                {
                    const Real sj = (Real)Jacobi::S(j);
                    const V Vq = O::fma(sj, q1, q0), Vp = O::fma(sj, p1, p0), Vm = O::fma(sj, m1, m0);
                    fit_point<4, Real>(s, i + j, Vq, Vp, Vm);
                    // |T1|^2 + (|TP|^2 + |TQ|^2) / 3 = 7/6 |q - p|^2 + 1/6 |2 m - p - q|^2
                    const double wv = Jacobi::W(i) * Jacobi::W(j) * (1.0 + Jacobi::S(i)) * (1.0 + Jacobi::S(j));
                    fit_square<4, Real>(s, wv * 7.0 / 6.0, O::sub(Vq, Vp));
                    fit_square<4, Real>(s, wv / 6.0, O::fma((Real)-2.0, Vm, O::add(Vp, Vq)));
                }
            }
        }
}

// sum over the Gauss points of |W|^2 (reference units).  3D: along the axis R that is neither P nor Q the
// coefficient of each of the monomials 1, t_P, t_Q is a quadratic W0 + W1 t + W2 t^2 of minors of the signed
// sums, whose mean square is (W0 + W2 / 3)^2 + W1^2 / 3 + 4/45 W2^2: the 21 minors once, 150 multiplies and
// adds an element (432 on the 12-point rule).
template <int D, typename Real>
__device__ __forceinline__ Real element_wedge(const Real2<Real> (&f)[1 << D])
{
    using O = Ops<Real>;
    using V = Real2<Real>;
    if constexpr (D == 3)
    {
        V d[8], Dm[3], E[3], Fn;
#pragma unroll
        for (int c = 1; c < 8; c++) d[c] = O::sub(f[c], f[0]);
        signed_sums<Real>(d, Dm, E, Fn);
        Real DE[3][3], DF[3], EF[3];
#pragma unroll
        for (int i = 0; i < 3; i++)
        {
#pragma unroll
            for (int j = 0; j < 3; j++) DE[i][j] = minor2<Real>(Dm[i], E[j]);
            DF[i] = minor2<Real>(Dm[i], Fn);
            EF[i] = minor2<Real>(E[i], Fn);
        }
        const Real third = (Real)(1.0 / 3.0);
        // mean squares of the monomial 1 (a) and of t_P, t_Q (b), by the three terms above
        Real a0 = 0, a1 = 0, a2 = 0, b0 = 0, b1 = 0, b2 = 0;
#pragma unroll
        for (int P = 1; P < 3; P++)
#pragma unroll
            for (int Q = 0; Q < P; Q++)
            {
                const int R = 3 - P - Q;
                auto add = [&](Real W0, Real W1, Real W2, Real &s0, Real &s1, Real &s2) {
                    const Real m = O::fma(third, W2, W0);
                    s0 = O::fma(m, m, s0);
                    s1 = O::fma(W1, W1, s1);
                    s2 = O::fma(W2, W2, s2);
                };
                const Real EPR = minor2<Real>(E[P], E[R]), EQR = minor2<Real>(E[Q], E[R]);
                // [D_Q + E_P t, D_P + E_Q t], [E_R + F t, D_P + E_Q t], [D_Q + E_P t, E_R + F t] with F = -Fn
                add(minor2<Real>(Dm[Q], Dm[P]), O::sub(DE[Q][Q], DE[P][P]), minor2<Real>(E[P], E[Q]), a0, a1, a2);
                add(-DE[P][R], O::sub(DF[P], EQR), EF[Q], b0, b1, b2);
                add(DE[Q][R], O::sub(EPR, DF[Q]), -EF[P], b0, b1, b2);
            }
        const Real p0 = O::fma(third, b0, a0), p1 = O::fma(third, b1, a1), p2 = O::fma(third, b2, a2);
        // each W carries 1/16 of the signed sums' minors
        return O::mul((Real)(1.0 / 256.0), O::fma((Real)(4.0 / 45.0), p2, O::fma(third, p1, p0)));
    }
    else
    {
        Real x[16], y[16];
#pragma unroll
        for (int c = 0; c < 16; c++) { x[c] = f[c].x; y[c] = f[c].y; }
        Real s = component_wedge<D, 0>(x, y) + component_wedge<D, 1>(x, y) + component_wedge<D, 2>(x, y);
        s += component_wedge<D, 3>(x, y) + component_wedge<D, 4>(x, y) + component_wedge<D, 5>(x, y);
        return s;
    }
}

// ---------------------------------------------------------------------------------------------
// Gauss-Newton products for corner 0 (canonical orientation): J = W(dx, y) + W(x, dy), acc += the sums
// (<J, V>, -<J, U>) in units of 4^D (the fit's linear part with J in the place of W)
// ---------------------------------------------------------------------------------------------
template <typename Real>
__device__ __forceinline__ Real minor_derivative(const Real2<Real> &u, const Real2<Real> &v, const Real2<Real> &du, const Real2<Real> &dv)
{
    using O = Ops<Real>;
    return O::sub(O::fma(du.x, v.y, O::mul(u.x, dv.y)), O::fma(du.y, v.x, O::mul(u.y, dv.x)));
}
template <typename Real>
__device__ __forceinline__ void gn_point(Real w, const Real2<Real> &q, const Real2<Real> &p, const Real2<Real> &m, const Real2<Real> &dq,
                                         const Real2<Real> &dp, const Real2<Real> &dm, Real2<Real> &acc)
{
    using O = Ops<Real>;
    const Real third = (Real)(1.0 / 3.0);
    const Real J1 = O::mul(w, minor_derivative<Real>(q, p, dq, dp));
    const Real JP = O::mul((Real)(w * third), minor_derivative<Real>(m, p, dm, dp)), JQ = O::mul((Real)(w * third), minor_derivative<Real>(q, m, dq, dm));
    acc = O::fma(J1, O::sub(q, p), acc);
    acc = O::fma(JQ, O::sub(q, m), acc);
    acc = O::fma(JP, O::sub(m, p), acc);
}
template <typename Real>
__device__ __forceinline__ void element_gn(const Real2<Real> (&d)[8], const Real2<Real> (&dd)[8], Real2<Real> &acc)
{
    using O = Ops<Real>;
    using V = Real2<Real>;
    V D[3], E[3], F, dD[3], dE[3], dF;
    signed_sums<Real>(d, D, E, F);
    signed_sums<Real>(dd, dD, dE, dF);
#pragma unroll
    for (int k = 0; k < 2; k++)
    {
        const Real t = (Real)Jacobi::S(k);
#pragma unroll
        for (int P = 1; P < 3; P++)
#pragma unroll
            for (int Q = 0; Q < P; Q++)
            {
                const int R = 3 - P - Q;
                gn_point<Real>((Real)Jacobi::W(k), O::fma(t, E[P], D[Q]), O::fma(t, E[Q], D[P]), O::fma(-t, F, E[R]), O::fma(t, dE[P], dD[Q]),
                               O::fma(t, dE[Q], dD[P]), O::fma(-t, dF, dE[R]), acc);
            }
    }
}
template <typename Real>
__device__ __forceinline__ void element_gn(const Real2<Real> (&d)[16], const Real2<Real> (&dd)[16], Real2<Real> &acc)
{
    using O = Ops<Real>;
    using V = Real2<Real>;
    V D[16], dD[16];
    signed_sums<Real>(d, D);
    signed_sums<Real>(dd, dD);
#pragma unroll
    for (int P = 1; P < 4; P++)
#pragma unroll
        for (int Q = 0; Q < P; Q++)
        {
            constexpr int ax[4] = {8, 4, 2, 1};
            const int R = Q > 0 ? 0 : (P > 1 ? 1 : 2), S = 6 - P - Q - R;
            const int p = ax[P], q = ax[Q], r = ax[R], t = ax[S];
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 2; j++)
                {
                    const Real si = (Real)Jacobi::S(i), sj = (Real)Jacobi::S(j);
                    auto at = [&](const V *T, int a) { return O::fma(sj, O::fma(si, T[a | r | t], T[a | t]), O::fma(si, T[a | r], T[a])); };
                    gn_point<Real>((Real)(Jacobi::W(i) * Jacobi::W(j)), at(D, q), at(D, p), at(D, p | q), at(dD, q), at(dD, p), at(dD, p | q), acc);
                }
        }
}

}  // namespace epr
