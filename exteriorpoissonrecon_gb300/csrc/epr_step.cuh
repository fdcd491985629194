// The node step of the paired and separate Gauss-Seidel updates and what goes with it, shared by the
// relaxation kernels of all levels.
#pragma once
#include <type_traits>

#include "epr_common.cuh"
#include "epr_df.cuh"
#include "epr_kernels.h"

namespace epr {

// Colours of a sweep follow each other as launches of a few microseconds.  Each lets the next one's blocks
// start as soon as its own have (next_may_start), which then load what no colour writes, the stencils and
// tables, and wait for the whole of it, its writes included, before they touch a coefficient
// (await_previous).  Chained that way a launch also waits for every one before: the one it waits for cannot
// end before its own wait.  Without the attribute (launch_colour's first) both do nothing.
__device__ __forceinline__ void next_may_start() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void await_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// a colour's launch of `grid` blocks, in clusters of nc (on SMs of their own where the device can).
// after: the launch before it on the stream is a colour too; the first of a sequence must follow what
// wrote the stencils in full
template <typename... P, typename... A>
void launch_colour(void (*kernel)(P...), dim3 grid, int nc, int threads, size_t smem, cudaStream_t s, bool after, A... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3((unsigned)threads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[3];
    int n = 0;
    if (nc > 1)
    {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)nc;
        attr[n].val.clusterDim.y = 1;
        attr[n++].val.clusterDim.z = 1;
        attr[n].id = cudaLaunchAttributeClusterSchedulingPolicyPreference;
        attr[n++].val.clusterSchedulingPolicyPreference = cudaClusterSchedulingPolicySpread;
    }
    if (after)
    {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n++].val.programmaticStreamSerializationAllowed = 1;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

template <typename Real>
__device__ __forceinline__ Real2<Real> ld2(const Real *xy, int64_t i)
{
    return reinterpret_cast<const Real2<Real> *>(xy)[i];
}

// a level's storage type <-> the arithmetic it computes in
template <typename Real, typename Store>
__device__ __forceinline__ Real widen(Store v)
{
    if constexpr (std::is_same<Real, Store>::value) return v;
    else return Real(v, 0.f);  // float in double-float
}
template <typename Store, typename Real>
__device__ __forceinline__ Store narrow(Real v)
{
    if constexpr (std::is_same<Real, Store>::value) return v;
    else return v.hi;  // v normalised: its rounding to float
}

// lane n's value within every group of W lanes
template <int W>
__device__ __forceinline__ float shfl_group(float v, int n) { return __shfl_sync(0xffffffffu, v, n, W); }
template <int W>
__device__ __forceinline__ double shfl_group(double v, int n) { return __shfl_sync(0xffffffffu, v, n, W); }
template <int W>
__device__ __forceinline__ df shfl_group(df v, int n) { return df(shfl_group<W>(v.hi, n), shfl_group<W>(v.lo, n)); }

// Whether the Gauss-Seidel step of node i is applied: every node of the regular grid, the active
// functions of the adaptive indexer (its colour lists hold those only, ExteriorPoisson.h:161-169)
template <typename Real>
__device__ __forceinline__ bool relaxed(const LevelPtrs<Real> &L, int64_t i)
{
    return L.status == nullptr || L.status[i] == 2;
}

// Comparisons and finiteness tests in a level's own arithmetic: a double-float tests its pair
// without converting to FP64 where the leading float decides.
template <typename Real>
__device__ __forceinline__ bool exceeds(Real v, double t)
{
    return v > (Real)t;
}
// a double-float compares by its leading float unless that is within a factor of two of t
template <>
__device__ __forceinline__ bool exceeds<df>(df v, double t)
{
    const float tf = (float)t;
    if (v.hi > 2.f * tf) return true;
    if (v.hi < 0.5f * tf) return false;
    return (double)v.hi + (double)v.lo > t;
}
template <typename Real>
__device__ __forceinline__ Real abs_value(Real v)
{
    return v < (Real)0 ? -v : v;
}
template <>
__device__ __forceinline__ df abs_value<df>(df v)
{
    return v.hi < 0.f ? -v : v;
}
template <typename Real>
__device__ __forceinline__ bool finite_value(Real v)
{
    return isfinite(v);
}
template <>
__device__ __forceinline__ bool finite_value<df>(df v)
{
    return isfinite(v.hi) && isfinite(v.lo);
}

// a b - c d; in float with the rounding errors of both products (Kahan's difference of products), since
// where the fields' gradients are nearly parallel det H is a small difference of large products
template <typename Real>
__device__ __forceinline__ Real product_difference(Real a, Real b, Real c, Real d)
{
    return a * b - c * d;
}
template <>
__device__ __forceinline__ float product_difference<float>(float a, float b, float c, float d)
{
    const float w = __fmul_rn(c, d);
    return __fadd_rn(__fmaf_rn(a, b, -w), __fmaf_rn(-c, d, w));
}

// Node step from the quadratic model q = (Q20, Q02, Q11, Q10, Q01) with H = [[2 Q20, Q11], [Q11, 2 Q02]]
// and grad = (Q10, Q01).  Paired (ExteriorPoissonSolvers.h:173-181): -H^{-1} grad / 2 when
// |det H| > 1e-20.  Separate (ExteriorPoissonSolvers.h:216-235): p0 = -grad0 / (2 H00) when
// H00 > 1e-20, then p1 = -((H10 + H01) p0 + grad1) / (2 H11) when H11 > 1e-20.
template <typename Real>
__device__ __forceinline__ bool node_step(const Real *q, int separate, Real &p0, Real &p1)
{
    Real h00 = (Real)2 * q[0], h11 = (Real)2 * q[1], h01 = q[2];
    if (separate)
    {
        p0 = 0;
        p1 = 0;
        if (exceeds<Real>(h00, 1e-20)) p0 = -((h01 + h01) * p1 + q[3]) / ((Real)2 * h00);
        if (exceeds<Real>(h11, 1e-20)) p1 = -((h01 + h01) * p0 + q[4]) / ((Real)2 * h11);
        return true;
    }
    const Real det = product_difference<Real>(h00, h11, h01, h01);
    if (!exceeds<Real>(abs_value<Real>(det), 1e-20)) return false;
    p0 = -product_difference<Real>(h11, q[3], h01, q[4]) / det / (Real)2;
    p1 = -product_difference<Real>(h00, q[4], h01, q[3]) / det / (Real)2;
    return true;
}

// node_step with the singularity tests in the level's own arithmetic
template <typename Real>
__device__ __forceinline__ bool node_step_tiny(const Real *q, int separate, Real &p0, Real &p1)
{
    Real h00 = (Real)2 * q[0], h11 = (Real)2 * q[1], h01 = q[2];
    if (separate)
    {
        p0 = 0;
        p1 = 0;
        if (exceeds<Real>(h00, 1e-20)) p0 = -((h01 + h01) * p1 + q[3]) / ((Real)2 * h00);
        if (exceeds<Real>(h11, 1e-20)) p1 = -((h01 + h01) * p0 + q[4]) / ((Real)2 * h11);
        return true;
    }
    Real det = h00 * h11 - h01 * h01;
    if (!exceeds<Real>(abs_value<Real>(det), 1e-20)) return false;
    // -H^{-1} grad / 2 with one division
    const Real m = (Real)-0.5 / det;
    p0 = (h11 * q[3] - h01 * q[4]) * m;
    p1 = (-h01 * q[3] + h00 * q[4]) * m;
    return true;
}

// Power-of-two shift that brings the largest stored magnitude |hi| of a double-float level into
// [1, 2), or 0 while it stays within [2^-8, 2^9) (or the level is zero).  The whole block calls it;
// it ends with a barrier.
__device__ __forceinline__ int df_rescale_shift(const df *v, int64_t n)
{
    __shared__ float wmax[32];
    __shared__ int shift;
    float m = 0.f;
    for (int64_t k = threadIdx.x; k < n; k += blockDim.x) m = fmaxf(m, fabsf(v[k].hi));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) wmax[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0)
    {
        float mm = 0.f;
        for (int w = 0; w < (int)((blockDim.x + 31) >> 5); w++) mm = fmaxf(mm, wmax[w]);
        const int e = mm > 0.f ? ilogbf(mm) : 0;
        shift = (mm > 0.f && (e < -8 || e > 8)) ? -e : 0;
    }
    __syncthreads();
    return shift;
}

}  // namespace epr
