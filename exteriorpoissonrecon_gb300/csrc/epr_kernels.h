// Host-side declarations of the CUDA launchers (instantiated for Dim 3/4 and double/float in
// epr_solve.cu and epr_setup.cu).  Only plain pointers and sizes cross this header.
#pragma once
#include <cstddef>
#include <cstdint>
#include <type_traits>
#include <cuda_runtime.h>

#include "epr_df.cuh"

namespace epr {

// One level of the hierarchy as the solve kernels see it.
template <typename Real>
struct LevelPtrs
{
    int level = 0;
    int64_t N = 0;            // nodes
    Real *xy = nullptr;       // 2N interleaved (x, y)
    const Real *A = nullptr;  // 3^Dim * N column stencil of R + dWeight K (offset-major)
    const Real *B = nullptr;  // 3^Dim * N column stencil of the frame constraint
    // double stencils, where a level keeps no natural copy in Real (A, B null: float pair levels, whose
    // relaxation reads the pair layout; the other float kernels round the entries as they load them)
    const double *A64 = nullptr;
    const double *B64 = nullptr;
    const Real *Acb = nullptr;  // optional colour-blocked copies of A and B (colour_block_base); on pair
    const Real *Bcb = nullptr;  // levels both in Acb (PairLayout)
    // adaptive indexer: per node 0 (no function), 1 (indexed, held fixed), 2 (active); the
    // Gauss-Seidel kernels update active nodes only.  Null for the regular grid (all active).
    const uint8_t *status = nullptr;
    // adaptive indexer: the active nodes of every parity colour as colour-local indices (the
    // Colour::node order), colour c at alist[aoff[c] .. aoff[c+1]); the large levels relax these
    // lists instead of the whole colour.  Null for the regular grid.
    const int *alist = nullptr;
    int aoff[17] = {0};
    int blocks3 = 8;  // blocks of level 3's cluster, 8 or 16 (the same bits)
};

// Scratch for deterministic two-pass reductions
struct Reduce
{
    double *partial = nullptr;  // >= kMaxBlocks * 4 doubles
    double *out = nullptr;      // >= 4 doubles
    static constexpr int kMaxBlocks = 4096;
};

template <int D, typename Real>
void launch_energy(const LevelPtrs<Real> &L, const Real *xy, const Reduce &red, cudaStream_t s);
// red.out[0] = sum_i (dE/dx_i)^2 + (dE/dy_i)^2
template <int D, typename Real>
void launch_grad_norm(const LevelPtrs<Real> &L, const Real *xy, const Reduce &red, cudaStream_t s);
// writes N x 5 doubles (Q20, Q02, Q11, Q10, Q01)
template <int D, typename Real>
void launch_quadfit(const LevelPtrs<Real> &L, const Real *xy, double *out, cudaStream_t s);
// separate != 0: the reference's SeparateGaussSeidelSolve update (x first, then y with the new x).  after: the
// launch before it on the stream is another colour of the level (launch_colour).  Returns whether it launched.
template <int D, typename Real>
bool launch_gs_colour(const LevelPtrs<Real> &L, int colour, unsigned int *err, cudaStream_t s, int separate = 0, bool after = false);
// double-float levels: pairs stored as x 2^-k with k = kexp[level] (epr_df.cuh)
void launch_df_push(const double *in, df *out, int64_t n, int *kexp, int level, cudaStream_t s);
void launch_df_pull(const df *in, double *out, int64_t n, const int *kexp, int level, cudaStream_t s);
void launch_d2df(const double *in, df *out, int64_t n, cudaStream_t s);
// The sweeps of a caller that runs them by itself, in float, on levels of more than 729 nodes (gauss_level): the Gauss
// rule's arithmetic, whose bits they keep (epr_gauss.cu).  The smaller levels run a solve's kernels, which are
// nearer to 64 bits; the nodes where the rules differ visibly, one in 10^5, are not found there.
template <int D>
bool gauss_level(int level) { return level >= (D == 3 ? 4 : 3); }
template <int D>
int launch_gauss_sweeps(const LevelPtrs<float> &L, int iters, unsigned int *err, cudaStream_t s, int separate);
// iters full sweeps (all 2^D colours in order) as a solve runs them; the small levels run all sweeps in one
// launch, larger ones launch one kernel per colour.  Returns the number of kernels launched.
template <int D, typename Real>
int launch_gs_sweeps(const LevelPtrs<Real> &L, int iters, unsigned int *err, cudaStream_t s, int separate = 0);

// The small 3D levels (epr_small.cu).  All sweeps in one launch: levels 0-2, and level 3 but in double;
// levels 3 and 4 in double by its per-colour launches (a lane per element leaves three of four FP64
// units without a warp there: level 4 14.5 us a colour against 9.7).
constexpr int kSmallLevels3 = 5;
template <typename Real>
constexpr bool small_level(int level) { return level < 3 || (level == 3 && !std::is_same<Real, double>::value); }
template <typename Real>
constexpr bool small_colour_level(int level) { return level < 4 || (level == 4 && std::is_same<Real, double>::value); }
// 4D in double: levels 0 and 1 in one launch, 2 and 3 by per-colour launches of the same lanes
constexpr bool small4_colour_level(int level) { return level == 2 || level == 3; }
bool launch_small4(const LevelPtrs<double> &L, int iters, unsigned int *err, cudaStream_t s, int separate);  // false: not a level it takes
void launch_small4_colour(const LevelPtrs<double> &L, int colour, unsigned int *err, cudaStream_t s, int separate, bool after);
// blocks3: the largest cluster of level 3 that the device holds, 16 or 8 blocks
cudaError_t prepare_small_kernels(int *blocks3);
template <typename Real>
void launch_small_level(const LevelPtrs<Real> &L, int iters, unsigned int *err, cudaStream_t s, int separate, int *kexp);
template <typename Real>
void launch_small_colour(const LevelPtrs<Real> &L, int colour, unsigned int *err, cudaStream_t s, int separate, const int *kexp,
                         bool after = false);
// sets the kernels' shared-memory limits and uploads the small levels' tables (once per device, before any
// stream capture)
cudaError_t prepare_gs_kernels(int *blocks3);
template <int D, typename Real>
void launch_gn_matvec(const LevelPtrs<Real> &L, const Real *xy, const Real *dxy, Real *out, cudaStream_t s);
// fine (2 N_f) = P coarse (2 N_c), pairs; add != 0 accumulates
template <int D, typename Real>
// fineStatus (adaptive indexer): fine nodes without a function (status 0) stay zero
void launch_prolong(int coarseLevel, const Real *coarse, Real *fine, int add, cudaStream_t s,
                    const uint8_t *fineStatus = nullptr);
// out = fine - P coarse, pairs in double (status as above: P coarse is zero where no function is)
template <int D>
void launch_hierarchical(int coarseLevel, const double *coarse, const double *fine, double *out, cudaStream_t s, const uint8_t *fineStatus);
// coarse = P^T fine, pairs
template <int D, typename Real>
void launch_restrict(int coarseLevel, const Real *fine, Real *coarse, cudaStream_t s);

// coarse = P^T fine P of a column stencil (offset-major, double), fine level -> fineLevel - 1; scratch holds
// galerkin_scratch(fineLevel) doubles (enough for every coarser level too)
template <int D>
size_t galerkin_scratch(int fineLevel);
template <int D>
void launch_galerkin(int fineLevel, const double *Mf, double *Mc, double *scratch, cudaStream_t s);

// colour-blocked copy (Real) of a natural offset-major double stencil of `level`
template <int D, typename Real>
void launch_to_colour_blocks(int level, const double *M, Real *out, cudaStream_t s);

// elementwise helpers
template <typename Real>
void launch_scale(Real *v, int64_t n, double s, cudaStream_t st);
template <typename Real>
void launch_axpy(Real *y, const Real *x, int64_t n, double a, cudaStream_t st);
void launch_convert_d2f(const double *in, float *out, int64_t n, cudaStream_t st);
// interleaved (x, y) pairs <-> two planar arrays
void launch_split_pairs(const double *xy, double *x, double *y, int64_t n, cudaStream_t st);
void launch_merge_pairs(const double *x, const double *y, double *xy, int64_t n, cudaStream_t st);
void launch_convert_f2d(const float *in, double *out, int64_t n, cudaStream_t st);

// ---------------------------------------------------------------------------------------------
// Lockstep batches (3D): one launch relaxes the same level and colour of many reconstructions,
// each with its own arrays, sweep count and error flag.  Every reconstruction's nodes see exactly
// the arithmetic of its own solve's kernels for that level, so the batch gives each one its own
// solve's bits.
// ---------------------------------------------------------------------------------------------
template <typename Real>
struct BatchJob
{
    LevelPtrs<Real> L;
    unsigned int *err = nullptr;
    int *kexp = nullptr;  // the reconstruction's exponent table (double-float levels), else null
    int iters = 0;        // sweeps of this level
    int separate = 0;
};
// a level-to-level transfer of one reconstruction: src and dst arrays of the transfer's types
struct XferJob
{
    const void *src = nullptr;
    void *dst = nullptr;
    int *kexp = nullptr;
};
// the block shapes a batch may pick for the large levels' colour kernels (none changes any node's
// arithmetic): threads per block.  Level 3 in double has one shape.
constexpr int kLanesTiles[3] = {64, 128, 256};
constexpr int kDefaultTile = 1;  // index into the table: the solo solve's shape (128 threads)
// all sweeps of a small level of `count` reconstructions (jobs[0..count))
template <typename Real>
void launch_small_level_batch(const BatchJob<Real> *jobs, int level, int count, int blocks3, cudaStream_t s);
// one colour of a level of jobs[0..count)
template <typename Real>
void launch_small_colour_batch(const BatchJob<Real> *jobs, int level, int colour, int count, cudaStream_t s, bool after);
template <typename Real>
bool launch_colour_batch(const BatchJob<Real> *jobs, int level, int colour, int count, int tile, cudaStream_t s, bool after);
// fine += P coarse for jobs[0..count) (src coarse, dst fine)
template <typename Real>
void launch_prolong_add_batch(const XferJob *jobs, int coarseLevel, int count, cudaStream_t s);
// elementwise n values: float -> double, double -> float, double-float -> double (the exponent of
// `level`), double -> double-float (a new exponent for `level`, one block per reconstruction)
void launch_f2d_batch(const XferJob *jobs, int64_t n, int count, cudaStream_t s);
void launch_d2f_batch(const XferJob *jobs, int64_t n, int count, cudaStream_t s);
void launch_df_pull_batch(const XferJob *jobs, int64_t n, int level, int count, cudaStream_t s);
void launch_df_push_batch(const XferJob *jobs, int64_t n, int level, int count, cudaStream_t s);

}  // namespace epr
