// pbf_solver.cu — solver iterations, scatter-back, finalize and foam of the
// single-scene PBF step for sm_100a: one thread per sorted slot, the work of
// each slot in pbf_items.cuh.
//
// Replaces densityLambdaSorted (engine/shaders/Constraints.metal:82-131),
// applyDeltaSorted (:140-199), sphereCollision (:262-277),
// scatterPositionsToOriginal (:205-213), finalizeStep (:305-353) and
// computeFoam (:287-299), dispatched by engine/src/Engine.cpp:728-810.
//
//   lambda, first  sorted_a (absolute x, y, z) -> sorted_b (l, lambda), scell
//   delta          sorted_b (l, lambda) -> sorted_a (l')
//   lambda         sorted_a (l) -> sorted_b (l, lambda)
//   last delta     also scatter-back + finalize + foam into original order.
#include "pbf_team.cuh"

namespace mpb {
namespace {

inline uint32_t cdiv(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

// Launch shape of the solver kernels, measured on the 1,003,520-particle dam
// break: blocks of 128 threads (64 and 256 are within 0.5%), and at least 8 of
// them per SM, which caps registers at 64: 1285 us per step (with 9 blocks, 56
// registers, the lambda passes cost a step 1.5% more and the delta passes 3.5%;
// fewer blocks 10% and more).
#ifndef MPB_SOLVER_BLOCK
#define MPB_SOLVER_BLOCK 128
#endif
constexpr uint32_t kSB = MPB_SOLVER_BLOCK;
#ifndef MPB_LAMBDA_MIN_BLOCKS
#define MPB_LAMBDA_MIN_BLOCKS 8
#endif
#ifndef MPB_DELTA_MIN_BLOCKS
#define MPB_DELTA_MIN_BLOCKS 8
#endif
#ifndef MPB_DELTA_MID_MIN_BLOCKS
#define MPB_DELTA_MID_MIN_BLOCKS 8
#endif

template <bool LAST>
__global__ void __launch_bounds__(kSB, MPB_LAMBDA_MIN_BLOCKS)
k_lambda_first(StepConsts c, const float4* __restrict__ cur, const uint32_t* __restrict__ qpos, float4* __restrict__ nxt,
               uint32_t* __restrict__ scell, const uint32_t* __restrict__ cstart,
               const uint32_t* __restrict__ sidx, float* __restrict__ lambdas,
               uint32_t* __restrict__ ncount, RowMasks rm) {
    __shared__ uint2 queue[kQueue * kSB];
    const uint32_t s = blockIdx.x * kSB + threadIdx.x;
    if (s < c.n)
        lambda_first_item<LAST, true, kSB>(c, c, s, cur, qpos, nxt, scell, cstart, sidx, lambdas, ncount, rm, queue);
}

template <bool LAST>
__global__ void __launch_bounds__(kSB, MPB_LAMBDA_MIN_BLOCKS)
k_lambda(StepConsts c, const float4* __restrict__ cur, const uint32_t* __restrict__ qpos, float4* __restrict__ nxt,
         const uint32_t* __restrict__ scell, const uint32_t* __restrict__ cstart,
         const uint32_t* __restrict__ sidx, float* __restrict__ lambdas, RowMasks rm) {
    __shared__ uint2 queue[kQueue * kSB];
    const uint32_t s = blockIdx.x * kSB + threadIdx.x;
    if (s < c.n) lambda_item<LAST, true, kSB>(c, c, s, cur, qpos, nxt, scell, cstart, sidx, lambdas, rm, queue);
}

// SN = 4: the reference's s_corr exponent, fixed at compile time (the host
// launches this instance when scorr_n == 4); SN = 0 reads it from c.
template <bool LAST, uint32_t SN>
__global__ void __launch_bounds__(kSB, LAST ? MPB_DELTA_MIN_BLOCKS : MPB_DELTA_MID_MIN_BLOCKS)
k_delta(StepConsts c, const float4* __restrict__ src, float4* __restrict__ dst, uint32_t* __restrict__ qpos,
        const float* __restrict__ xa,
        const uint32_t* __restrict__ scell, const uint32_t* __restrict__ cstart,
        const uint32_t* __restrict__ sidx, const SphereState* __restrict__ sphere,
        float4* __restrict__ pos, float4* __restrict__ vel, const float4* __restrict__ prev,
        const uint32_t* __restrict__ ncount, float* __restrict__ foam, uint32_t* err, RowMasks rm) {
    __shared__ uint2 queue[kQueue * kSB];
    const uint32_t s = blockIdx.x * kSB + threadIdx.x;
    if (s < c.n)
        delta_item<LAST, SN, true, kSB>(c, c, s, src, dst, qpos, xa, scell, cstart, sidx, sphere, pos, vel, prev, ncount,
                                  foam, err, rm, nullptr, queue);
}

// The same with a team of G lanes per slot (pbf_team.cuh).
constexpr uint32_t kTB = 64;

template <bool LAST, uint32_t G>
__global__ void __launch_bounds__(kTB)
k_lambda_first_team(StepConsts c, const float4* __restrict__ cur, const uint32_t* __restrict__ qpos,
                    float4* __restrict__ nxt, uint32_t* __restrict__ scell, const uint32_t* __restrict__ cstart,
                    const uint32_t* __restrict__ sidx, float* __restrict__ lambdas,
                    uint32_t* __restrict__ ncount, RowMasks rm) {
    __shared__ TeamBuf bufs[kTB / G];
    const uint32_t s = (blockIdx.x * kTB + threadIdx.x) / G;
    if (s < c.n)
        team_lambda_first<LAST, true, G>(c, s, cur, qpos, nxt, scell, cstart, sidx, lambdas, ncount, rm, bufs);
}

template <bool LAST, uint32_t G>
__global__ void __launch_bounds__(kTB)
k_lambda_team(StepConsts c, const float4* __restrict__ cur, const uint32_t* __restrict__ qpos,
              float4* __restrict__ nxt, const uint32_t* __restrict__ scell, const uint32_t* __restrict__ cstart,
              const uint32_t* __restrict__ sidx, float* __restrict__ lambdas, RowMasks rm) {
    __shared__ TeamBuf bufs[kTB / G];
    const uint32_t s = (blockIdx.x * kTB + threadIdx.x) / G;
    if (s < c.n) team_lambda<LAST, true, G>(c, s, cur, qpos, nxt, scell, cstart, sidx, lambdas, rm, bufs);
}

template <bool LAST, uint32_t SN, uint32_t G>
__global__ void __launch_bounds__(kTB)
k_delta_team(StepConsts c, const float4* __restrict__ src, float4* __restrict__ dst, uint32_t* __restrict__ qpos,
             const float* __restrict__ xa, const uint32_t* __restrict__ scell,
             const uint32_t* __restrict__ cstart, const uint32_t* __restrict__ sidx,
             const SphereState* __restrict__ sphere, float4* __restrict__ pos, float4* __restrict__ vel,
             const float4* __restrict__ prev, const uint32_t* __restrict__ ncount, float* __restrict__ foam,
             uint32_t* err, RowMasks rm) {
    __shared__ TeamBuf bufs[kTB / G];
    const uint32_t s = (blockIdx.x * kTB + threadIdx.x) / G;
    if (s < c.n)
        team_delta<LAST, SN, true, G>(c, s, src, dst, qpos, xa, scell, cstart, sidx, sphere, pos, vel, prev, ncount,
                                foam, err, rm, nullptr, bufs);
}

template <uint32_t G, bool LAST>
void launch_lambda(const StepConsts& c, const DevState& d, bool first, const RowMasks& rm, cudaStream_t s) {
    const dim3 grid(cdiv(c.n, (G ? kTB / (G ? G : 1) : kSB)));
    if constexpr (G != 0) {
        if (first)
            k_lambda_first_team<LAST, G><<<grid, kTB, 0, s>>>(c, d.sorted_a, d.qpos, d.sorted_b, d.scell, d.cstart,
                                                              d.sidx, d.lambdas, d.ncount, rm);
        else
            k_lambda_team<LAST, G><<<grid, kTB, 0, s>>>(c, d.sorted_a, d.qpos, d.sorted_b, d.scell, d.cstart,
                                                        d.sidx, d.lambdas, rm);
    } else {
        if (first)
            k_lambda_first<LAST><<<grid, kSB, 0, s>>>(c, d.sorted_a, d.qpos, d.sorted_b, d.scell, d.cstart,
                                                      d.sidx, d.lambdas, d.ncount, rm);
        else
            k_lambda<LAST><<<grid, kSB, 0, s>>>(c, d.sorted_a, d.qpos, d.sorted_b, d.scell, d.cstart, d.sidx,
                                                d.lambdas, rm);
    }
}

template <uint32_t G, bool LAST, uint32_t SN>
void launch_delta_n(const StepConsts& c, const DevState& d, const RowMasks& rm, cudaStream_t s) {
    const dim3 grid(cdiv(c.n, (G ? kTB / (G ? G : 1) : kSB)));
    if constexpr (G != 0)
        k_delta_team<LAST, SN, G><<<grid, kTB, 0, s>>>(c, d.sorted_b, d.sorted_a, d.qpos, d.xa, d.scell, d.cstart,
                                                       d.sidx, d.sphere, d.pos, d.vel, d.prev, d.ncount, d.foam,
                                                       d.err, rm);
    else
        k_delta<LAST, SN><<<grid, kSB, 0, s>>>(c, d.sorted_b, d.sorted_a, d.qpos, d.xa, d.scell, d.cstart, d.sidx,
                                               d.sphere, d.pos, d.vel, d.prev, d.ncount, d.foam, d.err, rm);
}

template <uint32_t G, bool LAST>
void launch_iteration(const StepConsts& c, const DevState& d, bool first, const RowMasks& rm, cudaStream_t s,
                      KernelTimer* t) {
    tbegin(t, s);
    launch_lambda<G, LAST>(c, d, first, rm, s);
    tend(t, first ? "lambda_count" : "lambda", s);
    tbegin(t, s);
    if (c.scorr_n == 4)
        launch_delta_n<G, LAST, 4>(c, d, rm, s);
    else
        launch_delta_n<G, LAST, 0>(c, d, rm, s);
    tend(t, LAST ? "delta_finalize" : "delta", s);
}

template <uint32_t G>
void launch_iterations(const StepConsts& c, const DevState& d, uint32_t iterations, cudaStream_t s,
                       KernelTimer* t) {
    const RowMasks rm{d.row_masks, d.mask_overflow, d.mask_stride};  // 9 x u32 per slot
    for (uint32_t it = 0; it < iterations; ++it) {
        if (it + 1 == iterations)
            launch_iteration<G, true>(c, d, it == 0, rm, s, t);
        else
            launch_iteration<G, false>(c, d, it == 0, rm, s, t);
    }
}

__global__ void __launch_bounds__(256)
k_finalize_sorted(StepConsts c, const float4* __restrict__ sorted,
                  const uint32_t* __restrict__ sidx, float4* __restrict__ pos,
                  float4* __restrict__ vel, const float4* __restrict__ prev,
                  const uint32_t* __restrict__ ncount, float* __restrict__ foam, uint32_t* err) {
    const uint32_t s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s < c.n) finalize_sorted_item(c, s, sorted, sidx, pos, vel, prev, ncount, foam, err);
}

}  // namespace

cudaError_t launch_solver(const StepConsts& c, const DevState& d, uint32_t iterations,
                          cudaStream_t s, KernelTimer* t) {
    const uint32_t n = c.n;
    if (n == 0) return cudaSuccess;
    const uint32_t grid = cdiv(n, 256);
    if (iterations == 0) {
        cudaError_t e = launch_count_neighbors(c, d, s, t);
        if (e != cudaSuccess) return e;
        tbegin(t, s);
        k_finalize_sorted<<<grid, 256, 0, s>>>(c, d.sorted_a, d.sidx, d.pos, d.vel, d.prev, d.ncount,
                                               d.foam, d.err);
        tend(t, "finalize", s);
        return cudaGetLastError();
    }
    if (team_lanes(n, n))
        launch_iterations<kTeam>(c, d, iterations, s, t);
    else
        launch_iterations<0>(c, d, iterations, s, t);
    return cudaGetLastError();
}

uint32_t step_launch_count(uint32_t iterations) {
    // predict+hash, scan, scatter, sort+gather, then 2 per iteration (or count +
    // finalize for zero iterations).
    return 4u + (iterations ? 2u * iterations : 2u);
}

}  // namespace mpb
