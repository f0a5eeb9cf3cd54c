// pbf_adjoint.h — the adjoint (reverse-mode derivative) of one recorded PBF
// step of a batch of scenes.  No reference counterpart: the reference engine
// is not differentiable.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "pbf_batch.h"

namespace mpb {

// Per-scene gradient accumulators (FP64): d/d s_corr k, the sphere's center
// (3), velocity (3) and radius.  During the reverse sweep the sphere entries
// hold the adjoint of the sphere state at the current step.
constexpr uint32_t kGradStride = 8;
constexpr uint32_t kGradK = 0, kGradCenter = 1, kGradVel = 4, kGradRadius = 7;

// One recorded step, as the forward step kept it (pbf_batch.h BatchRecord
// plus the per-step arrays the record owns).
struct AdjStep {
    const SceneDev* scenes;       // scene table: sub-grids and sphere of the step
    const SphereState* sphere0;   // spheres before the step's kinematic advance
    const float4* x0;             // positions at the start of the step (original order)
    const float4* x1;             // positions at the end of the step (original order)
    const uint32_t* sidx;         // slot -> particle
    const uint32_t* scell;        // slot -> hash cell (sub-grid local id)
    const uint32_t* cstart;       // cell starts of the step's grids
    const float4* lam;            // iterations x stride: (l, lambda)
    const float4* delta;          // iterations x stride: unclamped corrections
    const uint32_t* masks;        // iterations x 9 x mask_stride row masks
    const uint32_t* overflow;     // iterations x mask_stride: bit r set for a long row r
};

#ifdef __CUDACC__
#define MPB_BOTH __host__ __device__ __forceinline__
#else
#define MPB_BOTH inline
#endif

// Dense cell coordinates packed 11 / 11 / 10 bits (x, y, z); the host checks
// that the dense grid fits.
MPB_BOTH uint32_t pack_cell(int x, int y, int z) {
    return uint32_t(x) | (uint32_t(y) << 11) | (uint32_t(z) << 22);
}

// Whether two packed cells are within one cell of each other on every axis.
// With each field's difference plus one in a field of its own, that is every
// field 0, 1 or 2: no bit above a field's low two, also after adding one more.
// The fields of the subtraction cannot borrow their way into that unless two
// cells are 2046 (x, y) or 1023 (z) apart; `wide` grids, which reach that far,
// compare axis by axis.
MPB_BOTH bool cells_adjacent(uint32_t a, uint32_t b, bool wide) {
    if (!wide) {
        constexpr uint32_t one = 1u | (1u << 11) | (1u << 22), low2 = 3u * one;
        const uint32_t d = a - (b - one);
        return ((d | (d + one)) & ~low2) == 0u;
    }
    const int dx = int(a & 0x7ffu) - int(b & 0x7ffu);
    const int dy = int((a >> 11) & 0x7ffu) - int((b >> 11) & 0x7ffu);
    const int dz = int(a >> 22) - int(b >> 22);
    return dx * dx <= 1 && dy * dy <= 1 && dz * dz <= 1;
}

// Whether a grid of these dense dims is wide in that sense.
inline bool wide_grid(int dx, int dy, int dz) { return dx > 2045 || dy > 2045 || dz > 1021; }

// Pair terms that a particle's sweep owes another particle whose own sweep
// does not see the pair (one-way pairs) are posted to the receiver's inbox:
// kInbox slots per receiver, then a shared pool of overflow entries linked
// into a list per receiver.  The next kernel then adds each receiver's
// posts in ascending order of the sender's slot, so the sums do not depend
// on the order the posts arrived in (no float atomics: two backward passes
// give the same bytes).
constexpr uint32_t kInbox = 4;
constexpr uint32_t kInboxOverflow = 1u << 18;  // pooled entries beyond kInbox, all receivers together
constexpr uint32_t kNoPost = 0xffffffffu;      // end of a receiver's overflow list
// The per-scene sums of the sphere gradient run over chunks of this many slots.
constexpr uint32_t kSumChunk = 2048;

struct AdjArgs {
    AdjStep t;
    const uint32_t* scene_of;     // scene of every particle / slot
    uint32_t n, nscenes, iterations, stride, mask_stride;
    float4* xbar;                 // in: dL/dx(t+1), out: dL/dx(t) (original order)
    float4* vbar;                 // in: dL/dv(t+1), out: dL/dv(t)
    // per-slot scratch (sorted order)
    float4 *pbar, *qbar, *lbar, *gd, *p_extra;
    float4* dbar;                 // dL/d delta; w: the packed current cell
    float2* qc;                   // (dL/d squared-gradient sum, packed current cell)
    float* lam_part;
    uint32_t* cpred;
    float* xa;                    // x anchor of each slot's hash cell
    uint32_t wide;                // 1: some scene's grid is too wide for the packed cell comparison
    uint32_t common;              // 1: every scene has the pair constants `pair`
    PairConsts pair;
    uint32_t scorr4;              // 1: every scene's s_corr exponent is 4
    // one-way pair posts: per receiver slot a count and kInbox (sender,
    // value) entries (entry e of receiver j at e * stride + j); further posts
    // take pooled entries (sender, value, next) linked from ovf_head[j]
    uint32_t *inbox_count, *inbox_src;
    float4* inbox_val;
    uint32_t *ovf_head, *ovf_count, *ovf_src, *ovf_next;
    float4* ovf_val;
    // per-slot FP64 accumulators of the scene gradients, reduced per scene in
    // a fixed order: dL/dk (over the whole backward pass) and the sphere's
    // center (xyz) and radius (w) (over one step, summed per chunk of
    // kSumChunk slots into spart[scene * sum_chunks + chunk])
    double* kacc;
    double4 *sacc, *spart;
    uint32_t sum_chunks;
    uint32_t* err;                // device error word (kDevErrIndex: a post was dropped)
    const uint32_t* abort;        // set: a recorded step was stopped, its record is not whole
    double* grads;                // nscenes x kGradStride
};

// Enqueue the reverse of one step: finalize, every solver iteration in
// reverse order, predict, and the sphere kinematics.  inbox_count and sacc must
// be zero and ovf_head kNoPost on entry (they are left so); kacc accumulates.
cudaError_t launch_adjoint_step(const AdjArgs& a, cudaStream_t s);
// grads[scene][kGradK] = the sum of kacc over the scene's slots (fixed order);
// kacc is cleared.
cudaError_t launch_adjoint_finish(const AdjArgs& a, cudaStream_t s);

// Kernel launches per reversed step.
uint32_t adjoint_launch_count(uint32_t iterations);

}  // namespace mpb
