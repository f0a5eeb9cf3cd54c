// pbf_adjoint.cu — adjoint kernels of the PBF step for sm_100a.  No
// reference counterpart: the reference engine (engine/src/Engine.cpp:685-811)
// is not differentiable.
//
// The reverse of one recorded step of a batch of scenes, every kernel one
// thread per sorted slot of every scene, in this order:
//   finalize   dL/d(solved position) and the prev-position term from dL/dx',
//              dL/dv' (finalizeStep, Constraints.metal:305-353, wall masks,
//              friction and the speed cap held at their forward states)
//   K x, last iteration first:
//     pre      through the sphere push (+ dL/d sphere center, radius), the box
//              clamp and the |delta| clamp: dL/d(delta)
//     delta    pair sweep: dL/d lambda, the direct position terms of
//              applyDelta (Constraints.metal:140-199) and dL/dk of s_corr;
//              recomputes the particle's density sums
//     lbar     dL/d(density, gradient sums) from dL/d lambda
//     lambda   pair sweep: position terms of densityLambda (:82-131)
//   predict    dL/dx, dL/dv of predictPositions (:54-66)
//   sphere     dL/d sphere state through its kinematic advance
//              (Engine.cpp:694-707), one thread per scene
//
// The pair sweeps walk exactly the pairs of the forward iteration: the row
// masks its lambda pass recorded (long rows distance-tested past their first
// 32 candidates, as the forward delta pass does).  The reference's neighbour
// search makes those lists asymmetric once particles leave their predicted
// cells (j is in i's list iff j's predicted cell is next to i's current
// cell), so each pair term of i's list is delivered to j by j's own sweep
// when i is in j's list too (a test on the two cells).  Otherwise (a one-way
// pair, ~0.4% of pairs in a 60-step cube drop) i posts the term to j's inbox
// and the next kernel over j adds its posts in ascending order of the sender's
// slot.  The scene gradients (dL/dk, the sphere's center and radius) are
// accumulated per slot and summed per scene in a fixed order.  Nothing is
// added with float atomics, so the gradients are the same bytes on every run.
#include "pbf_adjoint.h"
#include "pbf_team.cuh"

namespace mpb {
namespace {

constexpr uint32_t kBlock = 256;

inline uint32_t cdiv(uint32_t a, uint32_t b) { return (a + b - 1) / b; }

// x^n; N = 4 is s_corr's exponent fixed at compile time (n - 1 = 3), with the
// roundings of the loop.
template <uint32_t N>
__device__ __forceinline__ float pow_u(float x, uint32_t n) {
    if (N == 4u) return __fmul_rn(__fmul_rn(x, x), x);
    float r = 1.0f;
    for (uint32_t e = 0; e < n; ++e) r = __fmul_rn(r, x);
    return r;
}

// The pair terms below are written with explicit roundings, so that the sweeps
// with one lane and with a team of lanes per slot give the same bits.

__device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by, float bz) {
    return __fmaf_rn(az, bz, __fmaf_rn(ay, by, __fmul_rn(ax, bx)));
}

// Kernel values of a pair at offset r with 1e-12 < |r|^2 = r2 < h^2:
// spiky gradient g = f r, its Jacobian H v = f v + fp (r . v) r, d = h^2 - r2
// (poly6 weight W = w d, grad W = -6 poly6 d^2 r).
struct PairTerms {
    float d, f, fp, w;
    __device__ __forceinline__ PairTerms(const PairConsts& c, float r2) {
        d = __fsub_rn(c.h2, r2);
        const float rinv = rsqrt_normal(r2);
        const float hd = fmaxf(__fmaf_rn(-r2, rinv, c.h), 0.0f);
        f = __fmul_rn(__fmul_rn(__fmul_rn(-c.spiky, hd), hd), rinv);
        fp = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(c.spiky, d), rinv), rinv), rinv);
        w = __fmul_rn(__fmul_rn(c.poly6, d), d);
    }
    __device__ __forceinline__ float3 hess(float rx, float ry, float rz, float vx, float vy,
                                           float vz) const {
        const float a = __fmul_rn(fp, dot3(rx, ry, rz, vx, vy, vz));
        return make_float3(__fmaf_rn(a, rx, __fmul_rn(f, vx)), __fmaf_rn(a, ry, __fmul_rn(f, vy)),
                           __fmaf_rn(a, rz, __fmul_rn(f, vz)));
    }
};

// Posts the term v that sender slot `from` owes receiver slot `to` (a
// one-way pair): into one of the receiver's kInbox entries, or a pooled
// entry linked into the receiver's overflow list; a post that finds the pool
// exhausted sets kDevErrIndex.
__device__ __forceinline__ void post(const AdjArgs& a, uint32_t to, uint32_t from, const float4& v) {
    const uint32_t e = atomicAdd(&a.inbox_count[to], 1u);
    if (e < kInbox) {
        a.inbox_src[size_t(e) * a.stride + to] = from;
        a.inbox_val[size_t(e) * a.stride + to] = v;
        return;
    }
    const uint32_t o = atomicAdd(a.ovf_count, 1u);
    if (o < kInboxOverflow) {
        a.ovf_src[o] = from;
        a.ovf_val[o] = v;
        a.ovf_next[o] = atomicExch(&a.ovf_head[to], o);
    } else {
        atomicOr(a.err, kDevErrIndex);
    }
}

// The sum of the terms posted to receiver slot j by the last sweep, in ascending
// order of the sender's slot (a sender posts to a receiver at most once per
// sweep); empties its inbox.  Posts beyond the inbox are looked up in the
// overflow list.
__device__ __forceinline__ float4 collect(const AdjArgs& a, uint32_t j) {
    float sx = 0.0f, sy = 0.0f, sz = 0.0f, sw = 0.0f;
    const uint32_t cnt = a.inbox_count[j];
    if (cnt != 0) {
        a.inbox_count[j] = 0;
        const uint32_t nin = min(cnt, kInbox);
        const uint32_t head = cnt > kInbox ? a.ovf_head[j] : kNoPost;
        uint32_t last = 0;
        for (uint32_t done = 0; done < cnt; ++done) {
            uint32_t best = 0xffffffffu;
            float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            for (uint32_t e = 0; e < nin; ++e) {
                const uint32_t src = a.inbox_src[size_t(e) * a.stride + j];
                if ((done == 0 || src > last) && src < best) {
                    best = src;
                    v = a.inbox_val[size_t(e) * a.stride + j];
                }
            }
            for (uint32_t o = head; o != kNoPost; o = a.ovf_next[o]) {
                const uint32_t src = a.ovf_src[o];
                if ((done == 0 || src > last) && src < best) {
                    best = src;
                    v = a.ovf_val[o];
                }
            }
            if (best == 0xffffffffu) break;  // posts dropped with the pool exhausted
            sx += v.x;
            sy += v.y;
            sz += v.z;
            sw += v.w;
            last = best;
        }
        if (head != kNoPost) a.ovf_head[j] = kNoPost;
    }
    return make_float4(sx, sy, sz, sw);
}

// ---- finalize --------------------------------------------------------------

__global__ void __launch_bounds__(kBlock) k_adj_finalize(AdjArgs a) {
    const uint32_t s = blockIdx.x * kBlock + threadIdx.x;
    if (s >= a.n) return;
    // loads first (in flight together), stores after
    const uint32_t sc = __ldg(&a.scene_of[s]);
    const uint32_t cell = __ldg(&a.t.scell[s]);
    const uint32_t j = __ldg(&a.t.sidx[s]);
    const float4 X4 = __ldg(&a.t.x1[j]), P4 = __ldg(&a.t.x0[j]), xb = a.xbar[j], vb = a.vbar[j];
    const StepConsts& c = a.t.scenes[sc].c;
    int px, py, pz;
    decode_cell(c.g, cell, px, py, pz);
    a.cpred[s] = pack_cell(px + c.g.lx, py + c.g.ly, pz + c.g.lz);
    a.xa[s] = anchor_x(c.g, px);
    const double X[3] = {X4.x, X4.y, X4.z}, P[3] = {P4.x, P4.y, P4.z};
    const double lo_b[3] = {c.bminx, c.bminy, c.bminz}, hi_b[3] = {c.bmaxx, c.bmaxy, c.bmaxz};
    const double kd = double(c.damping) / double(c.dt);
    bool lo[3], hi[3], keep[3];
    double b[3];
    for (int k = 0; k < 3; ++k) {
        const double u = (X[k] - P[k]) * kd;
        lo[k] = X[k] <= lo_b[k] + double(c.wall_eps);
        hi[k] = X[k] >= hi_b[k] - double(c.wall_eps);
        keep[k] = !((lo[k] && u < 0.0) || (hi[k] && u > 0.0));
        b[k] = keep[k] ? u : 0.0;
    }
    double fr[3] = {1.0, 1.0, 1.0};
    if (lo[1]) {
        fr[0] = fr[2] = c.floor_fric;
    } else if (lo[0] || hi[0] || lo[2] || hi[2]) {
        fr[0] = fr[1] = fr[2] = c.wall_fric;
    }
    for (int k = 0; k < 3; ++k) b[k] *= fr[k];
    const double vmax = double(c.vmax_frac) * double(c.h) / double(c.dt);
    const double bl = sqrt(b[0] * b[0] + b[1] * b[1] + b[2] * b[2]);
    double bb[3] = {vb.x, vb.y, vb.z};
    if (bl > vmax) {  // v = b vmax / |b|
        const double dot = (b[0] * bb[0] + b[1] * bb[1] + b[2] * bb[2]) / bl;
        for (int k = 0; k < 3; ++k) bb[k] = (vmax / bl) * (bb[k] - dot * b[k] / bl);
    }
    double ub[3];
    for (int k = 0; k < 3; ++k) ub[k] = keep[k] ? bb[k] * fr[k] * kd : 0.0;
    a.pbar[s] = make_float4(float(xb.x + ub[0]), float(xb.y + ub[1]), float(xb.z + ub[2]), 0.0f);
    a.xbar[j] = make_float4(float(-ub[0]), float(-ub[1]), float(-ub[2]), 0.0f);
}

// ---- one solver iteration ---------------------------------------------------

// Through the sphere push, the box clamp and the |delta| clamp of iteration
// `it`, from the position adjoint left by the iteration after it (its sweeps'
// own sums and what they posted); the iterate's current cell goes beside dL/d
// delta for the pair sweeps.
__global__ void __launch_bounds__(kBlock) k_adj_pre(AdjArgs a, uint32_t it) {
    const uint32_t s = blockIdx.x * kBlock + threadIdx.x;
    if (s == 0) *a.ovf_count = 0;  // the delta sweep posts into an empty list
    if (s >= a.n) return;
    // every per-slot input first, so their loads are in flight together
    const size_t off = size_t(it) * a.stride;
    const uint32_t sc = __ldg(&a.scene_of[s]);
    const float4 l = __ldg(&a.t.lam[off + s]);
    const float4 dr = __ldg(&a.t.delta[off + s]);
    const uint32_t cell = __ldg(&a.t.scell[s]);
    const bool first = it + 1 == a.iterations;  // no sweep has run in this step
    float4 pe = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (!first) pe = a.p_extra[s];
    const float4 pb4 = a.pbar[s];
    const SceneDev& sd = a.t.scenes[sc];
    const StepConsts& c = sd.c;
    int pcx, pcy, pcz;
    decode_cell(c.g, cell, pcx, pcy, pcz);
    const float ax = anchor_x(c.g, pcx), ay = anchor_y(c.g, pcy), az = anchor_z(c.g, pcz);
    int cx, cy, cz;
    cell_of(c.g, __fadd_rn(ax, l.x), __fadd_rn(ay, l.y), __fadd_rn(az, l.z), cx, cy, cz);
    const uint32_t ccur = pack_cell(cx + c.g.lx, cy + c.g.ly, cz + c.g.lz);
    if (!first) {
        const float4 more = collect(a, s);
        pe = make_float4(pe.x + more.x, pe.y + more.y, pe.z + more.z, 0.0f);
    }

    // the forward update (delta_item): clamp |delta|, A + (l + delta) in FP64
    const float dl = __fsqrt_rn(dist2(dr.x, dr.y, dr.z));
    const bool big = dl > c.max_step;
    const float f = big ? __fdiv_rn(c.max_step, dl) : 1.0f;
    const float dx = big ? __fmul_rn(dr.x, f) : dr.x;
    const float dy = big ? __fmul_rn(dr.y, f) : dr.y;
    const float dz = big ? __fmul_rn(dr.z, f) : dr.z;
    const double q[3] = {__dadd_rn(double(ax), double(__fadd_rn(l.x, dx))),
                         __dadd_rn(double(ay), double(__fadd_rn(l.y, dy))),
                         __dadd_rn(double(az), double(__fadd_rn(l.z, dz)))};
    const double lo_b[3] = {c.bminx, c.bminy, c.bminz}, hi_b[3] = {c.bmaxx, c.bmaxy, c.bmaxz};
    bool inside[3];
    double qc[3];
    for (int k = 0; k < 3; ++k) {
        inside[k] = q[k] >= lo_b[k] && q[k] <= hi_b[k];
        qc[k] = fmin(fmax(q[k], lo_b[k]), hi_b[k]);
    }

    float pb[3] = {pb4.x + pe.x, pb4.y + pe.y, pb4.z + pe.z};
    if (c.sphere) {
        const double ex = qc[0] - sd.sphere.c[0], ey = qc[1] - sd.sphere.c[1], ez = qc[2] - sd.sphere.c[2];
        const double e2 = ex * ex + ey * ey + ez * ez, r = sd.sphere.r;
        if (e2 < r * r) {  // x = center + e r / |e|
            const double el = sqrt(fmax(e2, double(1e-8f)));
            const double e[3] = {ex / el, ey / el, ez / el};
            const double dot = e2 > double(1e-8f) ? e[0] * pb[0] + e[1] * pb[1] + e[2] * pb[2] : 0.0;
            double cb[3], eb[3];
            for (int k = 0; k < 3; ++k) {
                eb[k] = (r / el) * (pb[k] - e[k] * dot);
                cb[k] = pb[k] - eb[k];
            }
            const double rb = e[0] * pb[0] + e[1] * pb[1] + e[2] * pb[2];
            double4 sa = a.sacc[s];  // this slot's share of the step's sphere gradient
            sa.x += cb[0];
            sa.y += cb[1];
            sa.z += cb[2];
            sa.w += rb;
            a.sacc[s] = sa;
            for (int k = 0; k < 3; ++k) pb[k] = float(eb[k]);
        }
    }
    for (int k = 0; k < 3; ++k)
        if (!inside[k]) pb[k] = 0.0f;
    a.qbar[s] = make_float4(pb[0], pb[1], pb[2], 0.0f);
    if (big) {  // delta = d max_step / |d|
        const float ux = dr.x / dl, uy = dr.y / dl, uz = dr.z / dl;
        const float dot = ux * pb[0] + uy * pb[1] + uz * pb[2];
        pb[0] = f * (pb[0] - ux * dot);
        pb[1] = f * (pb[1] - uy * dot);
        pb[2] = f * (pb[2] - uz * dot);
    }
    a.dbar[s] = make_float4(pb[0], pb[1], pb[2], __uint_as_float(ccur));
}

// Pair sweep of applyDelta's adjoint.  With dbar = dL/d delta:
//   lambdabar_i = sum_j g_ij . (dbar_i - dbar_j) / rho0
//   pbar_i     += sum_j ((lambda_i + lambda_j + s_ij) H_ij (dbar_i - dbar_j)
//                        + grad s_ij g_ij . (dbar_i - dbar_j)) / rho0
//   kbar       += sum_j -(W_ij / W(dq))^n g_ij . dbar_i / rho0
// (dbar_j and the j-side terms only for pairs in both lists; the j-side
// terms of a one-way pair are posted to j, and the next kernel over j adds
// them), and the particle's density sums for the lambda adjoint.
// Both pair sweeps walk their pairs through a PairQueue (pbf_items.cuh), one
// loop per slot instead of one per stencil row (10 -> 26 of 32 threads active),
// and keep the scene's constants in registers.  Bound by issue and load latency.
// 7 blocks of 128 per SM (72 registers, a small spill): gradients of eight lakes
// (386,000 particles) 8.0 ms, of the 97,336-particle cube 6.6 ms (5 blocks: 8.3 and
// 7.3, 6: 8.05 and 6.55, 8: 8.0 and 6.65 ms).
#ifndef MPB_ADJ_SWEEP_MIN_BLOCKS
#define MPB_ADJ_SWEEP_MIN_BLOCKS 7
#endif
constexpr int kSweepMinBlocks = MPB_ADJ_SWEEP_MIN_BLOCKS;
constexpr uint32_t kSweepBlock = 128;

// What a slot's delta sweep reads of its own.
struct DeltaSlot {
    float4 l, dm;
    uint32_t pm;
    float ax, ay, az;
    int cx, cy, cz;
    __device__ __forceinline__ DeltaSlot(const AdjArgs& a, const StepConsts& c, const float4* src, uint32_t m) {
        l = src[m];
        dm = a.dbar[m];
        pm = a.cpred[m];
        int pcx, pcy, pcz;
        decode_cell(c.g, a.t.scell[m], pcx, pcy, pcz);
        ax = anchor_x(c.g, pcx);
        ay = anchor_y(c.g, pcy);
        az = anchor_z(c.g, pcz);
        cell_of(c.g, __fadd_rn(ax, l.x), __fadd_rn(ay, l.y), __fadd_rn(az, l.z), cx, cy, cz);
    }
};

// A pair's terms in the delta sweep of slot m (1e-12 < r2 < h^2): the gradient
// sums' (f r, f^2 r2), dL/dk's (-rn gdm), dL/d lambda's (gdd) and dL/d position's
// (v).
struct DeltaTerms {
    float f, f2, rn, gdm, gdd, vx, vy, vz;
};

template <uint32_t SN>
__device__ __forceinline__ DeltaTerms delta_terms(const AdjArgs& a, const PairConsts& pc, uint32_t n, float sgk,
                                                  float li, const float4& dm, uint32_t pm, uint32_t m, uint32_t k,
                                                  const float4& q, float rx, float ry, float rz, float r2) {
    DeltaTerms r;
    const float4 di = __ldg(&a.dbar[k]);
    const PairTerms t(pc, r2);
    r.f = t.f;
    r.f2 = __fmul_rn(t.f, t.f);
    const float fx = __fmul_rn(t.f, rx), fy = __fmul_rn(t.f, ry), fz = __fmul_rn(t.f, rz);  // g
    const float ratio = __fmul_rn(__fmul_rn(t.w, t.d), pc.inv_wq);
    const float rn1 = n ? pow_u<SN>(ratio, n - 1) : 0.0f;
    r.rn = n ? __fmul_rn(rn1, ratio) : 1.0f;
    const float coef = __fmaf_rn(-pc.scorr_k, r.rn, __fadd_rn(li, q.w));
    const float sg = __fmul_rn(__fmul_rn(__fmul_rn(sgk, rn1), t.d), t.d);  // grad s_ij = sg r
    r.gdm = dot3(fx, fy, fz, dm.x, dm.y, dm.z);
    // a pair in both lists carries the other particle's terms too; a
    // one-way pair owes it the negative of its own
    const bool both = cells_adjacent(__float_as_uint(di.w), pm, a.wide);
    const float ex = __fsub_rn(dm.x, both ? di.x : 0.0f), ey = __fsub_rn(dm.y, both ? di.y : 0.0f);
    const float ez = __fsub_rn(dm.z, both ? di.z : 0.0f);
    r.gdd = dot3(fx, fy, fz, ex, ey, ez);
    const float3 hv = t.hess(rx, ry, rz, ex, ey, ez);
    const float sgd = __fmul_rn(sg, r.gdd);
    r.vx = __fmaf_rn(coef, hv.x, __fmul_rn(sgd, rx));
    r.vy = __fmaf_rn(coef, hv.y, __fmul_rn(sgd, ry));
    r.vz = __fmaf_rn(coef, hv.z, __fmul_rn(sgd, rz));
    if (!both) {
        const float ir = pc.inv_rho0;
        post(a, k, m, make_float4(-r.vx * ir, -r.vy * ir, -r.vz * ir, r.gdd * ir));
    }
    return r;
}

// The sums of a slot's delta sweep, written out.
__device__ __forceinline__ void delta_out(const AdjArgs& a, const StepConsts& c, uint32_t m, float gx, float gy,
                                          float gz, float gsq, float kb, float lb, float px, float py, float pz) {
    const float ir = c.inv_rho0;
    const float4 qb = a.qbar[m];
    a.qbar[m] = make_float4(__fmaf_rn(px, ir, qb.x), __fmaf_rn(py, ir, qb.y), __fmaf_rn(pz, ir, qb.z), 0.0f);
    a.lam_part[m] = __fmul_rn(lb, ir);
    const float g2 = __fadd_rn(dot3(gx, gy, gz, gx, gy, gz), gsq);
    a.gd[m] = make_float4(gx, gy, gz, __fmaf_rn(__fmul_rn(ir, ir), g2, c.eps));
    a.kacc[m] += double(__fmul_rn(kb, ir));  // this slot's share of dL/dk
}

__device__ __forceinline__ float scorr_grad(const PairConsts& pc, uint32_t n) {
    return n ? 6.0f * pc.scorr_k * float(n) * pc.inv_wq * pc.poly6 : 0.0f;
}

// Whether a recorded step gave up at a barrier.  Its record may mix two steps', so
// the pair sweeps leave their sums alone (the kernels that follow one index per slot
// stay inside their arrays).  Loaded beside the slot's own values, where it is free.
__device__ __forceinline__ bool stopped(const AdjArgs& a) { return __ldg(a.abort) != 0u; }

__device__ __forceinline__ RowMasks recorded_masks(const AdjArgs& a, uint32_t it) {
    const uint32_t ms = a.mask_stride;
    return RowMasks{const_cast<uint32_t*>(a.t.masks) + size_t(it) * 9 * ms,
                    const_cast<uint32_t*>(a.t.overflow) + size_t(it) * ms, ms};
}

template <uint32_t SN, bool COMMON>
__global__ void __launch_bounds__(kSweepBlock, kSweepMinBlocks) k_adj_delta(AdjArgs a, uint32_t it) {
    __shared__ uint2 queue[kQueue * kSweepBlock];
    const uint32_t m = blockIdx.x * kSweepBlock + threadIdx.x;
    if (m >= a.n) return;
    const bool stop = stopped(a);
    const StepConsts& c = a.t.scenes[a.scene_of[m]].c;
    const float4* src = a.t.lam + size_t(it) * a.stride;
    const DeltaSlot o(a, c, src, m);
    // a kernel argument, or kept in registers: a post would otherwise make every
    // pair load them again
    const PairConsts pc = COMMON ? a.pair : pair_consts(c);
    const uint32_t n = SN ? SN : pc.scorr_n;
    const float sgk = scorr_grad(pc, n);
    float gx = 0.0f, gy = 0.0f, gz = 0.0f, gsq = 0.0f;
    float kb = 0.0f, lb = 0.0f, px = 0.0f, py = 0.0f, pz = 0.0f;
    auto body = [&](uint32_t k, const float4& q, float rx, float ry, float rz, float r2) {
        if (!(r2 < pc.h2 && r2 > 1e-12f)) return;
        const DeltaTerms t = delta_terms<SN>(a, pc, n, sgk, o.l.w, o.dm, o.pm, m, k, q, rx, ry, rz, r2);
        gx = __fmaf_rn(t.f, rx, gx);
        gy = __fmaf_rn(t.f, ry, gy);
        gz = __fmaf_rn(t.f, rz, gz);
        gsq = __fmaf_rn(t.f2, r2, gsq);
        kb = __fmaf_rn(-t.rn, t.gdm, kb);
        lb = __fadd_rn(lb, t.gdd);
        px = __fadd_rn(px, t.vx);
        py = __fadd_rn(py, t.vy);
        pz = __fadd_rn(pz, t.vz);
    };
    if (stop) return;
    queued_pairs<true, kSweepBlock>(c, src, a.xa, a.t.cstart, recorded_masks(a, it), m, o.l, o.ax, o.ay, o.az, o.cx,
                              o.cy, o.cz, PairQueue<kSweepBlock>(queue), body);
    delta_out(a, c, m, gx, gy, gz, gsq, kb, lb, px, py, pz);
}

// The same with a team of kTeam lanes per slot (pbf_team.cuh): 8,000 slots, 25 -> 9
// us a sweep; ten steps forward and backward 4.16 -> 3.21 ms.
constexpr uint32_t kTeamBlock = 64;

template <uint32_t SN>
__global__ void __launch_bounds__(kTeamBlock) k_adj_delta_team(AdjArgs a, uint32_t it) {
    __shared__ TeamBufOf<9> bufs[kTeamBlock / kTeam];
    const uint32_t m = (blockIdx.x * kTeamBlock + threadIdx.x) / kTeam;
    if (m >= a.n) return;
    const Team<kTeam, TeamBufOf<9>> team(bufs);
    const bool stop = stopped(a);
    const StepConsts& c = a.t.scenes[a.scene_of[m]].c;
    const float4* src = a.t.lam + size_t(it) * a.stride;
    const DeltaSlot o(a, c, src, m);
    const PairConsts pc = pair_consts(c);
    const uint32_t n = SN ? SN : pc.scorr_n;
    const float sgk = scorr_grad(pc, n);
    const RowMasks rm = recorded_masks(a, it);
    const TeamWalk<true> walk{c, src, a.xa, rm, m, o.l, o.ax, o.ay, o.az, o.cy - 1, o.cz - 1};
    auto terms = [&](uint32_t k, uint32_t y, uint32_t z, float2* out) {
        const float4 q = __ldg(&src[k]);
        float rx, ry, rz;
        walk.offset(k, q, y, z, rx, ry, rz);
        const float r2 = dist2(rx, ry, rz);
        DeltaTerms t{};
        const bool apart = r2 < pc.h2 && r2 > 1e-12f;
        if (apart) t = delta_terms<SN>(a, pc, n, sgk, o.l.w, o.dm, o.pm, m, k, q, rx, ry, rz, r2);
        auto put = [&](uint32_t i, float x, float y) {
            out[i * kTermStride] = apart ? make_float2(x, y) : make_float2(0.0f, 0.0f);
        };
        put(0, t.f, rx);
        put(1, t.f, ry);
        put(2, t.f, rz);
        put(3, t.f2, r2);
        put(4, -t.rn, t.gdm);
        put(5, t.gdd, 1.0f);
        put(6, t.vx, 1.0f);
        put(7, t.vy, 1.0f);
        put(8, t.vz, 1.0f);
    };
    float sum = 0.0f;
    if (stop) return;
    team_pairs<kTeam, 9>(
        team, c, a.t.cstart, o.cx, o.cy, o.cz, sum,
        [&](uint32_t row, uint32_t c0, uint32_t b0, uint32_t b3) { return walk.bits(row, c0, b0, b3); },
        [](uint32_t) {}, terms);
    float r[9];
#pragma unroll
    for (uint32_t i = 0; i < 9; ++i) r[i] = team.from(sum, i);
    if (team.lane == 0) delta_out(a, c, m, r[0], r[1], r[2], r[3], r[4], r[5], r[6], r[7], r[8]);
}

// dL/d(density sum, gradient sum, squared-gradient sum) of each particle's
// lambda = -(rho / rho0 - 1) / (|G|^2 + Q) / rho0^2 + eps):
//   rhobar = -lambdabar / (D rho0), Dbar = -lambdabar lambda / D,
//   Gbar = 2 Dbar G / rho0^2, Qbar = Dbar / rho0^2.
__global__ void __launch_bounds__(kBlock) k_adj_lbar(AdjArgs a, uint32_t it) {
    const uint32_t s = blockIdx.x * kBlock + threadIdx.x;
    if (s == 0) *a.ovf_count = 0;  // the lambda sweep posts into an empty list
    if (s >= a.n) return;
    const StepConsts& c = a.t.scenes[a.scene_of[s]].c;
    const uint32_t ccur = __float_as_uint(a.dbar[s].w);
    const float4 posts = collect(a, s);  // of the delta sweep
    a.p_extra[s] = posts;
    const float lb = a.lam_part[s] + posts.w;
    const float4 gd = a.gd[s];
    const float lam = a.t.lam[size_t(it) * a.stride + s].w;
    const float ir = c.inv_rho0;
    const float Db = -lb * lam / gd.w;
    const float gG = 2.0f * Db * ir * ir;
    a.lbar[s] = make_float4(gG * gd.x, gG * gd.y, gG * gd.z, -lb * ir / gd.w);
    a.qc[s] = make_float2(Db * ir * ir, __uint_as_float(ccur));
}

// A pair's position term in the lambda sweep of slot m (1e-12 < r2 < h^2).
__device__ __forceinline__ float3 lambda_term(const AdjArgs& a, const PairConsts& pc, const float4& lm, float qm,
                                              uint32_t pm, uint32_t m, uint32_t k, float rx, float ry, float rz,
                                              float r2) {
    const float4 li = __ldg(&a.lbar[k]);
    const float2 qi = __ldg(&a.qc[k]);
    const PairTerms t(pc, r2);
    const float gw = __fmul_rn(__fmul_rn(__fmul_rn(-6.0f, pc.poly6), t.d), t.d);  // grad W = gw r
    const bool both = cells_adjacent(__float_as_uint(qi.y), pm, a.wide);
    const float qs = __fmul_rn(__fmul_rn(2.0f, __fadd_rn(qm, both ? qi.x : 0.0f)), t.f);
    const float3 hv = t.hess(rx, ry, rz, __fmaf_rn(qs, rx, __fsub_rn(lm.x, both ? li.x : 0.0f)),
                             __fmaf_rn(qs, ry, __fsub_rn(lm.y, both ? li.y : 0.0f)),
                             __fmaf_rn(qs, rz, __fsub_rn(lm.z, both ? li.z : 0.0f)));
    const float w = __fmul_rn(__fadd_rn(lm.w, both ? li.w : 0.0f), gw);
    const float3 v = make_float3(__fmaf_rn(w, rx, hv.x), __fmaf_rn(w, ry, hv.y), __fmaf_rn(w, rz, hv.z));
    if (!both) post(a, k, m, make_float4(-v.x, -v.y, -v.z, 0.0f));
    return v;
}

// Pair sweep of densityLambda's adjoint:
//   pbar_i += sum_j (rhobar_i + rhobar_j) grad W_ij
//             + H_ij (Gbar_i - Gbar_j + 2 (Qbar_i + Qbar_j) g_ij)
// (j-side terms of one-way pairs are posted to j, as in the delta sweep).
template <bool COMMON>
__global__ void __launch_bounds__(kSweepBlock, kSweepMinBlocks) k_adj_lambda(AdjArgs a, uint32_t it) {
    __shared__ uint2 queue[kQueue * kSweepBlock];
    const uint32_t m = blockIdx.x * kSweepBlock + threadIdx.x;
    if (m >= a.n) return;
    const bool stop = stopped(a);
    const StepConsts& c = a.t.scenes[a.scene_of[m]].c;
    const float4* src = a.t.lam + size_t(it) * a.stride;
    const DeltaSlot o(a, c, src, m);
    const float4 lm = a.lbar[m];
    const float qm = a.qc[m].x;
    const float4 qb = a.qbar[m];
    float px = qb.x, py = qb.y, pz = qb.z;
    const PairConsts pc = COMMON ? a.pair : pair_consts(c);
    auto body = [&](uint32_t k, const float4&, float rx, float ry, float rz, float r2) {
        if (!(r2 < pc.h2 && r2 > 1e-12f)) return;
        const float3 v = lambda_term(a, pc, lm, qm, o.pm, m, k, rx, ry, rz, r2);
        px = __fadd_rn(px, v.x);
        py = __fadd_rn(py, v.y);
        pz = __fadd_rn(pz, v.z);
    };
    if (stop) return;
    queued_pairs<true, kSweepBlock>(c, src, a.xa, a.t.cstart, recorded_masks(a, it), m, o.l, o.ax, o.ay, o.az, o.cx,
                              o.cy, o.cz, PairQueue<kSweepBlock>(queue), body);
    a.pbar[m] = make_float4(px, py, pz, 0.0f);
}

__global__ void __launch_bounds__(kTeamBlock) k_adj_lambda_team(AdjArgs a, uint32_t it) {
    __shared__ TeamBufOf<3> bufs[kTeamBlock / kTeam];
    const uint32_t m = (blockIdx.x * kTeamBlock + threadIdx.x) / kTeam;
    if (m >= a.n) return;
    const Team<kTeam, TeamBufOf<3>> team(bufs);
    const bool stop = stopped(a);
    const StepConsts& c = a.t.scenes[a.scene_of[m]].c;
    const float4* src = a.t.lam + size_t(it) * a.stride;
    const DeltaSlot o(a, c, src, m);
    const float4 lm = a.lbar[m];
    const float qm = a.qc[m].x;
    const float4 qb = a.qbar[m];
    const PairConsts pc = pair_consts(c);
    const RowMasks rm = recorded_masks(a, it);
    const TeamWalk<true> walk{c, src, a.xa, rm, m, o.l, o.ax, o.ay, o.az, o.cy - 1, o.cz - 1};
    auto terms = [&](uint32_t k, uint32_t y, uint32_t z, float2* out) {
        float rx, ry, rz;
        walk.offset(k, __ldg(&src[k]), y, z, rx, ry, rz);
        const float r2 = dist2(rx, ry, rz);
        float3 v = make_float3(0.0f, 0.0f, 0.0f);
        if (r2 < pc.h2 && r2 > 1e-12f) v = lambda_term(a, pc, lm, qm, o.pm, m, k, rx, ry, rz, r2);
        out[0] = make_float2(v.x, 1.0f);
        out[kTermStride] = make_float2(v.y, 1.0f);
        out[2 * kTermStride] = make_float2(v.z, 1.0f);
    };
    float sum = team.lane == 0 ? qb.x : team.lane == 1 ? qb.y : qb.z;
    if (stop) return;
    team_pairs<kTeam, 3>(
        team, c, a.t.cstart, o.cx, o.cy, o.cz, sum,
        [&](uint32_t row, uint32_t c0, uint32_t b0, uint32_t b3) { return walk.bits(row, c0, b0, b3); },
        [](uint32_t) {}, terms);
    const float px = team.from(sum, 0), py = team.from(sum, 1), pz = team.from(sum, 2);
    if (team.lane == 0) a.pbar[m] = make_float4(px, py, pz, 0.0f);
}

// ---- scene sums ------------------------------------------------------------------

// Fixed-order block sum of one double per thread (blockDim.x == kBlock).
__device__ __forceinline__ double block_sum(double v, double* sh) {
    sh[threadIdx.x] = v;
    __syncthreads();
    for (uint32_t w = kBlock / 2; w > 0; w >>= 1) {
        if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    const double r = sh[0];
    __syncthreads();
    return r;
}

// Block (chunk, scene): the step's sphere gradient summed, in a fixed order,
// over the chunk's kSumChunk slots of a sphere scene into spart; the per-slot
// accumulators are cleared.  k_adj_sphere adds the chunks in order.
__global__ void __launch_bounds__(kBlock) k_adj_sphere_sum(AdjArgs a) {
    __shared__ double sh[kBlock];
    const uint32_t chunk = blockIdx.x, sc = blockIdx.y;
    const SceneDev& sd = a.t.scenes[sc];
    if (!sd.c.sphere) return;  // only sphere scenes accumulate
    const uint32_t first = chunk * kSumChunk, n = sd.c.n;
    const uint32_t end = min(n, first + kSumChunk);
    // kSumChunk / kBlock = 8 entries per thread, loaded 4 at a time before
    // they are added (in index order) and cleared
    static_assert(kSumChunk == 8 * kBlock, "two rounds of four loads per thread");
    double cx = 0.0, cy = 0.0, cz = 0.0, r = 0.0;
    double4* acc = a.sacc + sd.p0;
#pragma unroll
    for (uint32_t round = 0; round < 2; ++round) {
        double4 v[4];
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            const uint32_t i = first + (round * 4 + u) * kBlock + threadIdx.x;
            v[u] = i < end ? acc[i] : make_double4(0.0, 0.0, 0.0, 0.0);
        }
#pragma unroll
        for (uint32_t u = 0; u < 4; ++u) {
            const uint32_t i = first + (round * 4 + u) * kBlock + threadIdx.x;
            cx += v[u].x;
            cy += v[u].y;
            cz += v[u].z;
            r += v[u].w;
            if (i < end) acc[i] = make_double4(0.0, 0.0, 0.0, 0.0);
        }
    }
    cx = block_sum(cx, sh);
    cy = block_sum(cy, sh);
    cz = block_sum(cz, sh);
    r = block_sum(r, sh);
    if (threadIdx.x == 0) a.spart[size_t(sc) * a.sum_chunks + chunk] = make_double4(cx, cy, cz, r);
}

// dL/dk of every scene: block (chunk, scene) sums the chunk's per-slot
// accumulators into spart and clears them; k_adj_k_sum, one warp per scene, adds
// the chunks.  Both in a fixed order.  (One block per scene walked 80,000 slots
// in 92 us; the two kernels take 8.)
__global__ void __launch_bounds__(kBlock) k_adj_k_part(AdjArgs a) {
    __shared__ double sh[kBlock];
    const uint32_t chunk = blockIdx.x, sc = blockIdx.y;
    const SceneDev& sd = a.t.scenes[sc];
    const uint32_t first = chunk * kSumChunk, end = min(sd.c.n, first + kSumChunk);
    double* acc = a.kacc + sd.p0;
    double k = 0.0;
    for (uint32_t i = first + threadIdx.x; i < end; i += kBlock) {
        k += acc[i];
        acc[i] = 0.0;
    }
    k = block_sum(k, sh);
    if (threadIdx.x == 0) a.spart[size_t(sc) * a.sum_chunks + chunk].x = k;
}

__global__ void __launch_bounds__(32) k_adj_k_sum(AdjArgs a) {
    const uint32_t sc = blockIdx.x;
    const uint32_t chunks = (a.t.scenes[sc].c.n + kSumChunk - 1) / kSumChunk;
    double k = 0.0;
    for (uint32_t i = threadIdx.x; i < chunks; i += 32) k += a.spart[size_t(sc) * a.sum_chunks + i].x;
    for (int o = 16; o > 0; o >>= 1) k += __shfl_down_sync(kFull, k, o);
    if (threadIdx.x == 0) a.grads[size_t(sc) * kGradStride + kGradK] = k;
}

// ---- predict, sphere ----------------------------------------------------------

__global__ void __launch_bounds__(kBlock) k_adj_predict(AdjArgs a) {
    const uint32_t s = blockIdx.x * kBlock + threadIdx.x;
    if (s >= a.n) return;
    // loads first (in flight together), stores after
    const uint32_t sc = __ldg(&a.scene_of[s]);
    const uint32_t j = __ldg(&a.t.sidx[s]);
    const float4 pb = a.pbar[s];
    const float4 xb = a.xbar[j];
    const float dt = a.t.scenes[sc].c.dt;
    float4 pe = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (a.iterations) {  // what the last iteration's sweeps posted
        pe = a.p_extra[s];
        const float4 more = collect(a, s);
        pe = make_float4(pe.x + more.x, pe.y + more.y, pe.z + more.z, 0.0f);
    }
    const float bx = pb.x + pe.x, by = pb.y + pe.y, bz = pb.z + pe.z;
    a.xbar[j] = make_float4(xb.x + bx, xb.y + by, xb.z + bz, 0.0f);
    a.vbar[j] = make_float4(bx * dt, by * dt, bz * dt, 0.0f);
}

// The sphere's kinematic advance of this step (sphere_advance) reversed:
// the adjoint of the advanced state -> the adjoint of the state before it.
__global__ void __launch_bounds__(128) k_adj_sphere(AdjArgs a) {
    const uint32_t sc = blockIdx.x * 128 + threadIdx.x;
    if (sc >= a.nscenes) return;
    const StepConsts& c = a.t.scenes[sc].c;
    if (!c.sphere) return;
    {  // this step's push terms, chunk by chunk in order (k_adj_sphere_sum)
        // added in chunk order in registers (the same sums as adding each
        // chunk into g), loads four chunks ahead
        double* g = a.grads + size_t(sc) * kGradStride;
        const uint32_t chunks = (c.n + kSumChunk - 1) / kSumChunk;
        const double4* part = a.spart + size_t(sc) * a.sum_chunks;
        double gx = g[kGradCenter], gy = g[kGradCenter + 1], gz = g[kGradCenter + 2], gr = g[kGradRadius];
        for (uint32_t k0 = 0; k0 < chunks; k0 += 4) {
            double4 v[4];
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u)
                v[u] = k0 + u < chunks ? part[k0 + u] : make_double4(0.0, 0.0, 0.0, 0.0);
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                if (k0 + u >= chunks) break;
                gx += v[u].x;
                gy += v[u].y;
                gz += v[u].z;
                gr += v[u].w;
            }
        }
        g[kGradCenter] = gx;
        g[kGradCenter + 1] = gy;
        g[kGradCenter + 2] = gz;
        g[kGradRadius] = gr;
    }
    const SphereState s0 = a.t.sphere0[sc];
    // forward branch decisions, as sphere_advance computes them
    float v[3] = {s0.v[0], __fadd_rn(s0.v[1], __fmul_rn(c.sph_gravity, c.dt)), s0.v[2]};
    float p[3];
    const float lo_b[3] = {c.bminx, c.bminy, c.bminz}, hi_b[3] = {c.bmaxx, c.bmaxy, c.bmaxz};
    bool lo[3], hi[3];
    for (int k = 0; k < 3; ++k) {
        v[k] = __fmul_rn(v[k], c.sph_drag);
        p[k] = __fadd_rn(s0.c[k], __fmul_rn(v[k], c.dt));
        lo[k] = __fsub_rn(p[k], s0.r) < lo_b[k];
        if (lo[k]) p[k] = __fadd_rn(lo_b[k], s0.r);
        hi[k] = __fadd_rn(p[k], s0.r) > hi_b[k];
    }
    double* g = a.grads + size_t(sc) * kGradStride;
    double cb[3] = {g[kGradCenter], g[kGradCenter + 1], g[kGradCenter + 2]};
    double vb[3] = {g[kGradVel], g[kGradVel + 1], g[kGradVel + 2]};
    double rb = g[kGradRadius];
    const double rest = c.sph_rest;
    for (int k = 2; k >= 0; --k) {
        if (hi[k]) {  // p = hi - r, v = -v rest
            rb -= cb[k];
            cb[k] = 0.0;
            vb[k] *= -rest;
        }
        if (lo[k]) {  // p = lo + r, v = -v rest
            rb += cb[k];
            cb[k] = 0.0;
            vb[k] *= -rest;
        }
    }
    for (int k = 0; k < 3; ++k) {
        vb[k] = (vb[k] + cb[k] * double(c.dt)) * double(c.sph_drag);  // p = c + v dt, v = v drag
        g[kGradCenter + k] = cb[k];
        g[kGradVel + k] = vb[k];
    }
    g[kGradRadius] = rb;
}

}  // namespace

cudaError_t launch_adjoint_step(const AdjArgs& a, cudaStream_t s) {
    if (a.n == 0) return cudaSuccess;
    const uint32_t grid = cdiv(a.n, kBlock), sweep_grid = cdiv(a.n, kSweepBlock);
    const bool team = team_lanes(a.n, a.n) != 0;
    const uint32_t team_grid = cdiv(a.n, kTeamBlock / kTeam);
    k_adj_finalize<<<grid, kBlock, 0, s>>>(a);
    for (uint32_t it = a.iterations; it-- > 0;) {
        k_adj_pre<<<grid, kBlock, 0, s>>>(a, it);
        if (team && a.scorr4)
            k_adj_delta_team<4><<<team_grid, kTeamBlock, 0, s>>>(a, it);
        else if (team)
            k_adj_delta_team<0><<<team_grid, kTeamBlock, 0, s>>>(a, it);
        else if (a.common)
            k_adj_delta<4, true><<<sweep_grid, kSweepBlock, 0, s>>>(a, it);
        else if (a.scorr4)
            k_adj_delta<4, false><<<sweep_grid, kSweepBlock, 0, s>>>(a, it);
        else
            k_adj_delta<0, false><<<sweep_grid, kSweepBlock, 0, s>>>(a, it);
        k_adj_lbar<<<grid, kBlock, 0, s>>>(a, it);
        if (team)
            k_adj_lambda_team<<<team_grid, kTeamBlock, 0, s>>>(a, it);
        else if (a.common)
            k_adj_lambda<true><<<sweep_grid, kSweepBlock, 0, s>>>(a, it);
        else
            k_adj_lambda<false><<<sweep_grid, kSweepBlock, 0, s>>>(a, it);
    }
    k_adj_predict<<<grid, kBlock, 0, s>>>(a);
    if (a.nscenes && a.sum_chunks) k_adj_sphere_sum<<<dim3(a.sum_chunks, a.nscenes), kBlock, 0, s>>>(a);
    k_adj_sphere<<<cdiv(a.nscenes, 128), 128, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_adjoint_finish(const AdjArgs& a, cudaStream_t s) {
    if (a.n == 0 || a.nscenes == 0) return cudaSuccess;
    k_adj_k_part<<<dim3(a.sum_chunks, a.nscenes), kBlock, 0, s>>>(a);
    k_adj_k_sum<<<a.nscenes, 32, 0, s>>>(a);
    return cudaGetLastError();
}

uint32_t adjoint_launch_count(uint32_t iterations) { return 4u + 4u * iterations; }

}  // namespace mpb
