// pbf_items.cuh — the per-particle and per-slot operations of the PBF step as
// device functions, shared by the single-scene kernels (pbf_hash.cu,
// pbf_solver.cu) and the persistent multi-scene kernel (pbf_batch.cu).
//
//   sphere_advance   Engine.cpp:694-707 (host-side sphere kinematics)
//   predict_item     predictPositions, Constraints.metal:54-66
//   count_cell       hashCells + countCells, Spatial.metal:49-70
//   scatter_item     scatterParticles, Spatial.metal:169-180 (rank from the count)
//   sort_gather_item stable order + gatherPositions, Spatial.metal:190-198
//   long_segment     the same for cells of more than kSegMax particles
//   count_neighbors_item  countNeighbors, Spatial.metal:207-243
//   lambda_*_item    densityLambdaSorted, Constraints.metal:82-131
//   delta_item       applyDeltaSorted + sphereCollision (+ scatter-back,
//                    finalizeStep, computeFoam for the last iteration),
//                    Constraints.metal:140-213, 262-353
//
// Solver state (cell-anchored local coordinates): each particle's position is
// A(c) + l, with c its hash cell (fixed for the step), A(c) = origin +
// c * cellSize per axis in FP32 and l a small FP32 offset.  Neighbour vectors
// are ((A_i - A_cell(k)) + l_i) - l_k with A_i - A_cell(k) exact (Sterbenz:
// neighbouring anchors of one sign are within a factor of two of each other,
// except next to a zero coordinate, where the difference is off by at most
// half an ulp of 0.1 m, ~4e-9 m), so they carry ~1e-8 m of rounding instead of
// the ~5e-7 m of FP32 absolute coordinates at 4-8 m, while each candidate is
// still one 16-byte load.  Box clamps, the sphere push and finalize run in
// FP64 on A + l.  The first lambda pass runs on the absolute FP32 predicted
// positions exactly as the reference does (so the neighbour count it fuses in
// is bit-exact) and converts them to offsets, which is exact for the
// particle's own cell.
#pragma once

#include "pbf_kernels.h"

namespace mpb {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kPassAll = 1 << 30;  // a prefilter threshold every candidate passes

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// ---- hash ------------------------------------------------------------------

// Sphere kinematics (Engine.cpp:694-707), in FP32 with one rounding per
// operation, run by one thread before the hash.
__device__ inline void sphere_advance(const StepConsts& c, SphereState* s) {
    float vx = s->v[0], vy = s->v[1], vz = s->v[2];
    vy = __fadd_rn(vy, __fmul_rn(c.sph_gravity, c.dt));
    vx = __fmul_rn(vx, c.sph_drag);
    vy = __fmul_rn(vy, c.sph_drag);
    vz = __fmul_rn(vz, c.sph_drag);
    float p[3] = {__fadd_rn(s->c[0], __fmul_rn(vx, c.dt)), __fadd_rn(s->c[1], __fmul_rn(vy, c.dt)),
                  __fadd_rn(s->c[2], __fmul_rn(vz, c.dt))};
    float v[3] = {vx, vy, vz};
    const float lo[3] = {c.bminx, c.bminy, c.bminz};
    const float hi[3] = {c.bmaxx, c.bmaxy, c.bmaxz};
    const float r = s->r;
    for (int a = 0; a < 3; ++a) {
        if (__fsub_rn(p[a], r) < lo[a]) {
            p[a] = __fadd_rn(lo[a], r);
            v[a] = __fmul_rn(-v[a], c.sph_rest);
        }
        if (__fadd_rn(p[a], r) > hi[a]) {
            p[a] = __fsub_rn(hi[a], r);
            v[a] = __fmul_rn(-v[a], c.sph_rest);
        }
    }
    for (int a = 0; a < 3; ++a) {
        s->c[a] = p[a];
        s->v[a] = v[a];
    }
}

// prev = p; v' = v + g dt; p' = p + v' dt (each one fused multiply-add);
// writes p' over pos[i] and returns it.  A non-finite input would survive as
// a finite clamped position (the reference's clamp semantics), so it is
// flagged here, on entry.
__device__ __forceinline__ float4 predict_item(const StepConsts& c, uint32_t i,
                                               float4* __restrict__ pos,
                                               const float4* __restrict__ vel,
                                               float4* __restrict__ prev, uint32_t* err) {
    float4 p = pos[i];
    const float4 v = vel[i];
    if (!isfinite(p.x + p.y + p.z + v.x + v.y + v.z)) atomicOr(err, kDevErrNaN);
    prev[i] = p;
    const float vx = __fmaf_rn(c.gravx, c.dt, v.x);
    const float vy = __fmaf_rn(c.gravy, c.dt, v.y);
    const float vz = __fmaf_rn(c.gravz, c.dt, v.z);
    p.x = __fmaf_rn(vx, c.dt, p.x);
    p.y = __fmaf_rn(vy, c.dt, p.y);
    p.z = __fmaf_rn(vz, c.dt, p.z);
    pos[i] = p;
    return p;
}

// Warp-aggregated count: every lane of the warp calls it (active or not);
// each active lane gets its rank among the particles of cell `cell` counted
// so far, in *rank.  One atomic per distinct cell in the warp.
__device__ __forceinline__ void count_cell(bool active, uint32_t cell, uint32_t* __restrict__ counts,
                                           uint32_t* rank) {
    const unsigned act = __ballot_sync(kFull, active);
    if (active) {
        const unsigned peers = __match_any_sync(act, cell);
        const int leader = __ffs(peers) - 1;
        const int lane = threadIdx.x & 31;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(&counts[cell], uint32_t(__popc(peers)));
        base = __shfl_sync(act, base, leader);
        *rank = base + uint32_t(__popc(peers & lanemask_lt()));
    }
}

// scatterParticles without the second atomic: slot = cellStart + rank.
__device__ __forceinline__ void scatter_item(uint32_t i, const uint32_t* __restrict__ hash,
                                             const uint32_t* __restrict__ off,
                                             const uint32_t* __restrict__ cstart,
                                             uint32_t* __restrict__ tmp) {
    tmp[cstart[hash[i]] + off[i]] = i;
}

// A particle's place in sorted order: its index, predicted position, quantized
// position and the x anchor of its cell.  strays (may be NULL) is set to 1 when the
// position lies outside the cell.
__device__ __forceinline__ void place(const StepConsts& c, uint32_t d, uint32_t j, const float4& p,
                                      uint32_t* __restrict__ sidx, float4* __restrict__ sorted,
                                      uint32_t* __restrict__ qpos, float* __restrict__ xa,
                                      uint32_t* strays) {
    int cx, cy, cz;
    cell_of(c.g, p.x, p.y, p.z, cx, cy, cz);
    sidx[d] = j;
    sorted[d] = p;
    const float ax = anchor_x(c.g, cx);
    xa[d] = ax;
    const float lx = __fsub_rn(p.x, ax), ly = __fsub_rn(p.y, anchor_y(c.g, cy));
    const float lz = __fsub_rn(p.z, anchor_z(c.g, cz));
    qpos[d] = quantize<false>(c, cx + c.g.lx, cy + c.g.ly, cz + c.g.lz, lx, ly, lz);
    // (count_neighbors_item) a position outside its cell, or not finite
    if (strays && !(fminf(fminf(lx, ly), lz) >= -c.q_slack && fmaxf(fmaxf(lx, ly), lz) <= c.g.cs + c.q_slack &&
                    lx + ly + lz < 1e30f))  // (fminf and fmaxf drop a NaN)
        *strays = 1u;
}

// Stable re-rank inside the cell segment + gatherPositions: the slot's
// particle j moves to cellStart + (number of particles of its cell with a
// smaller index).  A cell of more than kSegMax particles is left to
// long_segment: on_long(cell) is called once, by its first slot.
template <class OnLong>
__device__ __forceinline__ void sort_gather_item(const StepConsts& sc, uint32_t s,
                                                 const uint32_t* __restrict__ tmp,
                                                 const uint32_t* __restrict__ hash,
                                                 const uint32_t* __restrict__ cstart,
                                                 const float4* __restrict__ pos,
                                                 uint32_t* __restrict__ sidx,
                                                 float4* __restrict__ sorted,
                                                 uint32_t* __restrict__ qpos, float* __restrict__ xa,
                                                 uint32_t* strays, OnLong&& on_long) {
    const uint32_t j = tmp[s];
    const uint32_t c = hash[j];
    const uint32_t a = cstart[c], b = cstart[c + 1];
    if (b - a > kSegMax) {
        if (s == a) on_long(c);
        return;
    }
    uint32_t rank = 0;
    for (uint32_t k = a; k < b; ++k) rank += (tmp[k] < j) ? 1u : 0u;
    place(sc, a + rank, j, pos[j], sidx, sorted, qpos, xa, strays);
}

// A long segment, by the whole block: rank(j) = number of particles j' < j of
// cell c, from a block-wide scan over the particle indices [p0, p1) that can
// hold the cell's particles.  s_warp: blockDim.x / 32 words of shared memory.
__device__ inline void long_segment(const StepConsts& sc, uint32_t c, uint32_t p0, uint32_t p1,
                                    const uint32_t* __restrict__ hash,
                                    const uint32_t* __restrict__ cstart,
                                    const float4* __restrict__ pos, uint32_t* __restrict__ sidx,
                                    float4* __restrict__ sorted, uint32_t* __restrict__ qpos,
                                    float* __restrict__ xa, uint32_t* strays, uint32_t* s_warp) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t a = cstart[c], len = cstart[c + 1] - a;
    uint32_t running = 0;
    for (uint32_t base = p0; base < p1 && running < len; base += blockDim.x) {
        const uint32_t j = base + threadIdx.x;
        const bool f = j < p1 && hash[j] == c;
        const unsigned m = __ballot_sync(kFull, f);
        if (lane == 0) s_warp[warp] = __popc(m);
        __syncthreads();
        uint32_t before = 0, blk = 0;
        for (uint32_t w = 0; w < blockDim.x / 32; ++w) {
            if (w < warp) before += s_warp[w];
            blk += s_warp[w];
        }
        if (f)
            place(sc, a + running + before + __popc(m & lanemask_lt()), j, pos[j], sidx, sorted, qpos, xa,
                  strays);
        running += blk;
        __syncthreads();
    }
}

// ---- solver ------------------------------------------------------------------

// In-range masks of one lambda pass.  For each particle and each of the 9
// stencil rows [b0, b3), bit i is set when candidate slot (b0 & ~3) + i lies
// within h (the row's first slot rounded down to a 16-byte boundary of the
// quantized positions).  The delta pass of the same iteration sees the same
// positions and the same stencil, hence exactly the same in-range pairs, so it
// walks these bits instead of sweeping the 27 cells again.  Row-major layout
// (row r of slot s at r * stride + s): the warp's stores and loads of one row
// coalesce.  A row that does not end within 32 slots of its rounded start keeps
// those bits and sets bit r of overflow[s]; the delta pass distance-tests that
// row's remaining candidates again.
struct RowMasks {
    uint32_t* rows;
    uint32_t* overflow;
    uint32_t stride;
};

// The solver arithmetic below is written with explicit round-to-nearest
// operations (__fmaf_rn, __fmul_rn, __fadd_rn, and their FP64 forms): the
// compiler may not fuse or split them, so every kernel that inlines these
// functions (the single-scene kernels, the persistent batch kernel) rounds
// identically and gives bit-identical results.

// 1 / sqrt(x) of a normal x (the value of rsqrtf without its handling of
// subnormal arguments).
__device__ __forceinline__ float rsqrt_normal(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Two FP32 values in one 64-bit register, and the packed operations on them: each
// half rounds exactly as the single operation does.  They save the lambda pass's
// pair body three of about 50 instructions (1M-particle dam break: 1463 -> 1440 us
// per step); packing the neighbour vector's x and y too, or the delta pass's sums,
// costs as many register moves as it saves.
struct F2 {
    unsigned long long v;
    F2() = default;
    __device__ __forceinline__ F2(float a, float b) { asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(a), "f"(b)); }
    __device__ __forceinline__ void get(float& a, float& b) const {
        asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    }
};
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
// The pair functions take the constants as C: StepConsts, or PairConsts where a
// batch's scenes share them.

// densityLambdaSorted's sums for one particle (Constraints.metal:99-121): the
// density starts at the particle's own W(0) whether or not its slot lies in
// the stencil of its current cell (a particle can drift two cells from its
// hash cell within a step), and add() takes the terms of every other
// in-range candidate at offset r, r2 = |r|^2 < h^2, in slot order.  A
// candidate at the particle's own position (r2 = 0) adds W(0) and no gradient.
struct LambdaAcc {
    float dens = 0.0f, gx = 0.0f, gy = 0.0f, gz = 0.0f, gsq = 0.0f;
    // the particle's own W(0)
    template <class C>
    __device__ __forceinline__ void self(const C& c) {
        dens = __fmul_rn(__fmul_rn(__fmul_rn(c.poly6, c.h2), c.h2), c.h2);
    }
    // no effect unless r2 < h^2
    template <class C>
    __device__ __forceinline__ void add(const C& c, float rx, float ry, float rz, float r2) {
        const float d = __fsub_rn(c.h2, r2);
        const float rinv = rsqrt_normal(r2);
        const float hd = fmaxf(__fsub_rn(c.h, __fmul_rn(r2, rinv)), 0.0f);
        float w, s1;  // poly6 d d and -spiky hd hd
        const F2 dh(d, hd);
        mul2(mul2(F2(c.poly6, -c.spiky), dh), dh).get(w, s1);
        const float sc = __fmul_rn(s1, rinv);
        const float sc2 = __fmul_rn(sc, sc);
        if (r2 < c.h2) dens = __fmaf_rn(w, d, dens);
        if (r2 < c.h2 && r2 > 1e-12f) {
            fma2(F2(sc, sc), F2(rx, ry), F2(gx, gy)).get(gx, gy);
            fma2(F2(sc, sc2), F2(rz, r2), F2(gz, gsq)).get(gz, gsq);
        }
    }
    __device__ __forceinline__ float lambda(const StepConsts& c) const {
        const float C = __fmaf_rn(dens, c.inv_rho0, -1.0f);
        const float g2 = __fmaf_rn(gz, gz, __fmaf_rn(gy, gy, __fmaf_rn(gx, gx, gsq)));
        const float denom = __fmaf_rn(__fmul_rn(c.inv_rho0, c.inv_rho0), g2, c.eps);
        return __fdiv_rn(-C, denom);
    }
};

// ratio^n of s_corr; N = 4 fixes the exponent at compile time (the
// reference's, Constraints.metal:179), N = 0 takes c.scorr_n.  Both give
// the same bits for n = 4.
template <uint32_t N>
__device__ __forceinline__ float scorr_pow(float x, uint32_t n) {
    if (N == 4u || (N == 0u && n == 4u)) {
        const float x2 = __fmul_rn(x, x);
        return __fmul_rn(x2, x2);
    }
    float r = 1.0f;
    for (uint32_t e = 0; e < n; ++e) r = __fmul_rn(r, x);
    return r;
}

// Position-correction term of one in-range candidate (Constraints.metal:
// 170-181) with the common factor -spiky / rho0 left out (delta_item
// applies c.delta_scale once to the sum):
//   (lambda_i + lambda_j - k (W / W(dq))^n) (h - r)^2 / r  r
// W / W(dq) = d^3 poly6 / W(dq) (c.scorr_pq); the sum of lambdas and s_corr is
// one fused multiply-add.  No effect unless r2 < h^2.
template <uint32_t N, class C>
__device__ __forceinline__ float delta_coef(const C& c, float li, float lj, float r2) {
    const float d = __fsub_rn(c.h2, r2);
    const float ratio = __fmul_rn(__fmul_rn(__fmul_rn(d, d), d), c.scorr_pq);
    const float rinv = rsqrt_normal(r2);
    const float hd = fmaxf(__fsub_rn(c.h, __fmul_rn(r2, rinv)), 0.0f);
    return __fmul_rn(__fmaf_rn(-c.scorr_k, scorr_pow<N>(ratio, c.scorr_n), __fadd_rn(li, lj)),
                     __fmul_rn(__fmul_rn(hd, hd), rinv));
}

template <uint32_t N, class C>
__device__ __forceinline__ void delta_add(const C& c, float li, float lj, float rx, float ry,
                                          float rz, float r2, float& dx, float& dy, float& dz) {
    const float coef = delta_coef<N>(c, li, lj, r2);
    if (r2 < c.h2 && r2 > 1e-12f) {
        dx = __fmaf_rn(coef, rx, dx);
        dy = __fmaf_rn(coef, ry, dy);
        dz = __fmaf_rn(coef, rz, dz);
    }
}

// A load of an array that other kernels write.  RO: nothing in this launch writes it,
// so it may go through the read-only path.  The persistent batch kernel writes these
// arrays in one phase and reads them in another, which only an ordinary load may do
// (its grid barrier orders those).  Written as instructions: as plain C++ loads the
// compiler moves and splits them, spills more (144 -> 232 bytes of spill loads) and a
// step of 256 cubes takes 4.28 ms instead of 4.00.
__device__ __forceinline__ float load_ordinary(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 load_ordinary(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ uint4 load_ordinary(const uint4* p) {
    uint4 v;
    asm volatile("ld.global.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}
template <bool RO, class T>
__device__ __forceinline__ T load(const T* p) {
    if constexpr (RO)
        return __ldg(p);
    else
        return load_ordinary(p);
}

// First slot of a row mask: the row's first slot, rounded down to a 16-byte
// boundary of the quantized positions.
__device__ __forceinline__ uint32_t row_base(uint32_t b0) { return b0 & ~3u; }

// Offsets of a particle to the three stencil rows along y and along z.
struct RowOffsets {
    float y0, y1, y2, z0, z1, z2;
    // (A_i - A_row) + l_i for the rows around cell (cy, cz)
    __device__ __forceinline__ static RowOffsets anchored(const GridDev& g, int cy, int cz, float ay, float az,
                                                          float ly, float lz) {
        return RowOffsets{__fadd_rn(__fsub_rn(ay, anchor_y(g, cy - 1)), ly),
                          __fadd_rn(__fsub_rn(ay, anchor_y(g, cy)), ly),
                          __fadd_rn(__fsub_rn(ay, anchor_y(g, cy + 1)), ly),
                          __fadd_rn(__fsub_rn(az, anchor_z(g, cz - 1)), lz),
                          __fadd_rn(__fsub_rn(az, anchor_z(g, cz)), lz),
                          __fadd_rn(__fsub_rn(az, anchor_z(g, cz + 1)), lz)};
    }
};

// Whether p holds on any lane that is here too.  Lanes that walk full queues do so
// together: each on its own, while the others of its warp wait, 50,000 particles in a
// cloud with clumps of thousands took 31.4 ms per step; together, 13.5.
__device__ __forceinline__ bool warp_any(bool p) { return __any_sync(__activemask(), p); }

// Per-thread queue of row chunks with candidates to visit, in shared memory:
// entry e of thread t at (e * BS + t), 8 bytes: the chunk's bits (first
// candidate in bit 31), and 4 times its first slot (a multiple of 4, below 2^30) with
// the row's y index in bits 0-1 and its z index in bits 2-3.  The lanes of a warp have
// very different numbers of candidates per row but similar totals: walking all
// rows' bits in one loop, each lane moving to its next chunk by itself with a
// predicated load, takes 38 iterations where row by row takes 87 (lattice or
// disordered fluid at rest density, 31 pairs per particle).  k_lambda on the
// 1,003,520-particle dam break: 214 M -> 150 M warp instructions, 17 -> 25 of 32
// threads active, 281 -> 184 us; k_delta 161 M -> 95 M, 14 -> 27, 150-171 -> 130 us.
// 16-byte entries that hold the two offsets instead of the row's indices leave
// too little of the SM's memory for L1 (k_delta 258 us, 13% hits).  With the rows
// in a loop of nine fixed ones, their bounds a row ahead (lambda) or all loads up
// front (delta): 167 and 107 us.
//
// 9 rows and 6 more chunks of long ones.  A lane whose queue is full walks it in the
// middle of the sweep while its warp waits: with 10 entries a few such warps
// decided the time of a scene that fits the GPU at once (97,336 particles: 31 us
// per lambda pass on the slowest SM, 20 on average).  15 is the most that leaves L1
// as large as 10 do (eight blocks of 128 use 131 KB).
constexpr uint32_t kQueue = 15;
static_assert(kQueue >= 10, "room for every row's first chunk and an empty one");

template <uint32_t BS>
struct PairQueue {
    uint32_t base;       // shared-memory address of this thread's entry 0
    uint32_t tail;       // where the next entry goes
    uint32_t pairs = 0;  // bits in the queue

    __device__ __forceinline__ explicit PairQueue(uint2* shared)
        : base(uint32_t(__cvta_generic_to_shared(shared + threadIdx.x))), tail(base) {}
    // whether fewer than `entries` more fit
    __device__ __forceinline__ bool short_of(uint32_t entries) const {
        return tail + entries * (BS * 8u) > base + kQueue * BS * 8u;
    }
    // code: y | z << 2.  An empty mask takes no entry.
    __device__ __forceinline__ void push(uint32_t mask, uint32_t first, uint32_t code) {
        asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(tail), "r"(mask), "r"(first * 4u | code));
        tail += mask ? BS * 8u : 0u;
        pairs += __popc(mask);
    }
    // The next bit's slot and offsets; `at`, `mask`, `first` are the walk's state.
    __device__ __forceinline__ uint32_t next(const RowOffsets& o, uint32_t& at, uint32_t& mask, uint32_t& first,
                                             float& oy, float& oz) const {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.eq.u32 p, %0, 0;\n\t"
            "@p ld.shared.v2.b32 {%0, %1}, [%2];\n\t"
            "@p add.u32 %2, %2, %3;\n\t}"
            : "+r"(mask), "+r"(first), "+r"(at)
            : "n"(BS * 8u));
        uint32_t t;
        asm("bfind.shiftamt.u32 %0, %1;" : "=r"(t) : "r"(mask));
        mask &= 0x7fffffffu >> t;
        oy = (first & 2u) ? o.y2 : ((first & 1u) ? o.y1 : o.y0);
        oz = (first & 8u) ? o.z2 : ((first & 4u) ? o.z1 : o.z0);
        return (first >> 4) * 4u + t;
    }
    // visit(slot, fetch(slot), oy, oz) for every bit, in the order queued; empties
    // the queue.  PIPE: each candidate is fetched while the one before it is
    // visited (1-2% of a step; not for walks in the middle of a sweep, whose
    // registers it would spill)
    template <bool PIPE, class Fetch, class Visit>
    __device__ __forceinline__ void drain(const RowOffsets& o, Fetch&& fetch, Visit&& visit) {
        uint32_t at = base, mask = 0, first = 0;
        float oy = 0.0f, oz = 0.0f;
        if (!PIPE) {
            for (; pairs > 0; --pairs) {
                const uint32_t k = next(o, at, mask, first, oy, oz);
                visit(k, fetch(k), oy, oz);
            }
        } else if (pairs) {
            uint32_t k = next(o, at, mask, first, oy, oz);
            auto q = fetch(k);
            while (--pairs) {
                const float y = oy, z = oz;
                const uint32_t kn = next(o, at, mask, first, oy, oz);
                const auto qn = fetch(kn);
                visit(k, q, y, z);
                k = kn;
                q = qn;
            }
            visit(k, q, oy, oz);
        }
        tail = base;
    }
};

// The 9 rows of the stencil around cell (cx, cy, cz), z outer, y inner: row
// (cy - 1 + y, cz - 1 + z) is number 3 z + y and starts at cell `base`, advanced by
// next_y after each row and by next_z after each plane.  Rows outside the grid are
// not valid (all of them for a particle that drifted more than a cell past a
// scene's sub-grid in x).
struct StencilRows {
    uint32_t base, nx, next_y, next_z;
    int gy, gz;
    __device__ __forceinline__ StencilRows(const GridDev& g, int cx, int cy, int cz) {
        const int x0 = max(cx - 1, 0), n = min(cx + 1, g.gx - 1) - x0 + 1;
        nx = uint32_t(n);
        gy = n > 0 ? g.gy : 0;
        gz = g.gz;
        next_y = uint32_t(g.gx);
        next_z = uint32_t(g.gx) * uint32_t(g.gy - 3);
        base = cell_hash(g, x0, cy - 1, cz - 1);
    }
    __device__ __forceinline__ bool valid(int y, int z) const {
        return uint32_t(y) < uint32_t(gy) && uint32_t(z) < uint32_t(gz);
    }
};

// Phase 1 of a sweep: the prefilter's bits of slots [c0, c1), c0 a multiple of 4, at
// most 32 of them (first one in bit 31), without slot s.  Reads up to 3 slots past
// c1 (whole groups of four).
template <bool RO>
__device__ __forceinline__ uint32_t row_bits(const uint32_t* __restrict__ qsrc, uint32_t qi, int nthr, uint32_t c0,
                                             uint32_t c1, uint32_t s) {
    uint32_t mask = 0, k = c0;
    auto test = [&](uint32_t w) {
        const int d = int(qi - w);
        mask = __funnelshift_l(uint32_t(__dp4a(d, d, nthr)), mask, 1);
    };
    for (; k < c1; k += 4) {
        const uint4 q = load<RO>(reinterpret_cast<const uint4*>(qsrc + k));
        test(q.x);
        test(q.y);
        test(q.z);
        test(q.w);
    }
    mask <<= 32u - (k - c0);
    mask &= 0xffffffffu << (32u - (c1 - c0));
    if (s - c0 < 32u) mask &= ~(0x80000000u >> (s - c0));
    return mask;
}

// Two-phase sweep of the 27-cell stencil around cell (cx, cy, cz).  Each row
// (3 consecutive cells, one contiguous slot range) is taken in chunks of 32
// candidates.
//
// Phase 1 tests the byte-quantized positions qsrc (quantize() above): per
// candidate one 32-bit subtraction, one __dp4a whose sum starts at -threshold
// and one funnel shift that collects its sign bit; one 16-byte load brings four
// candidates.  The threshold admits every pair the exact test could accept
// (set_prefilter), about 9% more than are in range.  Phase 2 visits just the
// set bits of all rows, loads the candidate's position and calls
// body(k, q, rx, ry, rz, r2), k the candidate's slot, in slot order row by row;
// the body ignores a candidate that fails the exact test r2 < h^2.  So counts
// and sums are those of the exact test alone.
//
// ANCHORED = false: (px, py, pz) is the absolute FP32 position and r = p - q.
// ANCHORED = true:  (px, py, pz) is the offset l from the anchor (aix, aiy,
// aiz) of the particle's hash cell and each candidate carries the x anchor of
// its own hash cell in w (the delta pass's output):
// r = ((A_i - A_cell(k)) + l_i) - l_k, A_i - A_cell(k) exact.
//
// Every row of the stencil stores the bits of its first chunk (the particle's
// own bit cleared) for the delta pass, and a row longer than one chunk sets
// its bit in the overflow word.
template <bool ANCHORED, bool RO, uint32_t BS, class Body>
__device__ __forceinline__ void sweep(const StepConsts& c, const float4* __restrict__ src,
                                      const uint32_t* __restrict__ qsrc,
                                      const uint32_t* __restrict__ cstart, int cx, int cy, int cz,
                                      float px, float py, float pz, float aix, float aiy, float aiz,
                                      uint32_t qi, int nthr, uint32_t s, const RowMasks& masks,
                                      PairQueue<BS> queue, Body&& body) {
    auto fetch = [&](uint32_t k) { return load<RO>(&src[k]); };
    auto visit = [&](uint32_t k, const float4& q, float oy, float oz) {
        const float ox = ANCHORED ? __fadd_rn(__fsub_rn(aix, q.w), px) : px;
        const float rx = __fsub_rn(ox, q.x), ry = __fsub_rn(oy, q.y), rz = __fsub_rn(oz, q.z);
        body(k, q, rx, ry, rz, dist2(rx, ry, rz));
    };
    RowOffsets o{py, py, py, pz, pz, pz};
    if (ANCHORED) o = RowOffsets::anchored(c.g, cy, cz, aiy, aiz, py, pz);
    const StencilRows rows(c.g, cx, cy, cz);
    uint32_t over = 0, base = rows.base, b0 = 0, b3 = 0;
    uint32_t* out = masks.rows + s;
    // bits of slots [c0, c1), c0 a multiple of 4, at most 32 of them, in row (y, z)
    auto bits = [&](uint32_t c0, uint32_t c1, int y, int z) {
        if (nthr != -kPassAll) return row_bits<RO>(qsrc, qi, nthr, c0, c1, s);
        // nothing the prefilter could tell apart: the exact test decides, or the
        // queue would carry every candidate (100,000 particles 300 m outside the box
        // 5.6 ms per step, this way 2.1)
        const float oy = y == 0 ? o.y0 : (y == 1 ? o.y1 : o.y2), oz = z == 0 ? o.z0 : (z == 1 ? o.z1 : o.z2);
        uint32_t mask = 0;
#pragma unroll 1
        for (uint32_t k = c0; k < c1; ++k) {
            const float4 q = fetch(k);
            const float ox = ANCHORED ? __fadd_rn(__fsub_rn(aix, q.w), px) : px;
            const float r2 = dist2(__fsub_rn(ox, q.x), __fsub_rn(oy, q.y), __fsub_rn(oz, q.z));
            mask |= r2 < c.h2 && k != s ? 0x80000000u >> (k - c0) : 0u;
        }
        return mask;
    };
    if (rows.valid(cy - 1, cz - 1)) {
        b0 = cstart[base];
        b3 = cstart[base + rows.nx];
    }
#pragma unroll 1  // (unrolled, the rows' code no longer fits the instruction cache)
    for (int z = 0; z < 3; ++z) {
#pragma unroll 1
        for (int y = 0; y < 3; ++y, out += masks.stride) {
            // the next row's bounds are on their way while this one is tested
            const int y1 = y < 2 ? y + 1 : 0, z1 = y < 2 ? z : z + 1;
            base += rows.next_y + (y < 2 ? 0u : rows.next_z);
            uint32_t n0 = 0, n3 = 0;
            if (z1 < 3 && rows.valid(cy - 1 + y1, cz - 1 + z1)) {
                n0 = cstart[base];
                n3 = cstart[base + rows.nx];
            }
            uint32_t mask = 0;
            const uint32_t a0 = row_base(b0);
            if (b0 < b3) mask = bits(a0, min(a0 + 32u, b3), y, z) & (0xffffffffu >> (b0 - a0));
            // the bits of the row's first chunk (the whole row if b3 - a0 <= 32)
            *out = mask;
            const uint32_t code = uint32_t(y) | (uint32_t(z) << 2);
            queue.push(mask, a0, code);
            if (__builtin_expect(b3 > a0 + 32u, 0)) {  // (never an empty row)
                const uint32_t row = uint32_t(3 * z + y);
                over |= 1u << row;
                for (uint32_t c0 = a0 + 32u; c0 < b3; c0 += 32) {
                    // Room for this chunk and the first ones of the rows to come.  A vote
                    // here costs the single-scene kernels 1-2% of ordinary states (the
                    // batch kernel nothing), so there the lanes, which mostly walk one
                    // row, meet at every eighth chunk of it, where those with room for
                    // less than four more walk their queues.
                    const bool meet = RO && ((c0 - a0) & 224u) == 32u;
                    const bool full = queue.short_of(meet ? 13u - row : 9u - row);
                    if (RO ? full : warp_any(full)) queue.template drain<false>(o, fetch, visit);
                    queue.push(bits(c0, min(c0 + 32u, b3), y, z), c0, code);
                }
            }
            b0 = n0;
            b3 = n3;
        }
    }
    masks.overflow[s] = over;
    queue.template drain<true>(o, fetch, visit);
}

// The prefilter's arguments of a particle at offset l from the corner of its
// hash cell (dense coordinates): its quantized word, and minus the threshold.  A
// particle far outside the grid (or not finite) tests every candidate exactly.
__device__ __forceinline__ int prefilter(const StepConsts& c, int hx, int hy, int hz, float lx, float ly,
                                         float lz, uint32_t& qi) {
    qi = quantize<true>(c, hx, hy, hz, lx, ly, lz);
    const bool near = fabsf(lx) < c.q_lim && fabsf(ly) < c.q_lim && fabsf(lz) < c.q_lim;
    return near ? -c.q_thr : -kPassAll;
}

// countNeighbors in sorted order.  Most candidates are decided by their quantized
// distance: more than q_thr is out of range, at most q_in is in range (when no
// particle lies outside its cell, so that no byte difference wraps to a small
// value: `strays` is 0), and only the shell in between, a sixth of the
// neighbours, is tested exactly.

// The same where that inner threshold does not hold: strays, or a particle that the
// prefilter cannot place.  All that passes the outer threshold is tested exactly,
// and where that is most of a row, the row goes straight through the exact test
// (50,000 particles in a cloud with clumps of thousands, some outside the box: 3.24 ms
// for buildSpatialHash with every candidate queued, 0.49 this way).  A function of
// its own: inlined, it costs the ordinary count 5 of 59 us (500,009 particles).
template <bool RO, uint32_t BS>
__device__ __noinline__ uint32_t count_neighbors_exact(const StepConsts& c, uint32_t s, float4 p,
                                                       const float4* __restrict__ sorted,
                                                       const uint32_t* __restrict__ qsrc,
                                                       const uint32_t* __restrict__ cstart, int cx, int cy, int cz,
                                                       uint32_t qi, int nthr, PairQueue<BS> queue) {
    const int x0 = max(cx - 1, 0), x1 = min(cx + 1, c.g.gx - 1);
    const int y0 = max(cy - 1, 0), y1 = min(cy + 1, c.g.gy - 1);
    const int z0 = max(cz - 1, 0), z1 = min(cz + 1, c.g.gz - 1);
    uint32_t cnt = 0;
    auto fetch = [&](uint32_t k) { return load<RO>(&sorted[k]); };
    auto near = [&](const float4& q) { return dist2(q.x - p.x, q.y - p.y, q.z - p.z) < c.h2; };
    auto visit = [&](uint32_t, const float4& q, float, float) { cnt += near(q) ? 1u : 0u; };
    const RowOffsets none{};
    const bool blind = nthr == -kPassAll;
    bool crowded = blind;
    for (int z = z0; z <= z1; ++z)
        for (int y = y0; y <= y1; ++y) {
            const uint32_t b0 = cstart[cell_hash(c.g, x0, y, z)];
            const uint32_t b3 = cstart[cell_hash(c.g, x1, y, z) + 1];
            const uint32_t a0 = row_base(b0);
            for (uint32_t c0 = b0 < b3 ? a0 : b3; c0 < b3; c0 += 32) {
                const uint32_t c1 = min(c0 + 32u, b3);
                if (warp_any(crowded)) {
                    uint32_t hits = 0;
#pragma unroll 4
                    for (uint32_t i = max(b0, c0); i < c1; ++i) hits += near(fetch(i)) && i != s ? 1u : 0u;
                    cnt += hits;
                    crowded = blind || hits >= 8u;
                    continue;
                }
                const uint32_t maybe = row_bits<RO>(qsrc, qi, nthr, c0, c1, s) & (0xffffffffu >> (max(b0, c0) - c0));
                crowded = __popc(maybe) >= 16;
                if (warp_any(queue.short_of(1u))) queue.template drain<false>(none, fetch, visit);
                queue.push(maybe, c0, 0u);
            }
        }
    queue.template drain<false>(none, fetch, visit);
    return cnt;
}

template <bool RO, uint32_t BS>
__device__ __forceinline__ void count_neighbors_item(const StepConsts& c, uint32_t s,
                                                     const float4* __restrict__ sorted,
                                                     const uint32_t* __restrict__ qsrc,
                                                     const uint32_t* __restrict__ cstart,
                                                     const uint32_t* __restrict__ sidx,
                                                     uint32_t* __restrict__ ncount, uint32_t strays,
                                                     PairQueue<BS> queue) {
    const float4 p = sorted[s];
    int cx, cy, cz;
    cell_of(c.g, p.x, p.y, p.z, cx, cy, cz);
    uint32_t qi;
    const int nthr = prefilter(c, cx + c.g.lx, cy + c.g.ly, cz + c.g.lz, __fsub_rn(p.x, anchor_x(c.g, cx)),
                               __fsub_rn(p.y, anchor_y(c.g, cy)), __fsub_rn(p.z, anchor_z(c.g, cz)), qi);
    if (strays || nthr != -c.q_thr || c.q_thr == kPassAll) {
        ncount[sidx[s]] = count_neighbors_exact<RO, BS>(c, s, p, sorted, qsrc, cstart, cx, cy, cz, qi, nthr, queue);
        return;
    }
    const int up = c.q_thr - c.q_in;
    const int x0 = max(cx - 1, 0), x1 = min(cx + 1, c.g.gx - 1);
    const int y0 = max(cy - 1, 0), y1 = min(cy + 1, c.g.gy - 1);
    const int z0 = max(cz - 1, 0), z1 = min(cz + 1, c.g.gz - 1);
    uint32_t cnt = 0;
    auto fetch = [&](uint32_t k) { return load<RO>(&sorted[k]); };
    auto visit = [&](uint32_t, const float4& q, float, float) {
        cnt += dist2(q.x - p.x, q.y - p.y, q.z - p.z) < c.h2 ? 1u : 0u;
    };
    const RowOffsets none{};
    for (int z = z0; z <= z1; ++z)
        for (int y = y0; y <= y1; ++y) {
            const uint32_t b0 = cstart[cell_hash(c.g, x0, y, z)];
            const uint32_t b3 = cstart[cell_hash(c.g, x1, y, z) + 1];
            const uint32_t a0 = row_base(b0);
            for (uint32_t c0 = b0 < b3 ? a0 : b3; c0 < b3; c0 += 32) {
                const uint32_t c1 = min(c0 + 32u, b3);
                uint32_t maybe = 0, in = 0, k = c0;
                for (; k < c1; k += 4) {
                    const uint4 q = load<RO>(reinterpret_cast<const uint4*>(qsrc + k));
                    const int d0 = int(qi - q.x), d1 = int(qi - q.y);
                    const int d2 = int(qi - q.z), d3 = int(qi - q.w);
                    const int s0 = __dp4a(d0, d0, nthr), s1 = __dp4a(d1, d1, nthr);
                    const int s2 = __dp4a(d2, d2, nthr), s3 = __dp4a(d3, d3, nthr);
                    maybe = __funnelshift_l(uint32_t(s0), maybe, 1);
                    in = __funnelshift_l(uint32_t(s0 + up), in, 1);
                    maybe = __funnelshift_l(uint32_t(s1), maybe, 1);
                    in = __funnelshift_l(uint32_t(s1 + up), in, 1);
                    maybe = __funnelshift_l(uint32_t(s2), maybe, 1);
                    in = __funnelshift_l(uint32_t(s2 + up), in, 1);
                    maybe = __funnelshift_l(uint32_t(s3), maybe, 1);
                    in = __funnelshift_l(uint32_t(s3 + up), in, 1);
                }
                const uint32_t left = 32u - (k - c0);
                uint32_t row = (0xffffffffu >> (max(b0, c0) - c0)) & (0xffffffffu << (32u - (c1 - c0)));
                if (s - c0 < 32u) row &= ~(0x80000000u >> (s - c0));
                in = (in << left) & row;
                maybe = (maybe << left) & row & ~in;
                cnt += __popc(in);
                if (warp_any(queue.short_of(1u))) queue.template drain<false>(none, fetch, visit);
                queue.push(maybe, c0, 0u);
            }
        }
    queue.template drain<false>(none, fetch, visit);
    ncount[sidx[s]] = cnt;
}

// First lambda pass: absolute FP32 predicted positions (reference arithmetic,
// so the fused neighbour count equals countNeighbors bit for bit); converts
// the state to anchored offsets for the following passes.
template <bool LAST, bool RO, uint32_t BS, class C>
__device__ __forceinline__ void lambda_first_item(const StepConsts& c, const C& pc, uint32_t s,
                                                  const float4* __restrict__ cur,
                                                  const uint32_t* __restrict__ qpos,
                                                  float4* __restrict__ nxt,
                                                  uint32_t* __restrict__ scell,
                                                  const uint32_t* __restrict__ cstart,
                                                  const uint32_t* __restrict__ sidx,
                                                  float* __restrict__ lambdas,
                                                  uint32_t* __restrict__ ncount, const RowMasks& rm,
                                                  uint2* queue) {
    const float4 p = cur[s];
    int cx, cy, cz;
    cell_of(c.g, p.x, p.y, p.z, cx, cy, cz);
    // l = p - A(c): exact for the particle's own cell (Sterbenz) unless the
    // cell reaches a zero coordinate from below, where it rounds once, by at
    // most half an ulp of the cell size; so the anchored state starts equal to
    // the FP32 predicted position.
    const float lx = __fsub_rn(p.x, anchor_x(c.g, cx)), ly = __fsub_rn(p.y, anchor_y(c.g, cy));
    const float lz = __fsub_rn(p.z, anchor_z(c.g, cz));
    uint32_t qi;
    const int nthr = prefilter(c, cx + c.g.lx, cy + c.g.ly, cz + c.g.lz, lx, ly, lz, qi);
    LambdaAcc acc;
    acc.self(pc);
    uint32_t cnt = 0;
    sweep<false, RO, BS>(c, cur, qpos, cstart, cx, cy, cz, p.x, p.y, p.z, 0.0f, 0.0f, 0.0f, qi, nthr, s, rm,
                     PairQueue<BS>(queue),
                     [&](uint32_t, const float4&, float rx, float ry, float rz, float r2) {
                         cnt += r2 < pc.h2 ? 1u : 0u;
                         acc.add(pc, rx, ry, rz, r2);
                     });
    const float lambda = acc.lambda(c);
    nxt[s] = make_float4(lx, ly, lz, lambda);
    scell[s] = cell_local(c.g, cx, cy, cz);
    const uint32_t j = sidx[s];
    ncount[j] = cnt;
    if (LAST) lambdas[j] = lambda;
}

// Later lambda passes on the anchored state: cur is the previous delta pass's
// output, (l, x anchor of the hash cell) per slot.
template <bool LAST, bool RO, uint32_t BS, class C>
__device__ __forceinline__ void lambda_item(const StepConsts& c, const C& pc, uint32_t s,
                                            const float4* __restrict__ cur,
                                            const uint32_t* __restrict__ qpos, float4* __restrict__ nxt,
                                            const uint32_t* __restrict__ scell,
                                            const uint32_t* __restrict__ cstart,
                                            const uint32_t* __restrict__ sidx,
                                            float* __restrict__ lambdas, const RowMasks& rm, uint2* queue) {
    const float4 l = cur[s];
    int pcx, pcy, pcz, cx, cy, cz;
    decode_cell(c.g, scell[s], pcx, pcy, pcz);
    const float ax = anchor_x(c.g, pcx), ay = anchor_y(c.g, pcy), az = anchor_z(c.g, pcz);
    cell_of(c.g, __fadd_rn(ax, l.x), __fadd_rn(ay, l.y), __fadd_rn(az, l.z), cx, cy, cz);
    uint32_t qi;
    const int nthr = prefilter(c, pcx + c.g.lx, pcy + c.g.ly, pcz + c.g.lz, l.x, l.y, l.z, qi);
    LambdaAcc acc;
    acc.self(pc);
    sweep<true, RO, BS>(c, cur, qpos, cstart, cx, cy, cz, l.x, l.y, l.z, ax, ay, az, qi, nthr, s, rm,
                    PairQueue<BS>(queue),
                    [&](uint32_t, const float4&, float rx, float ry, float rz, float r2) {
                        acc.add(pc, rx, ry, rz, r2);
                    });
    const float lambda = acc.lambda(c);
    nxt[s] = make_float4(l.x, l.y, l.z, lambda);
    if (LAST) lambdas[sidx[s]] = lambda;
}

// finalizeStep (Constraints.metal:305-353) + computeFoam (:287-299) in FP64
// for particle j at solved position X.
__device__ __forceinline__ void finalize_particle(const StepConsts& c, uint32_t j, double X, double Y,
                                                  double Z, float4* __restrict__ pos,
                                                  float4* __restrict__ vel,
                                                  const float4* __restrict__ prev,
                                                  const uint32_t* __restrict__ ncount,
                                                  float* __restrict__ foam, uint32_t* err) {
    const double bx0 = c.bminx, by0 = c.bminy, bz0 = c.bminz;
    const double bx1 = c.bmaxx, by1 = c.bmaxy, bz1 = c.bmaxz;
    X = fmin(fmax(X, bx0), bx1);
    Y = fmin(fmax(Y, by0), by1);
    Z = fmin(fmax(Z, bz0), bz1);
    const float4 pr = prev[j];
    const double k = __dmul_rn(__drcp_rn(double(c.dt)), double(c.damping));
    double vx = __dmul_rn(__dsub_rn(X, double(pr.x)), k);
    double vy = __dmul_rn(__dsub_rn(Y, double(pr.y)), k);
    double vz = __dmul_rn(__dsub_rn(Z, double(pr.z)), k);
    const double we = c.wall_eps;
    const bool xMin = X <= __dadd_rn(bx0, we), xMax = X >= __dsub_rn(bx1, we);
    const bool yMin = Y <= __dadd_rn(by0, we), yMax = Y >= __dsub_rn(by1, we);
    const bool zMin = Z <= __dadd_rn(bz0, we), zMax = Z >= __dsub_rn(bz1, we);
    if (xMin) vx = fmax(vx, 0.0);
    if (xMax) vx = fmin(vx, 0.0);
    if (yMin) vy = fmax(vy, 0.0);
    if (yMax) vy = fmin(vy, 0.0);
    if (zMin) vz = fmax(vz, 0.0);
    if (zMax) vz = fmin(vz, 0.0);
    if (yMin) {
        vx = __dmul_rn(vx, double(c.floor_fric));
        vz = __dmul_rn(vz, double(c.floor_fric));
    } else if (xMin || xMax || zMin || zMax) {
        vx = __dmul_rn(vx, double(c.wall_fric));
        vy = __dmul_rn(vy, double(c.wall_fric));
        vz = __dmul_rn(vz, double(c.wall_fric));
    }
    const double vmax = __ddiv_rn(__dmul_rn(double(c.vmax_frac), double(c.h)), double(c.dt));
    double vl = __dsqrt_rn(__fma_rn(vz, vz, __fma_rn(vy, vy, __dmul_rn(vx, vx))));
    if (vl > vmax) {
        const double f = __ddiv_rn(vmax, vl);
        vx = __dmul_rn(vx, f);
        vy = __dmul_rn(vy, f);
        vz = __dmul_rn(vz, f);
        vl = __dsqrt_rn(__fma_rn(vz, vz, __fma_rn(vy, vy, __dmul_rn(vx, vx))));
    }
    pos[j] = make_float4(float(X), float(Y), float(Z), 1.0f);
    vel[j] = make_float4(float(vx), float(vy), float(vz), 0.0f);
    const float surface = __fsub_rn(1.0f, fminf(fmaxf(__fdiv_rn(float(ncount[j]), c.foam_maxn), 0.0f), 1.0f));
    foam[j] = __fmul_rn(surface, smoothstep_f(c.foam_lo, c.foam_hi, float(vl)));
    if (!(isfinite(X + Y + Z) && isfinite(vx + vy + vz))) atomicOr(err, kDevErrNaN);
}

// The pairs a lambda pass recorded in its row masks (the particle's own bit
// cleared), walked through a PairQueue with the neighbour vector of sweep<true>:
// body(k, q, rx, ry, rz, r2) for each, the ones out of range included, in
// sweep<true>'s order (rows in stencil order, slots ascending).  The candidates
// of a long row past its first chunk are distance-tested again.  (cx, cy, cz):
// the stencil cell of the particle at offset l from anchor (ax, ay, az).  xa: the
// x anchor of every slot's hash cell, so that a candidate's neighbour vector does
// not need the row's cell bounds.
template <bool RO, uint32_t BS, class Body>
__device__ __forceinline__ void queued_pairs(const StepConsts& c, const float4* __restrict__ src,
                                             const float* __restrict__ xa,
                                             const uint32_t* __restrict__ cstart, const RowMasks& rm,
                                             uint32_t s, const float4& l, float ax, float ay, float az,
                                             int cx, int cy, int cz, PairQueue<BS> queue, Body&& body) {
    const uint32_t longrows = rm.overflow[s];
    struct Candidate {
        float4 q;
        float a;
    };
    auto fetch = [&](uint32_t k) { return Candidate{load<RO>(&src[k]), load<RO>(&xa[k])}; };
    auto visit = [&](uint32_t k, const Candidate& f, float oy, float oz) {
        const float4& q = f.q;
        const float ox = __fadd_rn(__fsub_rn(ax, f.a), l.x);
        const float rx = __fsub_rn(ox, q.x), ry = __fsub_rn(oy, q.y), rz = __fsub_rn(oz, q.z);
        body(k, q, rx, ry, rz, dist2(rx, ry, rz));
    };
    const RowOffsets o = RowOffsets::anchored(c.g, cy, cz, ay, az, l.y, l.z);
    const StencilRows rows(c.g, cx, cy, cz);
    uint32_t base = rows.base;
    const uint32_t* in = rm.rows + s;
    if (longrows == 0u) {
        // all masks and row starts on their way at once
        uint32_t mask[9], b0[9];
#pragma unroll
        for (uint32_t r = 0; r < 9; ++r) {
            mask[r] = in[size_t(r) * rm.stride];  // (9 rows of 2^30 slots pass 2^32)
            b0[r] = rows.valid(cy - 1 + int(r % 3u), cz - 1 + int(r / 3u))
                        ? cstart[base + r * rows.next_y + (r / 3u) * rows.next_z]
                        : 0u;
        }
#pragma unroll
        for (uint32_t r = 0; r < 9; ++r) queue.push(mask[r], row_base(b0[r]), (r % 3u) | ((r / 3u) << 2));
    } else {
#pragma unroll 1
        for (int z = 0; z < 3; ++z, base += rows.next_z) {
#pragma unroll 1
            for (int y = 0; y < 3; ++y, base += rows.next_y, in += rm.stride) {
                const uint32_t mask = *in;
                const uint32_t row = uint32_t(3 * z + y);
                const bool long_row = (longrows >> row) & 1u;
                if (mask == 0u && !long_row) continue;
                const uint32_t a0 = row_base(cstart[base]);
                const uint32_t code = uint32_t(y) | (uint32_t(z) << 2);
                queue.push(mask, a0, code);
                if (long_row) {
                    const float oy = y == 0 ? o.y0 : (y == 1 ? o.y1 : o.y2);
                    const float oz = z == 0 ? o.z0 : (z == 1 ? o.z1 : o.z2);
                    const uint32_t b3 = cstart[base + rows.nx];
                    for (uint32_t c0 = a0 + 32u; c0 < b3; c0 += 32) {
                        uint32_t more = 0;
                        for (uint32_t k = c0; k < min(c0 + 32u, b3); ++k) {
                            const float4 q = load<RO>(&src[k]);
                            const float ox = __fadd_rn(__fsub_rn(ax, load<RO>(&xa[k])), l.x);
                            const float r2 = dist2(__fsub_rn(ox, q.x), __fsub_rn(oy, q.y), __fsub_rn(oz, q.z));
                            more |= r2 < c.h2 && k != s ? 0x80000000u >> (k - c0) : 0u;
                        }
                        if (warp_any(queue.short_of(9u - row))) queue.template drain<false>(o, fetch, visit);
                        queue.push(more, c0, code);
                    }
                }
            }
        }
    }
    queue.template drain<true>(o, fetch, visit);
}

// The position update of one particle whose pair sums are (dx, dy, dz): box
// clamp and sphere push in FP64; the last iteration also scatters back, finalizes
// and writes foam.  drec (may be NULL): receives the unclamped correction, for
// the adjoint.
template <bool LAST>
__device__ __forceinline__ void delta_apply(const StepConsts& c, uint32_t s, const float4& l, float ax, float ay,
                                            float az, int pcx, int pcy, int pcz, float dx, float dy, float dz,
                                            float4* __restrict__ dst, uint32_t* __restrict__ qpos,
                                            const uint32_t* __restrict__ sidx,
                                            const SphereState* __restrict__ sphere,
                                            float4* __restrict__ pos, float4* __restrict__ vel,
                                            const float4* __restrict__ prev,
                                            const uint32_t* __restrict__ ncount, float* __restrict__ foam,
                                            uint32_t* err, float4* __restrict__ drec) {
    dx = __fmul_rn(dx, c.delta_scale);
    dy = __fmul_rn(dy, c.delta_scale);
    dz = __fmul_rn(dz, c.delta_scale);
    if (drec) drec[s] = make_float4(dx, dy, dz, 0.0f);
    const float dl = __fsqrt_rn(dist2(dx, dy, dz));
    if (dl > c.max_step) {
        const float f = __fdiv_rn(c.max_step, dl);
        dx = __fmul_rn(dx, f);
        dy = __fmul_rn(dy, f);
        dz = __fmul_rn(dz, f);
    }
    // new position A + (l + delta), box clamp (and sphere push) in FP64
    double X = __dadd_rn(double(ax), double(__fadd_rn(l.x, dx)));
    double Y = __dadd_rn(double(ay), double(__fadd_rn(l.y, dy)));
    double Z = __dadd_rn(double(az), double(__fadd_rn(l.z, dz)));
    X = fmin(fmax(X, double(c.bminx)), double(c.bmaxx));
    Y = fmin(fmax(Y, double(c.bminy)), double(c.bmaxy));
    Z = fmin(fmax(Z, double(c.bminz)), double(c.bmaxz));
    if (c.sphere) {
        const double scx = sphere->c[0], scy = sphere->c[1], scz = sphere->c[2], sr = sphere->r;
        const double ex = __dsub_rn(X, scx), ey = __dsub_rn(Y, scy), ez = __dsub_rn(Z, scz);
        const double e2 = __fma_rn(ez, ez, __fma_rn(ey, ey, __dmul_rn(ex, ex)));
        if (e2 < __dmul_rn(sr, sr)) {
            const double inv = __ddiv_rn(sr, __dsqrt_rn(fmax(e2, double(1e-8f))));
            X = __fma_rn(ex, inv, scx);
            Y = __fma_rn(ey, inv, scy);
            Z = __fma_rn(ez, inv, scz);
        }
    }
    if (!LAST) {
        // w: the x anchor of the particle's hash cell, for the next lambda
        // pass's neighbour vectors
        const float lx = float(__dsub_rn(X, double(ax))), ly = float(__dsub_rn(Y, double(ay)));
        const float lz = float(__dsub_rn(Z, double(az)));
        dst[s] = make_float4(lx, ly, lz, ax);
        qpos[s] = quantize<false>(c, pcx + c.g.lx, pcy + c.g.ly, pcz + c.g.lz, lx, ly, lz);
        return;
    }
    finalize_particle(c, sidx[s], X, Y, Z, pos, vel, prev, ncount, foam, err);
}

// applyDeltaSorted + sphereCollision on the anchored state; the last
// iteration also scatters back, finalizes and writes foam.  drec (may be
// NULL): receives the particle's unclamped correction, for the adjoint.
// SN: the s_corr exponent when fixed at compile time (4), else 0.
template <bool LAST, uint32_t SN, bool RO, uint32_t BS, class C>
__device__ __forceinline__ void delta_item(const StepConsts& c, const C& pc, uint32_t s,
                                           const float4* __restrict__ src, float4* __restrict__ dst,
                                           uint32_t* __restrict__ qpos, const float* __restrict__ xa,
                                           const uint32_t* __restrict__ scell,
                                           const uint32_t* __restrict__ cstart,
                                           const uint32_t* __restrict__ sidx,
                                           const SphereState* __restrict__ sphere,
                                           float4* __restrict__ pos, float4* __restrict__ vel,
                                           const float4* __restrict__ prev,
                                           const uint32_t* __restrict__ ncount,
                                           float* __restrict__ foam, uint32_t* err,
                                           const RowMasks& rm, float4* __restrict__ drec, uint2* queue) {
    const float4 l = src[s];
    int pcx, pcy, pcz;
    decode_cell(c.g, scell[s], pcx, pcy, pcz);
    const float ax = anchor_x(c.g, pcx), ay = anchor_y(c.g, pcy), az = anchor_z(c.g, pcz);
    int cx, cy, cz;
    cell_of(c.g, __fadd_rn(ax, l.x), __fadd_rn(ay, l.y), __fadd_rn(az, l.z), cx, cy, cz);
    float dx = 0.0f, dy = 0.0f, dz = 0.0f;
    auto body = [&](uint32_t, const float4& q, float rx, float ry, float rz, float r2) {
        delta_add<SN>(pc, l.w, q.w, rx, ry, rz, r2, dx, dy, dz);
    };
    queued_pairs<RO, BS>(c, src, xa, cstart, rm, s, l, ax, ay, az, cx, cy, cz, PairQueue<BS>(queue), body);
    delta_apply<LAST>(c, s, l, ax, ay, az, pcx, pcy, pcz, dx, dy, dz, dst, qpos, sidx, sphere, pos, vel, prev,
                      ncount, foam, err, drec);
}

// Zero solver iterations: scatter-back + finalize + foam of the predicted
// positions.
__device__ __forceinline__ void finalize_sorted_item(const StepConsts& c, uint32_t s,
                                                     const float4* __restrict__ sorted,
                                                     const uint32_t* __restrict__ sidx,
                                                     float4* __restrict__ pos, float4* __restrict__ vel,
                                                     const float4* __restrict__ prev,
                                                     const uint32_t* __restrict__ ncount,
                                                     float* __restrict__ foam, uint32_t* err) {
    const float4 p = sorted[s];
    finalize_particle(c, sidx[s], p.x, p.y, p.z, pos, vel, prev, ncount, foam, err);
}

}  // namespace mpb
