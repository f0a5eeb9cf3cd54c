// pbf_team.cuh — the solver passes with a team of G lanes per particle, for
// scenes too small to fill the GPU with one lane each.
//
// With one lane per particle a pass is one long chain of dependent
// instructions (about 4,000 for 31 pairs); a small scene leaves most warp slots
// empty and waits for it.  Here the lanes of a team test the candidates of
// different stencil rows, expand the hits into one list in slot order, compute
// the terms of different pairs, and then add them up: each sum is owned by one
// lane, which adds its terms in list order with the one-lane pass's operations.
// So the results are the same bits, and who runs which variant is a question of
// speed only (team_lanes()).
//
// Bound by latency: 2,197 particles at K = 3, k_lambda 16 -> 7 us, k_delta 12 -> 6; the step
// 97 -> 54 us.
//
//   team_lambda_first, team_lambda   lambda_first_item, lambda_item
//   team_delta                       delta_item
#pragma once

#include "pbf_items.cuh"

namespace mpb {

constexpr uint32_t kTeamChunks = 10;  // row chunks (of 32 candidates) expanded at a time
constexpr uint32_t kTeamPairs = 32;   // pairs whose terms are computed at a time

// Shared memory of one team that adds up SUMS sums.
template <uint32_t SUMS>
struct TeamBufOf {
    uint32_t b0[9], b3[9], chunks[9];      // rows: slot range, number of chunks
    uint32_t list[kTeamChunks * 32];       // slot (below kTeamMaxSlots) | y << 28 | z << 30
    float2 term[SUMS][kTeamPairs + 1];     // per sum: the factors of each pair's term
};
using TeamBuf = TeamBufOf<5>;

template <uint32_t G, class Buf = TeamBuf>
struct Team {
    uint32_t lane, mask;  // lane in the team; the team's lanes in the warp
    Buf* buf;
    __device__ __forceinline__ explicit Team(Buf* bufs)
        : lane(threadIdx.x % G),
          mask((G == 32 ? 0xffffffffu : (1u << G) - 1u) << ((threadIdx.x & 31u) & ~(G - 1u))),
          buf(bufs + threadIdx.x / G) {}
    __device__ __forceinline__ void sync() const { __syncwarp(mask); }
    // the value of the team's lane l, to all its lanes
    template <class T>
    __device__ __forceinline__ T from(T v, uint32_t l) const {
        return __shfl_sync(mask, v, int(l), int(G));
    }
};

// The candidates of the 27-cell stencil around (cx, cy, cz), in slot order row
// by row: bits(row, c0, b0, b3) gives the mask (first candidate in bit 31) of the
// chunk of row `row` that starts at slot c0, to the lane that owns the chunk;
// terms(k, y, z, t) writes the NT term factors of candidate slot k (t[i * stride],
// i < NT), and lane i adds x * y of factor pair i over all candidates to `sum`.
// empty(row) is called for rows without candidates.
template <uint32_t G, uint32_t NT, class Buf, class Bits, class Empty, class Terms>
__device__ __forceinline__ void team_pairs(const Team<G, Buf>& team, const StepConsts& c,
                                           const uint32_t* __restrict__ cstart, int cx, int cy, int cz,
                                           float& sum, Bits&& bits, Empty&& empty, Terms&& terms) {
    static_assert(NT <= G, "one lane per sum");
    Buf& buf = *team.buf;
    const StencilRows rows(c.g, cx, cy, cz);
    team.sync();  // the buffer may still be read for the team's previous slot
    for (uint32_t row = team.lane; row < 9; row += G) {
        const uint32_t y = row % 3u, z = row / 3u;
        uint32_t b0 = 0, b3 = 0;
        if (rows.valid(cy - 1 + int(y), cz - 1 + int(z))) {
            const uint32_t base = rows.base + row * rows.next_y + z * rows.next_z;
            b0 = cstart[base];
            b3 = cstart[base + rows.nx];
        }
        if (b0 >= b3) empty(row);
        buf.b0[row] = b0;
        buf.b3[row] = b3;
        buf.chunks[row] = b0 < b3 ? (b3 - row_base(b0) + 31u) / 32u : 0u;
    }
    team.sync();
    uint32_t total = 0;
#pragma unroll
    for (uint32_t row = 0; row < 9; ++row) total += buf.chunks[row];
    for (uint32_t t0 = 0; t0 < total; t0 += kTeamChunks) {
        const uint32_t t1 = min(t0 + kTeamChunks, total);
        uint32_t pairs = 0;
        for (uint32_t ti = t0; ti < t1; ti += G) {
            uint32_t mask = 0, first = 0, code = 0;
            if (ti + team.lane < t1) {
                uint32_t t = ti + team.lane, row = 0;
                while (t >= buf.chunks[row]) t -= buf.chunks[row++];
                const uint32_t b0 = buf.b0[row], b3 = buf.b3[row];
                first = row_base(b0) + 32u * t;
                code = ((row % 3u) << 28) | ((row / 3u) << 30);
                mask = bits(row, first, b0, b3);
            }
            uint32_t upto = uint32_t(__popc(mask));
            const uint32_t own = upto;
#pragma unroll
            for (uint32_t o = 1; o < G; o <<= 1) {
                const uint32_t below = __shfl_up_sync(team.mask, upto, o, int(G));
                if (team.lane >= o) upto += below;
            }
            uint32_t at = pairs + upto - own;
            pairs += team.from(upto, G - 1u);
            while (mask) {
                uint32_t b;
                asm("bfind.shiftamt.u32 %0, %1;" : "=r"(b) : "r"(mask));
                mask &= 0x7fffffffu >> b;
                buf.list[at++] = (first + b) | code;
            }
        }
        team.sync();
        for (uint32_t p0 = 0; p0 < pairs; p0 += kTeamPairs) {
            const uint32_t n = min(kTeamPairs, pairs - p0);
            for (uint32_t p = team.lane; p < n; p += G) {
                const uint32_t e = buf.list[p0 + p];
                terms(e & (kTeamMaxSlots - 1u), (e >> 28) & 3u, e >> 30, &buf.term[0][p]);
            }
            team.sync();
            if (team.lane < NT) {
                const float2* t = buf.term[team.lane];
#pragma unroll 4
                for (uint32_t p = 0; p < n; ++p) sum = __fmaf_rn(t[p].x, t[p].y, sum);
            }
            team.sync();
        }
    }
}

constexpr uint32_t kTermStride = kTeamPairs + 1;

// LambdaAcc::add's factors of one candidate (all zero unless r2 < h^2).
__device__ __forceinline__ void lambda_terms(const StepConsts& c, float rx, float ry, float rz, float r2,
                                             float2* t) {
    const float d = __fsub_rn(c.h2, r2);
    const float rinv = rsqrt_normal(r2);
    const float hd = fmaxf(__fsub_rn(c.h, __fmul_rn(r2, rinv)), 0.0f);
    const float sc = __fmul_rn(__fmul_rn(__fmul_rn(-c.spiky, hd), hd), rinv);
    const bool in = r2 < c.h2, apart = in && r2 > 1e-12f;
    const float2 zero = make_float2(0.0f, 0.0f);
    t[0] = in ? make_float2(__fmul_rn(__fmul_rn(c.poly6, d), d), d) : zero;
    t[kTermStride] = apart ? make_float2(sc, rx) : zero;
    t[2 * kTermStride] = apart ? make_float2(sc, ry) : zero;
    t[3 * kTermStride] = apart ? make_float2(sc, rz) : zero;
    t[4 * kTermStride] = apart ? make_float2(__fmul_rn(sc, sc), r2) : zero;
}

// The sums of a lambda pass for slot s (see sweep()).  Returns the number of
// in-range candidates other than the particle; acc is complete on every lane.
template <uint32_t G, bool ANCHORED, bool RO>
__device__ __forceinline__ uint32_t team_sweep(const Team<G>& team, const StepConsts& c,
                                               const float4* __restrict__ src,
                                               const uint32_t* __restrict__ qsrc,
                                               const uint32_t* __restrict__ cstart, int cx, int cy, int cz,
                                               float px, float py, float pz, float aix, float aiy, float aiz,
                                               uint32_t qi, int nthr, uint32_t s, const RowMasks& masks,
                                               LambdaAcc& acc) {
    const int y0 = cy - 1, z0 = cz - 1;
    uint32_t hits = 0, over = 0;
    auto offset = [&](const float4& q, uint32_t y, uint32_t z, float& rx, float& ry, float& rz) {
        float ox = px, oy = py, oz = pz;
        if (ANCHORED) {
            ox = __fadd_rn(__fsub_rn(aix, q.w), px);
            oy = __fadd_rn(__fsub_rn(aiy, anchor_y(c.g, y0 + int(y))), py);
            oz = __fadd_rn(__fsub_rn(aiz, anchor_z(c.g, z0 + int(z))), pz);
        }
        rx = __fsub_rn(ox, q.x);
        ry = __fsub_rn(oy, q.y);
        rz = __fsub_rn(oz, q.z);
        return dist2(rx, ry, rz);
    };
    auto bits = [&](uint32_t row, uint32_t c0, uint32_t b0, uint32_t b3) {
        const uint32_t c1 = min(c0 + 32u, b3);
        uint32_t mask = 0;
        if (nthr != -kPassAll) {
            mask = row_bits<RO>(qsrc, qi, nthr, c0, c1, s);
        } else {  // as sweep() does
#pragma unroll 1
            for (uint32_t k = c0; k < c1; ++k) {
                float rx, ry, rz;
                const float r2 = offset(load<RO>(&src[k]), row % 3u, row / 3u, rx, ry, rz);
                mask |= r2 < c.h2 && k != s ? 0x80000000u >> (k - c0) : 0u;
            }
        }
        mask &= 0xffffffffu >> (max(b0, c0) - c0);
        if (c0 == row_base(b0)) {
            masks.rows[size_t(row) * masks.stride + s] = mask;
            if (b3 - c0 > 32u) over |= 1u << row;
        }
        return mask;
    };
    auto empty = [&](uint32_t row) { masks.rows[size_t(row) * masks.stride + s] = 0u; };
    auto terms = [&](uint32_t k, uint32_t y, uint32_t z, float2* t) {
        float rx, ry, rz;
        const float r2 = offset(load<RO>(&src[k]), y, z, rx, ry, rz);
        hits += r2 < c.h2 ? 1u : 0u;
        lambda_terms(c, rx, ry, rz, r2, t);
    };
    acc.self(c);
    float sum = team.lane == 0 ? acc.dens : 0.0f;
    team_pairs<G, 5>(team, c, cstart, cx, cy, cz, sum, bits, empty, terms);
    acc.dens = team.from(sum, 0);
    acc.gx = team.from(sum, 1);
    acc.gy = team.from(sum, 2);
    acc.gz = team.from(sum, 3);
    acc.gsq = team.from(sum, 4);
    over = __reduce_or_sync(team.mask, over);
    if (team.lane == 0) masks.overflow[s] = over;
    return __reduce_add_sync(team.mask, hits);
}

template <bool LAST, bool RO, uint32_t G>
__device__ __forceinline__ void team_lambda_first(const StepConsts& c, uint32_t s,
                                                  const float4* __restrict__ cur,
                                                  const uint32_t* __restrict__ qpos,
                                                  float4* __restrict__ nxt, uint32_t* __restrict__ scell,
                                                  const uint32_t* __restrict__ cstart,
                                                  const uint32_t* __restrict__ sidx,
                                                  float* __restrict__ lambdas,
                                                  uint32_t* __restrict__ ncount, const RowMasks& rm,
                                                  TeamBuf* bufs) {
    const Team<G> team(bufs);
    const float4 p = cur[s];
    int cx, cy, cz;
    cell_of(c.g, p.x, p.y, p.z, cx, cy, cz);
    const float lx = __fsub_rn(p.x, anchor_x(c.g, cx)), ly = __fsub_rn(p.y, anchor_y(c.g, cy));
    const float lz = __fsub_rn(p.z, anchor_z(c.g, cz));
    uint32_t qi;
    const int nthr = prefilter(c, cx + c.g.lx, cy + c.g.ly, cz + c.g.lz, lx, ly, lz, qi);
    LambdaAcc acc;
    const uint32_t cnt = team_sweep<G, false, RO>(team, c, cur, qpos, cstart, cx, cy, cz, p.x, p.y, p.z, 0.0f, 0.0f,
                                              0.0f, qi, nthr, s, rm, acc);
    if (team.lane != 0) return;
    const float lambda = acc.lambda(c);
    nxt[s] = make_float4(lx, ly, lz, lambda);
    scell[s] = cell_local(c.g, cx, cy, cz);
    const uint32_t j = sidx[s];
    ncount[j] = cnt;
    if (LAST) lambdas[j] = lambda;
}

template <bool LAST, bool RO, uint32_t G>
__device__ __forceinline__ void team_lambda(const StepConsts& c, uint32_t s, const float4* __restrict__ cur,
                                            const uint32_t* __restrict__ qpos, float4* __restrict__ nxt,
                                            const uint32_t* __restrict__ scell,
                                            const uint32_t* __restrict__ cstart,
                                            const uint32_t* __restrict__ sidx, float* __restrict__ lambdas,
                                            const RowMasks& rm, TeamBuf* bufs) {
    const Team<G> team(bufs);
    const float4 l = cur[s];
    int pcx, pcy, pcz, cx, cy, cz;
    decode_cell(c.g, scell[s], pcx, pcy, pcz);
    const float ax = anchor_x(c.g, pcx), ay = anchor_y(c.g, pcy), az = anchor_z(c.g, pcz);
    cell_of(c.g, __fadd_rn(ax, l.x), __fadd_rn(ay, l.y), __fadd_rn(az, l.z), cx, cy, cz);
    uint32_t qi;
    const int nthr = prefilter(c, pcx + c.g.lx, pcy + c.g.ly, pcz + c.g.lz, l.x, l.y, l.z, qi);
    LambdaAcc acc;
    team_sweep<G, true, RO>(team, c, cur, qpos, cstart, cx, cy, cz, l.x, l.y, l.z, ax, ay, az, qi, nthr, s, rm, acc);
    if (team.lane != 0) return;
    const float lambda = acc.lambda(c);
    nxt[s] = make_float4(l.x, l.y, l.z, lambda);
    if (LAST) lambdas[sidx[s]] = lambda;
}

// Neighbour vectors and chunk masks of a pass that walks recorded row masks, for a
// particle at offset l from anchor (ax, ay, az) (see queued_pairs()).
template <bool RO>
struct TeamWalk {
    const StepConsts& c;
    const float4* __restrict__ src;
    const float* __restrict__ xa;
    const RowMasks& rm;
    uint32_t s;
    float4 l;
    float ax, ay, az;
    int y0, z0;
    __device__ __forceinline__ void offset(uint32_t k, const float4& q, uint32_t y, uint32_t z, float& rx,
                                           float& ry, float& rz) const {
        const float ox = __fadd_rn(__fsub_rn(ax, load<RO>(&xa[k])), l.x);
        const float oy = __fadd_rn(__fsub_rn(ay, anchor_y(c.g, y0 + int(y))), l.y);
        const float oz = __fadd_rn(__fsub_rn(az, anchor_z(c.g, z0 + int(z))), l.z);
        rx = __fsub_rn(ox, q.x);
        ry = __fsub_rn(oy, q.y);
        rz = __fsub_rn(oz, q.z);
    }
    __device__ __forceinline__ uint32_t bits(uint32_t row, uint32_t c0, uint32_t b0, uint32_t b3) const {
        if (c0 == row_base(b0)) return rm.rows[size_t(row) * rm.stride + s];
        uint32_t more = 0;
        for (uint32_t k = c0; k < min(c0 + 32u, b3); ++k) {
            float rx, ry, rz;
            offset(k, load<RO>(&src[k]), row % 3u, row / 3u, rx, ry, rz);
            more |= dist2(rx, ry, rz) < c.h2 && k != s ? 0x80000000u >> (k - c0) : 0u;
        }
        return more;
    }
};

template <bool LAST, uint32_t SN, bool RO, uint32_t G>
__device__ __forceinline__ void team_delta(const StepConsts& c, uint32_t s, const float4* __restrict__ src,
                                           float4* __restrict__ dst, uint32_t* __restrict__ qpos,
                                           const float* __restrict__ xa, const uint32_t* __restrict__ scell,
                                           const uint32_t* __restrict__ cstart,
                                           const uint32_t* __restrict__ sidx,
                                           const SphereState* __restrict__ sphere, float4* __restrict__ pos,
                                           float4* __restrict__ vel, const float4* __restrict__ prev,
                                           const uint32_t* __restrict__ ncount, float* __restrict__ foam,
                                           uint32_t* err, const RowMasks& rm, float4* __restrict__ drec,
                                           TeamBuf* bufs) {
    const Team<G> team(bufs);
    const float4 l = src[s];
    int pcx, pcy, pcz;
    decode_cell(c.g, scell[s], pcx, pcy, pcz);
    const float ax = anchor_x(c.g, pcx), ay = anchor_y(c.g, pcy), az = anchor_z(c.g, pcz);
    int cx, cy, cz;
    cell_of(c.g, __fadd_rn(ax, l.x), __fadd_rn(ay, l.y), __fadd_rn(az, l.z), cx, cy, cz);
    const TeamWalk<RO> walk{c, src, xa, rm, s, l, ax, ay, az, cy - 1, cz - 1};
    auto bits = [&](uint32_t row, uint32_t c0, uint32_t b0, uint32_t b3) { return walk.bits(row, c0, b0, b3); };
    auto terms = [&](uint32_t k, uint32_t y, uint32_t z, float2* t) {
        const float4 q = load<RO>(&src[k]);
        float rx, ry, rz;
        walk.offset(k, q, y, z, rx, ry, rz);
        const float r2 = dist2(rx, ry, rz);
        const float coef = delta_coef<SN>(c, l.w, q.w, r2);
        const bool apart = r2 < c.h2 && r2 > 1e-12f;
        const float2 zero = make_float2(0.0f, 0.0f);
        t[0] = apart ? make_float2(coef, rx) : zero;
        t[kTermStride] = apart ? make_float2(coef, ry) : zero;
        t[2 * kTermStride] = apart ? make_float2(coef, rz) : zero;
    };
    float sum = 0.0f;
    team_pairs<G, 3>(team, c, cstart, cx, cy, cz, sum, bits, [](uint32_t) {}, terms);
    const float dx = team.from(sum, 0), dy = team.from(sum, 1), dz = team.from(sum, 2);
    if (team.lane != 0) return;
    delta_apply<LAST>(c, s, l, ax, ay, az, pcx, pcy, pcz, dx, dy, dz, dst, qpos, sidx, sphere, pos, vel, prev,
                      ncount, foam, err, drec);
}

}  // namespace mpb
