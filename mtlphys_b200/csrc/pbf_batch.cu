// pbf_batch.cu — many independent scenes of uneven particle counts advanced by
// one persistent, cooperative launch per step (no reference counterpart: the
// reference runs one scene per Engine).
//
// Every scene keeps its own parameters (dt, epsilon, box, ...) and its own
// hash grid.  To keep the cell arrays proportional to the particles instead of
// to (scenes x box volume), each step stores only the bounding box of the
// scene's predicted cells: the same dense cell coordinates as a single-scene
// engine, the same x-fastest order inside the box, so a scene's sorted order,
// neighbour sets and arithmetic are exactly those of a single-scene step.
// Scenes' particles and slots are contiguous ranges of the global arrays, and
// each scene's boxes are laid end to end in the global cell arrays.
//
// Phases of one step, separated by a grid-wide barrier (bounded spin: a
// block that gives up sets MP_DEVERR_SPIN_LIMIT and an abort flag, and every
// block leaves the launch at its next barrier, so no phase ever runs on the
// incomplete output of an earlier one):
//   0  per scene: advance the sphere; in the same phase
//   1  per particle: predict, dense cell -> scene bounding box (atomics,
//      reduced per warp first)
//   2  one block: per-scene sub-grid dims and cell offsets (exclusive scan); blocks
//      that only a larger box would have needed leave
//   3  per particle: cell id in the scene's box, warp-aggregated count; per
//      scene: the bounding box emptied for the next step
//   4  exclusive scan of the counts (tile sums, scan of the sums, tile scan)
//   5  scatter, 6 stable re-rank + gather, 7 long segments
//   8+ K x (lambda, delta); the last delta finalizes.
// The per-particle work is the single-scene engine's (pbf_items.cuh).  The
// serial mode launches this same kernel once per scene.
#include "pbf_batch.h"
#include "pbf_team.cuh"

namespace mpb {
namespace {

constexpr uint32_t kScanItems = kBatchScanItems;

// Grid-wide barrier.  Every block calls it the same number of times.  All blocks
// count their arrivals on the word that they then poll: the first block adds bit 31
// less the number of the others, those add 1, so the last one to arrive flips bit 31
// and leaves the other bits zero, and nothing has to be reset or passed on (the
// arithmetic of the grid barrier in the CUDA toolkit's cooperative groups).  With
// `last`, the arrivals are counted elsewhere, and the block that completes them runs
// last() before it flips the polled word, with everything the others wrote before
// the barrier visible: work for one block costs no barrier of its own.
//
// Latency of the chain of fences, atomics and polls is all there is to it, so it has
// as few links as can be: a fence, one atomic and the poll that sees it (2 us between
// the last arrival and the others' return).  One scene of 8,000 particles 109 -> 92 us
// per step (11 barriers), 12 of 61,000 in all 156 -> 137, 64 scenes of 4,000 to 20,000
// on all 1,184 blocks 636 -> 615, against arrivals at counters of 32 blocks each,
// their sums at a root and a generation word behind it (three atomics and four fences
// in a row); that form with the blocks polling the root: 101, 147, 624.  The length of
// the pause between polls makes no difference (0 to 200 ns).
//
// The wait is bounded: a block that waits more than a.spin_limit polls sets the
// error bit and the abort flag, the other half of the polled word.  Returns false (to
// every thread of the block) when the launch is aborted, by this block or another one;
// the block must then return.  A barrier only completes once every block has arrived,
// i.e. finished the phase before it, so a block that returns true works on complete
// data; a block that left early never arrives at the next barrier, so nobody passes
// that one.
constexpr unsigned kBarPhase = 0x80000000u;

struct BarrierState {
    unsigned phase;  // bit 31 of the phase word until the next barrier completes
    unsigned blocks;  // that take part
    unsigned passed;  // barriers so far (counted by the first block, for bar_pass only)
    int last, ok;
};

__device__ __forceinline__ uint2 bar_word(const BatchArgs& a) {
    uint2 w;
    asm volatile("ld.volatile.global.v2.u32 {%0, %1}, [%2];" : "=r"(w.x), "=r"(w.y) : "l"(a.bar + kBarGen));
    return w;
}

// Thread 0: this block is at the barrier that `word` counts.  Returns whether that
// completes it.
__device__ __forceinline__ bool arrive(const BatchArgs& a, uint32_t word, BarrierState* state) {
    __threadfence();
    unsigned inc = 1u;
    if (blockIdx.x == 0u) {
        inc = kBarPhase - (state->blocks - 1u);
        if (a.bar_extra && state->passed++ >= a.bar_pass) inc -= a.bar_extra;
    }
    const unsigned old = atomicAdd(a.bar + word, inc);
    return ((old + inc) ^ old) & kBarPhase;
}

// Thread 0: waits for the barrier's phase to end.
__device__ __forceinline__ void wait_phase(const BatchArgs& a, BarrierState* state) {
    int ok = 1;
    uint32_t spins = 0;
    uint2 w = bar_word(a);
    while (((w.x ^ state->phase) & kBarPhase) == 0u && !w.y) {
        if (++spins > a.spin_limit) {
            atomicOr(a.err, kDevErrSpin);
            atomicExch(a.abort, 1u);
            ok = 0;
            break;
        }
        __nanosleep(32);
        w = bar_word(a);
    }
    state->ok = ok && !w.y;
    state->phase ^= kBarPhase;
    __threadfence();
}

__device__ __forceinline__ bool grid_barrier(const BatchArgs& a, BarrierState* state) {
    __syncthreads();
    if (threadIdx.x == 0) {
        arrive(a, kBarGen, state);
        wait_phase(a, state);
    }
    __syncthreads();
    return state->ok != 0;
}

template <class Last>
__device__ __forceinline__ bool grid_barrier(const BatchArgs& a, BarrierState* state, Last&& last) {
    __syncthreads();
    if (threadIdx.x == 0) {
        state->last = arrive(a, kBarRoot, state);
        if (state->last) __threadfence();
    }
    __syncthreads();
    if (state->last) {
        last();
        __syncthreads();
        if (threadIdx.x == 0) {
            __threadfence();
            atomicAdd(a.bar + kBarGen, kBarPhase);
        }
    }
    if (threadIdx.x == 0) wait_phase(a, state);
    __syncthreads();
    return state->ok != 0;
}

template <uint32_t BS>
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* s_warp, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFull, incl, o);
        if (lane >= uint32_t(o)) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = lane < BS / 32 ? s_warp[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFull, wi, o);
            if (lane >= uint32_t(o)) wi += y;
        }
        if (lane < BS / 32) s_warp[lane] = wi - w;
        if (lane == BS / 32 - 1) s_warp[BS / 32] = wi;
    }
    __syncthreads();
    const uint32_t r = s_warp[warp] + incl - v;
    total = s_warp[BS / 32];
    __syncthreads();
    return r;
}

// Resident blocks of BS threads per SM the step kernel is compiled for: its
// registers are capped at 64 per thread (left alone, the compiler takes ~108
// for the inlined phases and fits a single 512-thread block per SM; at 64 the
// ensemble step is ~25% faster despite a small spill).
template <uint32_t BS>
constexpr int batch_min_blocks() {
    return int(65536u / (BS * 64u));
}

template <bool COMMON>
__device__ __forceinline__ const auto& pair_constants(const BatchArgs& a, const StepConsts& c) {
    if constexpr (COMMON)
        return a.pair;
    else
        return c;
}

// SN: the s_corr exponent fixed at compile time (4, when every scene uses
// the reference's) or read per scene (0); both give the same bits for 4.
// G: lanes per particle of the solver phases (kTeam) or 0 for one each
// (team_lanes(); the same bits).
// COMMON: every scene has the constants a.pair, which as an argument need no
// registers; per scene they are loads and a register each, of which the solver
// phases at 64 have none to spare (spill loads 368 -> 140 bytes with REC fixed
// too, 164 recording; 256 cubes, 4.2 M particles: 4.44 -> 4.23 ms; 12 small ones
// 182 -> 168 us).
// REC: whether the step is recorded, fixed at compile time (0, 1) or read from
// the arguments (2).
template <uint32_t BS, uint32_t SN, uint32_t G, bool COMMON, int REC>
__global__ void __launch_bounds__(BS, batch_min_blocks<BS>()) k_batch_step(BatchArgs a) {
    __shared__ uint32_t s_warp[BS / 32 + 1];
    __shared__ BarrierState s_bar;
    // one lane per particle: kQueue entries per thread; teams: a TeamBuf each
    extern __shared__ uint2 shared[];
    uint2* queue = shared;
    TeamBuf* bufs = reinterpret_cast<TeamBuf*>(shared);
    const uint32_t gtid = blockIdx.x * BS + threadIdx.x;
    // an earlier launch gave up on a barrier and left the barrier counter
    // mid-count: do nothing until the host has re-armed the batch
    if (*static_cast<volatile uint32_t*>(a.abort)) {
        if (gtid == 0) atomicOr(a.err, kDevErrSpin);
        return;
    }
    // (no barrier completes before this block arrives, so none has yet)
    if (threadIdx.x == 0) {
        s_bar.phase = bar_word(a).x;
        s_bar.passed = 0;
        s_bar.blocks = gridDim.x;
    }
    uint32_t nblocks = gridDim.x, gsize = nblocks * BS;
    const uint32_t pb = a.p_begin, pe = a.p_end;
    // loops over particles run in whole warps (warp-level operations inside)
    const uint32_t pe_round = pb + ((pe - pb + 31u) & ~31u);
    SceneDev* sc = a.scenes;

    // 0: advance the spheres (the solver reads them), clear the long-segment queue
    for (uint32_t s = a.scene_begin + gtid; s < a.scene_end; s += gsize) {
        if (a.rec.sphere0) a.rec.sphere0[s] = sc[s].sphere;
        if (sc[s].c.sphere) sphere_advance(sc[s].c, &sc[s].sphere);
    }
    if (gtid == 0) *a.long_count = 0;

    // 1: predict + dense cell of the predicted position -> scene bounding box
    for (uint32_t i = pb + gtid; i < pe_round; i += gsize) {
        const bool active = i < pe;
        uint32_t scene = 0xffffffffu, dx = 0, dy = 0, dz = 0;
        if (active) {
            scene = a.scene_of[i];
            const StepConsts& c = sc[scene].c;
            const float4 p = predict_item(c, i, a.pos, a.vel, a.prev, a.err);
            dx = uint32_t(cell_axis(p.x, c.g.ox, c.g.inv, c.g.dgx));
            dy = uint32_t(cell_axis(p.y, c.g.oy, c.g.inv, c.g.dgy));
            dz = uint32_t(cell_axis(p.z, c.g.oz, c.g.inv, c.g.dgz));
        }
        const unsigned act = __ballot_sync(kFull, active);
        if (active) {
            const unsigned peers = __match_any_sync(act, scene);
            const uint32_t mnx = __reduce_min_sync(peers, dx), mxx = __reduce_max_sync(peers, dx);
            const uint32_t mny = __reduce_min_sync(peers, dy), mxy = __reduce_max_sync(peers, dy);
            const uint32_t mnz = __reduce_min_sync(peers, dz), mxz = __reduce_max_sync(peers, dz);
            if (int(threadIdx.x & 31) == __ffs(peers) - 1) {
                uint32_t* bb = sc[scene].bb;
                atomicMin(&bb[0], mnx);
                atomicMin(&bb[1], mny);
                atomicMin(&bb[2], mnz);
                atomicMax(&bb[3], mxx);
                atomicMax(&bb[4], mxy);
                atomicMax(&bb[5], mxz);
            }
        }
    }
    // 2: sub-grid of every scene and its offset in the cell arrays, by the block
    // that completes the barrier
    auto lay_out = [&] {
        uint32_t running = 0;
        for (uint32_t s0 = a.scene_begin; s0 < a.scene_end; s0 += BS) {
            const uint32_t s = s0 + threadIdx.x;
            uint32_t cells = 0;
            if (s < a.scene_end) {
                const uint32_t* bb = sc[s].bb;
                GridDev& g = sc[s].c.g;
                if (bb[0] <= bb[3]) {
                    g.lx = int(bb[0]);
                    g.ly = int(bb[1]);
                    g.lz = int(bb[2]);
                    g.gx = int(bb[3] - bb[0]) + 1;
                    g.gy = int(bb[4] - bb[1]) + 1;
                    g.gz = int(bb[5] - bb[2]) + 1;
                } else {  // no particles
                    g.lx = g.ly = g.lz = 0;
                    g.gx = g.gy = g.gz = 0;
                }
                cells = uint32_t(g.gx) * uint32_t(g.gy) * uint32_t(g.gz);
                g.cells = cells;
            }
            uint32_t total = 0;
            const uint32_t excl = block_exclusive_scan<BS>(cells, s_warp, total);
            if (s < a.scene_end) sc[s].c.g.cell0 = running + excl;
            running += total;
        }
        if (threadIdx.x == 0) *a.total_cells = running;
    };
    if (!grid_barrier(a, &s_bar, lay_out)) return;
    if (a.particle_blocks < nblocks) {
        // blocks launched for the scan of cells that there could have been leave
        const uint32_t round = BS * kScanItems * kBatchScanRounds;
        nblocks = min(nblocks, max(a.particle_blocks, *a.total_cells / round + 1u));
        if (blockIdx.x >= nblocks) return;
        gsize = nblocks * BS;
        if (threadIdx.x == 0) s_bar.blocks = nblocks;
    }

    // 3: cell id inside the scene's box + warp-aggregated count; the boxes are
    // empty again for the next step
    for (uint32_t s = a.scene_begin + gtid; s < a.scene_end; s += gsize) {
        if (a.rec.scenes) a.rec.scenes[s] = sc[s];
        empty_box(sc[s].bb);
    }
    const uint32_t ncells = *a.total_cells;
    if (ncells > a.max_cells && gtid == 0) atomicOr(a.err, kDevErrIndex);
    const bool cells_ok = ncells <= a.max_cells;
    for (uint32_t i = pb + gtid; i < pe_round; i += gsize) {
        const bool active = i < pe && cells_ok;
        uint32_t cell = 0;
        if (active) {
            const StepConsts& c = sc[a.scene_of[i]].c;
            const float4 p = a.pos[i];
            int cx, cy, cz;
            cell_of(c.g, p.x, p.y, p.z, cx, cy, cz);
            cell = cell_hash(c.g, cx, cy, cz);
            a.hash[i] = cell;
        }
        uint32_t rank = 0;
        count_cell(active, cell, a.counts, &rank);
        if (active) a.off[i] = rank;
    }
    if (!grid_barrier(a, &s_bar)) return;

    // 4: exclusive scan of counts[0, ncells] into cstart (counts left zero)
    const uint32_t len = cells_ok ? ncells + 1u : 0u;
    const uint32_t tile = BS * kScanItems;
    const uint32_t tiles = (len + tile - 1) / tile;
    for (uint32_t t = blockIdx.x; t < tiles; t += nblocks) {
        uint32_t sum = 0;
        for (uint32_t k = 0; k < kScanItems; ++k) {
            const uint32_t idx = t * tile + k * BS + threadIdx.x;
            if (idx < len) sum += a.counts[idx];
        }
        uint32_t total = 0;
        block_exclusive_scan<BS>(sum, s_warp, total);
        if (threadIdx.x == 0) a.tile_sums[t] = total;
    }
    // tile offsets, by the block that completes the barrier; slots of this launch
    // start at its first particle (a scene's range in serial mode)
    auto scan_tiles = [&] {
        uint32_t running = pb;
        for (uint32_t t0 = 0; t0 < tiles; t0 += BS) {
            const uint32_t t = t0 + threadIdx.x;
            const uint32_t v = t < tiles ? a.tile_sums[t] : 0u;
            uint32_t total = 0;
            const uint32_t excl = block_exclusive_scan<BS>(v, s_warp, total);
            if (t < tiles) a.tile_sums[t] = running + excl;
            running += total;
        }
    };
    if (!grid_barrier(a, &s_bar, scan_tiles)) return;
    for (uint32_t t = blockIdx.x; t < tiles; t += nblocks) {
        // each thread owns kScanItems consecutive items of the tile
        uint32_t v[kScanItems], sum = 0;
        const uint32_t first = t * tile + threadIdx.x * kScanItems;
#pragma unroll
        for (uint32_t k = 0; k < kScanItems; ++k) {
            v[k] = first + k < len ? a.counts[first + k] : 0u;
            sum += v[k];
        }
        uint32_t total = 0;
        uint32_t run = a.tile_sums[t] + block_exclusive_scan<BS>(sum, s_warp, total);
#pragma unroll
        for (uint32_t k = 0; k < kScanItems; ++k)
            if (first + k < len) {
                a.cstart[first + k] = run;
                a.counts[first + k] = 0u;
                run += v[k];
            }
    }
    if (!grid_barrier(a, &s_bar)) return;

    // 5: scatter; 6: stable re-rank + gather; 7: long segments
    if (cells_ok)
        for (uint32_t i = pb + gtid; i < pe; i += gsize) scatter_item(i, a.hash, a.off, a.cstart, a.tmp);
    if (!grid_barrier(a, &s_bar)) return;
    if (cells_ok)
        for (uint32_t s = pb + gtid; s < pe; s += gsize)
            sort_gather_item(sc[a.scene_of[s]].c, s, a.tmp, a.hash, a.cstart, a.pos, a.sidx, a.sorted_a,
                             a.qpos, a.xa, nullptr,
                             [&](uint32_t cell) { a.long_list[atomicAdd(a.long_count, 1u)] = cell; });
    if (!grid_barrier(a, &s_bar)) return;
    const uint32_t nl = cells_ok ? *static_cast<volatile uint32_t*>(a.long_count) : 0u;
    if (nl) {  // the same for every block: long_count is written before the barrier only
        for (uint32_t li = blockIdx.x; li < nl; li += nblocks) {
            const uint32_t cell = a.long_list[li];
            const SceneDev& sd = sc[a.scene_of[a.tmp[a.cstart[cell]]]];
            long_segment(sd.c, cell, sd.p0, sd.p0 + sd.c.n, a.hash, a.cstart, a.pos, a.sidx, a.sorted_a,
                         a.qpos, a.xa, nullptr, s_warp);
        }
        if (!grid_barrier(a, &s_bar)) return;
    }

    // 8+: solver
    const RowMasks rm{a.row_masks, a.mask_overflow, a.mask_stride};
    if (!cells_ok) return;  // every block takes this branch together
    if (a.iterations == 0) {
        if constexpr (G == 0)
            for (uint32_t s = pb + gtid; s < pe; s += gsize)
                count_neighbors_item<false, BS>(sc[a.scene_of[s]].c, s, a.sorted_a, a.qpos, a.cstart, a.sidx, a.ncount,
                                         1u, PairQueue<BS>(queue));
        if (!grid_barrier(a, &s_bar)) return;
        for (uint32_t s = pb + gtid; s < pe; s += gsize)
            finalize_sorted_item(sc[a.scene_of[s]].c, s, a.sorted_a, a.sidx, a.pos, a.vel, a.prev,
                                 a.ncount, a.foam, a.err);
        return;
    }
    // a recorded step keeps every lambda pass's output, row masks and
    // corrections in the record instead of overwriting one buffer
    const bool record = REC == 2 ? a.rec.lam != nullptr : REC == 1;
    for (uint32_t it = 0; it < a.iterations; ++it) {
        const bool last = it + 1 == a.iterations;
        float4* lam_out = record ? a.rec.lam + size_t(it) * a.rec.stride : a.sorted_b;
        const RowMasks rmi =
            record ? RowMasks{a.rec.masks + size_t(it) * 9 * a.mask_stride,
                              a.rec.overflow + size_t(it) * a.mask_stride, a.mask_stride}
                   : rm;
        float4* drec = record ? a.rec.delta + size_t(it) * a.rec.stride : nullptr;
        constexpr uint32_t lanes = G ? G : 1u;
        for (uint32_t s = pb + gtid / lanes; s < pe; s += gsize / lanes) {
            const StepConsts& c = sc[a.scene_of[s]].c;
            const auto& pc = pair_constants<COMMON>(a, c);
            if constexpr (G != 0) {
                if (it == 0) {
                    if (last)
                        team_lambda_first<true, false, G>(c, s, a.sorted_a, a.qpos, lam_out, a.scell, a.cstart, a.sidx,
                                                   a.lambdas, a.ncount, rmi, bufs);
                    else
                        team_lambda_first<false, false, G>(c, s, a.sorted_a, a.qpos, lam_out, a.scell, a.cstart, a.sidx,
                                                    a.lambdas, a.ncount, rmi, bufs);
                } else if (last) {
                    team_lambda<true, false, G>(c, s, a.sorted_a, a.qpos, lam_out, a.scell, a.cstart, a.sidx, a.lambdas,
                                         rmi, bufs);
                } else {
                    team_lambda<false, false, G>(c, s, a.sorted_a, a.qpos, lam_out, a.scell, a.cstart, a.sidx, a.lambdas,
                                          rmi, bufs);
                }
            } else if (it == 0) {
                if (last)
                    lambda_first_item<true, false, BS>(c, pc, s, a.sorted_a, a.qpos, lam_out, a.scell, a.cstart, a.sidx,
                                                a.lambdas, a.ncount, rmi, queue);
                else
                    lambda_first_item<false, false, BS>(c, pc, s, a.sorted_a, a.qpos, lam_out, a.scell, a.cstart, a.sidx,
                                                 a.lambdas, a.ncount, rmi, queue);
            } else if (last) {
                lambda_item<true, false, BS>(c, pc, s, a.sorted_a, a.qpos, lam_out, a.scell, a.cstart, a.sidx, a.lambdas,
                                      rmi, queue);
            } else {
                lambda_item<false, false, BS>(c, pc, s, a.sorted_a, a.qpos, lam_out, a.scell, a.cstart, a.sidx, a.lambdas,
                                       rmi, queue);
            }
        }
        if (!grid_barrier(a, &s_bar)) return;
        for (uint32_t s = pb + gtid / lanes; s < pe; s += gsize / lanes) {
            const SceneDev& sd = sc[a.scene_of[s]];
            const auto& pc = pair_constants<COMMON>(a, sd.c);
            if constexpr (G != 0) {
                if (last)
                    team_delta<true, SN, false, G>(sd.c, s, lam_out, a.sorted_a, a.qpos, a.xa, a.scell, a.cstart, a.sidx,
                                            &sd.sphere, a.pos, a.vel, a.prev, a.ncount, a.foam, a.err, rmi, drec,
                                            bufs);
                else
                    team_delta<false, SN, false, G>(sd.c, s, lam_out, a.sorted_a, a.qpos, a.xa, a.scell, a.cstart, a.sidx,
                                             &sd.sphere, a.pos, a.vel, a.prev, a.ncount, a.foam, a.err, rmi, drec,
                                             bufs);
            } else if (last) {
                delta_item<true, SN, false, BS>(sd.c, pc, s, lam_out, a.sorted_a, a.qpos, a.xa, a.scell, a.cstart, a.sidx,
                                         &sd.sphere, a.pos, a.vel, a.prev, a.ncount, a.foam, a.err, rmi, drec,
                                         queue);
            } else {
                delta_item<false, SN, false, BS>(sd.c, pc, s, lam_out, a.sorted_a, a.qpos, a.xa, a.scell, a.cstart, a.sidx,
                                          &sd.sphere, a.pos, a.vel, a.prev, a.ncount, a.foam, a.err, rmi, drec,
                                          queue);
            }
        }
        if (!last && !grid_barrier(a, &s_bar)) return;
    }
}

// Dynamic shared memory of a launch: the threads' pair queues or the teams'
// buffers (beyond the 48 KB a kernel may use unasked at BS = 512).
template <uint32_t BS>
constexpr size_t shared_bytes(bool team) {
    return team ? sizeof(TeamBuf) * (BS / kTeam) : sizeof(uint2) * kQueue * BS;
}

// The step kernel for a launch with these properties (common implies scorr4).
template <uint32_t BS>
const void* batch_kernel(bool scorr4, bool common, bool team, bool record) {
    if (team)
        return scorr4 ? reinterpret_cast<const void*>(&k_batch_step<BS, 4, kTeam, false, 2>)
                      : reinterpret_cast<const void*>(&k_batch_step<BS, 0, kTeam, false, 2>);
    if (common)
        return record ? reinterpret_cast<const void*>(&k_batch_step<BS, 4, 0, true, 1>)
                      : reinterpret_cast<const void*>(&k_batch_step<BS, 4, 0, true, 0>);
    return scorr4 ? reinterpret_cast<const void*>(&k_batch_step<BS, 4, 0, false, 2>)
                  : reinterpret_cast<const void*>(&k_batch_step<BS, 0, 0, false, 2>);
}

cudaError_t allow_shared(const void* fn, size_t bytes) {
    if (bytes <= 48 * 1024) return cudaSuccess;
    return cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes));
}

template <uint32_t BS>
cudaError_t launch_bs(const BatchArgs& args, uint32_t blocks, cudaStream_t s) {
    void* kargs[] = {const_cast<BatchArgs*>(&args)};
    const bool team = args.iterations && team_lanes(args.p_end - args.p_begin, args.p_end) != 0;
    const void* fn = batch_kernel<BS>(args.scorr4 != 0, args.common != 0, team, args.rec.lam != nullptr);
    const size_t bytes = shared_bytes<BS>(team);
    const cudaError_t e = allow_shared(fn, bytes);
    if (e != cudaSuccess) return e;
    return cudaLaunchCooperativeKernel(fn, dim3(blocks), dim3(BS), kargs, bytes, s);
}

// Blocks of every instance that fit on one SM at once (the smallest count).
template <uint32_t BS>
int occupancy_bs() {
    int least = 1 << 30;
    for (int i = 0; i < 6; ++i) {
        // two instances each: teams, shared constants, neither
        const bool team = i < 2, common = i / 2 == 1, odd = i & 1;
        const void* fn = batch_kernel<BS>(common || odd, common, team, common && odd);
        int n = 0;
        if (allow_shared(fn, shared_bytes<BS>(team)) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, BS, shared_bytes<BS>(team)) != cudaSuccess)
            return 0;
        least = n < least ? n : least;
    }
    return least;
}

}  // namespace

int batch_max_blocks_per_sm(uint32_t block) {
    switch (block) {
        case 128: return occupancy_bs<128>();
        case 256: return occupancy_bs<256>();
        case 512: return occupancy_bs<512>();
        default: return 0;
    }
}

cudaError_t launch_batch_step(const BatchArgs& args, uint32_t block, uint32_t blocks, cudaStream_t s) {
    switch (block) {
        case 128: return launch_bs<128>(args, blocks, s);
        case 256: return launch_bs<256>(args, blocks, s);
        case 512: return launch_bs<512>(args, blocks, s);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace mpb
