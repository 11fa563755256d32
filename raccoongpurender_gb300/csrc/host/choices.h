// choices.h — the rules by which calls choose their kernels and launch shapes: plain
// functions of sizes and settings, without CUDA, so that they can be tested on the host.
#pragma once
#include <algorithm>
#include <cstdint>

namespace rgr {

// From this many paths in flight on (the pool's, or the sample budget where that is less) a
// render's bounces take the persistent refilling cast and, inside a run, no logic pass
// (launch_inner_queues); fewer take the fused cast + logic kernel, as a bounce is then
// bound by its launches' latency and its longest rays.  Time of the fused bounces over that of
// the others, whole renders (8 spp, depth 6) in pools of 2^18 / 3 * 2^17 / 2^19 / 2^20 paths:
// 36 triangles 0.97 / 1.04 / 1.10 / 1.22, 5 K 0.95 / 1.08 / 1.13 / 1.31; single bounces 0.92 /
// 1.00 / 0.99 / 1.04 and 1.02 / 1.13 / 1.13 / 1.23; renders that train a guide 0.99 / 1.10 / 1.08 /
// 1.12.  1.31M triangles in 2^14 / 2^16 / 2^17 / 2^18 / 3 * 2^17: 0.85 / 0.86 / 0.85 / 0.86 / 0.93.  A
// budget below the pool: 2^14 / 2^17 / 2^18 samples in 2^20 paths 0.96 / 0.85 / 0.88 (36
// triangles), 0.95 / 0.87 / 0.93 (5 K), 0.92 / 0.86 / 0.79 (1.31M), guided 0.96 / 0.92 / 0.93.
constexpr uint64_t kPersistentMinPaths = 3ull << 17;

// samples: the render's budget, 0 for none
inline uint64_t paths_in_flight(uint64_t pool, uint64_t samples) { return samples ? std::min(pool, samples) : pool; }

// mode: rgr_set_render_trace's
inline bool persistent_cast(int mode, uint64_t pool, uint64_t samples) {
    if (mode >= 0) return mode != 0;
    return paths_in_flight(pool, samples) >= kPersistentMinPaths;
}

// Scenes of at most so many primitives take the fused kernel with one thread a slot: a ray is
// over before a list of the live slots pays.  Time with the list (k_cast_logic) over time with
// one thread a slot, whole renders (8 spp, depth 6) in pools of 2^12 / 2^14 / 2^16 / 2^17 / 2^18
// paths: 36 triangles 1.13 / 1.12 / 1.08 / 1.05 / 1.04, 600 spheres 1.12 / 1.11 / 1.07 / 1.05 / 1.07, 320
// triangles 1.09 / 1.09 / 1.08 / 1.05 / 0.99; 1280 triangles in 2^14 / 2^16 / 2^17 / 2^18 1.05 / 1.04 /
// 1.02 / 0.95, 5 K 1.00 / 0.99 / 0.99 / 0.91.
constexpr uint32_t kPerSlotMaxPrims = 1024;
inline bool per_slot_cast(uint32_t prims) { return prims <= kPerSlotMaxPrims; }

// The blocks of the fused kernel (k_cast_logic) take kCastSpan slots each, those below
// cast_half_end half as many: while the blocks of the paths in flight are one wave then (half
// against all at 2^17 paths: 2596 / 2646 us in 5 K triangles, 1775 / 1851 in 80 K; at 2^18
// 3807 / 3400 and 2538 / 2243).  A budget below the pool lives in the pool's first slots:
// 20,440 samples in 649,316 paths of 5 K triangles 687 us with whole spans and 574 so; 131,072 in
// 2^24 of 36 triangles 1483 with whole spans, 1997 with half ones over all the pool, 1507 so.
constexpr uint32_t kCastSpan = 512;
inline uint32_t cast_half_end(uint64_t pool, uint64_t samples, uint32_t resident_blocks, uint32_t tile) {
    const uint64_t paths = paths_in_flight(pool, samples);
    if (paths > (uint64_t)(kCastSpan / 2) * resident_blocks) return 0u;
    return (uint32_t)((paths + tile - 1) / tile * tile);  // a block's slots lie in one tile
}
// blocks that cover the pool
inline uint32_t cast_blocks(uint64_t pool, uint32_t half_end) {
    const uint64_t half = std::min<uint64_t>(pool, half_end), rest = pool - half;
    return (uint32_t)((half + kCastSpan / 2 - 1) / (kCastSpan / 2) + (rest + kCastSpan - 1) / kCastSpan);
}

// A warp of the closest-hit kernels takes new rays when `refill` of its lanes are idle, and its
// lanes take node steps while `search` of them still search for their leaf; in large calls
// (not sorted, staged or across the link) a warp whose rays head into several octants goes by
// the mixed pair.  The defaults: 24 and 8 the best of 1..32 and 1..24 for camera rays (3702 Mrays/s;
// 3319 with every lane waiting for the last), 12 and 12 for rays in all directions (k_trace_rays).
struct CastTuning {
    int refill = 24, search = 8, mixed_refill = 12, mixed_search = 12;
};
// A caller's value holds for every warp; the default value gives both pairs theirs back.
inline void set_refill(CastTuning& t, int refill) {
    const CastTuning d;
    t.refill = refill;
    t.mixed_refill = refill == d.refill ? d.mixed_refill : refill;
}
inline void set_search(CastTuning& t, int search) {
    const CastTuning d;
    t.search = search;
    t.mixed_search = search == d.search ? d.mixed_search : search;
}

// Blocks of the closest-hit kernels: with staged nodes, and without (calls of few rays, sorted
// ones and those across the link stage none, whatever is set).  blocks: resident ones an SM
// asked for, 0 for as many as fit.
struct TraceGrids {
    int staged, plain;
};
inline TraceGrids trace_grids(int sms, int blocks, int fit_staged, int fit_plain) {
    auto grid = [&](int fit) { return sms * (blocks ? std::min(blocks, fit) : fit); };
    return TraceGrids{grid(fit_staged), grid(fit_plain)};
}

// Resident blocks an SM of the shading kernels until rgr_set_render_tuning: what is resident.  A
// preview frame 2604 us with 8, 2566 with 4, the mixed render 69.45 and 69.07 ms.
constexpr int kShadeBlocksPerSm = 4;

}  // namespace rgr
