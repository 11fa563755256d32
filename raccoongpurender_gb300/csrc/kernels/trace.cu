// trace.cu — closest hit for a batch of rays (extension_ray_cast as a
// service), the kernel of the ray-cast microbenchmark.
//
// Rays arrive as structure-of-arrays FP32 (ox, oy, oz, dx, dy, dz, tmax:
// 28 bytes per ray); results are the primitive id (-1 on a miss), t (tmax on
// a miss) and optionally the geometric normal.
//
// Persistent warps: each warp keeps 32 rays in flight and, between traversal
// rounds, hands finished lanes new rays from a global counter (one atomic per
// refill per warp).  Within a round the lanes take node steps while at least
// `search` of them still search for their next leaf; the others wait at
// theirs.  A warp left with a few rays, and a call of few rays, which is spread
// over the warps instead, go on lane by lane (kTailLanes, spread).  Rays are read
// and results written with streaming (evict-first) cache hints; the tree is
// read with an L2 evict-last policy.  Each ray's traversal is unchanged, so results
// do not depend on the schedule.
//
// Ray reordering (optional, for incoherent rays): a counting sort by a 16-bit
// key puts rays that start close together and head the same way next to each
// other, so that the 32 lanes of a warp walk similar paths through the tree.
// The key is a 6-D Morton code of the ray's origin and of the point half the
// scene's diagonal along it, three bits per coordinate over the scene's box
// (the far point's box widened by that reach), top 16 of the 18 bits.  Three
// passes: the key histogram (rays read once), its exclusive scan (one block),
// and the scatter of each ray as a 32-byte record (origin, tmax, direction,
// its index) to its bucket; the traversal then takes the records in bucket
// order and writes each hit at the ray's own index.  Within a bucket the
// order is that of the atomic cursor, which changes nothing but the schedule.
#include <algorithm>
#include <type_traits>

#include "wavefront.cuh"
#include "traverse.cuh"

#ifndef RGR_TRACE_MIN_BLOCKS
#define RGR_TRACE_MIN_BLOCKS 5  // resident 256-thread blocks per SM the register budget must allow
#endif

namespace rgr {
namespace dev {
namespace {

struct RayBatch {
    const float *ox, *oy, *oz, *dx, *dy, *dz, *tmax;
    const float4* packed;        // reordered records (kPacked): 2 float4 per ray
    uint64_t n;
    int32_t* prim;
    float* t;
    float* ng;                   // optional, 3 floats per ray
    uint32_t* nodes;             // optional counters (instrumented kernel)
    uint32_t* prims;
    uint32_t* err;
    unsigned long long* next;    // work counter, zero at launch (share = 0)
    uint32_t share;              // rays of a warp in a call of few, without the counter; 0 otherwise
    CastTuning tune;
    uint32_t stage;              // inner nodes copied to shared memory (kStaged)
};

// 32-byte read of a reordered ray record, not kept in L1 and first out of L2
RGR_DEV void ld_record(const float4* ptr, float4& a, float4& b) {
    asm("ld.global.nc.L1::no_allocate.L2::evict_first.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(a.x), "=f"(a.y), "=f"(a.z), "=f"(a.w), "=f"(b.x), "=f"(b.y), "=f"(b.z), "=f"(b.w)
        : "l"(ptr));
}

// Results in host memory (kLink) cross the link in runs: the rays of one refill are
// consecutive, and their hits wait in shared memory until the last of them is known.
// Single 4-byte stores keep the link busy: 1M random rays in 330 K triangles took 400 us with
// only the results across it, 342 with only the rays (320 with neither), the whole call
// 502 and now 400 us; 2M rays in 1.31M triangles 957 and 762.  (The rays' reads hide behind the
// traversal: copying them to shared memory a batch ahead was slower, 549, as every
// warp's first rays then share the link with the others' second.)  A warp keeps up to
// kRuns runs open (all of a run in shared memory: its words in registers spilled, 407 and 787);
// to begin another it writes what the oldest has, and that one's missing
// rays write their own.
constexpr int kRuns = 4;
struct LinkRuns {
    int32_t prim[kRuns][32];
    float t[kRuns][32];
    uint64_t base[kRuns];  // the run's first ray
    uint32_t rays[kRuns];  // a bit per ray of it (0: free)
    uint32_t done[kRuns];  // the finished ones
};

// From this many rays on a warp's octants choose its thresholds (CastTuning): a warp of a call
// of fewer takes rays a few times only (300,000 random rays in 20 K triangles 112 us, 116 with
// thresholds of its own).
constexpr uint64_t kMixedMinRays = 1ull << 19;

// kFew: each lane takes one ray of its warp's share, without the rounds
template <bool kCount, bool kStaged, bool kPacked, bool kFew, bool kLink>
__global__ void __launch_bounds__(256, RGR_TRACE_MIN_BLOCKS) k_trace_rays(SceneView sc, RayBatch b) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    if (kFew) follow();  // calls of few, one after another: the next one's blocks are there already
    const uint64_t pol = l2_evict_last_policy();
    extern __shared__ float4 s_nodes[];
    StagedNodes stn{s_nodes, 0u};
    if (kStaged) {
        stn.n = min(b.stage, sc.num_nodes);
        for (uint32_t i = threadIdx.x; i < 4u * stn.n; i += blockDim.x) s_nodes[i] = __ldg(sc.nodes + i);
        __syncthreads();
    }
    __shared__ uint32_t s_stack[(kSmemStack + 1) * kStackThreads];  // the last row: see touch
    TraceState s;
    s.sstk = s_stack + threadIdx.x;
    TraceCounters cnt;
    uint64_t ray = ~0ull;  // ~0: idle
    __shared__ LinkRuns s_runs[kLink ? kStackThreads / 32 : 1];
    LinkRuns& runs = s_runs[kLink ? threadIdx.x >> 5 : 0];
    if (kLink && lane < kRuns) runs.rays[lane] = runs.done[lane] = 0u;
    __syncwarp();
    int place = -1;  // this lane's ray's run << 5 | its place there, or it writes its own hit
    int oldest = 0;
    // writes the finished rays of run k, which is free then
    auto flush = [&](int k) {
        if ((runs.done[k] >> lane) & 1u) {
            const uint64_t r = runs.base[k] + lane;
            __stcs(b.prim + r, runs.prim[k][lane]);
            __stcs(b.t + r, runs.t[k][lane]);
        }
        __syncwarp();
        if (lane == 0) runs.rays[k] = runs.done[k] = 0u;
        __syncwarp();
    };
    auto take = [&](uint64_t r) {
        if (kPacked) {
            float4 o4, d4;
            ld_record(b.packed + 2 * r, o4, d4);
            const uint32_t idx = __float_as_uint(d4.w);
            if (idx < b.n) {  // every record holds one of the n rays
                ray = idx;
                trace_begin(sc, s, xyz(o4), xyz(d4), o4.w);
            }
        } else {
            ray = r;
            trace_begin(sc, s, mk(__ldcs(b.ox + r), __ldcs(b.oy + r), __ldcs(b.oz + r)),
                        mk(__ldcs(b.dx + r), __ldcs(b.dy + r), __ldcs(b.dz + r)), __ldcs(b.tmax + r));
        }
        if (kCount) cnt = TraceCounters();
    };
    auto put = [&]() {
        const int32_t prim = hit_id(s.prim);
        if (kLink && place >= 0) {
            runs.prim[place >> 5][place & 31] = prim;
            runs.t[place >> 5][place & 31] = s.tmin;
            atomicOr(&runs.done[place >> 5], 1u << (place & 31));
        } else {
            __stcs(b.prim + ray, prim);
            __stcs(b.t + ray, s.tmin);
        }
        if (b.ng) {
            f3 n = prim >= 0 ? hit_normal(sc, prim, s.ro, s.rd, s.tmin) : mk(0.0f, 0.0f, 0.0f);
            b.ng[3 * ray + 0] = n.x;
            b.ng[3 * ray + 1] = n.y;
            b.ng[3 * ray + 2] = n.z;
        }
        if (kCount) {
            b.nodes[ray] = cnt.nodes;
            b.prims[ray] = cnt.prims;
        }
        ray = ~0ull;
    };
    uint32_t err = 0;
    if (kFew) {
        const uint64_t r = ((uint64_t)blockIdx.x * (kStackThreads / 32) + (threadIdx.x >> 5)) * b.share + lane;
        if ((uint32_t)lane < b.share && r < b.n) take(r);
    }
    bool exhausted = false;
    // kMixed: a compile-time constant, so that each loop's thresholds are operands and not registers
    auto rounds = [&](auto which) {
        constexpr bool kMixed = decltype(which)::value;
        for (;;) {
            const unsigned idle = __ballot_sync(full, ray == ~0ull);
            if (!exhausted && (int)__popc(idle) >= (kMixed ? b.tune.mixed_refill : b.tune.refill)) {
                const uint32_t need = __popc(idle);
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(b.next, (unsigned long long)need);
                base = __shfl_sync(full, base, 0);
                if (base + need >= b.n) exhausted = true;
                if (kLink && base < b.n) {  // a run of the new rays
                    const int k = oldest;
                    oldest = (oldest + 1) % kRuns;
                    const bool open = runs.rays[k] != 0u;
                    __syncwarp();  // every lane has read it before lane 0 writes it
                    if (open) {
                        flush(k);
                        if ((place >> 5) == k) place = -1;
                    }
                    if (lane == 0) {
                        runs.base[k] = base;
                        runs.rays[k] =
                            b.n - base >= need ? (need < 32u ? (1u << need) - 1u : full) : (1u << (b.n - base)) - 1u;
                    }
                    if (ray == ~0ull) place = k << 5 | __popc(idle & lt);
                }
                if (ray == ~0ull) {
                    const uint64_t r = base + __popc(idle & lt);
                    if (r < b.n) take(r);
                }
            }
            const unsigned held = __ballot_sync(full, ray != ~0ull);
            if (exhausted && __popc(held) <= kTailLanes) break;
            if (held == 0u) continue;
            trace_warp_round<kCount, kStaged, kSmemStack>(sc, s, ray != ~0ull && s.link != kDone,
                                                          kMixed ? b.tune.mixed_search : b.tune.search, &cnt, err, pol, stn);
            if (ray != ~0ull && s.link == kDone) put();
            if (kLink) {
                __syncwarp();
                const bool whole = lane < kRuns && runs.rays[lane] != 0u && runs.done[lane] == runs.rays[lane];
                for (unsigned m = __ballot_sync(full, whole); m != 0u; m &= m - 1u) flush(__ffs(m) - 1);
            }
        }
    };
    if (!kFew) {
        // Rays of one octant keep together in large batches (4M camera rays in 1.31M triangles, calls in
        // a row: refill / search 24 / 8 658 us, 12 / 12 721); others part at once, and full lanes
        // count for more (random rays 1098 and 1036; in a scene of 1280 triangles 700 and 633).  The
        // warp looks at rays about where its first will be; chosen anew at each refill it cost
        // registers, and a tenth of the camera rays' time.  Sorted rays: 999 with 24 / 8, 1040 with 12 / 12.
        bool mixed = false;
        if (!kCount && !kStaged && !kLink && !kPacked && b.n >= kMixedMinRays) {
            const uint64_t r = (uint64_t)blockIdx.x * kStackThreads + threadIdx.x;
            const bool has = r < b.n;
            f3 d = mk(0.0f, 0.0f, 0.0f);
            if (has) d = mk(__ldg(b.dx + r), __ldg(b.dy + r), __ldg(b.dz + r));
            const unsigned rays = __ballot_sync(full, has), x = __ballot_sync(full, d.x < 0.0f),
                           y = __ballot_sync(full, d.y < 0.0f), z = __ballot_sync(full, d.z < 0.0f);
            mixed = (x != 0u && x != rays) || (y != 0u && y != rays) || (z != 0u && z != rays);
        }
        if (mixed)
            rounds(std::true_type());
        else
            rounds(std::false_type());
    }
    if (kLink) {  // the last rays write their own
        __syncwarp();
#pragma unroll
        for (int k = 0; k < kRuns; ++k) flush(k);
        place = -1;
    }
    if (ray != ~0ull) {
        while (s.link != kDone) trace_round<kCount, kStaged, kSmemStack, true>(sc, s, &cnt, err, pol, stn);
        put();
        touch_done();
    }
    if (err) atomicOr(b.err, err);
}

// ---------------------------------------------------------------- reordering
struct RaySoA {
    const float *ox, *oy, *oz, *dx, *dy, *dz, *tmax;
};

// one coordinate in 3 bits: floor((x - lo) * scale) clamped to [0, 7]; NaN
// goes to 0 (fmaxf returns the other operand), infinities to an end.  Explicit
// roundings: the histogram and the scatter must compute the same key.
RGR_DEV uint32_t key3(float x, float lo, float scale) {
    return (uint32_t)fminf(fmaxf(floorf(__fmul_rn(__fsub_rn(x, lo), scale)), 0.0f), 7.0f);
}

RGR_DEV uint32_t ray_key(const RayKeyBox& kb, f3 o, f3 d) {
    const uint32_t c[6] = {key3(o.x, kb.lo[0], kb.scale[0]),
                           key3(o.y, kb.lo[1], kb.scale[1]),
                           key3(o.z, kb.lo[2], kb.scale[2]),
                           key3(__fmaf_rn(d.x, kb.reach, o.x), kb.lo_far[0], kb.scale_far[0]),
                           key3(__fmaf_rn(d.y, kb.reach, o.y), kb.lo_far[1], kb.scale_far[1]),
                           key3(__fmaf_rn(d.z, kb.reach, o.z), kb.lo_far[2], kb.scale_far[2])};
    uint32_t k = 0;
#pragma unroll
    for (int bit = 2; bit >= 0; --bit)
#pragma unroll
        for (int j = 0; j < 6; ++j) k = (k << 1) | ((c[j] >> bit) & 1u);
    return k >> (18 - kRayKeyBits);
}

// The histogram and the scatter: a warp takes kKeyRays x 32 consecutive rays
// at a time, lane l the rays l, l + 32, ... (coalesced loads, kKeyRays of
// each array in flight per thread; full tiles without predicates).  Lanes
// past n form a suffix of the warp and take no part.  Equal keys are
// gathered per run of consecutive lanes: the run's first lane takes the
// run's atomic (camera rays share keys in long runs; for incoherent rays
// each lane is its own run).
constexpr int kKeyRays = 4;

// this lane's run of equal keys among the valid lanes (a prefix of `nvalid`):
// its first lane and its length
RGR_DEV void key_run(uint32_t key, int lane, int nvalid, int& head, int& len) {
    const unsigned full = 0xffffffffu;
    const uint32_t prev = __shfl_up_sync(full, key, 1);
    const unsigned heads = __ballot_sync(full, lane < nvalid && (lane == 0 || prev != key));
    head = 31 - __clz(heads & ((2u << lane) - 1u));
    const unsigned after = heads & ~((2u << head) - 1u);
    len = (after ? __ffs(after) - 1 : nvalid) - head;
}

template <bool kStream>
RGR_DEV float ld_ray(const float* p) {
    return kStream ? __ldcs(p) : __ldg(p);
}

// the kKeyRays rays of this lane, arrays a[0..kArrays-1]; lanes past n get zeros
template <int kArrays, bool kStream>
RGR_DEV void load_rays(const float* const* a, uint64_t i0, uint64_t n, int lane, float (&v)[kArrays][kKeyRays]) {
    if (i0 + 32 * kKeyRays <= n) {
#pragma unroll
        for (int j = 0; j < kKeyRays; ++j)
#pragma unroll
            for (int c = 0; c < kArrays; ++c) v[c][j] = ld_ray<kStream>(a[c] + i0 + lane + 32 * j);
    } else {
#pragma unroll
        for (int j = 0; j < kKeyRays; ++j) {
            const uint64_t i = i0 + lane + 32 * j;
#pragma unroll
            for (int c = 0; c < kArrays; ++c) v[c][j] = i < n ? ld_ray<kStream>(a[c] + i) : 0.0f;
        }
    }
}

// The counts of the keys, and each ray's rank among the rays of its key: the
// run's atomic returns the rays of that key counted before it
__global__ void __launch_bounds__(256) k_ray_bins(RaySoA r, uint64_t n, RayKeyBox kb, uint32_t* __restrict__ bins,
                                                 uint32_t* __restrict__ rank) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const float* const a[6] = {r.ox, r.oy, r.oz, r.dx, r.dy, r.dz};
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x * kKeyRays;
    for (uint64_t i0 = ((uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) * kKeyRays; i0 < n; i0 += stride) {
        float v[6][kKeyRays];
        load_rays<6, false>(a, i0, n, lane, v);
        uint32_t base[kKeyRays];
        int off[kKeyRays], head[kKeyRays];
#pragma unroll
        for (int j = 0; j < kKeyRays; ++j) {
            const uint64_t left = n - (i0 + 32 * j);
            const int nvalid = i0 + 32 * j >= n ? 0 : (left >= 32 ? 32 : (int)left);
            base[j] = 0u;
            head[j] = 0;
            off[j] = -1;
            if (nvalid == 0) continue;
            const uint32_t key = ray_key(kb, mk(v[0][j], v[1][j], v[2][j]), mk(v[3][j], v[4][j], v[5][j]));
            int len;
            key_run(key, lane, nvalid, head[j], len);
            if (lane == head[j] && lane < nvalid) base[j] = atomicAdd(bins + key, (uint32_t)len);
            if (lane < nvalid) off[j] = lane - head[j];
        }
        // the ranks, once the atomics of all kKeyRays rows are in flight
#pragma unroll
        for (int j = 0; j < kKeyRays; ++j) {
            const uint32_t b = __shfl_sync(full, base[j], head[j]);
            if (off[j] >= 0) rank[i0 + lane + 32 * j] = b + (uint32_t)off[j];
        }
    }
}

// Exclusive scan of the kRayBins counts into the cursors: 32 blocks of 1024
// threads, block b the bins [2048 b, 2048 b + 2048), two per thread.  Each
// block first sums all the bins before its own (at most 62 K reads from L2,
// the blocks in parallel), so no block waits for another.
constexpr int kScanBlocks = 32;
RGR_DEV uint32_t block_sum_1024(uint32_t v, uint32_t* s_warp) {
    v = __reduce_add_sync(0xffffffffu, v);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = v;
    __syncthreads();
    uint32_t t = 0;
#pragma unroll
    for (int w = 0; w < 32; ++w) t += s_warp[w];
    __syncthreads();  // s_warp reused
    return t;
}

__global__ void __launch_bounds__(1024) k_ray_bins_scan(const uint32_t* __restrict__ bins,
                                                        uint32_t* __restrict__ cursor) {
    static_assert(kRayBins == kScanBlocks * 2048, "32 blocks of 2048 bins");
    const unsigned full = 0xffffffffu;
    __shared__ uint32_t s_warp[32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint4* p4 = reinterpret_cast<const uint4*>(bins);
    uint32_t pre = 0;
    for (uint32_t q = threadIdx.x; q < 512u * blockIdx.x; q += 1024u) {
        const uint4 v = p4[q];
        pre += v.x + v.y + v.z + v.w;
    }
    pre = block_sum_1024(pre, s_warp);
    const uint2 v = reinterpret_cast<const uint2*>(bins)[1024 * blockIdx.x + threadIdx.x];
    const uint32_t t = v.x + v.y;
    uint32_t x = t;  // inclusive scan over the warp
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(full, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    uint32_t wpre = 0;
    for (int w = 0; w < warp; ++w) wpre += s_warp[w];
    const uint32_t e = pre + wpre + x - t;
    reinterpret_cast<uint2*>(cursor)[1024 * blockIdx.x + threadIdx.x] = make_uint2(e, e + v.x);
}

// each ray's 32-byte record to its place: the start of its key's bucket (the
// scanned counts) plus its rank there
__global__ void __launch_bounds__(256) k_ray_scatter(RaySoA r, uint64_t n, RayKeyBox kb,
                                                    const uint32_t* __restrict__ start,
                                                    const uint32_t* __restrict__ rank, float4* __restrict__ packed) {
    const int lane = threadIdx.x & 31;
    const float* const a[7] = {r.ox, r.oy, r.oz, r.dx, r.dy, r.dz, r.tmax};
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x * kKeyRays;
    for (uint64_t i0 = ((uint64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31u)) * kKeyRays; i0 < n; i0 += stride) {
        float v[7][kKeyRays];
        load_rays<7, true>(a, i0, n, lane, v);
#pragma unroll
        for (int j = 0; j < kKeyRays; ++j) {
            const uint64_t i = i0 + lane + 32 * j;
            if (i >= n) continue;
            const uint32_t key = ray_key(kb, mk(v[0][j], v[1][j], v[2][j]), mk(v[3][j], v[4][j], v[5][j]));
            const uint32_t pos = __ldg(start + key) + __ldcs(rank + i);
            // pos < n always (both passes compute the same key)
            if (pos >= n) continue;
            float4* q = packed + 2 * (size_t)pos;
            asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(q), "f"(v[0][j]),
                         "f"(v[1][j]), "f"(v[2][j]), "f"(v[6][j]), "f"(v[3][j]), "f"(v[4][j]), "f"(v[5][j]),
                         "f"(__uint_as_float((uint32_t)i))
                         : "memory");
        }
    }
}

}  // namespace

namespace {
// A call of few rays (at most kFewRays a warp of the grid) is bound by the latency of its
// longest ray's steps, so its rays are spread over the warps, ceil(n / warps) each,
// without the counter and its reset, and go on lane by lane: 1000 / 6000 / 20000 random
// rays in a 20 K-triangle scene, calls in a row, 57.5 / 69.2 / 70.7 us in whole warps,
// 35.1 / 43.3 / 60.0 spread, 24.9 / 34.9 / 53.7 with the next links brought into L1 (touch),
// 21.7 / 31.3 / 49.4 as dependent launches.
// 30,000 / 40,000: 58.5 / 60.5 us in whole warps, 52.0 / 57.9 so (1.31M triangles 99.7 / 100.3 and
// 89.2 / 92.4); from there on whole warps win (55,000: 64 us, 71.5 spread ten a warp; 156 and 165).
// Returns the rays a warp, 0 for the counter, which it resets; *blocks: at most `grid`.
constexpr uint64_t kFewRays = 8;
uint32_t spread(uint64_t n, int grid, int* blocks, unsigned long long* counter, cudaStream_t st) {
    const uint64_t per = kStackThreads / 32, warps = (uint64_t)grid * per;
    *blocks = grid;
    if (n > kFewRays * warps) {
        cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st);
        return 0u;
    }
    const uint64_t share = (n + warps - 1) / warps;
    *blocks = (int)((n + per * share - 1) / (per * share));
    return (uint32_t)share;
}
}  // namespace

void launch_trace_rays(const SceneView& sc, const float* ox, const float* oy, const float* oz, const float* dx,
                       const float* dy, const float* dz, const float* tmax, uint64_t n, int32_t* prim, float* t,
                       float* ng, uint32_t* err, unsigned long long* counter, const CastTuning& tune,
                       const TraceGrids& grids, uint32_t stage, cudaStream_t st) {
    if (n == 0) return;
    int blocks;
    const uint32_t share = spread(n, grids.plain, &blocks, counter, st);
    RayBatch b{ox, oy, oz, dx, dy, dz, tmax, nullptr, n, prim, t, ng, nullptr, nullptr, err, counter, share, tune,
               stage};
    if (share)
        chain(k_trace_rays<false, false, false, true, false>, blocks, kStackThreads, 0, st, sc, b);
    else if (stage > 0)
        k_trace_rays<false, true, false, false, false><<<grids.staged, kStackThreads, 64 * (size_t)stage, st>>>(sc, b);
    else
        k_trace_rays<false, false, false, false, false><<<blocks, kStackThreads, 0, st>>>(sc, b);
}

// rays and results in host memory
void launch_trace_rays_link(const SceneView& sc, const float* const* rays, uint64_t n, int32_t* prim, float* t,
                            uint32_t* err, unsigned long long* counter, const CastTuning& tune, int grid,
                            cudaStream_t st) {
    if (n == 0) return;
    int blocks;
    const uint32_t share = spread(n, grid, &blocks, counter, st);
    RayBatch b{rays[0], rays[1], rays[2], rays[3], rays[4], rays[5], rays[6], nullptr, n, prim, t, nullptr,
               nullptr, nullptr, err, counter, share, tune, 0u};
    if (share)
        chain(k_trace_rays<false, false, false, true, false>, blocks, kStackThreads, 0, st, sc, b);
    else
        k_trace_rays<false, false, false, false, true><<<blocks, kStackThreads, 0, st>>>(sc, b);
}

void launch_trace_rays_counts(const SceneView& sc, const float* ox, const float* oy, const float* oz, const float* dx,
                              const float* dy, const float* dz, const float* tmax, uint64_t n, int32_t* prim,
                              float* t, uint32_t* nodes, uint32_t* prims, uint32_t* err, unsigned long long* counter,
                              int grid, cudaStream_t st) {
    if (n == 0) return;
    int blocks;
    const uint32_t share = spread(n, grid, &blocks, counter, st);
    RayBatch b{ox, oy, oz, dx, dy, dz, tmax, nullptr, n, prim, t, nullptr, nodes, prims, err, counter, share, CastTuning{16, 1, 16, 1},
               0u};
    if (share)
        chain(k_trace_rays<true, false, false, true, false>, blocks, kStackThreads, 0, st, sc, b);
    else
        k_trace_rays<true, false, false, false, false><<<blocks, kStackThreads, 0, st>>>(sc, b);
}

// the per-triangle table of a scene (its tri_normals still null): the normal,
// and in w the triangle's material type (the queue of its next stage)
__global__ void k_tri_normals(SceneView sc, uint32_t ntri, float4* __restrict__ out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= ntri) return;
    const f3 n = triangle_normal(sc, (int32_t)i);
    out[i] = make_float4(n.x, n.y, n.z, __int_as_float(__ldg(sc.materials + i).x));
}

void launch_tri_normals(const SceneView& sc, uint32_t ntri, float4* out, cudaStream_t st) {
    if (ntri == 0) return;
    k_tri_normals<<<(ntri + 255) / 256, 256, 0, st>>>(sc, ntri, out);
}

void launch_ray_reorder(const float* ox, const float* oy, const float* oz, const float* dx, const float* dy,
                        const float* dz, const float* tmax, uint64_t n, const RayKeyBox& kb, uint32_t* bins,
                        uint32_t* rank, float4* packed, int grid, cudaStream_t st) {
    if (n == 0) return;
    RaySoA r{ox, oy, oz, dx, dy, dz, tmax};
    // one pass of 256 x kKeyRays rays per block where the grid allows (the
    // block scheduler then overlaps one block's loads with another's work)
    const uint64_t tiles = (n + 256 * kKeyRays - 1) / (256 * kKeyRays);
    const int g = (int)std::min<uint64_t>(tiles, (uint64_t)grid);
    uint32_t* start = bins + kRayBins;
    cudaMemsetAsync(bins, 0, sizeof(uint32_t) * kRayBins, st);
    k_ray_bins<<<g, 256, 0, st>>>(r, n, kb, bins, rank);
    k_ray_bins_scan<<<kScanBlocks, 1024, 0, st>>>(bins, start);
    k_ray_scatter<<<g, 256, 0, st>>>(r, n, kb, start, rank, packed);
}

void launch_trace_packed(const SceneView& sc, const float4* packed, uint64_t n, int32_t* prim, float* t, float* ng,
                         uint32_t* err, unsigned long long* counter, const CastTuning& tune, int grid,
                         cudaStream_t st) {
    if (n == 0) return;
    cudaMemsetAsync(counter, 0, sizeof(unsigned long long), st);  // sorted calls are not few
    RayBatch b{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, packed, n, prim, t, ng, nullptr,
               nullptr, err, counter, 0u, tune, 0u};
    k_trace_rays<false, false, true, false, false><<<grid, kStackThreads, 0, st>>>(sc, b);
}

int trace_rays_max_blocks_per_sm(uint32_t stage) {
    int nb = 0;
    if (stage > 0) {
        cudaFuncSetAttribute(k_trace_rays<false, true, false, false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)(64 * kMaxStagedNodes));
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_trace_rays<false, true, false, false, false>, 256, 64 * (size_t)stage);
    } else {
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_trace_rays<false, false, false, false, false>, 256, 0);
    }
    return nb;
}

}  // namespace dev
}  // namespace rgr
