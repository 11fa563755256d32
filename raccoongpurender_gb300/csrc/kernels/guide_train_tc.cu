// guide_train_tc.cu — one training iteration of the path-guiding network on the
// 5th-generation tensor cores: forward, loss gradient, backward and the weight
// gradients as tcgen05.mma with the operands in shared memory and every
// accumulator in tensor memory (TMEM).
//
// A CTA (one per SM) holds kTrGroups groups of 256 row threads and three warps
// that only issue MMAs (one per group, one for every weight gradient).  A group works on tiles of 128 samples; two threads own a
// sample of the tile from its input encoding to its output gradient, each one half of
// its 64 columns (of its 8 lobes in the loss).  The layer
// inputs live in shared memory as one 128-byte line per sample (64 bf16,
// 128-byte swizzle, 8-line groups 1024 bytes apart), and that single layout
// is read three ways by the tensor core:
//  * as A of the forward product act . W (M = samples, K-major);
//  * as A of the weight gradient act^T . dY (M = layer inputs, K = samples,
//    MN-major), which accumulates in TMEM over every tile the CTA trains on;
//  * the output gradient dY, in the same layout, as A of dX = dY . W^T
//    (K-major) and as B of act^T . dY (MN-major).
// The weights stay in shared memory as W[in][out] lines, B of the forward
// product (MN-major) and of dX (K-major) alike.  The weight-gradient MMAs have
// M = 128: rows 0..63 are the layer's 64 inputs, rows 64..127 read a region of
// bf16 ones, so TMEM lanes 64..127 accumulate the column sums of dY, the bias
// gradient, in the same instructions.
//
// Per tile the group and the MMA warp take ten turns (the group writes an
// operand into shared memory and arrives on a_full; the MMA warp issues the
// turn's MMAs and commits them, D to d_full and dW to w_full; the group waits and
// reads the accumulators with tcgen05.ld):
//   0..4  forward, layer 0..4: D = act_l . W_l    (the group then adds the
//         bias, applies ReLU, rounds to bf16 and writes act_l+1; after layer 4
//         it computes the loss gradient of the 41 outputs and writes dY_4)
//   5..8  backward, layer 4..1: D = dY_l . W_l^T and dW_l += act_l^T . dY_l
//         (the group masks D by ReLU' of act_l and rounds while dW_l runs, then
//         writes dY_l-1)
//   9     dW_0 += act_0^T . dY_0
// Buffers per group: B1..B3 hold act_1..act_3; B0 holds act_0, then act_4
// once layer 0 has run, then act_0 again (re-encoded) a turn after dW_4; BY
// holds the output gradient of the current layer.  The two groups alternate on
// the tensor core: while one waits for its MMAs the other runs its epilogue.
//
// Bound by the chain of a tile's ten turns: shared memory holds two tiles' operands and
// no more, so a turn itself has to be short.  2^18 samples, CUDA events over 40
// iterations in a row: 133.6 us an iteration with one thread a sample and one warp
// issuing every MMA from run-time loops (the issuing warp set the pace: two threads
// a sample changed nothing then, 135 us a launch); 93 us a launch with the issue
// unrolled, warp-uniform and split over three warps, 92.5 us an iteration with bias and
// ReLU' operands loaded ahead of the waits, no timer read in a short wait, and the
// reduction, Adam and bookkeeping in one launch.  A tile takes 20.5k cycles: 3.9k waiting
// for the forward products, 3.4k for the dX, 1.4k for dW_0, 4.7k in the loss.
//
// After its last tile each CTA writes its weight and bias gradients and loss
// to its own slot of a partials buffer; a second kernel sums the slots in a
// fixed order (no atomics) and takes the Adam step.  Inside a CTA the two groups' tiles add into the
// same accumulators in the order their turns reach the tensor core, so FP32
// rounding differs slightly from run to run.  Every wait is
// bounded: on a timeout the CTA records an error, stops, waits (bounded) for
// the MMAs it issued and frees its TMEM.
//
// Arithmetic follows the mma.sync training kernel (guide_mlp.cu): BF16
// operands with FP32 accumulation, FP32 bias adds, layer inputs and output
// gradients rounded to bf16, ReLU' from the stored bf16 input.
#include <cuda_bf16.h>

#include "guide.cuh"

namespace rgr {
namespace dev {
namespace {

constexpr int kTrGroups = 2;                           // 128-sample tiles in flight per CTA
constexpr int kTrRows = 128;                           // samples per tile
constexpr int kTrHalves = 2;                           // row threads per sample
constexpr int kTrGroupWarps = kTrHalves * kTrRows / 32;
// the MMA-issuing warps: one per group for its forward and dX, then one for every dW
constexpr int kTrMmaWarp = kTrGroups * kTrGroupWarps;
constexpr int kTrMmaWarps = kTrGroups + 1;
constexpr int kTrThreads = 32 * (kTrMmaWarp + kTrMmaWarps);
constexpr uint32_t kTileBytes = kTrRows * 128u;        // a tile's lines: 16 KB
constexpr int kTrBufs = 5;                             // B0..B3 and BY
constexpr int kBufY = 4;
constexpr uint32_t kWLayerBytes = 64u * 128u;          // W[in][out] of a layer, 64 lines
// TMEM: dW of layer l in columns 64 l .. 64 l + 63 (lanes 0..63 dW[in][out],
// lanes 64..127 the bias gradient); group g's accumulator D at 320 + 64 g
constexpr uint32_t kDwCols = 64u * kGuideLayers;
constexpr int kTrCols = 512;
static_assert(kDwCols + 64u * kTrGroups <= (uint32_t)kTrCols, "TMEM columns");
constexpr uint32_t kWaitNs = 1000000000u;              // a wait gives up after 1 s (%globaltimer)
constexpr uint32_t kWaitPolls = 1u << 30;              // and after this many polls whatever the timer says
constexpr uint32_t kErrTrainTimeout = 2u;

struct __align__(1024) SmemTr {
    unsigned char w[kGuideLayers][kWLayerBytes];        // W[l][in][out], 128-byte swizzle (40 KB)
    unsigned char buf[kTrGroups][kTrBufs][kTileBytes];  // per group B0..B3, BY (160 KB)
    unsigned char ones[2048];                           // bf16 1.0: rows 64..127 of every dW MMA's A (16 lines)
    float4 xch[kTrGroups][2 * kTrHalves][kTrRows];      // per sample and half: its lobes' logits, densities
    float bias[kGuideLayers][kGuideWidth];
    unsigned long long a_full[kTrGroups];               // turns 0..8: the operand is written (one arrival per warp)
    unsigned long long b_full[kTrGroups];               // turns 5..9, for dW
    unsigned long long d_full[kTrGroups];               // the turn's D is done (one commit)
    unsigned long long w_full[kTrGroups];               // the turn's dW is done (one commit)
    unsigned long long x_full[kTrGroups][4];            // both halves of 32 samples have written xch
    unsigned long long fin;                             // every MMA the CTA issued is done
    uint32_t tmem_base;
    uint32_t error;
    uint32_t trained;                                   // the MMA warp issued every turn of at least one tile
    float loss;
};
// the ones sit above every activation buffer: the dW MMAs reach them with a
// positive leading-byte offset of at most 160 KB (14 bits of 16-byte units)
static_assert(sizeof(SmemTr) + 1024 <= 232448, "shared memory");

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// shared-memory descriptor, 128-byte swizzle, version 1 (bits 46-47), swizzle
// mode 2 (bits 61-63), start address >> 4 (bits 0-13), leading byte offset
// >> 4 (bits 16-29), stride byte offset >> 4 (bits 32-45).
//  K-major: lines are M (or N) rows of 64 K elements; SBO 1024 between
//    8-row groups; LBO unused (16).
//  MN-major: lines are K rows of 64 M (or N) elements; SBO 1024 between
//    8-line groups along K; LBO between 64-element groups along M (or N).
__device__ __forceinline__ uint64_t desc_sw128(uint32_t saddr, uint32_t lbo) {
    return (uint64_t)((saddr & 0x3ffffu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3fffu) << 16) |
           ((uint64_t)(1024 >> 4) << 32) | ((uint64_t)1 << 46) | ((uint64_t)2 << 61);
}
// instruction descriptors of kind::f16, D FP32 (bits 4-5 = 1), A and B BF16
// (bits 7-9, 10-12 = 1), N 64 (bits 17-22 = N >> 3), M 128 (bits 24-28 =
// M >> 4); bit 15 / 16 = A / B MN-major
constexpr uint32_t kIdescBase = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(64 >> 3) << 17) |
                                ((uint32_t)(128 >> 4) << 24);
constexpr uint32_t kIdescFwd = kIdescBase | (1u << 16);              // act (K-major) . W (MN-major)
constexpr uint32_t kIdescDx = kIdescBase;                             // dY (K-major) . W^T (K-major)
constexpr uint32_t kIdescDw = kIdescBase | (1u << 15) | (1u << 16);  // act^T (MN-major) . dY (MN-major)

__device__ __forceinline__ void mma_ss(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                       uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(tmem_d),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void mma_commit(uint32_t mbar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(mbar)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t mbar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    return ok != 0u;
}
__device__ __forceinline__ bool mbar_test(uint32_t mbar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(mbar), "r"(parity)
        : "memory");
    return ok != 0u;
}
__device__ __forceinline__ uint32_t global_ns() {
    uint32_t t;
    asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t));
    return t;
}
// bounded wait for the phase with the given parity: false after kWaitNs (or kWaitPolls
// polls); the timer, a slow register to read, is not read by a short wait
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
    uint32_t t0 = 0u;
    for (uint32_t i = 0; i < kWaitPolls; ++i) {
        if (mbar_try_wait(mbar, parity)) return true;
        if ((i & 63u) == 63u) {
            const uint32_t now = global_ns();
            if (i == 63u) t0 = now;
            else if (now - t0 > kWaitNs) return false;
        }
    }
    return false;
}
__device__ __forceinline__ void mbar_arrive(uint32_t mbar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(mbar) : "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
// generic-proxy shared-memory writes visible to the tensor core
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t* r) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory"); }

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
__device__ __forceinline__ uint32_t relu_pack2(float lo, float hi) {
    uint32_t d;
    asm("cvt.rn.relu.bf16x2.f32 %0, %1, %2;\n" : "=r"(d) : "f"(hi), "f"(lo));
    return d;
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld1(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];\n" : "=r"(r[0]) : "r"(taddr));
}

// chunk c (16 bytes, 8 bf16) of sample r's line in a tile buffer, at its swizzled place
__device__ __forceinline__ void store_chunk(unsigned char* tile, uint32_t r, uint32_t c, uint32_t w0, uint32_t w1,
                                            uint32_t w2, uint32_t w3) {
    *reinterpret_cast<uint4*>(tile + sw128_offset(r, c)) = make_uint4(w0, w1, w2, w3);
}

// Frequency encoding of the sample (as guide_mlp.cu and guide_tc.cu):
// coordinate i gives the features 4i .. 4i + 3 = sin(pi v), cos(pi v),
// sin(2 pi v), cos(2 pi v), the first octave by the SFU's sine and cosine
// (absolute error near 2^-21 for these arguments, far below the bf16 rounding
// that follows), the second by the double-angle identities; inputs 36..63 are
// zero.  Half 0 writes coordinates 0..5 (v[0..5]; chunks 0..2) and the line's last
// chunks, half 1 coordinates 6..8 (v[0..2]; chunks 3, 4) and chunk 5.
__device__ __forceinline__ void encode_words(float v, uint32_t& a, uint32_t& b) {
    float s, c;
    __sincosf(3.14159265358979f * v, &s, &c);
    a = pack_bf16(s, c);
    b = pack_bf16(2.0f * s * c, (c - s) * (c + s));
}
__device__ __forceinline__ void encode_half(const float* v, uint32_t half, unsigned char* tile, uint32_t r) {
    uint32_t w[4];
    if (half == 0u) {
#pragma unroll
        for (uint32_t c = 0; c < 3u; ++c) {
            encode_words(v[2 * c], w[0], w[1]);
            encode_words(v[2 * c + 1], w[2], w[3]);
            store_chunk(tile, r, c, w[0], w[1], w[2], w[3]);
        }
        store_chunk(tile, r, 6u, 0u, 0u, 0u, 0u);
        store_chunk(tile, r, 7u, 0u, 0u, 0u, 0u);
    } else {
        encode_words(v[0], w[0], w[1]);
        encode_words(v[1], w[2], w[3]);
        store_chunk(tile, r, 3u, w[0], w[1], w[2], w[3]);
        encode_words(v[2], w[0], w[1]);
        store_chunk(tile, r, 4u, w[0], w[1], 0u, 0u);
        store_chunk(tile, r, 5u, 0u, 0u, 0u, 0u);
    }
}

// One lobe of the mixture (guide.cuh's lobe_of) and its density, in the SFU's
// exponential, logarithm and reciprocal: the loss gradient is rounded to bf16
// right after, so their relative errors near 2^-21 do not show.  The weight
// logit keeps the accurate tanh, whose error would otherwise reach 2^-11.
struct LobeT {
    float mx, my, mz, kappa, inv_norm, norm, th, logit, sp;
};
__device__ __forceinline__ LobeT lobe_t(float o0, float o1, float o2, float o3, float o4) {
    LobeT L;
    const float ss = fmaxf(o0 * o0 + o1 * o1 + o2 * o2, 1.0e-24f);
    L.inv_norm = rsqrtf(ss);
    L.norm = ss * L.inv_norm;
    L.mx = o0 * L.inv_norm;
    L.my = o1 * L.inv_norm;
    L.mz = o2 * L.inv_norm;
    L.sp = o3 > 20.0f ? o3 : __logf(1.0f + __expf(o3));
    L.kappa = fminf(L.sp + 0.01f, kGuideKappaMax);
    L.th = tanhf(o4 * (1.0f / kGuideLogitBound));
    L.logit = kGuideLogitBound * L.th;
    return L;
}
__device__ __forceinline__ float vmf_t(float kappa, float c) {
    return __fdividef(kappa, 6.283185307179586f * (1.0f - __expf(-2.0f * kappa))) * __expf(kappa * (c - 1.0f));
}

// The loss of one sample, -wt log q(d), and its gradient with respect to the
// 41 raw outputs (field-major mixture outputs, then the selection logit,
// whose term -wt log(a q + (1 - a) pb) holds q fixed), into dY's line: the
// derivatives of guide.cuh's lobe_grad.  Half h has the raw outputs of lobes
// 4h .. 4h + 3 (o[4 f + j]: field f of lobe 4h + j) and writes their words; the
// halves trade their lobes' logits and densities through `xch` (`traded` waits for
// the other half) and both sum the mixture over the eight lobes in order.
template <class Trade>
__device__ __forceinline__ bool row_loss_half(const float* o, float sel, uint32_t half, float dx, float dy, float dz,
                                              float wt, float pb, float4 (*xch)[kTrRows], uint32_t r,
                                              unsigned char* tile, float& loss, Trade traded) {
    float lg[kGuideLobes], f[kGuideLobes];
    LobeT lobe[4];
    {
        float own[4], fo[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const LobeT L = lobe[j] = lobe_t(o[j], o[4 + j], o[8 + j], o[12 + j], o[16 + j]);
            own[j] = L.logit;
            fo[j] = vmf_t(L.kappa, L.mx * dx + L.my * dy + L.mz * dz);
        }
        xch[2u * half][r] = make_float4(own[0], own[1], own[2], own[3]);
        xch[2u * half + 1u][r] = make_float4(fo[0], fo[1], fo[2], fo[3]);
        if (!traded()) return false;
        const float4 a = xch[0][r], b = xch[2][r], c = xch[1][r], d = xch[3][r];
        lg[0] = a.x, lg[1] = a.y, lg[2] = a.z, lg[3] = a.w, lg[4] = b.x, lg[5] = b.y, lg[6] = b.z, lg[7] = b.w;
        f[0] = c.x, f[1] = c.y, f[2] = c.z, f[3] = c.w, f[4] = d.x, f[5] = d.y, f[6] = d.z, f[7] = d.w;
    }
    float mx = -3.0e38f;
#pragma unroll
    for (int i = 0; i < kGuideLobes; ++i) mx = fmaxf(mx, lg[i]);
    float den = 0.0f;
#pragma unroll
    for (int i = 0; i < kGuideLobes; ++i) {
        lg[i] = __expf(lg[i] - mx);
        den += lg[i];
    }
    const float rden = __fdividef(1.0f, den);
    float q = 0.0f;
#pragma unroll
    for (int i = 0; i < kGuideLobes; ++i) {
        lg[i] *= rden;  // the lobe's weight pi
        q += lg[i] * f[i];
    }
    q = fmaxf(q, 1.0e-30f);
    const float rq = __fdividef(1.0f, q);
    const bool live = wt > 0.0f;
    float pi4[4], f4_[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        pi4[j] = half ? lg[4 + j] : lg[j];
        f4_[j] = half ? f[4 + j] : f[j];
    }
    uint32_t w[2][5];  // lobes 4h + 2m, 4h + 2m + 1 of field k: word 4k + 2h + m of the line
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        float gg[2][5];
#pragma unroll
        for (int s2 = 0; s2 < 2; ++s2) {
            const int j = 2 * m + s2;
            const LobeT& L = lobe[j];
            const float pi = pi4[j], rr = pi * f4_[j] * rq;
            float* g = gg[s2];
            g[4] = -wt * (rr - pi) * (1.0f - L.th * L.th);
            const float k = L.kappa, e2 = __expf(-2.0f * k);
            const float md = L.mx * dx + L.my * dy + L.mz * dz;
            const float dlogf = __fdividef(1.0f, k) - __fdividef(2.0f * e2, 1.0f - e2) + (md - 1.0f);
            const float dk = (L.sp + 0.01f < kGuideKappaMax) ? __fdividef(1.0f, 1.0f + __expf(-o[12 + j])) : 0.0f;
            g[3] = -wt * rr * dlogf * dk;
            const float gx = -wt * rr * k * dx, gy = -wt * rr * k * dy, gz = -wt * rr * k * dz;
            const float gm = gx * L.mx + gy * L.my + gz * L.mz;
            const float pen = 2.0f * wt * kGuideNormPenalty * (L.norm - 1.0f);
            g[0] = (gx - gm * L.mx) * L.inv_norm + pen * L.mx;
            g[1] = (gy - gm * L.my) * L.inv_norm + pen * L.my;
            g[2] = (gz - gm * L.mz) * L.inv_norm + pen * L.mz;
        }
#pragma unroll
        for (int k = 0; k < 5; ++k) w[m][k] = live ? pack_bf16(gg[0][k], gg[1][k]) : 0u;
    }
#pragma unroll
    for (uint32_t k = 0; k < 5u; ++k)
        *reinterpret_cast<uint2*>(tile + sw128_offset(r, k) + 8u * half) = make_uint2(w[0][k], w[1][k]);
    if (half == 0u) {
        store_chunk(tile, r, 5u, live ? pack_bf16(selection_grad(sel, q, pb, wt), 0.0f) : 0u, 0u, 0u, 0u);
        if (live) loss += -wt * __logf(q);
    } else {
        store_chunk(tile, r, 6u, 0u, 0u, 0u, 0u);
        store_chunk(tile, r, 7u, 0u, 0u, 0u, 0u);
    }
    return true;
}

// true in one lane of the (converged) warp, the same one each time
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile(
        "{\n\t.reg .pred e;\n\t"
        "elect.sync _|e, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, e;\n\t}\n"
        : "=r"(p));
    return p != 0u;
}
// kSteps MMAs of one product, the descriptors advancing by a constant per K step.  With the
// steps unrolled and the operands warp-uniform (elected lane, shuffled warp index) an
// MMA costs a few issue slots; as a run-time loop under `lane == 0` the issuing
// warp, not the tensor pipe, set the pace of the kernel.
template <int kSteps>
__device__ __forceinline__ void issue_product(uint32_t d, uint64_t a, uint64_t a_step, uint64_t b, uint64_t b_step,
                                              uint32_t idesc, uint32_t accumulate) {
#pragma unroll
    for (int s = 0; s < kSteps; ++s)
        mma_ss(d, a + (uint64_t)s * a_step, b + (uint64_t)s * b_step, idesc, s > 0 ? 1u : accumulate);
}

// samples: 16 floats each (x, n, wo, wi, weight); loss weight = weight * scale,
// scale = weight_scale / *wsum (weight_scale without wsum).  part: this CTA's
// slot (kGuidePartStride floats) of the partials buffer.
// count: the number of samples on the device (at most cap), or null: cap samples.
__global__ void __launch_bounds__(kTrThreads, 1)
    k_guide_train_tc(GuideView gv, const float* __restrict__ samples, const uint32_t* __restrict__ count, uint32_t cap,
                     uint32_t min_count, const float* __restrict__ wsum, float weight_scale, float* __restrict__ part,
                     uint32_t* err) {
    const uint32_t n = count ? min(*count, cap) : cap;
    if (n < min_count) return;  // too few yet: the samples carry over (the reduction skips too)
    float* my_part = part + (size_t)blockIdx.x * kGuidePartStride;
    const uint32_t ntiles = (n + kTrRows - 1u) / kTrRows, stride = gridDim.x * kTrGroups;
    if (blockIdx.x * kTrGroups >= ntiles) {  // no tile here: an empty slot
        for (uint32_t i = threadIdx.x; i < kGuidePartStride; i += blockDim.x) my_part[i] = 0.0f;
        return;
    }
    extern __shared__ unsigned char smem_raw[];
    SmemTr& S = *reinterpret_cast<SmemTr*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const uint32_t t = threadIdx.x, lane = t & 31u;
    // the warp's group, TMEM lane quarter (its 32 samples of a tile) and half of their columns
    const uint32_t warp = __shfl_sync(0xffffffffu, t >> 5, 0), g = warp / kTrGroupWarps, quarter = warp & 3u,
                   half = (warp >> 2) & 1u;
    const uint32_t lt = 32u * quarter + lane;
    float scale = weight_scale;
    if (wsum) {
        const float s = *wsum;
        scale = s > 0.0f ? weight_scale / s : 0.0f;
    }
    // stage the weights as W[in][out] lines, the biases and the ones
    {
        const uint4* src = reinterpret_cast<const uint4*>(gv.wbf);
        for (uint32_t i = t; i < (uint32_t)kGuideLayers * 64u * 8u; i += blockDim.x) {
            const uint32_t l = i >> 9, in = (i >> 3) & 63u, c = i & 7u;
            *reinterpret_cast<uint4*>(S.w[l] + sw128_offset(in, c)) = src[i];
        }
        for (uint32_t i = t; i < (uint32_t)kGuideBiases; i += blockDim.x) (&S.bias[0][0])[i] = gv.b[i];
        for (uint32_t i = t; i < sizeof(S.ones) / 16u; i += blockDim.x)
            reinterpret_cast<uint4*>(S.ones)[i] = make_uint4(0x3f803f80u, 0x3f803f80u, 0x3f803f80u, 0x3f803f80u);
    }
    if (t == 0) {
        S.error = 0u;
        S.trained = 0u;
        S.loss = 0.0f;
        for (int i = 0; i < kTrGroups; ++i) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&S.a_full[i])), "r"(kTrGroupWarps)
                         : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&S.b_full[i])), "r"(kTrGroupWarps)
                         : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&S.d_full[i])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&S.w_full[i])) : "memory");
            for (int q = 0; q < 4; ++q)
                asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&S.x_full[i][q])),
                             "r"(kTrHalves)
                             : "memory");
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&S.fin)), "r"(kTrMmaWarps) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&S.tmem_base)),
                     "r"(kTrCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = S.tmem_base;
    auto tiles_of = [&](uint32_t gg) -> uint32_t {
        const uint32_t base = blockIdx.x * kTrGroups + gg;
        return base < ntiles ? (ntiles - base + stride - 1u) / stride : 0u;
    };

    if (warp >= (uint32_t)kTrMmaWarp) {
        // ------------------------------------------------------------ MMA warps
        const uint32_t role = warp - (uint32_t)kTrMmaWarp;
        const uint32_t w_addr = smem_u32(S.w);
        bool late = false;          // a group stopped arriving
        uint32_t dw_started = 0u;
        if (role < (uint32_t)kTrGroups) {
            // group `role`: forward of layers 0..4 (turns 0..4), dX of layers 4..1 (turns 5..8)
            const uint32_t b0 = smem_u32(S.buf[role][0]), b1 = b0 + kTileBytes, b2 = b1 + kTileBytes,
                           b3 = b2 + kTileBytes, by = smem_u32(S.buf[role][kBufY]);
            const uint32_t d = tmem + kDwCols + 64u * role;
            const uint32_t af = smem_u32(&S.a_full[role]), df = smem_u32(&S.d_full[role]);
            uint32_t ph = 0u;
            for (uint32_t k = tiles_of(role); k > 0u && !late; --k) {
#pragma unroll
                for (uint32_t turn = 0; turn < 9u; ++turn) {
                    if (late || !__all_sync(0xffffffffu, mbar_wait(af, ph))) {
                        late = true;
                        continue;
                    }
                    ph ^= 1u;
                    fence_after();
                    if (elect_one()) {
                        if (turn < 5u) {
                            // B0 holds act_0, then act_4; the encoding's 36 inputs fit in K = 48
                            const uint32_t act = turn == 1u ? b1 : turn == 2u ? b2 : turn == 3u ? b3 : b0;
                            const uint64_t a = desc_sw128(act, 16u), b = desc_sw128(w_addr + turn * kWLayerBytes, 8192u);
                            if (turn == 0u) issue_product<3>(d, a, 2u, b, 128u, kIdescFwd, 0u);
                            else issue_product<4>(d, a, 2u, b, 128u, kIdescFwd, 0u);
                        } else {
                            const uint32_t l = 9u - turn;
                            issue_product<4>(d, desc_sw128(by, 16u), 2u, desc_sw128(w_addr + l * kWLayerBytes, 16u), 2u,
                                             kIdescDx, 0u);
                        }
                        mma_commit(df);
                    }
                    __syncwarp();
                }
            }
        } else {
            // dW of both groups: one thread issues every MMA into the shared accumulators,
            // and one thread's tcgen05 operations run in issue order
            const uint32_t ones = smem_u32(S.ones);
            uint32_t left[kTrGroups], ph[kTrGroups], turn[kTrGroups];
#pragma unroll
            for (int i = 0; i < kTrGroups; ++i) {
                left[i] = (uint32_t)kGuideLayers * tiles_of(i);
                ph[i] = 0u;
                turn[i] = 5u;
            }
            uint32_t last = 0u, idle = 0u;  // when the warp fell idle, polls since
            for (;;) {
                bool any = false, progressed = false;
#pragma unroll
                for (int i = 0; i < kTrGroups; ++i) {
                    if (left[i] == 0u) continue;
                    any = true;
                    if (__shfl_sync(0xffffffffu, (uint32_t)mbar_test(smem_u32(&S.b_full[i]), ph[i]), 0) == 0u) continue;
                    ph[i] ^= 1u;
                    fence_after();
                    const uint32_t l = 9u - turn[i], act = smem_u32(S.buf[i][l == 4u ? 0u : l]),
                                   by = smem_u32(S.buf[i][kBufY]);
                    if (elect_one()) {
                        // A: 64 inputs of 16 samples (2048 bytes a K step), and the same 16 lines of
                        // ones after them (the leading byte offset shrinks as the start moves on)
                        issue_product<kTrRows / 16>(tmem + 64u * l, desc_sw128(act, ones - act),
                                                    128u - ((uint64_t)128u << 16), desc_sw128(by, 8192u), 128u, kIdescDw,
                                                    (dw_started >> l) & 1u);
                        mma_commit(smem_u32(&S.w_full[i]));
                    }
                    __syncwarp();
                    dw_started |= 1u << l;
                    turn[i] = turn[i] == 9u ? 5u : turn[i] + 1u;
                    --left[i];
                    progressed = true;
                }
                if (!any) break;
                idle = progressed ? 0u : idle + 1u;
                if (idle > 4u) __nanosleep(32);  // leave the issue slots to the row threads
                if ((idle & 63u) == 63u) {
                    const uint32_t now = global_ns();
                    if (idle == 63u) last = now;
                    if (idle >= kWaitPolls || now - last > kWaitNs) {
                        late = true;
                        break;
                    }
                }
            }
        }
        // every MMA issued above has completed before TMEM is read or freed
        if (elect_one()) mma_commit(smem_u32(&S.fin));
        __syncwarp();
        const bool fin_ok = mbar_wait(smem_u32(&S.fin), 0u);
        if (lane == 0u) {
            if (!fin_ok || late) S.error = kErrTrainTimeout;
            if (dw_started == (1u << kGuideLayers) - 1u) S.trained = 1u;
        }
    } else {
        // ------------------------------------------------------------ row threads
        const uint32_t d = tmem + kDwCols + 64u * g + ((32u * quarter) << 16);  // this warp's 32 TMEM lanes
        unsigned char* B0 = S.buf[g][0];
        unsigned char* BY = S.buf[g][kBufY];
        const uint32_t af = smem_u32(&S.a_full[g]), df = smem_u32(&S.d_full[g]), wf = smem_u32(&S.w_full[g]),
                       xf = smem_u32(&S.x_full[g][quarter]);
        const uint32_t kt = tiles_of(g), base = blockIdx.x * kTrGroups + g;
        uint32_t pd = 0u, pw = 0u, px = 0u;
        bool timed_out = false;
        float lsum = 0.0f;
        // a bounded wait of the whole warp (the same answer in every lane)
        auto wait = [&](uint32_t bar, uint32_t& parity) -> bool {
            const bool ok = __all_sync(0xffffffffu, mbar_wait(bar, parity));
            parity ^= 1u;
            if (!ok) S.error = kErrTrainTimeout;
            fence_after();
            return ok;
        };
        const uint32_t bf = smem_u32(&S.b_full[g]);
        // hand the turn's operand to the MMA warps: of D (turns 0..8), of dW (turns 5..9)
        auto hand = [&](bool for_d, bool for_w) {
            fence_async_smem();  // the lines just written, to the tensor core
            fence_before();      // the accumulator reads just done, before the next MMAs
            __syncwarp();
            if (lane == 0u) {
                if (for_d) mbar_arrive(af);
                if (for_w) mbar_arrive(bf);
            }
        };
        // the 16 floats of tile k's sample (zeros past the end)
        float4 s0, s1, s2, s3;
        auto load = [&](uint32_t k) {
            const uint32_t r = (base + k * stride) * (uint32_t)kTrRows + lt;
            s0 = s1 = s2 = s3 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (k < kt && r < n) {
                const float4* p4 = reinterpret_cast<const float4*>(samples + 16 * (size_t)r);
                s0 = __ldg(p4), s1 = __ldg(p4 + 1), s2 = __ldg(p4 + 2), s3 = __ldg(p4 + 3);
            }
        };
        load(0u);
        for (uint32_t k = 0; k < kt; ++k) {
            // this half's coordinates: position and normal, or the outgoing direction
            float v[6];
            if (half == 0u) {
                const float p3[3] = {s0.x, s0.y, s0.z};
#pragma unroll
                for (int c = 0; c < 3; ++c) v[c] = (p3[c] - gv.params.lo[c]) * gv.params.inv_ext[c];
                v[3] = 0.5f * (s0.w + 1.0f), v[4] = 0.5f * (s1.x + 1.0f), v[5] = 0.5f * (s1.y + 1.0f);
            } else {
                v[0] = 0.5f * (s1.z + 1.0f), v[1] = 0.5f * (s1.w + 1.0f), v[2] = 0.5f * (s2.x + 1.0f);
                v[3] = v[4] = v[5] = 0.0f;
            }
            const float dx = s2.y, dy = s2.z, dz = s2.w, wt = s3.x * scale, pb = s3.y;
            encode_half(v, half, B0, lt);
            // forward: turns 0..4
#pragma unroll 1
            for (uint32_t l = 0; l + 1u < (uint32_t)kGuideLayers; ++l) {
                hand(true, false);
                float4 bias[8];
#pragma unroll
                for (int c = 0; c < 8; ++c) bias[c] = reinterpret_cast<const float4*>(S.bias[l] + 32u * half)[c];
                if (!wait(df, pd)) {
                    timed_out = true;
                    break;
                }
                unsigned char* next = l + 1u < 4u ? S.buf[g][l + 1u] : B0;  // act_4 into B0
                uint32_t x[32], y[16];
                tmem_ld32(d + 32u * half, x);
                tmem_wait_ld();
#pragma unroll
                for (int c = 0; c < 8; ++c) {
                    const float4 bb = bias[c];
                    y[2 * c] = relu_pack2(__uint_as_float(x[4 * c]) + bb.x, __uint_as_float(x[4 * c + 1]) + bb.y);
                    y[2 * c + 1] =
                        relu_pack2(__uint_as_float(x[4 * c + 2]) + bb.z, __uint_as_float(x[4 * c + 3]) + bb.w);
                }
#pragma unroll
                for (uint32_t c = 0; c < 4u; ++c)
                    store_chunk(next, lt, 4u * half + c, y[4 * c], y[4 * c + 1], y[4 * c + 2], y[4 * c + 3]);
            }
            if (timed_out) break;
            hand(true, false);
            if (!wait(df, pd)) {
                timed_out = true;
                break;
            }
            // loss gradient: dY_4 (turn 5)
            {
                uint32_t x[20], z = 0u;
#pragma unroll
                for (uint32_t f = 0; f < 5u; ++f) tmem_ld4(d + 8u * f + 4u * half, x + 4 * f);
                tmem_ld1(d + (uint32_t)kGuideSelOutput, &z);
                tmem_wait_ld();
                float o[20];
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    const float4 bb = *reinterpret_cast<const float4*>(S.bias[kGuideLayers - 1] + 8 * f + 4 * half);
                    o[4 * f] = __uint_as_float(x[4 * f]) + bb.x;
                    o[4 * f + 1] = __uint_as_float(x[4 * f + 1]) + bb.y;
                    o[4 * f + 2] = __uint_as_float(x[4 * f + 2]) + bb.z;
                    o[4 * f + 3] = __uint_as_float(x[4 * f + 3]) + bb.w;
                }
                const float sel = __uint_as_float(z) + S.bias[kGuideLayers - 1][kGuideSelOutput];
                const bool ok = row_loss_half(o, sel, half, dx, dy, dz, wt, pb, S.xch[g], lt, BY, lsum, [&] {
                    __syncwarp();
                    if (lane == 0u) mbar_arrive(xf);
                    return wait(xf, px);
                });
                if (!ok) {
                    timed_out = true;
                    break;
                }
            }
            // backward: turns 5..8 give dX of layers 4..1; masked by ReLU' of the layer's
            // input (read back from this sample's line: act_l is > 0 where its bf16 is
            // not zero), it is dY of layers 3..0
#pragma unroll 1
            for (int l = 4; l >= 1; --l) {
                hand(true, true);
                const unsigned char* act = l == 4 ? B0 : S.buf[g][l];
                uint4 a4[4];  // this thread wrote them
#pragma unroll
                for (uint32_t c = 0; c < 4u; ++c)
                    a4[c] = *reinterpret_cast<const uint4*>(act + sw128_offset(lt, 4u * half + c));
                if (!wait(df, pd)) {
                    timed_out = true;
                    break;
                }
                uint32_t x[32], y[16];
                tmem_ld32(d + 32u * half, x);
                tmem_wait_ld();
#pragma unroll
                for (uint32_t c = 0; c < 4u; ++c) {
                    const uint4 a = a4[c];
                    const uint32_t aw[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int i = 4 * (int)c + j;  // word i of the half: inputs 32 h + 2i, + 1
                        y[i] = pack_bf16((aw[j] & 0xffffu) ? __uint_as_float(x[2 * i]) : 0.0f,
                                         (aw[j] >> 16) ? __uint_as_float(x[2 * i + 1]) : 0.0f);
                    }
                }
                if (!wait(wf, pw)) {  // dW_l has read dY_l and act_l
                    timed_out = true;
                    break;
                }
#pragma unroll
                for (uint32_t c = 0; c < 4u; ++c)
                    store_chunk(BY, lt, 4u * half + c, y[4 * c], y[4 * c + 1], y[4 * c + 2], y[4 * c + 3]);
                // act_0 back into B0 for dW_0.  It writes chunks whose act_4 the other half's
                // thread reads above, at l = 4: that read comes before its warp's arrival at the
                // next turn, and so before this turn's D
                if (l == 3) encode_half(v, half, B0, lt);
            }
            if (timed_out) break;
            // turn 9: dW_0; its end frees B0 and BY for the next tile
            hand(false, true);
            load(k + 1u);
            if (!wait(wf, pw)) {
                timed_out = true;
                break;
            }
        }
        // this group's loss
        for (int off = 16; off > 0; off >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, off);
        if ((t & 31u) == 0u) atomicAdd(&S.loss, lsum);
    }
    fence_before();
    __syncthreads();
    fence_after();
    // the CTA's gradients: dW rows from TMEM lanes 0..63 (quarters 0 and 1), the bias
    // gradient from lane 64; zeros if a timeout left them incomplete
    const bool ok = S.trained != 0u && S.error == 0u;
    if (warp < (uint32_t)kTrMmaWarp && quarter < 3u) {
        for (uint32_t l = warp >> 2; l < (uint32_t)kGuideLayers; l += (uint32_t)kTrMmaWarp / 4u) {
            for (uint32_t h = 0; h < 2u; ++h) {
                uint32_t x[32];
                tmem_ld32(tmem + 64u * l + 32u * h + ((32u * quarter) << 16), x);
                tmem_wait_ld();
                float* row = quarter < 2u ? my_part + (size_t)l * 4096u + (size_t)lt * 64u
                                          : my_part + kGuideWeights + l * 64u;
                if (quarter < 2u || lane == 0u) {
                    float4* dst = reinterpret_cast<float4*>(row + 32u * h);
#pragma unroll
                    for (int c = 0; c < 8; ++c)
                        dst[c] = ok ? make_float4(__uint_as_float(x[4 * c]), __uint_as_float(x[4 * c + 1]),
                                                  __uint_as_float(x[4 * c + 2]), __uint_as_float(x[4 * c + 3]))
                                    : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                }
            }
        }
    }
    if (t == 0) my_part[kGuideParams] = ok ? S.loss : 0.0f;
    fence_before();
    __syncthreads();
    if (warp == 0) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kTrCols) : "memory");
    }
    if (t == 0 && S.error && err) atomicOr(err, S.error);
}

// The gradients and the loss as the sums of the CTAs' slots, in a fixed order: a
// block covers 32 parameters; its 8 warps each sum every 8th slot (a warp's
// loads are 32 consecutive floats of one slot), then one warp adds the 8
// partial sums in warp order, and takes the Adam step with them.  The last block to
// finish does the iteration's bookkeeping.  The slots are 12.7 MB in L2: one pass over
// them is what this costs (9 us; as separate reduction, Adam and bookkeeping launches
// 8.5 + 5.6 + 4.0 us).
constexpr int kReduceParams = 32, kReduceWarps = 8;
__global__ void __launch_bounds__(32 * kReduceWarps)
    k_guide_update_tc(GuideView g, const float* part, uint32_t nparts, const uint32_t* count, uint32_t cap,
                      float* __restrict__ grads, int step, GuideAdam adam, GuideTrainD t, float* host_loss) {
    // the training kernel's slots are written from here on (and so not read through the read-only path)
    follow();
    const uint32_t n = count ? *count : cap;
    if (n == 0u || (step && n < t.min_count)) {  // no iteration
        if (step && blockIdx.x == 0 && threadIdx.x == 0) finish_iteration(g, t, n);
        return;
    }
    __shared__ float partial[kReduceWarps][kReduceParams];
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t i = blockIdx.x * kReduceParams + lane;
    const float iter = step ? (float)(*t.iter + 1u) : 0.0f;
    float s = 0.0f;
    if (i <= (uint32_t)kGuideParams)
#pragma unroll 4
        for (uint32_t c = w; c < nparts; c += kReduceWarps) s += __ldcg(part + (size_t)c * kGuidePartStride + i);
    partial[w][lane] = s;
    __syncthreads();
    if (w != 0u) return;
    float sum = 0.0f;
#pragma unroll
    for (int k = 0; k < kReduceWarps; ++k) sum += partial[k][lane];
    if (i < (uint32_t)kGuideParams) {
        if (grads) grads[i] = sum;
        if (step) adam_update(g, i, sum, iter, adam);
    } else if (i == (uint32_t)kGuideParams) {
        g.loss[0] = step ? sum : 0.0f;
        g.loss[1] = sum;
        if (host_loss) *host_loss = sum;
    }
    if (!step) return;
    __threadfence();
    __syncwarp();
    uint32_t* ticket = reinterpret_cast<uint32_t*>(g.loss) + 2;
    if (lane == 0u && atomicAdd(ticket, 1u) + 1u == gridDim.x) {  // every block has read *t.iter
        __threadfence();
        *ticket = 0u;
        finish_iteration(g, t, n);
    }
}

}  // namespace

size_t guide_train_tc_smem() { return sizeof(SmemTr) + 1024; }

int guide_train_tc_attributes() {
    return (int)cudaFuncSetAttribute(k_guide_train_tc, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)guide_train_tc_smem());
}

void launch_guide_train_tc(const GuideView& g, const float* samples, const uint32_t* count, uint32_t cap,
                           uint32_t min_count, const float* wsum, float weight_scale, int grid, float* part,
                           uint32_t* err, cudaStream_t st) {
    k_guide_train_tc<<<grid, kTrThreads, guide_train_tc_smem(), st>>>(g, samples, count, cap, min_count, wsum,
                                                                      weight_scale, part, err);
}

void launch_guide_update_tc(const GuideView& g, const float* part, uint32_t nparts, const uint32_t* count,
                            uint32_t cap, float* grads, bool step, const GuideAdam& adam, const GuideTrainD& t,
                            float* host_loss, cudaStream_t st) {
    chain(k_guide_update_tc, (kGuideParams + kReduceParams) / kReduceParams, 32 * kReduceWarps, 0, st, g, part, nparts,
          count, cap, grads, step ? 1 : 0, adam, t, host_loss);
}

}  // namespace dev
}  // namespace rgr
