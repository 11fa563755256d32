// wavefront.cu — the per-bounce kernels of the wavefront path tracer (sm_103a).
//
// One reference step() (common/wavefront_path_tracing.hpp:591-939) is about
// twenty launches of 2^22 work items.  Here a bounce by itself is:
//   1. compact_new  — ordered compaction of the slots logic marked "new path"
//      (slot order, so pixels are assigned exactly as a sequential run of
//      new_path.cl:41-43 over that queue would);
//   2. shade        — persistent kernel draining the new-path queue and the six
//      material queues back to back; per item it runs, in the reference stage
//      order, new_path / strategy_selection / envmap sample / BSDF sample or
//      pdf / envmap pdf / material stage / homogeneous_volume_through, keeping
//      IncidentSample and ShadingResult in registers;
//   3. trace_paths  — the closest hits, by persistent refilling warps (large pools);
//   4. trace_logic  — logic.cl (after casting the rays itself in small pools):
//      throughput update, envmap on miss, Russian roulette, FP64 per-pixel
//      accumulation, and the appends to the next step's material queues, aggregated
//      per warp (match_any) and per block (shared-memory counts, one global atomic
//      per queue per block).
// Inside a run of several bounces the logic is not a pass of its own: the cast
// finds where each path goes next, k_classify builds the queues from a byte per
// slot, k_new_paths finishes the ended paths and starts the new ones, k_shade_inner
// does the logic's share of the others (launch_inner_queues in wavefront.cuh).  At 2^24 paths of
// the mixed 1080p render a bounce was 1.15 ms shading, 2.25 cast and 1.15 logic; it is
// 0.06 classification, 0.48 new paths, 0.81 shading and 2.3 cast: 91.5 to 73.3 ms.
// Every slot's arithmetic is the reference kernels' arithmetic (see the
// file:line notes); the translation unit is built with --fmad=false.
#include <cuda_fp16.h>

#include <algorithm>

#include "wavefront.cuh"
#include "traverse.cuh"
#include "guide.cuh"

namespace rgr {
namespace dev {
namespace {

using namespace rgr::fm;

constexpr float kPiF = 3.14159274f;                 // (float)(M_PI)
constexpr float kPdfUniformSphere = 0.0795774683f;  // (float)(1.0 / (M_PI * 4.0))
constexpr float kFourPiF = 12.566371f;              // (float)(4.0 * M_PI)
constexpr double kPiD = 3.14159265358979323846;     // M_PI
constexpr float kFltMax = 3.40282347e+38f;

enum { kBxdf = 0, kEnv = 1, kNone = 2, kGuide = 3 };

RGR_DEV f3 mix3(f3 a, f3 b, float t) { return mk(mix_(a.x, b.x, t), mix_(a.y, b.y, t), mix_(a.z, b.z, t)); }
RGR_DEV float sqr(float x) { return x * x; }
RGR_DEV int to_int(float x) {
    if (isnan(x)) return 0;
    if (x >= 2147483648.0f) return 2147483647;
    if (x <= -2147483648.0f) return (-2147483647 - 1);
    return (int)x;
}

// ------------------------------------------------------------ envmap
// cartesian_to_polar (envmap_sampling.cl:25-34)
RGR_DEV void cartesian_to_polar(f3 rd, float& theta, float& phi) {
    float z = rd.y, x = rd.z, y = rd.x;
    theta = atan2_(sqrtf(x * x + y * y), z);
    phi = atan2_(y, x);
    if (!is_finite(phi)) phi = 0.0f;
}
// envmap_index (envmap_sampling.cl:75-95)
RGR_DEV int envmap_index(f3 wi, int width, int height) {
    float theta, phi;
    cartesian_to_polar(wi, theta, phi);
    float u = 1.0f - phi / (2.0f * kPiF);
    float v = theta / kPiF;
    int ix = to_int(floorf(u * (float)width));
    int iy = to_int(floorf(v * (float)height));
    int r = ix % width;
    ix = r < 0 ? r + width : r;
    iy = min(max(iy, 0), height - 1);
    return iy * width + ix;
}
RGR_DEV f3 texel(const SceneView& sc, int i, int j) { return xyz(__ldg(sc.env_rgba + (size_t)j * sc.env_w + i)); }
// get_envmap_value (envmap_sampling.cl:36-52): read_imagef with normalized
// coordinates, CLK_ADDRESS_REPEAT, nearest or bilinear (OpenCL 1.2 sampler
// formulas, FP32 weights)
RGR_DEV f3 envmap_value(const SceneView& sc, f3 rd, bool linear) {
    float theta, phi;
    cartesian_to_polar(rd, theta, phi);
    float su = 1.0f - phi / (2.0f * kPiF);
    float sv = theta / kPiF;
    const int w = sc.env_w, h = sc.env_h;
    float u = (su - floorf(su)) * (float)w;
    float v = (sv - floorf(sv)) * (float)h;
    if (!linear) {
        int i = to_int(floorf(u)), j = to_int(floorf(v));
        if (i > w - 1) i = i - w;
        if (j > h - 1) j = j - h;
        i = min(max(i, 0), w - 1);
        j = min(max(j, 0), h - 1);
        return texel(sc, i, j);
    }
    float uu = u - 0.5f, vv = v - 0.5f;
    int i0 = to_int(floorf(uu)), j0 = to_int(floorf(vv));
    int i1 = i0 + 1, j1 = j0 + 1;
    if (i0 < 0) i0 = w + i0;
    if (i1 > w - 1) i1 = i1 - w;
    if (j0 < 0) j0 = h + j0;
    if (j1 > h - 1) j1 = j1 - h;
    i0 = min(max(i0, 0), w - 1);
    i1 = min(max(i1, 0), w - 1);
    j0 = min(max(j0, 0), h - 1);
    j1 = min(max(j1, 0), h - 1);
    float a = uu - floorf(uu), b = vv - floorf(vv);
    float w00 = (1.0f - a) * (1.0f - b), w10 = a * (1.0f - b);
    float w01 = (1.0f - a) * b, w11 = a * b;
    return ((texel(sc, i0, j0) * w00 + texel(sc, i1, j0) * w10) + texel(sc, i0, j1) * w01) + texel(sc, i1, j1) * w11;
}
// alias_method (envmap_sampling.cl:54-66); table t of 7
RGR_DEV uint32_t alias_method(const SceneView& sc, size_t base, Rng& st, uint32_t count) {
    uint32_t idx = (uint32_t)(st.uniform_integer() % (uint64_t)count);
    int2 b = __ldg(sc.env_alias + base + idx);
    if (b.y < 0) return idx;
    float u = st.uniform();
    if (u < __int_as_float(b.x)) return idx;
    return (uint32_t)b.y;
}
// sample_from_fragment (envmap_sampling.cl:68-73, 158-167)
RGR_DEV f3 sample_from_fragment(const SceneView& sc, uint32_t idx, Rng& st) {
    float4 fr = __ldg(sc.env_frag + idx);
    float y = mix_(fr.x, fr.y, st.uniform());
    float phi = mix_(fr.z, fr.w, st.uniform());
    float sp, cp;
    sincos_(phi, &sp, &cp);
    f3 p = mk(sp, y, cp);
    float r_xz = sqrtf(fmax_(1.0f - p.y * p.y, 0.0f));
    p.x *= r_xz;
    p.z *= r_xz;
    return p;
}
RGR_DEV void six_axis_bases(size_t count, f3 n, size_t& xb, size_t& yb, size_t& zb) {
    xb = count * (0.0f < n.x ? 1 : 2);
    yb = count * (0.0f < n.y ? 3 : 4);
    zb = count * (0.0f < n.z ? 5 : 6);
}

// ------------------------------------------------------------ BSDFs
// cosine_weighted_hemisphere_z_up (lambertian.cl:9-20)
RGR_DEV f3 cosine_hemisphere(float a, float b) {
    float r = sqrtf(a);
    float theta = (float)((double)b * kPiD * 2.0);
    float s, c;
    sincos_(theta, &s, &c);
    return mk(r * c, r * s, sqrtf(fmax_(1.0f - a, 0.0f)));
}
// get_orthonormal_basis (lambertian.cl:26-32)
RGR_DEV void orthonormal_basis(f3 z, f3& xa, f3& ya) {
    const float sign = copysign_(1.0f, z.z);
    const float a = -1.0f / (sign + z.z);
    const float b = z.x * z.y * a;
    xa = mk(1.0f + sign * z.x * z.x * a, sign * b, -sign * z.x);
    ya = mk(b, sign + z.y * z.y * a, -z.y);
}
RGR_DEV f3 reflect(f3 d, f3 n) { return d - (2.0f * dot(d, n)) * n; }
// sample_ward (ward.cl:40-53)
RGR_DEV f3 sample_ward(f3 wo, f3 zaxis, float alpha, float u0, float u1) {
    float phiH = u0 * 2.0f * kPiF;
    float thetaH = atan_(alpha * sqrtf(-log_(u1)));
    float st, ct, sp, cp;
    sincos_(thetaH, &st, &ct);
    sincos_(phiH, &sp, &cp);
    f3 hl = mk(st * cp, st * sp, ct);
    f3 xa, ya;
    orthonormal_basis(zaxis, xa, ya);
    f3 h = xa * hl.x + ya * hl.y + zaxis * hl.z;
    return reflect(-wo, h);
}
// pdf_ward (ward.cl:55-74)
RGR_DEV float pdf_ward(f3 wo, f3 wi, f3 zaxis, float alpha) {
    if (dot(wo, zaxis) * dot(wi, zaxis) < 0.0f) return 0.0f;
    const float alpha2 = sqr(alpha);
    f3 h = normalize(wi + wo);
    float c = dot(h, zaxis);
    float c2 = sqr(c);
    float tan2 = (1.0f - c2) / c2;
    float k0 = 1.0f / (4.0f * kPiF * alpha2 * dot(h, wi) * (c * c * c));
    float k1 = exp_(-tan2 / alpha2);
    return k0 * k1;
}
// fresnel_dielectrics, refract (delta_materials.cl:11-32)
RGR_DEV float fresnel_dielectrics(float c, float eta_t, float eta_i) {
    float g = sqrtf(eta_t * eta_t / sqr(eta_i) - 1.0f + sqr(c));
    float a = 0.5f * sqr(g - c) / sqr(g + c);
    float b = 1.0f + sqr(c * (g + c) - 1.0f) / sqr(c * (g - c) + 1.0f);
    return a * b;
}
RGR_DEV bool refract(f3& out, f3 d, f3 n, float eta_i, float eta_t) {
    float eta = eta_i / eta_t;
    float NoD = dot(n, d);
    float k = 1.0f - eta * eta * (1.0f - NoD * NoD);
    if (k <= 0.0f) return false;
    out = eta * d - (eta * NoD + sqrtf(k)) * n;
    return true;
}
// uniform_on_unit_sphere (homogeneous_volume.cl:7-14)
RGR_DEV f3 uniform_sphere(float u0, float u1) {
    float phi = (float)((double)u0 * kPiD * 2.0);
    float z = mix_(-1.0f, 1.0f, u1);
    float r_xy = sqrtf(fmax_(1.0f - z * z, 0.0f));
    float s, c;
    sincos_(phi, &s, &c);
    return mk(r_xy * c, r_xy * s, z);
}
RGR_DEV uint32_t volume_hash(float4 v) {  // types.cl:104-106 (C, R.x, R.y, R.z)
    return __float_as_uint(v.w) ^ __float_as_uint(v.x) ^ __float_as_uint(v.y) ^ __float_as_uint(v.z);
}

// sel0/pdf0: BSDF (or phase function), sel1/pdf1: envmap, sel2/pdf2: the
// learned guide (guided renders only)
struct Incident {
    f3 wi;
    float sel0, sel1, pdf0, pdf1, sel2, pdf2;
    int strategy;
};
template <bool kGuided>
RGR_DEV float incident_pdf(const Incident& is) {  // types.cl:65-71
    float pdf = 0.0f;
    pdf = pdf + is.sel0 * is.pdf0;
    pdf = pdf + is.sel1 * is.pdf1;
    if (kGuided) pdf = pdf + is.sel2 * is.pdf2;
    return pdf;
}

// A slot's path state in registers, as the shading stages see it.
struct SlotState {
    f3 ro, rd, T, L, Ng;
    float tmin;
    int32_t hv, hs;      // volume hit (negative: none), surface hit
    uint32_t pixel;
    uint32_t logic_i;    // segments so far
    int vcount;          // volumes the path is inside; their ids in va, vb.xyz
    int4 va, vb;
    Rng rng;
};

// One slot's share of a step, from new_path to homogeneous_volume_through, on
// its state in registers.  k: the queue the slot came from (0 = new path, else
// its material type); a new path replaces everything but the RNG state and the
// volume list and reads the ended path's volume hit.
// Guided renders: gi is the slot's index among this bounce's guided items
// (its mixture in gd.lobes), ~0u when the vertex is not guided.
// Returns whether the stage changed L.
template <bool kGuided>
RGR_DEV bool shade_state(const RequestD& rq, int k, uint32_t slot, unsigned long long gpix, const GuideRenderD& gd,
                         uint32_t gi, SlotState& st) {
    const SceneView& sc = rq.sc;
    const bool fresh = k == 0;
    f3 &ro = st.ro, &rd = st.rd, &T = st.T, &L = st.L, &Ng = st.Ng;
    float& tmin = st.tmin;
    int32_t &hv = st.hv, &hs = st.hs;
    int& vcount = st.vcount;
    int4 &va = st.va, &vb = st.vb;
    Rng& rng = st.rng;

    if (k == 0) {  // new_path (new_path.cl:17-83)
        const CameraD& cam = rq.cam;
        T = mk(1, 1, 1);
        L = mk(0, 0, 0);
        st.logic_i = 0;
        uint32_t npix = cam.w * cam.h;
        const uint32_t pixel = (uint32_t)(gpix % (unsigned long long)npix);
        st.pixel = pixel;
        uint32_t x = pixel % cam.w, y = pixel / cam.w;
        float ux = rng.uniform();
        float uy = rng.uniform();
        f3 sop = mk(cam.o[0], cam.o[1], cam.o[2]) + mk(cam.r[0], cam.r[1], cam.r[2]) * ((float)x + ux) +
                 mk(cam.b[0], cam.b[1], cam.b[2]) * ((float)y + uy);
        float u0 = rng.uniform();
        float u1 = rng.uniform();
        float r = sqrtf(u0);
        float theta = (float)((double)u1 * kPiD * 2.0);
        float s, c;
        sincos_(theta, &s, &c);
        float lensx = rq.dof * r * c;
        float lensy = rq.dof * r * s;
        f3 lens = mk(cam.eye[0], cam.eye[1], cam.eye[2]) + mk(cam.up[0], cam.up[1], cam.up[2]) * lensx +
                  mk(cam.right[0], cam.right[1], cam.right[2]) * lensy;
        ro = lens;
        rd = normalize(sop - lens);
        vcount = 0;
        hs = -1;
        tmin = kFltMax;
        Ng = mk(0, 0, 0);
        if (kGuided) gd.nrec[slot] = 0;
    }
    f3 shLe = mk(0, 0, 0), shT = mk(1, 1, 1);

    // strategy_selection (mixture_density.cl:7-133)
    Incident is;
    is.wi = mk(0, 0, 0);
    is.sel0 = is.sel1 = is.pdf0 = is.pdf1 = is.sel2 = is.pdf2 = 0.0f;
    is.strategy = kNone;
    const bool surface_hit = 0 <= hs, volume_hit = 0 <= hv;
    int envq = -1;
    if (surface_hit || volume_hit) {
        const float env_p = sc.has_env ? rq.env_p : 0.0f;
        if (surface_hit) {
            int mt = __ldg(sc.materials + hs).x;
            if (mt == kMatLambertian || mt == kMatWard) {
                const float bxdf_p = 1.0f - env_p;
                is.sel0 = bxdf_p;
                is.sel1 = 1.0f - bxdf_p;
            } else {
                is.sel0 = 1.0f;
                is.sel1 = 0.0f;
            }
        } else {
            const float bxdf_p = 1.0f - env_p;
            is.sel0 = bxdf_p;
            is.sel1 = 1.0f - bxdf_p;
        }
        if (kGuided && gi != ~0u) {
            // the guide takes its share of the non-envmap probability: the sum of the
            // record's stored weights (the network's selection output, or the fixed
            // fraction), decoded identically wherever the record is read
            is.sel2 = is.sel0 * mixture_alpha(gd.lobes + (size_t)kGuideMixVecs * gi);
            is.sel0 = is.sel0 - is.sel2;
        }
        float u = rng.uniform();
        if (kGuided) {
            is.strategy = (u <= is.sel0) ? kBxdf : ((u <= is.sel0 + is.sel2) ? kGuide : kEnv);
        } else {
            is.strategy = (u <= is.sel0) ? kBxdf : kEnv;
        }
        if (is.sel1 != 0.0f) {
            const int sq = volume_hit ? 0 : 2, eq = volume_hit ? 1 : 3;
            envq = is.strategy == kEnv ? sq : eq;
        }
    }
    const uint4* mix = (kGuided && gi != ~0u) ? gd.lobes + (size_t)kGuideMixVecs * gi : nullptr;
    if (kGuided && gi != ~0u && is.strategy == kGuide) {
        const float u0 = rng.uniform();
        const float u1 = rng.uniform();
        const float u2 = rng.uniform();
        float d[3];
        mixture_sample(mix, u0, u1, u2, d);
        is.wi = mk(d[0], d[1], d[2]);
    }
    const size_t count = (size_t)sc.env_w * sc.env_h;
    // sample_envmap_6axis_stage / sample_envmap_stage (envmap_sampling.cl:169-248)
    if (envq == 2) {
        f3 n = Ng;
        if (dot(n, -rd) < 0.0f) n = -n;
        size_t xb, yb, zb;
        six_axis_bases(count, n, xb, yb, zb);
        float u = rng.uniform();
        f3 ap = n * n;
        size_t sel = (u < ap.x) ? xb : ((u < ap.x + ap.y) ? yb : zb);
        uint32_t idx = alias_method(sc, sel, rng, (uint32_t)count);
        float pdf = 0.0f;
        pdf = pdf + ap.x * __ldg(sc.env_pdf + xb + idx);
        pdf = pdf + ap.y * __ldg(sc.env_pdf + yb + idx);
        pdf = pdf + ap.z * __ldg(sc.env_pdf + zb + idx);
        is.wi = sample_from_fragment(sc, idx, rng);
        is.pdf1 = pdf;
    } else if (envq == 0) {
        uint32_t idx = alias_method(sc, 0, rng, (uint32_t)count);
        float pdf = __ldg(sc.env_pdf + idx);
        is.wi = sample_from_fragment(sc, idx, rng);
        is.pdf1 = pdf;
    }
    // BSDF sample or pdf
    int2 mref = make_int2(0, 0);
    if (k >= 1 && k <= 5) mref = __ldg(sc.materials + hs);
    if (k == kMatLambertian) {  // sample_or_eval_lambertian_stage (lambertian.cl:34-71)
        float cosTheta;
        f3 ns = Ng;  // the raw Ng, as the reference samples, unless two-sided sampling is on
        if ((kGuided || (rq.flags & kFlagTwoSidedLambertian)) && dot(ns, -rd) < 0.0f) ns = -ns;
        if (is.strategy == kBxdf) {
            float u0 = rng.uniform();
            float u1 = rng.uniform();
            f3 wl = cosine_hemisphere(u0, u1);
            f3 xa, ya;
            orthonormal_basis(ns, xa, ya);
            is.wi = xa * wl.x + ya * wl.y + ns * wl.z;
            cosTheta = wl.z;
        } else {
            cosTheta = dot(ns, is.wi);
        }
        is.pdf0 = fmax_(cosTheta, 0.0f) / kPiF;
    } else if (k == kMatWard) {  // sample_or_eval_ward_stage (ward.cl:76-117)
        float4 w0 = __ldg(sc.wards + 3 * (size_t)mref.y);
        f3 wo = -rd;
        f3 n = Ng;
        if (dot(n, wo) < 0.0f) n = -n;
        f3 wi;
        if (is.strategy == kBxdf) {
            float u0 = rng.uniform();
            float u1 = rng.uniform();
            wi = sample_ward(wo, n, w0.x, u0, u1);
        } else {
            wi = is.wi;
        }
        is.wi = wi;
        is.pdf0 = pdf_ward(wo, wi, n, w0.x);
    } else if (k == kMatVolumeInside) {  // homogeneous_volume.cl:66-88
        if (is.strategy == kBxdf) {
            float u0 = rng.uniform();
            float u1 = rng.uniform();
            is.wi = uniform_sphere(u0, u1);
        }
        is.pdf0 = kPdfUniformSphere;
    }
    // evaluate_envmap_6axis_pdf_stage / evaluate_envmap_pdf_stage (envmap_sampling.cl:250-281)
    if (envq == 3) {
        size_t xb, yb, zb;
        f3 n = Ng;  // the raw Ng, as the reference does, unless the backside fix is on
        if ((kGuided || (rq.flags & kFlagFixBacksideEnvPdf)) && dot(n, -rd) < 0.0f) n = -n;
        six_axis_bases(count, n, xb, yb, zb);
        f3 ap = n * n;
        int index = envmap_index(is.wi, sc.env_w, sc.env_h);
        float pdf = 0.0f;
        pdf = pdf + ap.x * __ldg(sc.env_pdf + xb + index);
        pdf = pdf + ap.y * __ldg(sc.env_pdf + yb + index);
        pdf = pdf + ap.z * __ldg(sc.env_pdf + zb + index);
        is.pdf1 = pdf;
    } else if (envq == 1) {
        is.pdf1 = __ldg(sc.env_pdf + envmap_index(is.wi, sc.env_w, sc.env_h));
    }
    if (kGuided && is.sel2 != 0.0f) is.pdf2 = mixture_pdf(mix, is.wi.x, is.wi.y, is.wi.z);
    // the guided vertex as the network saw it (before the stage moves ro)
    f3 gx = mk(0, 0, 0), gn = mk(0, 0, 0);
    if (kGuided && is.sel2 != 0.0f) {
        gx = ro + rd * tmin;
        if (hs >= 0) {
            gn = Ng;
            if (dot(gn, -rd) < 0.0f) gn = -gn;
        }
    }
    const f3 wo_in = -rd;
    // material stages
    if (k == kMatLambertian) {  // lambertian_stage (lambertian.cl:73-123)
        float4 le = __ldg(sc.lambertians + 2 * (size_t)mref.y), R = __ldg(sc.lambertians + 2 * (size_t)mref.y + 1);
        f3 n = Ng;
        if (dot(n, -rd) < 0.0f) n = -n;
        f3 wi = is.wi;
        float pdf = incident_pdf<kGuided>(is);
        float cosTheta = dot(wi, n);
        f3 Ts = mk(0, 0, 0);
        if (0.0f < cosTheta) Ts = xyz(R) / kPiF * cosTheta / pdf;
        shLe = xyz(le);
        shT = Ts;
        ro = ro + rd * tmin + wi * 1.0e-5f + n * 1.0e-5f;
        rd = wi;
    } else if (k == kMatWard) {  // ward_stage (ward.cl:119-186)
        float4 w0 = __ldg(sc.wards + 3 * (size_t)mref.y);
        float4 refl = __ldg(sc.wards + 3 * (size_t)mref.y + 1), edge = __ldg(sc.wards + 3 * (size_t)mref.y + 2);
        f3 n = Ng;
        f3 wo = -rd;
        if (dot(n, wo) < 0.0f) n = -n;
        f3 wi = is.wi;
        float pdf = incident_pdf<kGuided>(is);
        float cosTheta = dot(wi, n);
        f3 Ts = mk(0, 0, 0);
        if (0.0f < cosTheta) {
            f3 lv = wi + wo;
            f3 h = normalize(lv);
            float alpha2 = sqr(w0.x);
            float cth = dot(h, n);
            float cth2 = sqr(cth);
            float tan2 = (1.0f - cth2) / cth2;
            float mu = dot(h, wi);
            f3 rho = mix3(xyz(refl), xyz(edge), pow_(1.0f - mu, 1.0f / w0.y));
            f3 k0 = rho / (kPiF * alpha2);
            float k1 = exp_(-tan2 / alpha2);
            float dn = dot(lv, n);
            float k2 = dot(lv, lv) / sqr(sqr(dn));
            Ts = k0 * k1 * k2 * cosTheta / pdf;
        }
        shT = Ts;
        ro = ro + rd * tmin + wi * 1.0e-5f + n * 1.0e-5f;
        rd = wi;
    } else if (k == kMatVolume) {  // homogeneous_volume_stage (homogeneous_volume.cl:19-64)
        bool backside = dot(Ng, -rd) < 0.0f;
        int vols[8] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z, 0};
        if (backside) {  // inVolumeList_Remove (types.cl:115-132)
            uint32_t hsh = volume_hash(__ldg(sc.volumes + mref.y));
            bool move = false;
#pragma unroll
            for (int i = 0; i < 7; ++i) {  // constant indices keep the list in registers
                if (i < vcount) {
                    if (move) {
                        if (i > 0) vols[i - 1] = vols[i];
                    } else {
                        int2 mi = __ldg(sc.materials + vols[i]);
                        if (volume_hash(__ldg(sc.volumes + mi.y)) == hsh) move = true;
                    }
                }
            }
            if (move) vcount--;
        } else if (vcount < 7) {  // inVolumeList_Add (types.cl:108-114)
#pragma unroll
            for (int i = 0; i < 7; ++i)
                if (i == vcount) vols[i] = hs;
            vcount++;
        }
        va = make_int4(vols[0], vols[1], vols[2], vols[3]);
        vb = make_int4(vols[4], vols[5], vols[6], 0);
        ro = ro + rd * (tmin + 1.0e-5f);
    } else if (k == kMatVolumeInside) {  // homogeneous_volume_inside_stage (homogeneous_volume.cl:90-129)
        int2 mi = __ldg(sc.materials + hv);
        float4 vol = __ldg(sc.volumes + mi.y);
        float pdf = incident_pdf<kGuided>(is);
        shT = xyz(vol) / kFourPiF / pdf;
        ro = ro + rd * tmin;
        rd = is.wi;
    } else if (k == kMatSpecular) {  // delta_materials.cl:34-64
        f3 n = Ng;
        if (dot(n, -rd) < 0.0f) n = -n;
        f3 wi = reflect(rd, n);
        ro = ro + rd * tmin + wi * 1.0e-5f;
        rd = wi;
    } else if (k == kMatDielectric) {  // delta_materials.cl:66-121
        f3 n = Ng;
        f3 wo = -rd;
        bool backside = dot(n, wo) < 0.0f;
        float eta_i = 1.0f, eta_t = 1.5f;
        if (backside) {
            float e = eta_i;
            eta_i = eta_t;
            eta_t = e;
            n = -n;
        }
        float f = fresnel_dielectrics(fabs_(dot(n, wo)), eta_t, eta_i);
        float u = rng.uniform();
        float rc = 1.0f;
        f3 wi;
        if (u < f) {
            wi = reflect(rd, n);
        } else if (!refract(wi, rd, n, eta_i, eta_t)) {
            wi = reflect(rd, n);
        } else {
            rc = sqr(eta_t / eta_i);
        }
        shT = mk(rc, rc, rc);
        ro = ro + rd * tmin + wi * 1.0e-5f;
        rd = wi;
    }
    // logic.cl:31-33, applied here: the stage that made the shading result consumes it.
    // L + T * shLe leaves L's bits unchanged when shLe is zero and T finite (L is
    // never -0), so L counts as changed only otherwise, for new paths and in
    // guided renders (the training records carry it).
    const bool touch_L = fresh || kGuided || shLe.x != 0.0f || shLe.y != 0.0f || shLe.z != 0.0f ||
                         !is_finite(T.x) || !is_finite(T.y) || !is_finite(T.z);
    L = L + T * shLe;
    T = T * shT;
    if (kGuided && is.sel2 != 0.0f && gd.record && guide_training_open(gd.train)) {
        // training record: the vertex, the sampled direction, the path's (L, T) just
        // after this vertex, so that the logic can recover the radiance L_i that
        // arrived along wi when the path ends, and cos / pdf of the sample
        const uint32_t r = gd.nrec[slot];
        if (r < (uint32_t)kGuideRecords) {
            const float c = (hs >= 0) ? fmax_(dot(is.wi, gn), 0.0f) : 1.0f;
            const float cp = c / incident_pdf<kGuided>(is);
            float4* rec = gd.records + ((size_t)slot * kGuideRecords + r) * kGuideRecordVecs;
            st_v8(rec, make_float4(L.x, L.y, L.z, T.x),
                  make_float4(T.y, T.z, cp, is.pdf0));  // pdf0: the BSDF (phase) pdf of wi
            st_v8(rec + 2, make_float4(gx.x, gx.y, gx.z, gn.x), make_float4(gn.y, gn.z, wo_in.x, wo_in.y));
            st_v8(rec + 4, make_float4(wo_in.z, is.wi.x, is.wi.y, is.wi.z), make_float4(0.0f, 0.0f, 0.0f, 0.0f));
            gd.nrec[slot] = (uint8_t)(r + 1);
        }
    }

    // homogeneous_volume_through (homogeneous_volume_through.cl:7-44)
    hs = -1;
    hv = -1;
    if (0 < vcount) {
        uint64_t u = rng.uniform_integer();
        int sel = (int)(u % (uint64_t)vcount);
        const int vols[7] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z};
        hv = pick(vols, sel < 7 ? sel : 6);
    }
    tmin = kFltMax;
    if (0 <= hv) {
        int2 mi = __ldg(sc.materials + hv);
        float4 vol = __ldg(sc.volumes + mi.y);
        float u = rng.uniform();
        tmin = -1.0f / vol.w * log_(u);
    }
    return touch_L;
}

// What the logic does to a path that goes on (logic.cl:27-190): the Russian
// roulette's draw and T / cp (exactly T where the roulette is off: cp is 1).
RGR_DEV void logic_advance(const RequestD& rq, uint32_t logic_i, f3& T, Rng& rng) {
    float cp = 1.0f;
    if ((long long)rq.rr_depth < (long long)logic_i) cp = fmin_(0.2126f * T.x + 0.7152f * T.y + 0.0722f * T.z, 1.0f);
    rng.uniform();
    T = T / cp;
}

// Whether the logic ends a path whatever its ray meets: Russian roulette, a black
// throughput, or the depth limit (logic_decide without the miss).
RGR_DEV bool logic_ends(const RequestD& rq, const PathsView& P, uint32_t slot, f3 T, uint32_t logic_i) {
    const float lum = 0.2126f * T.x + 0.7152f * T.y + 0.0722f * T.z;
    bool ends = lum < 1.0e-5f || (rq.max_depth > 0 && (long long)logic_i >= (long long)rq.max_depth);
    if ((long long)rq.rr_depth < (long long)logic_i) {
        Rng rng = rng_load(P.rng, slot);
        ends = ends || !(rng.uniform() < fmin_(lum, 1.0f));
    }
    return ends;
}

// The volume list of a slot (its record's last sector).
RGR_DEV void load_volumes(const PathsView& P, uint32_t slot, SlotState& st) {
    float4 a, b;
    ld_sector<3>(P, slot, a, b);
    st.va = make_int4(__float_as_int(a.x), __float_as_int(a.y), __float_as_int(a.z), __float_as_int(a.w));
    st.vb = make_int4(__float_as_int(b.x), __float_as_int(b.y), __float_as_int(b.z), __float_as_int(b.w));
}
RGR_DEV void store_volumes(const PathsView& P, uint32_t slot, const SlotState& st) {
    const int4 va = st.va, vb = st.vb;
    st_sector<3>(P, slot,
                 make_float4(__int_as_float(va.x), __int_as_float(va.y), __int_as_float(va.z), __int_as_float(va.w)),
                 make_float4(__int_as_float(vb.x), __int_as_float(vb.y), __int_as_float(vb.z),
                             __int_as_float(st.vcount)));
}

// shade_state on a slot's record in memory.  kInner: the bounce before was a bounce
// inside a run, whose logic left the state of a path that goes on as the trace
// kernel did: its share (the hit, the draw, T / cp, the segment count) comes first.
template <bool kGuided, bool kInner = false>
RGR_DEV void shade_slot(const RequestD& rq, const PathsView& P, int k, uint32_t slot, unsigned long long gpix,
                        const GuideRenderD& gd, uint32_t gi) {
    // Path state moves by 32-byte sector of the slot record and only where this
    // item uses it (a material queue is a sparse subset of the slots, so each
    // sector touched costs a DRAM sector): a new path (k = 0) replaces everything
    // but its RNG state and the volume hit of the ended path, so it skips the
    // (T, L) sector and the volume list; L is stored only when the stage changes
    // it; the first half of the volume list is loaded only when the list is used.
    const bool fresh = k == 0;
    float4 ro4, rd4, ng4, rng4, T4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f), L4 = T4;
    SlotState st;
    st.va = make_int4(0, 0, 0, 0), st.vb = st.va;
    // the ray's sector and the (ng, rng) sector, each in one access; (T, L) likewise
    ld_sector<0>(P, slot, ro4, rd4);
    ld_sector<2>(P, slot, ng4, rng4);
    st.vcount = 0;
    if (!fresh) {
        ld_sector<1>(P, slot, T4, L4);
        st.vcount = vcount_of(__float_as_uint(L4.w));
        if (k == kMatVolume || st.vcount > 0) load_volumes(P, slot, st);
    } else {
        ro4 = ng4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    }
    st.rng = rng_of_bits(rng4);
    st.ro = xyz(ro4), st.rd = xyz(rd4), st.T = xyz(T4), st.L = xyz(L4), st.Ng = xyz(ng4);
    st.tmin = ro4.w;
    st.hv = __float_as_int(rd4.w);
    st.hs = __float_as_int(ng4.w);
    st.pixel = __float_as_uint(T4.w);
    st.logic_i = depth_of(__float_as_uint(L4.w));
    if (kInner) {
        int mtype;
        resolve_hit(rq.sc, ro4, rd4, st.hv, st.hs, ng4, mtype);
        st.Ng = xyz(ng4);
        logic_advance(rq, st.logic_i, st.T, st.rng);
        st.logic_i += 1;
    }
    // the volume stage changes the volume count, which L.w carries
    const bool store_L = shade_state<kGuided>(rq, k, slot, gpix, gd, gi, st) || k == kMatVolume || kInner;
    st_sector<0>(P, slot, f4(st.ro, st.tmin), f4(st.rd, __int_as_float(st.hv)));
    if (store_L)  // a new path's count is 0; its list keeps the stale ids
        st_sector<1>(P, slot, f4(st.T, __uint_as_float(st.pixel)),
                     f4(st.L, __uint_as_float(depth_word(st.logic_i, st.vcount))));
    else  // the sector was read above: this half store finds it in L2
        P.T[slot] = f4(st.T, __uint_as_float(st.pixel));
    if (k == kMatVolume) store_volumes(P, slot, st);
    st_sector<2>(P, slot, f4(st.Ng, __int_as_float(st.hs)), rng_bits(st.rng));
}

// ------------------------------------------------------------ kernels
// The pool of a new render: its counters, error word and, of a render of one request
// (table set), the request table.  (As three memsets, a copy and a wait for it they were
// 25 of the 43 us that a render of 65,536 pixels took to begin.)
__global__ void k_init(PathsView P, QueueView Q, uint32_t seed_offset, InitView w, RequestD one) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < 8u) {
        Q.counts[i] = Q.taken[i] = 0u;
        w.scalars[i] = 0ull;
        if (i < 4u) w.err[i] = 0u;
        if (i < 2u && w.done) w.done[i] = 0ull;
        if (i == 0u && w.table) *w.table = one;
    }
    if (i < Q.ntiles) {
        uint32_t beg = i * kTile;
        Q.tile_new[i] = min(kTile, P.n - beg);
    }
    if (i >= Q.ntiles * kTile) return;
    if (i >= P.n) {
        P.qid[i] = kQueueIdle;  // padding up to a whole tile
        return;
    }
    // random_initialize (peseudo_random.cl:48-64)
    unsigned long long x = (unsigned long long)seed_offset + i;
    unsigned long long r[2];
    for (int k = 0; k < 2; ++k) {
        unsigned long long z = (x += 0x9e3779b97f4a7c15ull);
        z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
        z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
        r[k] = z ^ (z >> 31);
    }
    uint4 s = make_uint4((uint32_t)r[0], (uint32_t)(r[0] >> 32), (uint32_t)r[1], (uint32_t)(r[1] >> 32));
    if ((s.x | s.y | s.z | s.w) == 0u) s.x = 1u;
    const float4 zero = make_float4(0, 0, 0, 0);
    st_sector<0>(P, i, make_float4(0, 0, 0, kFltMax), make_float4(0, 0, 0, __int_as_float(-1)));
    st_sector<1>(P, i, zero, zero);
    st_sector<2>(P, i, make_float4(0, 0, 0, __int_as_float(-1)), rng_bits(Rng{s.x, s.y, s.z, s.w}));
    st_sector<3>(P, i, zero, zero);
    P.qid[i] = 0;  // initialize_all_as_new_path (new_path.cl:9-15)
    P.req[i] = 0;
}

// Ordered compaction of new-path slots: block t owns slots [t*4096, (t+1)*4096).  The last
// block starts the bounce: it takes the queues' counts for the kernels up to the cast, and
// clears them for the logic, and the cast's counter; the shading kernel clears the tile
// counts.  Two memsets between a small pool's kernels cost 5 to 10 % of its renders: at 2^15 /
// 2^17 / 2^18 paths 939 / 1283 / 1783 us with them and 884 / 1160 / 1705 without (36
// triangles), 1963 / 2596 / 3400 and 1838 / 2460 / 3280 (5 K triangles).
__global__ void __launch_bounds__(256) k_compact_new(PathsView P, QueueView Q, unsigned long long* cast_counter) {
    follow();
    __shared__ uint32_t s_warp[8];
    __shared__ uint32_t s_prefix;
    const uint32_t t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // prefix of the tile counts before this tile
    uint32_t sum = 0;
    for (uint32_t j = tid; j < t; j += 256) sum += Q.tile_new[j];
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    if (lane == 0) s_warp[warp] = sum;
    __syncthreads();
    if (tid == 0) {
        uint32_t p = 0;
        for (int w = 0; w < 8; ++w) p += s_warp[w];
        s_prefix = p;
    }
    __syncthreads();
    const uint32_t prefix = s_prefix;
    // 16 consecutive slots per thread
    const uint32_t base = t * kTile + tid * 16;
    uint4 q = *reinterpret_cast<const uint4*>(P.qid + base);
    uint32_t words[4] = {q.x, q.y, q.z, q.w};
    uint32_t mask = 0;
    for (int k = 0; k < 16; ++k) {
        uint32_t b = (words[k >> 2] >> (8 * (k & 3))) & 0xffu;
        if (b == 0u) mask |= 1u << k;
    }
    uint32_t c = __popc(mask);
    // block exclusive scan of c
    uint32_t inc = c;
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t v = __shfl_up_sync(0xffffffffu, inc, o);
        if (lane >= (uint32_t)o) inc += v;
    }
    __syncthreads();
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    uint32_t woff = 0, total = 0;
    for (int w = 0; w < 8; ++w) {
        uint32_t v = s_warp[w];
        if (w < (int)warp) woff += v;
        total += v;
    }
    uint32_t pos = prefix + woff + inc - c;
    uint32_t* out = Q.items[0];
    while (mask) {
        int k = __ffs(mask) - 1;
        mask &= mask - 1;
        out[pos++] = base + k;
    }
    if (t == Q.ntiles - 1 && tid == 0) {
        uint32_t all = prefix + total;
        Q.counts[0] = Q.taken[0] = all;
#pragma unroll
        for (int k = 1; k < kNumQueues; ++k) {
            Q.taken[k] = Q.counts[k];
            Q.counts[k] = 0u;
        }
        *cast_counter = 0ull;
        unsigned long long np = *Q.next_pixel;
        *Q.step_base = np;
        *Q.next_pixel = np + all;  // finalize_new_path (new_path.cl:85-88)
    }
}

template <bool kGuided>
__device__ __forceinline__ void shade_items(const PathsView& P, const QueueView& Q, const RenderParams& rp) {
    uint32_t off[kNumQueues + 1];
    off[0] = 0;
#pragma unroll
    for (int k = 0; k < kNumQueues; ++k) off[k + 1] = off[k] + Q.taken[k];
    const uint32_t total = off[kNumQueues];
    // guided items are numbered Lambertian, Ward, in-volume (as the inference kernel does)
    const uint32_t g4 = off[kMatLambertian + 1] - off[kMatLambertian];
    const uint32_t g6 = g4 + (off[kMatWard + 1] - off[kMatWard]);
    const unsigned long long base_pixel = *Q.step_base;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < Q.ntiles; i += stride) Q.tile_new[i] = 0u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        int k = 0;
#pragma unroll
        for (int j = 1; j < kNumQueues; ++j) k += (i >= off[j]) ? 1 : 0;
        const uint32_t slot = queue_items(Q, k)[i - pick(off, k)];
        unsigned long long gpix = 0;
        int r;
        if (k == 0) {
            gpix = base_pixel + (i - off[0]);
            if (rp.sample_limit != 0ull && gpix >= rp.sample_limit) {
                P.qid[slot] = kQueueIdle;  // sample budget reached: the slot retires
                continue;
            }
            // the request whose sample range holds this global sample index
            r = 0;
            while (r + 1 < rp.nreq && gpix >= rp.reqs[r].sample_end) ++r;
            P.req[slot] = (uint16_t)r;
            gpix -= rp.reqs[r].sample_begin;
        } else {
            r = P.req[slot];
        }
        uint32_t gi = ~0u;
        if (kGuided) {
            if (k == kMatLambertian) gi = i - off[kMatLambertian];
            else if (k == kMatWard) gi = g4 + (i - off[kMatWard]);
            else if (k == kMatVolumeInside && rp.gd.volumes) gi = g6 + (i - off[kMatVolumeInside]);
            if (gi != ~0u && rp.gd.max_depth) gi = rp.gd.remap[gi];  // its inference row, or unguided
        }
        shade_slot<kGuided>(rp.reqs[r], P, k, slot, gpix, rp.gd, gi);
    }
}

// The completion time of each request whose paths have all finished, stamped
// once by the bounce in which its last path ended (after that bounce's logic
// kernel, when its accumulation is complete).  The logic kernel only counts
// finished paths: an atomic with a returned value per warp, to find the last
// one, queued the warps on the requests' counters.  Requests i, i + stride, ...
RGR_DEV void stamp_done(const RenderParams& rp, int i, int stride) {
    for (int r = i; r < rp.nreq; r += stride) {
        const RequestD& q = rp.reqs[r];
        if (q.done == nullptr || *q.done_ns != 0ull || *q.done != q.sample_end - q.sample_begin) continue;
        unsigned long long t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
        *q.done_ns = t;
    }
}
__global__ void k_stamp_done(RenderParams rp) {
    follow();
    stamp_done(rp, blockIdx.x * blockDim.x + threadIdx.x, gridDim.x * blockDim.x);
}

// The plain and guided shading kernels: one queue item per thread, all
// queues in one launch, held to 4 resident 256-thread blocks per SM (64
// registers, a few spilled: the mixed 1080p render 1370 against 1347 Mpaths/s
// with the compiler's 78 registers and 3 blocks; the guided render 1.6 %
// faster than at 3 blocks and 80 registers).
#ifndef RGR_SHADE_MIN_BLOCKS
#define RGR_SHADE_MIN_BLOCKS 4
#endif
#ifndef RGR_SHADE_GUIDED_MIN_BLOCKS
#define RGR_SHADE_GUIDED_MIN_BLOCKS 4
#endif
__global__ void __launch_bounds__(256, RGR_SHADE_MIN_BLOCKS) k_shade(PathsView P, QueueView Q, RenderParams rp) {
    follow();
    shade_items<false>(P, Q, rp);
}
// the material queues of a bounce inside a run (k_new_paths has taken the new paths)
template <bool kGuided>
__global__ void __launch_bounds__(256, kGuided ? RGR_SHADE_GUIDED_MIN_BLOCKS : RGR_SHADE_MIN_BLOCKS)
    k_shade_inner(PathsView P, QueueView Q, RenderParams rp) {
    follow();
    // the ended paths of the bounce before are finished and counted
    if (blockIdx.x == 0) stamp_done(rp, (int)threadIdx.x, (int)blockDim.x);
    uint32_t off[kNumQueues];  // off[k]: the first item of queue k + 1
    off[0] = 0;
#pragma unroll
    for (int k = 1; k < kNumQueues; ++k) off[k] = off[k - 1] + Q.taken[k];
    const uint32_t total = off[kNumQueues - 1];
    // guided items are numbered as in shade_items
    const uint32_t g4 = off[kMatLambertian] - off[kMatLambertian - 1];
    const uint32_t g6 = g4 + (off[kMatWard] - off[kMatWard - 1]);
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < total; i += stride) {
        int k = 1;
#pragma unroll
        for (int j = 1; j < kNumQueues - 1; ++j) k += (i >= off[j]) ? 1 : 0;
        const uint32_t slot = queue_items(Q, k)[i - pick(off, k - 1)];
        uint32_t gi = ~0u;
        if (kGuided) {
            const uint32_t o = i - pick(off, k - 1);  // its place in the queue
            if (k == kMatLambertian) gi = o;
            else if (k == kMatWard) gi = g4 + o;
            else if (k == kMatVolumeInside && rp.gd.volumes) gi = g6 + o;
            if (gi != ~0u && rp.gd.max_depth) gi = rp.gd.remap[gi];  // its inference row, or unguided
        }
        shade_slot<kGuided, true>(rp.reqs[P.req[slot]], P, k, slot, 0ull, rp.gd, gi);
    }
}
__global__ void __launch_bounds__(256, RGR_SHADE_GUIDED_MIN_BLOCKS) k_shade_guided(PathsView P, QueueView Q,
                                                                                  RenderParams rp) {
    follow();
    shade_items<true>(P, Q, rp);
}

// Depth-limited guiding: the guided items whose vertex is among the first
// max_depth of its path (logic_i counts the path's segments so far) become
// the inference rows, appended with one atomic per warp; the others keep
// BSDF and envmap sampling.  The row order does not matter: a row's mixture
// depends on that row alone.  ahead: 1 inside a run, whose logic has not counted the last
// segment yet.
__global__ void __launch_bounds__(256) k_guide_select(PathsView P, QueueView Q, GuideRenderD gd, uint32_t ahead) {
    const uint32_t n = guided_items(Q, gd);
    const int lane = threadIdx.x & 31;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); base < n; base += stride) {
        const uint32_t gi = base + lane;
        uint32_t slot = 0;
        bool take = false;
        if (gi < n) {
            slot = guided_item_slot(Q, gi);
            take = depth_of(__float_as_uint(P.L[slot].w)) + ahead <= gd.max_depth;
        }
        const unsigned m = __ballot_sync(0xffffffffu, take);
        uint32_t first = 0;
        if (lane == 0 && m) first = atomicAdd(gd.nsel, (uint32_t)__popc(m));
        first = __shfl_sync(0xffffffffu, first, 0);
        if (gi < n) {
            const uint32_t row = first + (uint32_t)__popc(m & ((1u << lane) - 1u));
            gd.remap[gi] = take ? row : ~0u;
            if (take) gd.sel[row] = slot;
        }
    }
}

RGR_DEV uint32_t mix32(uint32_t h) {  // murmur3 finaliser
    h ^= h >> 16;
    h *= 0x85ebca6bu;
    h ^= h >> 13;
    h *= 0xc2b2ae35u;
    h ^= h >> 16;
    return h;
}

// A guided path ended with radiance L: its training records become samples.
// Record r holds the vertex, the sampled wi, the (L, T) of the path just after
// the vertex (its emission added, its throughput factor applied) and cos / pdf
// of wi, so the radiance that arrived along wi is L_i = (L_end - L_r) / T_r
// per channel, and the sample's weight in the KL loss is lum(L_i) cos / pdf:
// the guide learns the cosine-weighted incident radiance, which the MIS
// combines with the BSDF (the network does not see the material).
// Records are offered with the acceptance probability the last iteration set
// (a hash of slot, record and iteration, not the path's RNG, so rendering is
// unchanged) until `cap` samples are in.  guide_offer decides a lane's records;
// the logic kernel gathers the counts per block (one atomic for the block's
// samples, one for its offered count) and guide_write stores them.
struct GuideOffer {
    uint32_t take = 0;     // bit r: record r is accepted
    uint32_t offered = 0;  // records with a positive, finite weight
    float w[kGuideRecords] = {};
};
RGR_DEV void guide_offer(const GuideRenderD& gd, uint32_t slot, f3 L, bool ending, GuideOffer& o) {
    const GuideTrainD& tr = gd.train;
    const uint32_t nr = ending ? min((uint32_t)gd.nrec[slot], (uint32_t)kGuideRecords) : 0u;
    if (!nr) return;
    const float accept = *tr.accept;
    const uint32_t it = *tr.iter;
    for (uint32_t r = 0; r < (uint32_t)kGuideRecords; ++r) {
        if (r >= nr) continue;
        const float4* rec = gd.records + ((size_t)slot * kGuideRecords + r) * kGuideRecordVecs;
        float4 d, e;
        ld_v8(rec, d, e);
        const float lx = d.w > 0.0f ? (L.x - d.x) / d.w : 0.0f;
        const float ly = e.x > 0.0f ? (L.y - d.y) / e.x : 0.0f;
        const float lz = e.y > 0.0f ? (L.z - d.z) / e.y : 0.0f;
        const float wr = (0.2126f * lx + 0.7152f * ly + 0.0722f * lz) * e.z;
        if (!(wr > 0.0f) || !is_finite(wr)) continue;
        ++o.offered;
        const uint32_t h = mix32(slot * 0x9e3779b1u ^ (r + 1u) * 0x85ebca77u ^ (it + 1u) * 0xc2b2ae3du);
        if ((float)(h >> 8) * (1.0f / 16777216.0f) >= accept) continue;
        o.w[r] = wr;
        o.take |= 1u << r;
    }
}
// The accepted records of a lane as samples idx, idx + 1, ... (those below
// the cap); returns the sum of their weights.
RGR_DEV float guide_write(const GuideRenderD& gd, uint32_t slot, const GuideOffer& o, uint32_t idx) {
    const GuideTrainD& tr = gd.train;
    float wsum = 0.0f;
    for (uint32_t r = 0; r < (uint32_t)kGuideRecords; ++r) {
        if (!((o.take >> r) & 1u)) continue;
        if (idx < tr.cap) {
            const float4* rec = gd.records + ((size_t)slot * kGuideRecords + r) * kGuideRecordVecs;
            float4* dst = reinterpret_cast<float4*>(tr.samples + 16 * (size_t)idx);  // 64 bytes
            float4 x, n, wi, d;
            ld_v8(rec + 2, x, n);
            ld_v8(rec + 4, wi, d);
            st_v8(dst, x, n);                                                // x, n.x | n.yz, wo.xy
            st_v8(dst + 2, wi, make_float4(o.w[r], rec[1].w, 0.0f, 0.0f));  // wo.z, wi | weight, BSDF pdf of wi
            wsum += o.w[r];
        }
        ++idx;
    }
    return wsum;
}

// extension_ray_cast (extension_ray_cast_stackless.cl:202-246) of the slots
// this bounce shaded — the items of the seven queues, concatenated as the
// shading kernel reads them, less the new-path slots it retired — by
// persistent warps that hand finished lanes the next items (one atomic per
// refill per warp), as the closest-hit service kernel does with rays.  Runs
// after the shading kernel.  A hit writes the ray's sector once: t into P.ro.w and the primitive, as -2 - prim, into the volume-hit
// field P.rd.w (its readers take a negative id as none); the logic kernel computes
// Ng into P.ng.  A miss leaves P.ng.w at the -1 the shading stage wrote.  Each slot may belong
// to another request (scene).
// kInner: a bounce inside a run (launch_inner_queues).  The cast also decides where the path
// goes next and writes it as the slot's queue id: what ends a path whatever its ray
// meets (logic_ends) is found as the ray is taken, from the sector beside the
// ray's in the same line, and kept in the slot word's top bit (slots are below 2^28).
// kOne: a render of one request; its scene `one` is a kernel argument (constant bank).
// Read through the request table, a lane's node pointer was loaded again at every
// step (mixed 1080p render at 2^22 paths 24.35 ms, 23.85 with the argument).
#ifndef RGR_TRACE_PATHS_MIN_BLOCKS  // 4 / 5 / 6 (64 / 48 / 40 registers, 6 spilling): 1428 / 1473 / 1442 Mpaths/s
#define RGR_TRACE_PATHS_MIN_BLOCKS 5
#endif
// Scenes by request spill at 48 registers: eight requests 3483 us with 5 blocks, 3351 with 4.
template <bool kInner, bool kOne>
__global__ void __launch_bounds__(256, kOne ? RGR_TRACE_PATHS_MIN_BLOCKS : 4)
    k_trace_paths(PathsView P, QueueView Q, RenderParams rp, unsigned long long* next, int refill, int search,
                  SceneView one) {
    follow();
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const uint64_t pol = l2_evict_last_policy();
    uint32_t off[kNumQueues + 1];
    off[0] = 0;
#pragma unroll
    for (int k = 0; k < kNumQueues; ++k) off[k + 1] = off[k] + Q.taken[k];
    const uint32_t total = off[kNumQueues];
    __shared__ uint32_t s_stack[(kSmemStack + 1) * kStackThreads];  // the last row: see touch
    TraceState s;
    s.sstk = s_stack + threadIdx.x;
    const SceneView* scp = kOne ? &one : &rp.reqs[0].sc;  // a valid scene on idle lanes too
    uint32_t slot = ~0u;  // ~0: idle
    constexpr uint32_t kEnds = 0x80000000u;
    bool vol = false;  // kInner: the path is in a volume that ends its ray
    bool exhausted = false;
    uint32_t err = 0;
    auto put = [&]() {
        const uint32_t id = kInner ? slot & ~kEnds : slot;
        if (kInner) {
            const int q = s.prim >= 0 ? hit_type(s.prim) : (vol ? (int)kMatVolumeInside : 0);
            P.qid[id] = (uint8_t)((slot & kEnds) ? 0 : q);
        }
        if (s.prim >= 0) {
            // the ray's whole sector in one store (a partial store to a line that is
            // not in L2 costs a read of the sector from DRAM); the hit primitive
            // rides where the volume-hit id goes (none after a surface hit: every
            // reader takes a negative id as none), and the logic kernel, which
            // writes the (ng, rng) sector anyway, computes the normal
            st_sector<0>(P, id, f4(s.ro, s.tmin), f4(s.rd, __int_as_float(-2 - hit_id(s.prim))));
        }
        slot = ~0u;
    };
    for (;;) {
        const unsigned idle = __ballot_sync(full, slot == ~0u);
        if (!exhausted && (int)__popc(idle) >= refill) {
            const uint32_t need = __popc(idle);
            unsigned long long base = 0;
            if (lane == 0) base = atomicAdd(next, (unsigned long long)need);
            base = __shfl_sync(full, base, 0);
            if (base + need >= total) exhausted = true;
            if (slot == ~0u) {
                const unsigned long long i = base + __popc(idle & lt);
                if (i < total) {
                    int k = 0;
#pragma unroll
                    for (int j = 1; j < kNumQueues; ++j) k += ((uint32_t)i >= off[j]) ? 1 : 0;
                    const uint32_t r = queue_items(Q, k)[(uint32_t)i - pick(off, k)];
                    // only a new-path item can have retired (sample budget reached in
                    // the shading kernel): material-queue items skip the check
                    if (k != 0 || P.qid[r] != kQueueIdle) {
                        slot = r;
                        const RequestD* rq = kOne ? rp.reqs : rp.reqs + P.req[r];
                        if (!kOne) scp = &rq->sc;
                        float4 ro4, rd4;
                        ld_sector<0>(P, r, ro4, rd4);
                        if (kInner) {
                            float4 T4, L4;
                            ld_sector<1>(P, r, T4, L4);
                            if (logic_ends(*rq, P, r, xyz(T4), depth_of(__float_as_uint(L4.w)))) slot |= kEnds;
                            vol = __float_as_int(rd4.w) >= 0;
                        }
                        trace_begin(kOne ? one : *scp, s, xyz(ro4), xyz(rd4), ro4.w);
                    }
                }
            }
        }
        const unsigned held = __ballot_sync(full, slot != ~0u);
        if (exhausted && __popc(held) <= kTailLanes) break;
        if (held == 0u) continue;
        trace_warp_round<false, false, kSmemStack>(kOne ? one : *scp, s, slot != ~0u && s.link != kDone, search,
                                                   nullptr, err, pol);
        if (slot != ~0u && s.link == kDone) put();
    }
    if (slot != ~0u) {  // the last few paths of the warp, lane by lane
        while (s.link != kDone) trace_round<false, false, kSmemStack, true>(kOne ? one : *scp, s, nullptr, err, pol);
        put();
        touch_done();
    }
    if (err) atomicOr(rp.err, err);
}

// logic.cl:27-190 up to the accumulation, without the envmap's radiance: throughput,
// Russian roulette, depth limit.  Returns whether the path ends; a path that
// left the scene (hs < 0 and hv < 0) ends and is still owed T * envmap.
RGR_DEV bool logic_decide(const RequestD& rq, int32_t hs, int32_t hv, uint32_t logic_i, f3& T, f3& L, Rng& rng) {
    bool newPath = hs < 0 && hv < 0;
    float lum = 0.2126f * T.x + 0.7152f * T.y + 0.0722f * T.z;
    float cp = 1.0f;
    if ((long long)rq.rr_depth < (long long)logic_i) cp = fmin_(lum, 1.0f);
    float u = rng.uniform();
    if (u < cp) {
        T = T / cp;
    } else {
        newPath = true;
    }
    if (lum < 1.0e-5f) newPath = true;
    // depth limit: end after segment max_depth, adding the emission that the
    // next material stage would add (lambertian.cl:395)
    if (rq.max_depth > 0 && !newPath && (long long)logic_i >= (long long)rq.max_depth) {
        if (0 <= hs) {
            const SceneView& sc = rq.sc;
            int2 m = __ldg(sc.materials + hs);
            f3 Le = mk(0, 0, 0);
            if (m.x == kMatLambertian) Le = xyz(__ldg(sc.lambertians + 2 * (size_t)m.y));
            L = L + T * Le;
        }
        newPath = true;
    }
    return newPath;
}

// an ended path's radiance into its pixel's FP64 sums, unless it is discarded
// (not finite, or at the clamp); returns whether it was kept
RGR_DEV bool accumulate(const RequestD& rq, uint32_t pixel, f3 L) {
    const float cl = rq.radiance_clamp;
    if (!(is_finite(L.x) && is_finite(L.y) && is_finite(L.z) && L.x < cl && L.y < cl && L.z < cl)) return false;
    double* a = rq.accum + 4 * (size_t)pixel;
    atomicAdd(a + 0, (double)L.x);
    atomicAdd(a + 1, (double)L.y);
    atomicAdd(a + 2, (double)L.z);
    atomicAdd(a + 3, 1.0);
    return true;
}

// finished paths per request (stamp_done takes the completion times); called by
// the lanes `active` of a warp, `ended` on those whose path of request req ended
RGR_DEV void count_done(const RequestD& rq, int req, bool ended, unsigned active) {
    const unsigned donemask = __ballot_sync(active, ended);
    if (ended && rq.done != nullptr) {
        const unsigned peers = __match_any_sync(donemask, req);
        if ((int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(rq.done, (unsigned long long)__popc(peers));
    }
}

// The logic of one live slot (logic.cl:27-190) after its extension ray;
// returns the queue of its next step (0: a new path; the caller counts and
// appends).  kPreTraced: k_trace_paths has cast the extension rays of this
// bounce and written the hit; otherwise it is the primitive `prim` (-1: none) at t.
template <bool kGuided, bool kPreTraced>
RGR_DEV int logic_slot(const PathsView& P, const QueueView& Q, const RenderParams& rp, uint32_t slot,
                       unsigned active, GuideOffer& go, int32_t prim = -1, float t = 0.0f) {
    const int req = P.req[slot];
    const RequestD& rq = rp.reqs[req];
    const SceneView& sc = rq.sc;
    float4 ro4, rd4, ng4, rng4, T4, L4;
    ld_sector<0>(P, slot, ro4, rd4);
    ld_sector<1>(P, slot, T4, L4);
    ld_sector<2>(P, slot, ng4, rng4);
    f3 rd = xyz(rd4);
    int32_t hv = __float_as_int(rd4.w);
    if (!kPreTraced && prim >= 0) {
        ro4.w = t;
        hv = -2 - prim;
        st_sector<0>(P, slot, ro4, f4(rd, __int_as_float(-1)));
    }
    int32_t hs = __float_as_int(ng4.w);
    int mtype = -1;  // the hit triangle's material type, where the triangle table gave it
    resolve_hit(sc, ro4, rd4, hv, hs, ng4, mtype);
    // logic (logic.cl:27-190)
    f3 T = xyz(T4), L = xyz(L4);
    const uint32_t lw = __float_as_uint(L4.w);  // segment count and volume count
    const uint32_t logic_i = depth_of(lw);
    Rng rng = rng_of_bits(rng4);
    const bool newPath = logic_decide(rq, hs, hv, logic_i, T, L, rng);
    if (hs < 0 && hv < 0 && sc.has_env) L = L + T * envmap_value(sc, rd, logic_i == 0);
    const bool kept = newPath && accumulate(rq, __float_as_uint(T4.w), L);
    // No samples once the sample budget is handed out: the paths still in
    // flight are the long ones, and a few iterations on that subset alone
    // undo much of what the guide learned (the same for every thread).
    if (kGuided && rp.gd.record && guide_training_open(rp.gd.train) &&
        !(rp.sample_limit != 0ull && *Q.next_pixel >= rp.sample_limit))
        guide_offer(rp.gd, slot, L, kept, go);
    st_sector<1>(P, slot, f4(T, T4.w), f4(L, __uint_as_float(depth_word(logic_i + 1, vcount_of(lw)))));
    st_sector<2>(P, slot, ng4, rng_bits(rng));
    int q;
    if (newPath) {
        q = 0;
    } else if (0 <= hs) {
        q = mtype >= 0 ? mtype : __ldg(sc.materials + hs).x;
    } else {
        q = kMatVolumeInside;
    }
    P.qid[slot] = (uint8_t)q;
    count_done(rq, req, newPath, active);
    return q;
}

// The logic of a block's slots, all of tile `tile`, one a thread (`live` where it has
// one); logic(active, go) runs a live slot's.  Material-queue appends are gathered
// per block (shared-memory counts, then one global atomic per queue), and so
// is the ray count: with one atomic per warp all warps of the launch queued on
// the same few counters.
constexpr int kLogicThreads = 256;
template <bool kGuided, typename Logic>
RGR_DEV void logic_block(const QueueView& Q, const RenderParams& rp, uint32_t slot, uint32_t tile, bool live,
                         Logic logic) {
    const unsigned full = 0xffffffffu;
    __shared__ uint32_t s_q[kNumQueues];  // items per queue, then the block's base in it
    __shared__ uint32_t s_samples, s_offered;  // guided recording: accepted samples (then their base), offered
    if (threadIdx.x < kNumQueues) s_q[threadIdx.x] = 0;
    if (kGuided && threadIdx.x == 32) s_samples = s_offered = 0u;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const unsigned active = __ballot_sync(full, live);
    int q = 0;
    GuideOffer go;
    if (live) q = logic(active, go);
    __syncthreads();  // s_q, s_samples, s_offered cleared
    uint32_t off = 0;
    if (live) {
        const unsigned peers = __match_any_sync(active, q);
        const int leader = __ffs(peers) - 1;
        uint32_t base = 0;
        if (lane == leader) base = atomicAdd(&s_q[q], (uint32_t)__popc(peers));
        off = __shfl_sync(peers, base, leader) + __popc(peers & lt);
    }
    uint32_t sidx = 0;  // this lane's first sample within the block's
    if (kGuided) {
        // exclusive prefix of the accepted counts (0..3: two ballots)
        const uint32_t mine = __popc(go.take);
        const unsigned b0 = __ballot_sync(full, mine & 1u), b1 = __ballot_sync(full, (mine >> 1) & 1u);
        const uint32_t wtot = __popc(b0) + 2u * __popc(b1);
        const uint32_t offered = __reduce_add_sync(full, go.offered);
        uint32_t wbase = 0;
        if (lane == 0 && wtot) wbase = atomicAdd(&s_samples, wtot);
        if (lane == 0 && offered) atomicAdd(&s_offered, offered);
        sidx = __shfl_sync(full, wbase, 0) + __popc(b0 & lt) + 2u * __popc(b1 & lt);
    }
    const int nlive = __syncthreads_count(live);
    if (threadIdx.x < kNumQueues) {
        const uint32_t n = s_q[threadIdx.x];
        // queue 0: new paths per tile, for the ordered compaction (a block's slots lie in one tile)
        if (n && threadIdx.x == 0) atomicAdd(Q.tile_new + tile, n);
        else if (n) s_q[threadIdx.x] = atomicAdd(Q.counts + threadIdx.x, n);
    }
    if (kGuided && threadIdx.x == 32) {
        if (s_samples) s_samples = atomicAdd(rp.gd.train.count, s_samples);
        if (s_offered) atomicAdd(rp.gd.train.candidates, (unsigned long long)s_offered);
    }
    if (threadIdx.x == 0 && nlive) atomicAdd(rp.rays, (unsigned long long)nlive);
    __syncthreads();
    if (live && q != 0) queue_items(Q, q)[s_q[q] + off] = slot;
    if (kGuided && __any_sync(full, go.take != 0u)) {
        float ws = go.take ? guide_write(rp.gd, slot, go, s_samples + sidx) : 0.0f;
        for (int o = 16; o > 0; o >>= 1) ws += __shfl_xor_sync(full, ws, o);
        if (lane == 0 && ws > 0.0f) atomicAdd(rp.gd.train.wsum, ws);
    }
}

// The logic kernel of a cast made before, one thread per slot.
// latency-bound: 6 resident blocks per SM for the logic alone (40 registers; the
// render 0.6 % faster than at 5), 5 while it records guide samples
#ifndef RGR_LOGIC_MIN_BLOCKS  // the plain pre-traced logic: 5 / 6 / 7 give 1464 / 1472 / 1436 Mpaths/s
#define RGR_LOGIC_MIN_BLOCKS 6
#endif
template <bool kGuided>
__global__ void __launch_bounds__(kLogicThreads, kGuided ? 5 : RGR_LOGIC_MIN_BLOCKS)
    k_logic(PathsView P, QueueView Q, RenderParams rp) {
    follow();
    const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = slot < P.n && P.qid[slot] != kQueueIdle;
    logic_block<kGuided>(Q, rp, slot, slot / kTile, live, [&](unsigned active, GuideOffer& go) {
        return logic_slot<kGuided, true>(P, Q, rp, slot, active, go);
    });
}

// Cast and logic of a bounce in one launch, for few paths.  A block takes the live ones
// of `span` consecutive slots of one tile: it lists them in shared memory, its warps cast
// their rays (a warp takes the next rays of the list as its lanes fall idle, and
// ends lane by lane, as in k_trace_paths), the hits stay in shared memory, and the logic
// goes over the list.  Bound by instruction issue at few lanes and by the longest rays: with
// one thread a slot (k_slot_logic), 6 to 8 of a warp's lanes are in use, here 12 to 15.  Whole
// renders (8 spp, depth 6) at 2^14 / 2^16 / 2^17 / 2^18 paths, time of one thread a slot over this:
// 5 K triangles 1.00 / 1.01 / 1.01 / 1.10, 80 K 1.09 / 1.08 / 1.08 / 1.16.
// 4 blocks an SM: 5 the same to 2 % slower.  half_end: the slots below it go half a span a block.
constexpr int kCastLogicBlocks = 4;
template <bool kGuided, bool kOne>
__global__ void __launch_bounds__(kLogicThreads, kCastLogicBlocks)
    k_cast_logic(PathsView P, QueueView Q, RenderParams rp, uint32_t half_end, int refill, int search, SceneView one) {
    follow();
    const unsigned full = 0xffffffffu;
    __shared__ uint32_t s_stack[(kSmemStack + 1) * kStackThreads];  // the last row: see touch
    __shared__ uint32_t s_slot[kCastSpan];
    __shared__ int32_t s_prim[kCastSpan];
    __shared__ float s_t[kCastSpan];
    __shared__ uint32_t s_n, s_next;
    const int lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    const uint32_t half_blocks = half_end / (kCastSpan / 2);
    const bool half = blockIdx.x < half_blocks;
    const uint32_t span = half ? kCastSpan / 2 : kCastSpan;
    const uint32_t first = half ? blockIdx.x * (kCastSpan / 2) : half_end + (blockIdx.x - half_blocks) * kCastSpan;
    if (threadIdx.x == 0) s_n = s_next = 0u;
    __syncthreads();
    for (uint32_t o = threadIdx.x; o < span; o += kLogicThreads) {
        const uint32_t slot = first + o;
        const bool live = slot < P.n && P.qid[slot] != kQueueIdle;
        const unsigned m = __ballot_sync(full, live);
        uint32_t base = 0;
        if (lane == 0 && m) base = atomicAdd(&s_n, (uint32_t)__popc(m));
        base = __shfl_sync(full, base, 0);
        if (live) s_slot[base + __popc(m & lt)] = slot;
    }
    __syncthreads();
    const uint32_t n = s_n;
    // extension_ray_cast (extension_ray_cast_stackless.cl:202-246)
    const uint64_t pol = l2_evict_last_policy();
    TraceState s;
    s.sstk = s_stack + threadIdx.x;
    const SceneView* scp = kOne ? &one : &rp.reqs[0].sc;  // a valid scene on idle lanes too
    uint32_t item = ~0u, err = 0;
    bool exhausted = false;
    auto put = [&]() {
        s_t[item] = s.tmin;
        s_prim[item] = hit_id(s.prim);
        item = ~0u;
    };
    for (;;) {
        const unsigned idle = __ballot_sync(full, item == ~0u);
        if (!exhausted && (int)__popc(idle) >= refill) {
            const uint32_t need = __popc(idle);
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&s_next, need);
            base = __shfl_sync(full, base, 0);
            if (base + need >= n) exhausted = true;
            const uint32_t i = base + __popc(idle & lt);
            if (item == ~0u && i < n) {
                item = i;
                float4 ro4, rd4;
                ld_sector<0>(P, s_slot[i], ro4, rd4);
                if (!kOne) scp = &rp.reqs[P.req[s_slot[i]]].sc;
                trace_begin(kOne ? one : *scp, s, xyz(ro4), xyz(rd4), ro4.w);
            }
        }
        const unsigned held = __ballot_sync(full, item != ~0u);
        if (exhausted && __popc(held) <= kTailLanes) break;
        if (held == 0u) continue;
        trace_warp_round<false, false, kSmemStack>(kOne ? one : *scp, s, item != ~0u && s.link != kDone, search,
                                                   nullptr, err, pol);
        if (item != ~0u && s.link == kDone) put();
    }
    if (item != ~0u) {  // the last few paths of the warp, lane by lane
        while (s.link != kDone) trace_round<false, false, kSmemStack, true>(kOne ? one : *scp, s, nullptr, err, pol);
        put();
        touch_done();
    }
    if (err) atomicOr(rp.err, err);
    __syncthreads();
    for (uint32_t o = 0; o < n; o += kLogicThreads) {
        const uint32_t i = o + threadIdx.x;
        const uint32_t slot = i < n ? s_slot[i] : 0u;
        logic_block<kGuided>(Q, rp, slot, first / kTile, i < n, [&](unsigned active, GuideOffer& go) {
            return logic_slot<kGuided, false>(P, Q, rp, slot, active, go, s_prim[i], s_t[i]);
        });
        __syncthreads();  // before the counts are cleared again
    }
}

// The same for scenes whose rays are over before a list pays (per_slot_cast): one thread a
// slot, from its ray to its queue.  Bound by latency: the longest ray of a warp, and the launches.
template <bool kGuided, bool kOne>
__global__ void __launch_bounds__(kLogicThreads, kCastLogicBlocks)
    k_slot_logic(PathsView P, QueueView Q, RenderParams rp, SceneView one) {
    follow();
    __shared__ uint32_t s_stack[(kSmemStack > 0 ? kSmemStack : 1) * kStackThreads];
    const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    const bool live = slot < P.n && P.qid[slot] != kQueueIdle;
    uint32_t err = 0;
    TraceState s;
    s.sstk = s_stack + threadIdx.x;
    if (live) {
        const SceneView& sc = kOne ? one : rp.reqs[P.req[slot]].sc;
        float4 ro4, rd4;
        ld_sector<0>(P, slot, ro4, rd4);
        const uint64_t pol = l2_evict_last_policy();
        trace_begin(sc, s, xyz(ro4), xyz(rd4), ro4.w);
        while (s.link != kDone) trace_round<false, false, kSmemStack>(sc, s, nullptr, err, pol);
    }
    if (err) atomicOr(rp.err, err);
    logic_block<kGuided>(Q, rp, slot, slot / kTile, live, [&](unsigned active, GuideOffer& go) {
        return logic_slot<kGuided, false>(P, Q, rp, slot, active, go, hit_id(s.prim), s.tmin);
    });
}

// The queues of a bounce inside a run, from the queue ids that the cast left: block t
// takes the tile [t*4096, (t+1)*4096), 8 consecutive slots a thread.  Counts per class as
// 9-bit fields of one word (a warp's 256 fit) are scanned over the warp, then warp k
// scans class k's over the warps; the tile's slots go to shared memory in class order and from there to the queues, one
// atomic per queue per block: 16 MB of ids for 2^24 slots instead of a pass over
// their records.  The ended paths' slots go to the tile's own stretch of I.ended, in
// slot order.  The last block to finish scans the tiles' counts of them, so that
// k_new_paths can number them (pixels are assigned as new_path.cl:41-43 would over
// the slots in order), hands the bounce's counts to the kernels that follow,
// advances the sample counter (finalize_new_path, new_path.cl:85-88) and clears what
// the next bounce counts in, so that a bounce needs no memset.
// Bound by its chain of steps (256 tiles 12.4 us with 16 slots a thread, 11.0 so).
constexpr uint32_t kClassifyThreads = 512, kClassifyWarps = kClassifyThreads / 32;
__global__ void __launch_bounds__(kClassifyThreads) k_classify(PathsView P, QueueView Q, InnerView I, RenderParams rp,
                                                               unsigned long long* trace_next, int boundary) {
    follow();
    const unsigned full = 0xffffffffu;
    __shared__ unsigned long long s_warp[kClassifyWarps];
    __shared__ uint32_t s_pos[kNumQueues][kClassifyWarps];  // where a warp's slots of a class go in s_list
    __shared__ uint32_t s_off[kNumQueues + 1], s_base[kNumQueues], s_last;
    __shared__ uint16_t s_list[kTile];
    constexpr uint32_t kEach = kTile / kClassifyThreads;
    const uint32_t t = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const uint2 q8 = *reinterpret_cast<const uint2*>(P.qid + t * kTile + tid * kEach);
    // the queue of the thread's slot k; idle ones are above
    auto queue = [&](uint32_t k) { return ((k < 4u ? q8.x : q8.y) >> (8 * (k & 3u))) & 0xffu; };
    unsigned long long f = 0ull;
#pragma unroll
    for (uint32_t k = 0; k < kEach; ++k)
        if (queue(k) < (uint32_t)kNumQueues) f += 1ull << (9 * queue(k));
    unsigned long long inc = f;  // inclusive over the warp
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned long long a = __shfl_up_sync(full, inc, o);
        if ((int)lane >= o) inc += a;
    }
    if (lane == 31) s_warp[warp] = inc;
    __syncthreads();
    uint32_t base = 0;
    if (warp < (uint32_t)kNumQueues) {
        const unsigned long long w = lane < kClassifyWarps ? s_warp[lane] : 0ull;
        uint32_t below = 0, n = (uint32_t)(w >> (9 * warp)) & 511u, sum = n;
#pragma unroll
        for (uint32_t k = 0; k + 1 < (uint32_t)kNumQueues; ++k)
            if (k < warp) below += (uint32_t)(w >> (9 * k)) & 511u;
        below = __reduce_add_sync(full, below);
        for (int o = 1; o < (int)kClassifyWarps; o <<= 1) {
            const uint32_t a = __shfl_up_sync(full, sum, o);
            if ((int)lane >= o) sum += a;
        }
        if (lane < kClassifyWarps) s_pos[warp][lane] = below + sum - n;
        const uint32_t total = __shfl_sync(full, sum, kClassifyWarps - 1);
        if (lane == 0) {
            s_off[warp] = below;
            if (warp == 0) {
                Q.tile_new[t] = total;
            } else if (total) {
                base = atomicAdd(Q.counts + warp, total);
            }
            if (warp + 1 == (uint32_t)kNumQueues) {
                s_off[kNumQueues] = below + total;
                if (below + total) atomicAdd(rp.rays, (unsigned long long)(below + total));
            }
        }
    }
    __syncthreads();
    uint32_t off[kNumQueues + 1];
#pragma unroll
    for (int k = 0; k <= kNumQueues; ++k) off[k] = s_off[k];
    if (off[kNumQueues] != 0u) {  // not an idle tile (the same in every thread)
        // the thread's slots into class order
        unsigned long long e = inc - f;
#pragma unroll
        for (uint32_t k = 0; k < kEach; ++k) {
            const uint32_t q = queue(k);
            if (q < (uint32_t)kNumQueues) {
                s_list[s_pos[q][warp] + ((uint32_t)(e >> (9 * q)) & 511u)] = (uint16_t)(tid * kEach + k);
                e += 1ull << (9 * q);
            }
        }
        if (lane == 0 && warp < (uint32_t)kNumQueues) s_base[warp] = base;
        __syncthreads();
        for (uint32_t j = tid; j < off[1]; j += kClassifyThreads) I.ended[t * kTile + j] = s_list[j];
        for (uint32_t j = off[1] + tid; j < off[kNumQueues]; j += kClassifyThreads) {
            int q = 1;
#pragma unroll
            for (int k = 2; k < kNumQueues; ++k) q += j >= off[k] ? 1 : 0;
            queue_items(Q, q)[s_base[q] + j - s_off[q]] = t * kTile + s_list[j];
        }
    }
    // the last block: every block's counts are in
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(I.words + InnerView::kTicket, 1u) + 1u == gridDim.x ? 1u : 0u;
    __syncthreads();
    if (!s_last) return;
    uint32_t went_on = 0;
    unsigned long long np = 0;
    if (tid == 0) {  // on their way while the block scans
        np = *Q.next_pixel;
#pragma unroll
        for (int k = 1; k < kNumQueues; ++k) {
            went_on |= I.words[k] = __ldcg(Q.counts + k);
            Q.counts[k] = 0u;
        }
    }
    uint32_t run = 0;
    __shared__ uint32_t s_sum[kClassifyWarps];
    for (uint32_t b0 = 0; b0 < Q.ntiles; b0 += 4 * kClassifyThreads) {  // four tiles a thread
        uint32_t v[4], x = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t i = b0 + 4 * tid + k;
            v[k] = i < Q.ntiles ? __ldcg(Q.tile_new + i) : 0u;
            x += v[k];
        }
        uint32_t inc = x;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(full, inc, o);
            if ((int)lane >= o) inc += y;
        }
        if (lane == 31) s_sum[warp] = inc;
        __syncthreads();
        uint32_t e = run + inc - x;
#pragma unroll
        for (uint32_t w = 0; w < kClassifyWarps; ++w) {
            if (w < warp) e += s_sum[w];
            run += s_sum[w];
        }
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const uint32_t i = b0 + 4 * tid + k;
            if (i < Q.ntiles) I.tile_first[i] = e;
            e += v[k];
        }
        __syncthreads();  // s_sum is read
    }
    if (tid == 0) {
        const bool over = boundary && went_on == 0u && np >= rp.sample_limit;
        I.words[InnerView::kEnded] = run;
        I.words[InnerView::kStop] = over ? 1u : 0u;
        I.words[InnerView::kTicket] = 0u;
        I.words[0] = over ? 0u : run;
        if (!over) {
            Q.counts[0] = run;
            *Q.step_base = np;
            *Q.next_pixel = np + run;
        }
        *trace_next = 0ull;
    }
}

// The paths that ended in a bounce inside a run, and the new ones in their slots: the
// logic of the ended path (its envmap radiance and accumulation; the cast has
// only found that it ends), then the new path's first ray.  One ended path per
// thread, numbered in slot order, so that every lane has work; the slots go to queue 0
// for the cast.
// Bound by the records' DRAM traffic (a 128-byte line read, 96 bytes written per slot)
// and, where paths leave the scene, the envmap look-up's arithmetic.
// When the render is over (launch_inner_queues' boundary) the paths are only finished.
constexpr int kNewPathsBlocks = 8;  // per SM
__global__ void __launch_bounds__(256) k_new_paths(PathsView P, QueueView Q, InnerView I, RenderParams rp) {
    follow();
    const unsigned full = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t total = I.words[InnerView::kEnded];
    const bool over = I.words[InnerView::kStop] != 0u;
    const unsigned long long np = *Q.step_base;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t j0 = blockIdx.x * blockDim.x + (threadIdx.x & ~31u); j0 < total; j0 += stride) {
        // the tile of the warp's first path: the last one whose first number is <= j0
        // (a 32-way search of the scanned counts), then each lane's own
        uint32_t lo = 0, n = Q.ntiles;
        while (n > 1u) {
            const uint32_t step = (n + 31u) / 32u, i = lo + lane * step;
            const unsigned m = __ballot_sync(full, lane * step < n && I.tile_first[i] <= j0);
            const uint32_t k = 31u - __clz(m);  // lane 0's is always
            lo += k * step;
            n = min(step, n - k * step);
        }
        const uint32_t j = j0 + lane;
        const unsigned have = __ballot_sync(full, j < total);
        if (j >= total) continue;
        uint32_t t = lo, tf = I.tile_first[lo];
        while (t + 1u < Q.ntiles) {
            const uint32_t next = I.tile_first[t + 1u];
            if (next > j) break;
            ++t;
            tf = next;
        }
        const uint32_t slot = t * kTile + I.ended[t * kTile + (j - tf)];
        // the ended path
        const int req = P.req[slot];
        const RequestD& old = rp.reqs[req];
        float4 ro4, rd4, T4, L4, ng4, rng4;
        ld_sector<0>(P, slot, ro4, rd4);
        ld_sector<1>(P, slot, T4, L4);
        ld_sector<2>(P, slot, ng4, rng4);
        SlotState st;
        const int32_t word = __float_as_int(rd4.w);  // the hit, or the volume hit
        st.hv = word <= -2 ? -1 : word;
        const int32_t hs = word <= -2 ? -2 - word : -1;
        const uint32_t lw = __float_as_uint(L4.w);
        st.T = xyz(T4), st.L = xyz(L4);
        st.rng = rng_of_bits(rng4);
        logic_decide(old, hs, st.hv, depth_of(lw), st.T, st.L, st.rng);
        if (hs < 0 && st.hv < 0 && old.sc.has_env)
            st.L = st.L + st.T * envmap_value(old.sc, xyz(rd4), depth_of(lw) == 0);
        accumulate(old, __float_as_uint(T4.w), st.L);
        count_done(old, req, true, have);
        unsigned long long gpix = np + j;
        const bool retire = rp.sample_limit != 0ull && gpix >= rp.sample_limit;
        if (!over) Q.items[0][j] = slot;
        if (over || retire) {  // the state as the plain logic leaves it
            int32_t h2 = __float_as_int(ng4.w), v2 = word;
            int mtype;
            resolve_hit(old.sc, ro4, rd4, v2, h2, ng4, mtype);
            st_sector<1>(P, slot, f4(st.T, T4.w),
                         f4(st.L, __uint_as_float(depth_word(depth_of(lw) + 1, vcount_of(lw)))));
            st_sector<2>(P, slot, ng4, rng_bits(st.rng));
            if (!over) P.qid[slot] = kQueueIdle;  // sample budget reached: the slot retires
            continue;
        }
        int r = 0;  // the request whose sample range holds this global sample index
        while (r + 1 < rp.nreq && gpix >= rp.reqs[r].sample_end) ++r;
        P.req[slot] = (uint16_t)r;
        gpix -= rp.reqs[r].sample_begin;
        st.va = make_int4(0, 0, 0, 0), st.vb = st.va;
        shade_state<false>(rp.reqs[r], 0, slot, gpix, rp.gd, ~0u, st);
        st_sector<0>(P, slot, f4(st.ro, st.tmin), f4(st.rd, __int_as_float(st.hv)));
        st_sector<1>(P, slot, f4(st.T, __uint_as_float(st.pixel)), f4(st.L, __uint_as_float(depth_word(0u, 0))));
        st_sector<2>(P, slot, f4(st.Ng, __int_as_float(st.hs)), rng_bits(st.rng));
    }
}

// The mean sum / count (count > 0) in double, rounded to float, then to half.  A double
// division is some twenty operations on the chip's few FP64 units, and the half keeps 11
// bits of it: where all within 2^-20 of the quotient in float rounds to one half, that is the
// half (the roundings are monotonic, and the quotient's error is below 2^-21: 2^-24 from each
// operand, 2 ulp from the division), else, for about one value in 500, the
// division decides.  Image readbacks of 1280x720 / 1920x1080 pixels 135 / 239 us with
// divisions alone, 72 / 111 so.
RGR_DEV unsigned short half_mean(double sum, double count) {
    const float q = __fdividef((float)sum, (float)count);
    const unsigned short lo = __half_as_ushort(__float2half_rn(q * (1.0f - 0x1p-20f)));
    const unsigned short hi = __half_as_ushort(__float2half_rn(q * (1.0f + 0x1p-20f)));
    return lo == hi ? lo : __half_as_ushort(__float2half_rn((float)(sum / count)));
}

// RGB16 intermediate (accumlation.cl:6-25) from FP64 sums: half_mean; count to 16 bits.
__global__ void k_readback(int fmt, const double* accum, uint32_t npix, void* out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= npix) return;
    const double2 rg = __ldcs(reinterpret_cast<const double2*>(accum) + 2 * (size_t)i);
    const double2 bc = __ldcs(reinterpret_cast<const double2*>(accum) + 2 * (size_t)i + 1);
    const double a[3] = {rg.x, rg.y, bc.x}, cnt = bc.y;
    unsigned short h[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) h[k] = cnt > 0.0 ? half_mean(a[k], cnt) : (unsigned short)0;
    if (fmt == 1) {
        ushort4 v = make_ushort4(h[0], h[1], h[2], (unsigned short)((unsigned long long)cnt & 0xffffull));
        reinterpret_cast<ushort4*>(out)[i] = v;
        return;
    }
    // tonemap (accumlation.cl:68-79)
    uchar4 px;
    unsigned char c[3];
    for (int k = 0; k < 3; ++k) {
        float v = __half2float(__ushort_as_half(h[k]));
        int iv = to_int(pow_(v * 1.0f, 1.0f / 2.2f) * 256.0f);
        iv = min(max(iv, 0), 255);
        c[k] = (unsigned char)iv;
    }
    px.x = c[0];
    px.y = c[1];
    px.z = c[2];
    px.w = 255;
    reinterpret_cast<uchar4*>(out)[i] = px;
}

// stat (stat.cl:6-39): total accumulated samples
__global__ void k_sum_counts(const double* accum, uint32_t npix, unsigned long long* out) {
    unsigned long long s = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += gridDim.x * blockDim.x)
        s += (unsigned long long)accum[4 * (size_t)i + 3];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

// merge_intermediate (accumlation.cl:27-49): count-weighted merge of two RGB16
// intermediates in FP32, result stored as half into a
__global__ void k_merge_intermediate(ushort4* a, const ushort4* b, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    ushort4 va = a[i], vb = b[i];
    const unsigned short sa = va.w, sb = vb.w;
    const unsigned short sab = (unsigned short)(sa + sb);
    if (sab == 0) {
        a[i] = make_ushort4(0, 0, 0, 0);
        return;
    }
    const float one_over_sab = 1.0f / (float)sab;
    const unsigned short ha[3] = {va.x, va.y, va.z}, hb[3] = {vb.x, vb.y, vb.z};
    unsigned short out[3];
    for (int k = 0; k < 3; ++k) {
        float m = (__half2float(__ushort_as_half(ha[k])) * (float)sa + __half2float(__ushort_as_half(hb[k])) * (float)sb) *
                  one_over_sab;
        out[k] = __half_as_ushort(__float2half_rn(m));
    }
    a[i] = make_ushort4(out[0], out[1], out[2], sab);
}

__global__ void k_accum_add(double* dst, const double* src, uint32_t n4) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n4) dst[i] += src[i];
}

__global__ void k_debug_slots(PathsView P, uint32_t* out) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= P.n) return;
    uint32_t* o = out + 34 * (size_t)i;
    float4 T = P.T[i], L = P.L[i], ro = P.ro[i], rd = P.rd[i], ng = P.ng[i];
    uint4 r = P.rng[i];
    int4 va = P.va[i], vb = P.vb[i];
    const float f[12] = {T.x, T.y, T.z, L.x, L.y, L.z, ro.x, ro.y, ro.z, rd.x, rd.y, rd.z};
    for (int k = 0; k < 12; ++k) o[k] = __float_as_uint(f[k]);
    o[12] = depth_of(__float_as_uint(L.w));
    o[13] = __float_as_uint(T.w);
    o[14] = r.x;
    o[15] = r.y;
    o[16] = r.z;
    o[17] = r.w;
    o[18] = __float_as_uint(ng.w);
    o[19] = __float_as_int(rd.w) < -1 ? 0xffffffffu : __float_as_uint(rd.w);  // no volume hit: -1
    o[20] = __float_as_uint(ro.w);
    o[21] = __float_as_uint(ng.x);
    o[22] = __float_as_uint(ng.y);
    o[23] = __float_as_uint(ng.z);
    uint8_t q = P.qid[i];
    o[24] = q == kQueueIdle ? 0xffffffffu : (uint32_t)q;
    o[25] = (uint32_t)vcount_of(__float_as_uint(L.w));
    const int v[7] = {va.x, va.y, va.z, va.w, vb.x, vb.y, vb.z};
    for (int k = 0; k < 7; ++k) o[26 + k] = (uint32_t)v[k];
    o[33] = 0;
}

}  // namespace

void launch_init(const PathsView& p, const QueueView& q, uint32_t seed_offset, const InitView& w, const RequestD& one,
                 cudaStream_t st) {
    uint32_t n = q.ntiles * kTile;
    k_init<<<(n + 255) / 256, 256, 0, st>>>(p, q, seed_offset, w, one);
}
void launch_compact_new(const PathsView& p, const QueueView& q, unsigned long long* cast_counter, cudaStream_t st) {
    chain(k_compact_new, q.ntiles, 256, 0, st, p, q, cast_counter);
}
void launch_guide_select(const PathsView& p, const QueueView& q, const GuideRenderD& gd, bool inner, int grid,
                         cudaStream_t st) {
    cudaMemsetAsync(gd.nsel, 0, sizeof(uint32_t), st);
    k_guide_select<<<grid, 256, 0, st>>>(p, q, gd, inner ? 1u : 0u);
}

void launch_shade(const PathsView& p, const QueueView& q, const RenderParams& rp, int grid, cudaStream_t st) {
    if (rp.gd.lobes)
        chain(k_shade_guided, grid, 256, 0, st, p, q, rp);
    else
        chain(k_shade, grid, 256, 0, st, p, q, rp);
}
template <bool kInner>
static void cast_paths(const PathsView& p, const QueueView& q, const RenderParams& rp, const TraceShape& ts,
                       cudaStream_t st) {
    if (ts.one && rp.nreq == 1)
        chain(k_trace_paths<kInner, true>, ts.grid, kStackThreads, 0, st, p, q, rp, ts.counter, ts.refill, ts.search,
              *ts.one);
    else
        chain(k_trace_paths<kInner, false>, ts.grid, kStackThreads, 0, st, p, q, rp, ts.counter, ts.refill, ts.search,
              SceneView{});
}

void launch_trace_paths(const PathsView& p, const QueueView& q, const RenderParams& rp, const TraceShape& ts,
                        cudaStream_t st) {
    if (ts.persistent) cast_paths<false>(p, q, rp, ts, st);
}

template <bool kGuided>
static void trace_logic(const PathsView& p, const QueueView& q, const RenderParams& rp, const TraceShape& ts,
                        int num_sms, cudaStream_t st) {
    if (ts.persistent) {
        chain(k_logic<kGuided>, (p.n + kLogicThreads - 1) / kLogicThreads, kLogicThreads, 0, st, p, q, rp);
        return;
    }
    if (ts.per_slot) {
        const unsigned nb = (p.n + kLogicThreads - 1) / kLogicThreads;
        if (ts.one && rp.nreq == 1)
            chain(k_slot_logic<kGuided, true>, nb, kLogicThreads, 0, st, p, q, rp, *ts.one);
        else
            chain(k_slot_logic<kGuided, false>, nb, kLogicThreads, 0, st, p, q, rp, SceneView{});
        return;
    }
    const uint32_t half_end = cast_half_end(p.n, rp.sample_limit, (uint32_t)(num_sms * kCastLogicBlocks), kTile);
    const unsigned nb = cast_blocks(p.n, half_end);
    if (ts.one && rp.nreq == 1)
        chain(k_cast_logic<kGuided, true>, nb, kLogicThreads, 0, st, p, q, rp, half_end, ts.refill, ts.search, *ts.one);
    else
        chain(k_cast_logic<kGuided, false>, nb, kLogicThreads, 0, st, p, q, rp, half_end, ts.refill, ts.search,
              SceneView{});
}

void launch_trace_logic(const PathsView& p, const QueueView& q, const RenderParams& rp, const TraceShape& ts,
                        int num_sms, cudaStream_t st) {
    // the guided variant differs only in recording training samples: a render
    // with a frozen guide runs the plain one (fewer registers)
    if (rp.gd.lobes && rp.gd.record)
        trace_logic<true>(p, q, rp, ts, num_sms, st);
    else
        trace_logic<false>(p, q, rp, ts, num_sms, st);
}

// what a bounce inside a run counts in
void launch_inner_reset(const InnerView& in, cudaStream_t st) {
    cudaMemsetAsync(in.words, 0, sizeof(uint32_t) * InnerView::kWords, st);
}

void launch_inner_cast(const PathsView& p, const QueueView& q, const RenderParams& rp, const TraceShape& ts,
                       cudaStream_t st) {
    cast_paths<true>(p, q, rp, ts, st);
}

void launch_inner_queues(const PathsView& p, const QueueView& q, const InnerView& in, const RenderParams& rp,
                         const TraceShape& ts, bool boundary, int num_sms, cudaStream_t st) {
    chain(k_classify, q.ntiles, kClassifyThreads, 0, st, p, q, in, rp, ts.counter, boundary ? 1 : 0);
    const int blocks = std::min((int)((p.n + 255) / 256), num_sms * kNewPathsBlocks);
    chain(k_new_paths, blocks, 256, 0, st, p, q, in, rp);
}

void launch_inner_shade(const PathsView& p, const QueueView& u, const RenderParams& rp, const TraceShape& ts,
                        int shade_grid, cudaStream_t st) {
    if (rp.gd.lobes)
        chain(k_shade_inner<true>, shade_grid, 256, 0, st, p, u, rp);
    else
        chain(k_shade_inner<false>, shade_grid, 256, 0, st, p, u, rp);
    cast_paths<true>(p, u, rp, ts, st);
}

void launch_stamp_done(const RenderParams& rp, cudaStream_t st) {
    if (rp.nreq > 0) chain(k_stamp_done, (rp.nreq + 127) / 128, 128, 0, st, rp);
}

int trace_paths_max_blocks_per_sm(bool one) {
    int nb = 0;
    if (one)
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_trace_paths<true, true>, 256, 0);
    else
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&nb, k_trace_paths<true, false>, 256, 0);
    return nb > 0 ? nb : 1;
}
void launch_readback(int fmt, const double* accum, uint32_t npix, void* out, cudaStream_t st) {
    k_readback<<<(npix + 255) / 256, 256, 0, st>>>(fmt, accum, npix, out);
}
void launch_sum_counts(const double* accum, uint32_t npix, unsigned long long* out, cudaStream_t st) {
    k_sum_counts<<<152 * 4, 256, 0, st>>>(accum, npix, out);
}
void launch_debug_slots(const PathsView& p, uint32_t* out, cudaStream_t st) {
    k_debug_slots<<<(p.n + 255) / 256, 256, 0, st>>>(p, out);
}
void launch_merge_intermediate(void* a, const void* b, uint32_t n, cudaStream_t st) {
    k_merge_intermediate<<<(n + 255) / 256, 256, 0, st>>>(reinterpret_cast<ushort4*>(a),
                                                          reinterpret_cast<const ushort4*>(b), n);
}
void launch_accum_add(double* dst, const double* src, uint32_t npix, cudaStream_t st) {
    uint32_t n4 = npix * 4;
    k_accum_add<<<(n4 + 255) / 256, 256, 0, st>>>(dst, src, n4);
}

}  // namespace dev
}  // namespace rgr
