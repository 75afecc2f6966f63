// Wavefront path-tracing pipeline for sm_100a.
//
// The reference runs one megakernel thread per pixel and sample
// (sampleAdaptiveKernel, PathTracerLib/src/PathTracer.cu:186-273, body
// tracePathRand, PathIntegratorRandCore.h:206-363).  Here the same estimator
// is split into stages over structure-of-arrays path state:
//
//   generate   camera ray per (pixel, sample): curand_init with the reference
//              seed, jitter + lens draws (PathTracer.cu:69-96)
//   extend     closest hit for every live path (pt_traverse.cuh), then k_route,
//              which splits the queue into miss and hit queues
//   shade      pending NEE resolve, miss/env MIS, emission, environment and
//              emissive NEE (shadow rays queued), BSDF sample, throughput,
//              subsurface tier B, Russian roulette, continuation ray
//   shadow     any-hit occlusion for the queued shadow rays
//   finalize   paths that ended with shadow rays in flight; the next bounce's
//              extend queue in slot order, from the slots the shade kernel marked
//   accumulate per pixel, the batch's samples in sample order: running mean,
//              Welford luminance variance, convergence every 4 samples
//              (PathTracer.cu:232-272)
//   compact    active-pixel list without converged pixels, where it changed
//
// Radiance is added in exactly the reference's order: emission, env NEE,
// emissive NEE (resolved after the shadow stage), then at the next bounce the
// miss term.  Random numbers are drawn in the reference's order from the same
// per-(pixel, sample) XORWOW stream, so a path takes the same decisions as the
// reference's; the state lives in registers within a stage and in the SoA
// between stages.
#include "pt_render.cuh"

#include "pt_bsdf.cuh"
#include "pt_path.cuh"
#include "pt_spectral.cuh"
#include "pt_traverse.cuh"

#include <atomic>
#include <cooperative_groups.h>
#include "pt_select.cuh"
#include <curand_kernel.h>

namespace cg = cooperative_groups;

namespace pt {

namespace {

__device__ __forceinline__ uint32_t warpPush(unsigned int* counter)
{
    cg::coalesced_group g = cg::coalesced_threads();
    unsigned int base = 0;
    if (g.thread_rank() == 0) {
        base = atomicAdd(counter, g.size());
    }
    base = g.shfl(base, 0);
    return base + g.thread_rank();
}

// Warp-granular work distribution: each warp takes the next 32 queue entries
// from a per-launch counter, so warps that drew cheap rays keep working
// instead of idling while others finish (no static grid-stride split).
__device__ __forceinline__ unsigned int warpFetch(unsigned int* counter)
{
    unsigned int base = 0;
    if ((threadIdx.x & 31) == 0) {
        base = atomicAdd(counter, 32u);
    }
    return __shfl_sync(0xffffffffu, base, 0) + (threadIdx.x & 31);
}

__device__ __forceinline__ void rngLoad(const PathSoA& P, uint32_t i, curandStateXORWOW& s)
{
    const uint4 a = P.rngA[i];
    const uint2 b = P.rngB[i];
    s.d = a.x;
    s.v[0] = a.y;
    s.v[1] = a.z;
    s.v[2] = a.w;
    s.v[3] = b.x;
    s.v[4] = b.y;
    s.boxmuller_flag = 0;
    s.boxmuller_flag_double = 0;
    s.boxmuller_extra = 0.0f;
    s.boxmuller_extra_double = 0.0;
}

__device__ __forceinline__ void rngStore(const PathSoA& P, uint32_t i, const curandStateXORWOW& s)
{
    P.rngA[i] = make_uint4(s.d, s.v[0], s.v[1], s.v[2]);
    P.rngB[i] = make_uint2(s.v[3], s.v[4]);
}

// Geometry of path i's scene.
__device__ __forceinline__ const DevScene& sceneOf(const LaunchCtx& c, uint32_t i)
{
    return c.sceneCount > 1 ? c.scenes[c.paths.scene[i]] : c.scene;
}

// --- per-path colour: RGB (NW = 0, the reference's integrator) or the
// radiance at NW hero wavelengths (spectral mode) -----------------------------
template <int NW> struct Col {
    float v[NW];
};
template <> struct Col<0> {
    float3 c;
};

template <int NW> __device__ __forceinline__ Col<NW> czero()
{
    Col<NW> r;
    if constexpr (NW == 0) {
        r.c = f3(0.0f, 0.0f, 0.0f);
    } else {
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            r.v[k] = 0.0f;
        }
    }
    return r;
}
template <int NW> __device__ __forceinline__ Col<NW> cadd(const Col<NW>& a, const Col<NW>& b)
{
    Col<NW> r;
    if constexpr (NW == 0) {
        r.c = add3(a.c, b.c);
    } else {
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            r.v[k] = a.v[k] + b.v[k];
        }
    }
    return r;
}
template <int NW> __device__ __forceinline__ Col<NW> cmul(const Col<NW>& a, const Col<NW>& b)
{
    Col<NW> r;
    if constexpr (NW == 0) {
        r.c = mul3(a.c, b.c);
    } else {
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            r.v[k] = a.v[k] * b.v[k];
        }
    }
    return r;
}
template <int NW> __device__ __forceinline__ Col<NW> cscl(const Col<NW>& a, float s)
{
    Col<NW> r;
    if constexpr (NW == 0) {
        r.c = scl3(a.c, s);
    } else {
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            r.v[k] = a.v[k] * s;
        }
    }
    return r;
}
template <int NW> __device__ __forceinline__ bool cnonzero(const Col<NW>& a)
{
    if constexpr (NW == 0) {
        return a.c.x != 0.0f || a.c.y != 0.0f || a.c.z != 0.0f;
    } else {
        bool nz = false;
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            nz = nz || a.v[k] != 0.0f;
        }
        return nz;
    }
}

// Wavelengths of a path (spectral mode): the hero draw, wavelength k derived
// on use (a few instructions, cheaper than keeping NW registers live).
template <int NW> struct Waves {
    float u;
    __device__ __forceinline__ float lam(int k) const { return spectral::heroLambda(u, k, NW); }
};
template <int NW> __device__ __forceinline__ Waves<NW> pathWaves(const LaunchCtx& c, uint32_t i)
{
    Waves<NW> w;
    if constexpr (NW > 0) {
        w.u = c.paths.hero[i];
    } else {
        w.u = 0.0f;
    }
    return w;
}

// The spectrum of coefficient record q at the path's wavelengths.  A grey
// record (c = 0) is the constant scale / 2 and a zero scale is 0, exactly what
// evalCoef gives for them, without its square root and division.
template <int NW> __device__ __forceinline__ Col<NW> coefCol(float4 q, const Waves<NW>& w)
{
    Col<NW> r;
    if (q.x == 0.0f && q.y == 0.0f && q.z == 0.0f) {
        const float v = __fmul_rn(0.5f, q.w);
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            r.v[k] = v;
        }
    } else {
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            r.v[k] = spectral::evalCoef(q, w.lam(k));
        }
    }
    return r;
}

// Colour of a float4 path field (xyz in RGB mode; the spectral words otherwise).
template <int NW> __device__ __forceinline__ Col<NW> loadCol(float4 rgb, const float4* spec, int cap, uint32_t i)
{
    Col<NW> r;
    if constexpr (NW == 0) {
        r.c = f3(rgb.x, rgb.y, rgb.z);
    } else {
        (void)rgb;
#pragma unroll
        for (int j = 0; j < NW / 4; ++j) {
            const float4 q = spec[static_cast<size_t>(j) * cap + i];
            r.v[4 * j] = q.x;
            r.v[4 * j + 1] = q.y;
            r.v[4 * j + 2] = q.z;
            r.v[4 * j + 3] = q.w;
        }
    }
    return r;
}
// Stores a colour with `w` in the RGB field's fourth word (the RGB field
// keeps only w in spectral mode).
template <int NW> __device__ __forceinline__ void storeCol(float4* rgb, float4* spec, int cap, uint32_t i, const Col<NW>& v,
    float w)
{
    if constexpr (NW == 0) {
        rgb[i] = make_float4(v.c.x, v.c.y, v.c.z, w);
    } else {
        if (rgb != nullptr) {
            rgb[i] = make_float4(0.0f, 0.0f, 0.0f, w);
        }
#pragma unroll
        for (int j = 0; j < NW / 4; ++j) {
            spec[static_cast<size_t>(j) * cap + i] =
                make_float4(v.v[4 * j], v.v[4 * j + 1], v.v[4 * j + 2], v.v[4 * j + 3]);
        }
    }
}
// Depth and medium IOR of a spectral path, in the place of its RGB radiance.
__device__ __forceinline__ float2* depthEta(const LaunchCtx& c) { return reinterpret_cast<float2*>(c.paths.rad); }
template <int NW> __device__ __forceinline__ Col<NW> pendingEnv(const LaunchCtx& c, uint32_t i)
{
    if constexpr (NW == 0) {
        return loadCol<0>(c.paths.neeEnv[i], nullptr, 0, i);
    } else {
        return loadCol<NW>(make_float4(0.0f, 0.0f, 0.0f, 0.0f), c.paths.neeEnvS, c.paths.capacity, i);
    }
}
template <int NW> __device__ __forceinline__ Col<NW> pendingEmis(const LaunchCtx& c, uint32_t i)
{
    if constexpr (NW == 0) {
        return loadCol<0>(c.paths.neeEmis[i], nullptr, 0, i);
    } else {
        return loadCol<NW>(make_float4(0.0f, 0.0f, 0.0f, 0.0f), c.paths.neeEmisS, c.paths.capacity, i);
    }
}

// Environment / background radiance in direction d (LightSamplingCore.h:56-77).
template <int NW> __device__ __forceinline__ Col<NW> envCol(const LaunchCtx& c, float3 d, const Waves<NW>& w)
{
    Col<NW> r;
    if constexpr (NW == 0) {
        r.c = envEval(c.env, c.params, d);
    } else {
        float4 q = c.specBackground;
        if (c.env.valid) {
            float u, v;
            dirToLatLong(d, u, v);
            const int x = min(max(static_cast<int>(u * static_cast<float>(c.env.width)), 0), c.env.width - 1);
            const int y = min(max(static_cast<int>(v * static_cast<float>(c.env.height)), 0), c.env.height - 1);
            q = c.env.spec[static_cast<size_t>(y) * c.env.width + x];
        }
        r = coefCol<NW>(q, w);
    }
    return r;
}

// --- distant light ---------------------------------------------------------------
// Is direction d (any length) inside the light's cone?  Tested through the
// sine (|d x dir|^2 <= sin^2 * |d|^2), which keeps its precision for the small
// half-angles of a sun.
__device__ __forceinline__ bool inSun(const DevSun& s, float3 d)
{
    const float3 x = cross3(d, s.dir);
    return dot3(d, s.dir) > 0.0f && dot3(x, x) <= s.sin2 * dot3(d, d);
}
// Uniform direction in the cone (u1 -> 1 - cos theta over [0, omc], u2 -> phi).
__device__ __forceinline__ float3 sunSample(const DevSun& s, float u1, float u2)
{
    const float h = u1 * s.omc;
    const float ct = 1.0f - h;
    const float st = sqrtf(fmax2(0.0f, h * (2.0f - h)));
    float sp, cp;
    sincosf(2.0f * kPi * u2, &sp, &cp);
    return normalize3(add3(add3(scl3(s.t, st * cp), scl3(s.b, st * sp)), scl3(s.dir, ct)));
}
// Density of the sky's next-event sample (the light with probability select,
// else the environment) in direction d.
__device__ __forceinline__ float skyPdf(const LaunchCtx& c, float3 d)
{
    const float ls = inSun(c.sun, d) ? c.sun.pdf : 0.0f;
    return c.sun.select * ls + (1.0f - c.sun.select) * envPdf(c.env, d);
}
// Relative blackbody spectral radiance (Planck's law, lambda in micrometres).
__device__ __forceinline__ float planckRel(float lambdaNm, float temperature)
{
    const float lu = lambdaNm * 1.0e-3f;
    const float l2 = lu * lu;
    return 1.0f / (l2 * l2 * lu * expm1f(14387.769f / (lu * temperature)));
}
template <int NW> __device__ __forceinline__ Col<NW> sunCol(const LaunchCtx& c, const Waves<NW>& w)
{
    Col<NW> r;
    if constexpr (NW == 0) {
        (void)w;
        r.c = c.sun.rgb;
    } else if (c.sun.temperature > 0.0f) {
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            r.v[k] = c.sun.scale * planckRel(w.lam(k), c.sun.temperature);
        }
    } else {
        r = coefCol<NW>(c.sun.coef, w);
    }
    return r;
}
// Sky radiance (environment plus the light where d is inside its cone).
template <int NW> __device__ __forceinline__ Col<NW> skyCol(const LaunchCtx& c, float3 d, const Waves<NW>& w)
{
    Col<NW> L = envCol<NW>(c, d, w);
    if (c.sun.enabled && inSun(c.sun, d)) {
        L = cadd(L, sunCol<NW>(c, w));
    }
    return L;
}

// No light comes from the sky at all: a black background, no distant light.
template <int NW> __device__ __forceinline__ bool skyIsBlack(const LaunchCtx& c)
{
    if (c.sun.enabled != 0 || c.env.valid) {
        return false;
    }
    if constexpr (NW == 0) {
        const float k = c.params.environment_intensity;
        return c.params.background_r * k == 0.0f && c.params.background_g * k == 0.0f && c.params.background_b * k == 0.0f;
    } else {
        const float4 q = c.specBackground;
        return q.x == 0.0f && q.y == 0.0f && q.z == 0.0f && q.w == 0.0f;
    }
}

// Spectrum coefficients of the base colour and scatter radii of the material
// at a hit, following resolveMaterial's albedo-texture rules.
__device__ __forceinline__ void matCoefs(const DevScene& S, uint32_t mi, const pt_material& src, float u, float v,
    float4& base, float4& scatter)
{
    if (S.matSpec == nullptr || S.materials == nullptr || mi >= S.materialCount) {
        base = make_float4(0.0f, 0.0f, 0.0f, 1.6f); // the fallback material's grey 0.8
        scatter = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    } else {
        base = S.matSpec[2 * mi];
        scatter = S.matSpec[2 * mi + 1];
    }
    const uint32_t ti = src.albedo_tex;
    if (ti != 0u && S.textures != nullptr && ti < S.textureCount) {
        const pt_texture& t = S.textures[ti];
        if (t.kind == 1) {
            base = S.texSpec[2 * ti];
        } else if (t.kind == 2) {
            const float fx = fractf(u * t.p0[0]);
            const float fy = fractf(v * t.p0[1]);
            base = S.texSpec[2 * ti + ((fx < t.p0[2] || fy < t.p0[2]) ? 1 : 0)];
        } else {
            base = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
}

// BSDF value (RGB), or at each wavelength.  The spectral value at lambda is
// the RGB BSDF of the material with every colour channel set to the colour's
// spectrum at lambda.  All lobes but a scattering subsurface lobe are affine in
// the base colour, f(rho) = f(0) + rho (f(1) - f(0)), so one RGB evaluation
// with base (0, 1, 1) gives every wavelength: in spectral mode the shade
// kernel keeps the material's base at (0, 1, 1) (sampling and pdfs do not read
// it).  With a scattering subsurface lobe (radius per wavelength) each
// wavelength is evaluated on its own, cx's colour fields modified in place and
// restored.
template <int NW>
__device__ __forceinline__ Col<NW> evalCol(Ctx& cx, float3 wi, const Col<NW>& rho, float4 scatter, const Waves<NW>& w)
{
    Col<NW> f;
    if constexpr (NW == 0) {
        (void)rho;
        (void)scatter;
        (void)w;
        f.c = bsdfEval(cx, wi);
    } else {
        if (cx.w.subsurface != 0.0f && maxScatter(cx.m) > kMinRadius) {
            const float sr = cx.m.scatterR, sg = cx.m.scatterG, sb = cx.m.scatterB;
#pragma unroll 1
            for (int k = 0; k < NW; ++k) {
                cx.m.r = cx.m.g = cx.m.b = rho.v[k];
                const float rk = spectral::evalCoef(scatter, w.lam(k));
                cx.m.scatterR = cx.m.scatterG = cx.m.scatterB = rk;
                f.v[k] = bsdfEval(cx, wi).x;
            }
            cx.m.r = 0.0f;
            cx.m.g = cx.m.b = 1.0f;
            cx.m.scatterR = sr;
            cx.m.scatterG = sg;
            cx.m.scatterB = sb;
        } else {
            const float3 e = bsdfEval(cx, wi);
            const float b = e.y - e.x;
#pragma unroll
            for (int k = 0; k < NW; ++k) {
                f.v[k] = e.x + b * rho.v[k];
            }
        }
    }
    return f;
}

template <int NW>
__device__ __forceinline__ Col<NW> throughCol(const Col<NW>& T, const Ctx& cx, const BsdfSample& smp, const Col<NW>& f,
    const Col<NW>& rho)
{
    Col<NW> r;
    if constexpr (NW == 0) {
        (void)rho;
        r.c = applyThroughput(T.c, cx, smp, f.c);
    } else {
        float k;
        bool tint;
        if (!throughputFactor(cx, smp, k, tint)) {
            return czero<NW>();
        }
#pragma unroll
        for (int j = 0; j < NW; ++j) {
            float sc = f.v[j] * k;
            if (tint) {
                sc = sc * rho.v[j];
            }
            r.v[j] = T.v[j] * sc;
        }
    }
    return r;
}

// Russian-roulette weight of a throughput: Rec. 709 luminance (RGB), the mean
// over the wavelengths (spectral).
template <int NW> __device__ __forceinline__ float pathWeight(const Col<NW>& T)
{
    if constexpr (NW == 0) {
        return lum709(T.c);
    } else {
        float s = 0.0f;
#pragma unroll
        for (int k = 0; k < NW; ++k) {
            s += T.v[k];
        }
        return s * (1.0f / static_cast<float>(NW));
    }
}

template <int NW>
__device__ __forceinline__ void writeSample(const LaunchCtx& c, uint32_t i, const Col<NW>& Lc, const Waves<NW>& w)
{
    float3 L;
    if constexpr (NW == 0) {
        (void)w;
        L = Lc.c;
    } else {
        // hero-wavelength estimate of linear sRGB: each wavelength is uniform
        // over the range, so sum_k L_k resp(lambda_k) (range / NW); a zero
        // spectrum (a path that left a black scene) gives exactly 0
        L = f3(0.0f, 0.0f, 0.0f);
        if (cnonzero(Lc)) {
            float3 a = f3(0.0f, 0.0f, 0.0f);
#pragma unroll
            for (int k = 0; k < NW; ++k) {
                a = add3(a, scl3(spectral::responseAt(c.specResp, w.lam(k)), Lc.v[k]));
            }
            L = scl3(a, spectral::kLambdaRange / static_cast<float>(NW));
        }
    }
    const uint32_t o = c.paths.outIdx[i];
    const float3 s = NW == 0 ? clampFirefly(L) : clampFireflySigned(L);
    c.acc.samples[o] = make_float4(s.x, s.y, s.z, 1.0f);
    if (c.record != nullptr) {
        // sample index = samples the pixel had at batch start + the job's slot
        const uint32_t pixel = c.paths.pixel[i];
        const uint32_t k = c.acc.counts[pixel] + o / static_cast<uint32_t>(c.q.batch->activeCount);
        if (k < static_cast<uint32_t>(c.recordSpp)) {
            c.record[static_cast<size_t>(k) * static_cast<size_t>(c.width) * static_cast<size_t>(c.height) + pixel] =
                make_float4(L.x, L.y, L.z, 0.0f);
        }
    }
}

// Camera path for job j of the current batch (PathTracer.cu:69-96): job
// j = slot * activeCount + listIndex draws sample `counts[pixel] + slot` of
// pixel active[listIndex] with the reference seed for wave waveBase + slot.
template <int NW> __device__ __forceinline__ void initPath(const LaunchCtx& c, uint32_t i, unsigned long long j)
{
    const BatchInfo& bt = *c.q.batch;
    const int activeCount = bt.activeCount;
    const int* active = c.acc.active[c.activeSel];
    int li;
    uint32_t slot;
    uint32_t local;
    const pt_camera* cam = &c.cam;
    uint32_t width = static_cast<uint32_t>(c.width), height = static_cast<uint32_t>(c.height);
    uint32_t pixel;
    if (c.sceneCount > 1) {
        // scene-major job order: all of a scene's jobs before the next scene's,
        // so that the paths in flight share few scenes' geometry
        int lo = 0, hi = c.sceneCount - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (c.sceneJobStart[mid] <= j) {
                lo = mid;
            } else {
                hi = mid - 1;
            }
        }
        const uint32_t a0 = c.sceneActiveStart[lo];
        const uint32_t n = c.sceneActiveStart[lo + 1] - a0;
        const unsigned long long q = j - c.sceneJobStart[lo];
        slot = static_cast<uint32_t>(q / n);
        li = static_cast<int>(a0 + static_cast<uint32_t>(q % n));
        pixel = static_cast<uint32_t>(active[li]);
        const SceneView& sv = c.views[lo];
        // seeds and film coordinates use the pixel's index within its own
        // image, so a scene renders the same in a batch as alone
        local = pixel - sv.pixelBase;
        cam = &sv.cam;
        width = static_cast<uint32_t>(sv.width);
        height = static_cast<uint32_t>(sv.height);
        c.paths.scene[i] = static_cast<uint16_t>(lo);
    } else {
        li = static_cast<int>(j % static_cast<unsigned long long>(activeCount));
        slot = static_cast<uint32_t>(j / static_cast<unsigned long long>(activeCount));
        pixel = static_cast<uint32_t>(active[li]);
        local = pixel;
    }
    const uint32_t sampleIndex = c.acc.counts[pixel] + slot;
    const uint32_t globalSeed = bt.waveBase + slot + 1u + static_cast<uint32_t>(c.seedOffset);
    curandStateXORWOW st;
    const uint32_t seed = pathSeed(c.params, local, width, sampleIndex, globalSeed);
    curand_init(seed, 0ull, 0ull, &st);
    const uint32_t x = local % width, y = local / width;
    const float ju = curand_uniform(&st);
    const float jv = curand_uniform(&st);
    const float u = (static_cast<float>(x) + ju) / static_cast<float>(width);
    const float v = (static_cast<float>(y) + jv) / static_cast<float>(height);
    const float l1 = curand_uniform(&st);
    const float l2 = curand_uniform(&st);
    float3 ro, rd;
    cameraRay(*cam, u, v, l1, l2, ro, rd);
    c.paths.pixel[i] = pixel;
    c.paths.outIdx[i] = slot * static_cast<uint32_t>(activeCount) + static_cast<uint32_t>(li);
    rngStore(c.paths, i, st);
    c.paths.orig[i] = make_float4(ro.x, ro.y, ro.z, 0.0f);
    c.paths.dir[i] = make_float4(rd.x, rd.y, rd.z, 0.0f);
    // The throughput, radiance, depth and next-event flags of a path at depth 0
    // are 1, 0, 0 and clear: the whole first launch of a generation is at depth 0
    // and they are not stored (generation is bound by its writes: 16.7M paths
    // 329 -> 281 us).
    if constexpr (NW > 0) {
        c.paths.hero[i] = spectral::heroU(seed);
    }
}

// Path i joins the next bounce's extend queue: marked for listMarked in
// slot-ordered mode, else pushed (one atomic per warp).
__device__ __forceinline__ void queueNext(const LaunchCtx& c, uint32_t i, unsigned int* nextCount, uint32_t* nextQueue)
{
    if (c.q.nextFlag != nullptr) {
        c.q.nextFlag[i] = 1;
    } else {
        const uint32_t s = warpPush(nextCount);
        nextQueue[s] = i;
    }
}

// Jobs jobOffset .. jobOffset + count - 1 of a batch into slots 0..count-1
// (extend queue = identity).
template <int NW>
__global__ void __launch_bounds__(256) k_generate(const LaunchCtx* __restrict__ cp, int count, int extendSel,
    unsigned long long jobOffset)
{
    const LaunchCtx& c = *cp;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        c.q.counts[extendSel] = static_cast<unsigned int>(count);
        c.q.counts[extendSel ^ 1] = 0u;
        c.q.counts[2] = 0u;
        c.q.counts[3] = 0u;
        c.q.counts[4] = 0u;
        c.q.counts[5] = 0u;
        c.q.counts[8] = 0u;  // fetch counters of the first extend and shadow stages
        c.q.counts[10] = 0u;
        c.q.counts[12] = 0u; // Q1 mark of the first extend stage
        c.acc.activeCount[1] = 0; // pixels that go on after the batch (k_accumulate)
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < count; i += gridDim.x * blockDim.x) {
        initPath<NW>(c, static_cast<uint32_t>(i), jobOffset + static_cast<unsigned long long>(i));
        if (c.q.nextFlag != nullptr) {
            c.q.nextFlag[i] = 0; // (a mark that a failed render left)
        }
    }
}

// Closest hit for every queued path; each path is then routed to the miss or
// the hit queue of this bounce so that the two shade kernels run coherent work.
// Counters: [4 + 2p] misses and [5 + 2p] hits of bounce parity p; this kernel
// zeroes the other parity's pair for the next bounce.
template <bool Count, bool Inst>
#ifndef PT_EXTEND_MIN_BLOCKS
#define PT_EXTEND_MIN_BLOCKS 4
#endif
__global__ void __launch_bounds__(256, PT_EXTEND_MIN_BLOCKS) k_extend(const LaunchCtx* __restrict__ cp, int sel, bool identity, int iter)
{
    const LaunchCtx& c = *cp;
    extern __shared__ uint2 smemStack[];
    const unsigned int count = c.q.counts[sel];
    const int par = iter & 1;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(&c.q.rays[0], static_cast<unsigned long long>(count));
        // output counters of the shade stage that follows, and next bounce's routing counters
        c.q.counts[sel ^ 1] = 0u;
        c.q.counts[2] = 0u;
        c.q.counts[3] = 0u;
        c.q.counts[4 + 2 * (par ^ 1)] = 0u;
        c.q.counts[5 + 2 * (par ^ 1)] = 0u;
        c.q.counts[8 + (par ^ 1)] = 0u; // next extend's fetch counter
    }
    const uint32_t* queue = c.q.extend[sel];
    unsigned int* fetch = &c.q.counts[8 + par];
    for (;;) {
        const unsigned int k = warpFetch(fetch);
        if (__shfl_sync(0xffffffffu, k, 0) >= count) {
            break;
        }
        if (k >= count) {
            continue;
        }
        const uint32_t i = identity ? k : queue[k];
        const float4 o4 = c.paths.orig[i];
        const float4 d4 = c.paths.dir[i];
        const float3 dn = xnormalize(f3(d4.x, d4.y, d4.z));
        HitRec h;
        const DevScene& S = sceneOf(c, i);
        const bool hit = traceRay<false, Count, Inst>(S, f3(o4.x, o4.y, o4.z), dn, o4.w, kRayTMax, h, c.q.overflow,
            c.q.visits, smemStack + threadIdx.x, blockDim.x);
        if (hit) {
            c.paths.hit[i] = make_float4(h.t, h.u, h.v, __uint_as_float(h.tri));
            if (Inst && S.instanceCount > 0) {
                c.paths.hitInst[i] = h.inst;
            }
            const uint32_t s = warpPush(&c.q.counts[5 + 2 * par]);
            c.q.hitQueue[s] = i;
        } else {
            const uint32_t s = warpPush(&c.q.counts[4 + 2 * par]);
            c.q.missQueue[s] = i;
        }
    }
}

#ifndef PT_EXTEND_LANE_MIN_BLOCKS
#define PT_EXTEND_LANE_MIN_BLOCKS 6
#endif
#ifndef PT_SHADOW_LANE_MIN_BLOCKS
#define PT_SHADOW_LANE_MIN_BLOCKS 7
#endif

// Closest hit of every queued path by the whole-warp traversal.  The result of
// queue entry k goes back into entry k (path index, bit 31 set for a miss, bit
// 30 for a ray of quirk Q1, which k_route traces: its call would cost this
// kernel registers) and k_route splits the queue into the miss and hit queues
// in queue order afterwards.
template <bool Inst, bool Multi>
__global__ void __launch_bounds__(kTraceThreads, PT_EXTEND_LANE_MIN_BLOCKS)
    k_extend_lane(const LaunchCtx* __restrict__ cp, int sel, bool identity, int iter)
{
    const LaunchCtx& c = *cp;
    extern __shared__ float4 traceSmem[];
    WarpTrace<Inst>& W = reinterpret_cast<WarpTrace<Inst>*>(traceSmem)[threadIdx.x >> 5];
    const unsigned int count = c.q.counts[sel];
    const int par = iter & 1;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(&c.q.rays[0], static_cast<unsigned long long>(count));
        c.q.counts[sel ^ 1] = 0u;
        c.q.counts[2] = 0u;
        c.q.counts[3] = 0u;
        c.q.counts[4 + 2 * (par ^ 1)] = 0u;
        c.q.counts[5 + 2 * (par ^ 1)] = 0u;
        c.q.counts[8 + (par ^ 1)] = 0u;
        c.q.counts[12 + (par ^ 1)] = 0u;
    }
    uint32_t* queue = c.q.extend[sel];
    warpTraversal<false, Inst, Multi>(c.scene, count, &c.q.counts[8 + par], W, c.q.overflow,
        [&](unsigned int k, LaneRay& r, uint32_t& i) -> bool {
            i = identity ? k : queue[k];
            r.S = Multi ? &sceneOf(c, i) : &c.scene;
            const float4 o4 = c.paths.orig[i];
            const float4 d4 = c.paths.dir[i];
            r.o = f3(o4.x, o4.y, o4.z);
            r.tMin = o4.w;
            r.tMax = kRayTMax;
            r.dn = xnormalize(f3(d4.x, d4.y, d4.z));
            if ((Inst && r.S->instanceCount > 0) || (r.S->nodeCount != 0 && !isDegenerateDir(r.dn))) {
                return true;
            }
            // empty scene: a miss; quirk Q1: left to k_route
            if (r.S->nodeCount != 0) {
                queue[k] = i | 0x40000000u;
                c.q.counts[12 + par] = 1u;
            } else {
                queue[k] = i | 0x80000000u;
            }
            return false;
        },
        [&](unsigned int k, uint32_t i, bool hit, float t, float u, float v, uint32_t tri, uint32_t inst) {
            if (hit) {
                c.paths.hit[i] = make_float4(t, u, v, __uint_as_float(tri));
                if (Inst) {
                    c.paths.hitInst[i] = inst;
                }
            }
            queue[k] = hit ? i : (i | 0x80000000u);
        });
}

// Occlusion of every queued shadow ray by the whole-warp traversal (any hit
// below the ray's tMax); unoccluded rays mark their path's pending NEE
// contribution visible.
template <bool Inst, bool Multi>
__global__ void __launch_bounds__(kTraceThreads, PT_SHADOW_LANE_MIN_BLOCKS)
    k_shadow_lane(const LaunchCtx* __restrict__ cp, int iter)
{
    const LaunchCtx& c = *cp;
    extern __shared__ float4 traceSmem[];
    WarpTrace<Inst>& W = reinterpret_cast<WarpTrace<Inst>*>(traceSmem)[threadIdx.x >> 5];
    const unsigned int count = c.q.counts[2];
    const int par = iter & 1;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(&c.q.rays[1], static_cast<unsigned long long>(count));
        c.q.counts[10 + (par ^ 1)] = 0u; // next shadow stage's fetch counter
    }
    auto visible = [&](uint32_t e) {
        const uint32_t i = e & 0x7FFFFFFFu;
        if (e & 0x80000000u) {
            c.paths.visEmis[i] = 1;
        } else {
            c.paths.visEnv[i] = 1;
        }
    };
    warpTraversal<true, Inst, Multi>(c.scene, count, &c.q.counts[10 + par], W, c.q.overflow,
        [&](unsigned int k, LaneRay& r, uint32_t& e) -> bool {
            e = c.q.shadowPath[k];
            r.S = Multi ? &sceneOf(c, e & 0x7FFFFFFFu) : &c.scene;
            const float4 o4 = c.q.shadowOrig[k];
            const float4 d4 = c.q.shadowDir[k];
            r.o = f3(o4.x, o4.y, o4.z);
            r.dn = xnormalize(f3(d4.x, d4.y, d4.z));
            r.tMin = kShadowBias;
            r.tMax = d4.w > 0.0f ? d4.w : kRayTMax; // emitter MIS rays end short of the light
            if (Inst && r.S->instanceCount > 0) {
                return true;
            }
            bool occluded = false;
            if (r.S->nodeCount != 0) {
                if (!isDegenerateDir(r.dn)) {
                    return true;
                }
                HitRec h;
                occluded = traceQ1(*r.S, r.o, r.dn, r.tMin, r.tMax, true, h, c.q.overflow);
            }
            if (!occluded) {
                visible(e);
            }
            return false;
        },
        [&](unsigned int, uint32_t e, bool occluded, float, float, float, uint32_t, uint32_t) {
            if (!occluded) {
                visible(e);
            }
        });
}

// Closest hit of a ray with a degenerate direction (quirk Q1); its queue entry.
static __device__ __noinline__ uint32_t routeQ1(const LaunchCtx& c, uint32_t i)
{
    const DevScene& S = sceneOf(c, i);
    const float4 o4 = c.paths.orig[i];
    const float4 d4 = c.paths.dir[i];
    HitRec h;
    if (!traceQ1(S, f3(o4.x, o4.y, o4.z), xnormalize(f3(d4.x, d4.y, d4.z)), o4.w, kRayTMax, false, h, c.q.overflow)) {
        return i | 0x80000000u;
    }
    c.paths.hit[i] = make_float4(h.t, h.u, h.v, __uint_as_float(h.tri));
    return i;
}

// Splits the queue that k_extend_lane marked into the miss and hit queues of
// this bounce.  Every warp takes one contiguous part of the queue, counts its
// hits, the block reserves both output ranges with one atomic each, and the
// warp reads its part again and writes it in order.  Bound by the atomics when
// a tile of 2048 entries had two of its own (they serialise on one address,
// about 10 ns each): 16.7M entries 162 -> 56 us, below 1M entries unchanged.
constexpr int kListThreads = 256;
constexpr int kListWarps = kListThreads / 32;
constexpr int kRouteRows = 8; // loads in flight per lane

__global__ void __launch_bounds__(kListThreads) k_route(const LaunchCtx* __restrict__ cp, int sel, int iter)
{
    const LaunchCtx& c = *cp;
    const unsigned int count = c.q.counts[sel];
    const int par = iter & 1;
    uint32_t* queue = c.q.extend[sel];
    __shared__ unsigned int sHit[kListWarps], sMiss[kListWarps]; // counts, then first output positions
    const unsigned int lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned int below = (1u << lane) - 1u;
    const unsigned int warps = gridDim.x * kListWarps;
    const unsigned int part = ((count + warps - 1u) / warps + 31u) & ~31u;
    if (blockIdx.x * kListWarps * part >= count) {
        return;
    }
    const unsigned int first = min((blockIdx.x * kListWarps + warp) * part, count), last = min(first + part, count);
    if (c.q.counts[12 + par] != 0u) {
        for (unsigned int k = first + lane; k < last; k += 32u) {
            if ((queue[k] & 0x40000000u) != 0u) {
                queue[k] = routeQ1(c, queue[k] & 0x3FFFFFFFu);
            }
        }
    }
    // (a lane reads the entries that it wrote)
    unsigned int hits = 0;
#pragma unroll kRouteRows
    for (unsigned int k = first + lane; k < last; k += 32u) {
        hits += 1u - (queue[k] >> 31);
    }
    hits = __reduce_add_sync(0xffffffffu, hits);
    if (lane == 0) {
        sHit[warp] = hits;
        sMiss[warp] = last - first - hits;
    }
    __syncthreads();
    if (warp == 0) {
        const unsigned int h = lane < kListWarps ? sHit[lane] : 0u, m = lane < kListWarps ? sMiss[lane] : 0u;
        unsigned int hs = h, ms = m;
#pragma unroll
        for (int d = 1; d < kListWarps; d <<= 1) {
            const unsigned int ho = __shfl_up_sync(0xffffffffu, hs, d);
            const unsigned int mo = __shfl_up_sync(0xffffffffu, ms, d);
            if (lane >= static_cast<unsigned int>(d)) {
                hs += ho;
                ms += mo;
            }
        }
        // (the last warp's lane holds the totals)
        unsigned int hb = 0, mb = 0;
        if (lane == kListWarps - 1) {
            hb = hs != 0u ? atomicAdd(&c.q.counts[5 + 2 * par], hs) : 0u;
            mb = ms != 0u ? atomicAdd(&c.q.counts[4 + 2 * par], ms) : 0u;
        }
        hb = __shfl_sync(0xffffffffu, hb, kListWarps - 1);
        mb = __shfl_sync(0xffffffffu, mb, kListWarps - 1);
        if (lane < kListWarps) {
            sHit[lane] = hb + hs - h;
            sMiss[lane] = mb + ms - m;
        }
    }
    __syncthreads();
    unsigned int hitAt = sHit[warp], missAt = sMiss[warp];
    for (unsigned int k0 = first; k0 < last; k0 += 32u * kRouteRows) {
        uint32_t e[kRouteRows];
#pragma unroll
        for (int r = 0; r < kRouteRows; ++r) {
            const unsigned int k = k0 + static_cast<unsigned int>(r) * 32u + lane;
            e[r] = k < last ? queue[k] : 0u;
        }
#pragma unroll
        for (int r = 0; r < kRouteRows; ++r) {
            const bool valid = k0 + static_cast<unsigned int>(r) * 32u + lane < last;
            const bool miss = (e[r] >> 31) != 0u;
            const unsigned int hm = __ballot_sync(0xffffffffu, valid && !miss);
            const unsigned int mm = __ballot_sync(0xffffffffu, valid && miss);
            if (valid) {
                if (miss) {
                    c.q.missQueue[missAt + __popc(mm & below)] = e[r] & 0x7FFFFFFFu;
                } else {
                    c.q.hitQueue[hitAt + __popc(hm & below)] = e[r];
                }
            }
            hitAt += __popc(hm);
            missAt += __popc(mm);
        }
    }
}

// Slot-ordered mode: lists the slots the shade kernels marked (bytes of 0 or
// 1) as the next bounce's extend queue and clears the marks.  Every warp takes
// one contiguous range of slots, 16 marks per load, as in k_route, so that the
// extend and shade kernels read the path state of consecutive slots.  One mark
// per load kept 8 KB per SM in flight: 16.7M slots 78 -> 22 us (69 -> 9 with
// no slot marked).
constexpr unsigned int kMarksPerRow = 512; // slots of one step of a warp
__device__ __forceinline__ uint4 loadMarks(const uint8_t* flag, unsigned int k, unsigned int n)
{
    if (k + 16u <= n) {
        return *reinterpret_cast<const uint4*>(flag + k);
    }
    uint32_t w[4] = {0u, 0u, 0u, 0u};
    for (unsigned int j = 0; k + j < n; ++j) {
        w[j >> 2] |= static_cast<uint32_t>(flag[k + j]) << (8u * (j & 3u));
    }
    return make_uint4(w[0], w[1], w[2], w[3]);
}
__device__ __forceinline__ void listMarked(const LaunchCtx& c, int sel)
{
    const unsigned int n = static_cast<unsigned int>(c.q.batch->slotCount);
    uint8_t* flag = c.q.nextFlag;
    uint32_t* out = c.q.extend[sel ^ 1];
    __shared__ unsigned int sAt[kListWarps]; // counts, then first output positions
    __shared__ uint16_t sSlot[kListWarps][kMarksPerRow];
    const unsigned int lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const unsigned int warps = gridDim.x * kListWarps;
    const unsigned int part = ((n + warps - 1u) / warps + kMarksPerRow - 1u) / kMarksPerRow * kMarksPerRow;
    if (blockIdx.x * kListWarps * part >= n) {
        return;
    }
    const unsigned int first = min((blockIdx.x * kListWarps + warp) * part, n), last = min(first + part, n);
    unsigned int marks = 0;
#pragma unroll 4
    for (unsigned int k = first + 16u * lane; k < last; k += kMarksPerRow) {
        const uint4 v = loadMarks(flag, k, last);
        // (bytes are 0 or 1: the four words' bits do not meet)
        marks += __popc(v.x | (v.y << 1) | (v.z << 2) | (v.w << 3));
    }
    marks = __reduce_add_sync(0xffffffffu, marks);
    if (lane == 0) {
        sAt[warp] = marks;
    }
    __syncthreads();
    if (warp == 0) {
        const unsigned int a = lane < kListWarps ? sAt[lane] : 0u;
        unsigned int s = a;
#pragma unroll
        for (int d = 1; d < kListWarps; d <<= 1) {
            const unsigned int o = __shfl_up_sync(0xffffffffu, s, d);
            if (lane >= static_cast<unsigned int>(d)) {
                s += o;
            }
        }
        unsigned int b = 0;
        if (lane == kListWarps - 1 && s != 0u) {
            b = atomicAdd(&c.q.counts[sel ^ 1], s);
        }
        b = __shfl_sync(0xffffffffu, b, kListWarps - 1);
        if (lane < kListWarps) {
            sAt[lane] = b + s - a;
        }
    }
    __syncthreads();
    if (marks == 0u) {
        return;
    }
    unsigned int at = sAt[warp];
    uint16_t* slots = sSlot[warp];
    for (unsigned int k0 = first; k0 < last; k0 += kMarksPerRow) {
        const unsigned int k = k0 + 16u * lane;
        const uint4 v = k < last ? loadMarks(flag, k, last) : make_uint4(0u, 0u, 0u, 0u);
        const uint32_t w[4] = {v.x, v.y, v.z, v.w};
        const unsigned int own = __popc(v.x | (v.y << 1) | (v.z << 2) | (v.w << 3));
        unsigned int s = own;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned int o = __shfl_up_sync(0xffffffffu, s, d);
            if (lane >= static_cast<unsigned int>(d)) {
                s += o;
            }
        }
        const unsigned int total = __shfl_sync(0xffffffffu, s, 31);
        if (total == 0u) {
            continue;
        }
        unsigned int o = s - own;
#pragma unroll
        for (unsigned int j = 0; j < 16u; ++j) {
            if (((w[j >> 2] >> (8u * (j & 3u))) & 1u) != 0u) {
                slots[o++] = static_cast<uint16_t>(16u * lane + j);
            }
        }
        if (own != 0u) {
            if (k + 16u <= last) {
                *reinterpret_cast<uint4*>(flag + k) = make_uint4(0u, 0u, 0u, 0u);
            } else {
                for (unsigned int j = 0; k + j < last; ++j) {
                    flag[k + j] = 0;
                }
            }
        }
        __syncwarp();
        for (unsigned int q = lane; q < total; q += 32u) {
            out[at + q] = k0 + slots[q];
        }
        __syncwarp(); // the list is rewritten by the next step
        at += total;
    }
}

// A path whose ray left the scene: previous bounce's NEE, then the
// environment / background term (PathIntegratorRandCore.h:215-216, 338-346).
template <int NW> __device__ __forceinline__ void shadeMiss(const LaunchCtx& c, uint32_t i, bool fresh)
{
    const Waves<NW> wv = pathWaves<NW>(c, i);
    const float4 d4 = c.paths.dir[i];
    const float3 d = f3(d4.x, d4.y, d4.z);
    float4 r4 = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(0));
    if (!fresh) {
        if constexpr (NW == 0) {
            r4 = c.paths.rad[i];
        } else {
            r4.w = depthEta(c)[i].x;
        }
    }
    const int depth = __float_as_int(r4.w);
    Col<NW> L;
    const bool sunOn = c.sun.enabled != 0;
    const bool black = skyIsBlack<NW>(c); // (adds exactly nothing)
    if (depth == 0) {
        L = black ? czero<NW>() : sunOn ? skyCol<NW>(c, d, wv) : envCol<NW>(c, d, wv);
    } else {
        L = loadCol<NW>(r4, c.paths.radS, c.paths.capacity, i);
        if (c.paths.visEnv[i]) {
            L = cadd(L, pendingEnv<NW>(c, i));
        }
        if (c.paths.visEmis[i]) {
            L = cadd(L, pendingEmis<NW>(c, i));
        }
        if (!black) {
            const Col<NW> T = loadCol<NW>(NW == 0 ? c.paths.thr[i] : r4, c.paths.thrS, c.paths.capacity, i);
            const Col<NW> Le = sunOn ? skyCol<NW>(c, d, wv) : envCol<NW>(c, d, wv);
            const float lp = sunOn ? skyPdf(c, d) : envPdf(c.env, d);
            const float w = misBalance(fabsf(d4.w), lp);
            L = cadd(L, cmul(T, cscl(Le, w)));
        }
    }
    writeSample<NW>(c, i, L, wv);
}

// Shading of the paths that hit a triangle, then of those that left the scene.
// One thread per queued path.  fresh: every path is at depth 0, where the state
// that initPath leaves out is known.  (The misses in this launch and not in one of
// their own: they start in the blocks that the hits leave idle, and a bounce of
// few paths has one launch less: 4 waves of 1024^2 pixels 7.1 -> 6.97 ms with the
// merged listing pass below.)
//
// Bound by instruction fetch: a path runs through about 30 KB of straight-line
// code (the kernel has 170 - 230 KB), and with warps spread over it a third of
// the stalls were fetches (issue slots 31% used, DRAM 26%; prefetching the next
// path's state into shared memory changed nothing).  So the block's warps are
// kept in phase by a barrier before each of the stretches below, and a block
// is large: 16 warps share what one of them fetches.  Measured: hit shading of
// the large frame (972k triangles, 1024^2, 256 spp, 8 wavelengths) 85.3 ms
// without barriers, 68.5 with one per path, 64.7 with one at 512 threads, 60.6
// with three (60.4 with five, which costs the forest view 4%); RGB: 6-tree
// batch 11.3 -> 8.5 ms, zoo under a sky 4.9 -> 3.6 ms.
constexpr int kShadeThreads = 512;
#ifndef PT_SHADE_MIN_BLOCKS
// (64 registers: at 3/4 of the warps and 80 registers the dependent loads of
// path state and materials are hidden less than the spills cost)
#define PT_SHADE_MIN_BLOCKS 2
#endif
template <int NW>
__global__ void __launch_bounds__(kShadeThreads, PT_SHADE_MIN_BLOCKS)
    k_shade(const LaunchCtx* __restrict__ cp, int sel, int iter, bool fresh)
{
    const LaunchCtx& c = *cp;
    const unsigned int count = c.q.counts[5 + 2 * (iter & 1)];
    const uint32_t* queue = c.q.hitQueue;
    unsigned int* nextCount = &c.q.counts[sel ^ 1];
    uint32_t* nextQueue = c.q.extend[sel ^ 1];
    const int debugFlags = c.params.brdf_debug_flags;
    const int cap = c.paths.capacity;
    __shared__ float4 sRad[NW == 0 ? 1 : NW / 4][kShadeThreads]; // a thread's own column
    // (the whole block runs the loop: barriers)
    for (unsigned int base = blockIdx.x * blockDim.x; base < count; base += gridDim.x * blockDim.x) {
        const unsigned int k = base + threadIdx.x;
        const bool valid = k < count;
        bool live = false; // hit below the depth limit
        uint32_t i = 0u;
        const DevScene* scene = &c.scene;
        Waves<NW> wv{};
        int depth = 0;
        Col<NW> L, T, rho;
        float4 r4, scatterCoef;
        float3 d, pos, n;
        float t = 0.0f, eta = 1.0f;
        Ctx cx;
        bool emitterMis = false, misVertex = false;
        bool pendEnv = false, pendEmis = false;
        bool visEnv = false, visEmis = false; // next-event terms of the previous bounce
        bool cont = false;
        curandStateXORWOW st;
        __syncthreads();
        if (valid) {
            i = queue[k];
            scene = &sceneOf(c, i);
            wv = pathWaves<NW>(c, i);
            r4 = make_float4(0.0f, 0.0f, 0.0f, __int_as_float(0));
            if (!fresh) {
                if constexpr (NW == 0) {
                    r4 = c.paths.rad[i];
                } else {
                    const float2 de = depthEta(c)[i];
                    r4.w = de.x;
                    eta = de.y;
                }
            }
            visEnv = !fresh && c.paths.visEnv[i] != 0;
            visEmis = !fresh && c.paths.visEmis[i] != 0;
            depth = __float_as_int(r4.w);
            // RGB: the radiance stays in registers through the bounce.  Spectral: it
            // waits in shared memory once the NEE of the previous bounce and the
            // emission are added.
            L = czero<NW>();
            if constexpr (NW == 0) {
                L = loadCol<NW>(r4, c.paths.radS, cap, i);
                // NEE contributions of the previous bounce, in the reference's order
                // (the flags are clear for a path that starts at this bounce).
                if (visEnv) {
                    L = cadd(L, pendingEnv<NW>(c, i));
                }
                if (visEmis) {
                    L = cadd(L, pendingEmis<NW>(c, i));
                }
            }
            live = depth < c.maxDepth;
        }
        const DevScene& S = *scene;
        if (live) {
            const float4 h4 = c.paths.hit[i];
            const uint32_t tri = __float_as_uint(h4.w);
            const float4 d4 = c.paths.dir[i];
            d = f3(d4.x, d4.y, d4.z);
            const float4 o4 = c.paths.orig[i];
            const float4 t4 = fresh ? make_float4(1.0f, 1.0f, 1.0f, 1.0f) : NW == 0 ? c.paths.thr[i] : make_float4(1.0f, 1.0f, 1.0f, eta);
            if constexpr (NW == 0) {
                T = loadCol<NW>(t4, c.paths.thrS, cap, i);
            } else {
                if (depth == 0) {
#pragma unroll
                    for (int q = 0; q < NW; ++q) {
                        T.v[q] = 1.0f;
                    }
                } else {
                    T = loadCol<NW>(t4, c.paths.thrS, cap, i);
                }
            }
            eta = t4.w;
            t = h4.x;
            pos = xadd(f3(o4.x, o4.y, o4.z), xscl(d, t));
            const float3 dn = xnormalize(d);
            const TriShade sh = S.shade[tri];
            float tu, tv;
            if (S.instanceCount == 0) {
                hitShading(sh, dn, h4.y, h4.z, n, tu, tv);
            } else {
                hitShadingAt(S, sh, c.paths.hitInst[i], dn, h4.y, h4.z, n, tu, tv);
            }
            const uint32_t mi = __float_as_uint(sh.d.w);
            const pt_material& srcMat =
                (S.materials != nullptr && mi < S.materialCount) ? S.materials[mi] : kFallbackMaterial;
            cx.m = resolveMaterial(srcMat, tu, tv, S.textures, S.textureCount);
            cx.w = computeLobes(cx.m);
            cx.n = n;
            cx.wo = scl3(d, -1.0f);
            cx.eta = eta;
            cx.debug = 0;
            // Emitter MIS mode: at a vertex that takes part (emitterMisVertex), the
            // emissive NEE and the BSDF-sampled emitter hits share the light by the
            // balance heuristic, outside the transmit cones and above the surface;
            // elsewhere the reference's estimator is kept.
            emitterMis = c.params.emitter_mis == 1;
            misVertex = emitterMis && S.instanceCount == 0 && debugFlags == 0 && emitterMisVertex(cx);
            // weight of this hit's emission: the previous vertex took part (pdf > 0) and
            // emissive NEE can pick this point (front face of a listed emitter)
            float emitW = 1.0f;
            if (emitterMis && depth > 0 && d4.w > 0.0f && S.emitPdfArea != nullptr && cx.m.emission != 0.0f) {
                const float pa = S.emitPdfArea[tri];
                if (pa > 0.0f) {
                    const float3 ev0 = loadOrigVertex(S, tri, 0), ev1 = loadOrigVertex(S, tri, 1),
                                 ev2 = loadOrigVertex(S, tri, 2);
                    const float3 ng = normalize3(cross3(sub3(ev1, ev0), sub3(ev2, ev0)));
                    const float cl = fmax2(0.0f, -dot3(ng, dn));
                    if (cl > 0.0f) {
                        const float lp = pa * (t * t * dot3(d, d)) / cl;
                        emitW = misBalance(d4.w, lp);
                    }
                }
            }
            const float emission = cx.m.emission * emitW;
            // base colour at the path's wavelengths (spectral mode)
            scatterCoef = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if constexpr (NW == 0) {
                rho.c = f3(cx.m.r, cx.m.g, cx.m.b);
                // emission (PathIntegratorRandCore.h:248)
                L = cadd(L, cmul(T, Col<0>{f3(cx.m.r * emission, cx.m.g * emission, cx.m.b * emission)}));
            } else {
                float4 baseCoef;
                matCoefs(S, mi, srcMat, tu, tv, baseCoef, scatterCoef);
                rho = coefCol<NW>(baseCoef, wv);
                cx.m.r = 0.0f; // evalCol's affine form (the RGB base is not read again)
                cx.m.g = 1.0f;
                cx.m.b = 1.0f;
                Col<NW> Lm = depth == 0 ? czero<NW>() : loadCol<NW>(r4, c.paths.radS, cap, i);
                if (visEnv) {
                    Lm = cadd(Lm, pendingEnv<NW>(c, i));
                }
                if (visEmis) {
                    Lm = cadd(Lm, pendingEmis<NW>(c, i));
                }
                // emission (PathIntegratorRandCore.h:248)
#pragma unroll
                for (int q = 0; q < NW; ++q) {
                    Lm.v[q] = Lm.v[q] + T.v[q] * (rho.v[q] * emission);
                }
                storeCol<NW>(nullptr, &sRad[0][threadIdx.x], kShadeThreads, 0u, Lm, 0.0f);
            }
            rngLoad(c.paths, i, st);
        }
        __syncthreads();
        if (live) {
            // environment NEE (PathIntegratorRandCore.h:65-108); with a distant
            // light, one more draw first picks the light or the environment
            if (!skipsEnvNee(cx.m)) {
                const bool sunOn = c.sun.enabled != 0;
                const float uSel = sunOn ? curand_uniform(&st) : 0.0f;
                const float u1 = curand_uniform(&st);
                const float u2 = curand_uniform(&st);
                float lp = 0.0f;
                float3 wi = f3(0.0f, 0.0f, 0.0f);
                if (skyIsBlack<NW>(c)) {
                    // (a light of exactly zero radiance adds nothing, whatever its sample)
                } else if (!sunOn) {
                    wi = envSample(c.env, u1, u2, lp);
                } else if (uSel < c.sun.select) {
                    wi = sunSample(c.sun, u1, u2);
                    lp = skyPdf(c, wi);
                } else {
                    wi = envSample(c.env, u1, u2, lp);
                    lp = lp > kMinPdf ? skyPdf(c, wi) : 0.0f;
                }
                if (lp > kMinPdf) {
                    const float ct = fmax2(0.0f, dot3(n, wi));
                    const Col<NW> Le = sunOn ? skyCol<NW>(c, wi, wv) : envCol<NW>(c, wi, wv);
                    // A light of exactly zero radiance (a black background) contributes
                    // exactly zero for any finite BSDF value: the BSDF is not evaluated.
                    if (ct > 0.0f && cnonzero(Le)) {
                        const Col<NW> f = evalCol<NW>(cx, wi, rho, scatterCoef, wv);
                        const float bp = bsdfPdf(cx, wi);
                        const float kw = misBalance(lp, bp) * ct / lp;
                        const Col<NW> contrib = cmul(T, cmul(f, cscl(Le, kw)));
                        // A contribution of exactly zero adds nothing whether or not the light
                        // is occluded, so its shadow ray is not traced (black backgrounds).
                        if (cnonzero(contrib)) {
                            storeCol<NW>(c.paths.neeEnv, c.paths.neeEnvS, cap, i, contrib, 0.0f);
                            const uint32_t s = warpPush(&c.q.counts[2]);
                            const float3 so = add3(pos, scl3(n, kShadowBias));
                            c.q.shadowPath[s] = i;
                            c.q.shadowOrig[s] = make_float4(so.x, so.y, so.z, 0.0f);
                            c.q.shadowDir[s] = make_float4(wi.x, wi.y, wi.z, 0.0f);
                            pendEnv = true;
                        }
                    }
                }
            }
        }
        if (live) {
            // emissive NEE (PathIntegratorRandCore.h:110-167)
            if (S.emissiveCount > 0) {
                const float uTri = curand_uniform(&st);
                const float u1 = curand_uniform(&st);
                const float u2 = curand_uniform(&st);
                float3 lpos, ln, LeRgb, ev0, ev1, ev2;
                float ap;
                uint32_t etri = 0u;
                if (sampleEmissive(S, &kFallbackMaterial, uTri, u1, u2, lpos, ln, LeRgb, ap, ev0, ev1, ev2, &etri)) {
                    const float3 tl = sub3(lpos, pos);
                    const float d2 = dot3(tl, tl);
                    if (d2 > kMinPdf) {
                        const float3 wi = normalize3(tl);
                        const float ct = fmax2(0.0f, dot3(n, wi));
                        const float cl = fmax2(0.0f, dot3(ln, scl3(wi, -1.0f)));
                        if (ct > 0.0f && cl > 0.0f) {
                            const float lp = ap * d2 / cl;
                            // The reference's emissive shadow ray runs to tMax = 1e6
                            // (LightSamplingCore.h:360-369), so the sampled emitter triangle
                            // itself occludes it whenever the ray hits that triangle.  An
                            // any-hit query is true as soon as one triangle is hit, so testing
                            // the emitter first (same origin, direction and rounding as the
                            // shadow stage) decides those rays without a traversal -- and
                            // without evaluating the BSDF for a term that adds nothing.
                            const float3 so = add3(pos, scl3(wi, kShadowBias));
                            const float3 sdn = xnormalize(wi);
                            bool occludedBySelf = false;
                            // emitter MIS: the shadow ray ends just short of the light
                            // sample, so the emitter (and coplanar neighbours) never block it
                            float shadowTMax = 0.0f; // 0: the reference's kRayTMax
                            if (misVertex && !inTransmitCones(cx, wi)) {
                                shadowTMax = (sqrtf(d2) - kShadowBias) * (1.0f - 1.0e-4f);
                            } else if (!isDegenerateDir(sdn)) {
                                float th, tu2, tv2;
                                occludedBySelf = intersectTriExact(so, sdn, ev0, ev1, ev2, kShadowBias, kRayTMax, th,
                                                     tu2, tv2) && th < kRayTMax;
                            }
                            if (lp > kMinPdf && !occludedBySelf) {
                                Col<NW> Le;
                                if constexpr (NW == 0) {
                                    Le.c = LeRgb;
                                } else {
                                    // the emitter's own material colour (no texture), as sampleEmissive
                                    const uint32_t emi = __float_as_uint(S.shade[etri].d.w);
                                    const bool ok = S.matSpec != nullptr && S.materials != nullptr &&
                                        emi < S.materialCount;
                                    const float4 q = ok ? S.matSpec[2 * emi] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                                    const float em = ok ? S.materials[emi].emission : 0.0f;
                                    Le = cscl(coefCol<NW>(q, wv), em);
                                }
                                const Col<NW> f = evalCol<NW>(cx, wi, rho, scatterCoef, wv);
                                const float bp = bsdfPdf(cx, wi);
                                const float kw = misBalance(lp, bp) * ct / lp;
                                const Col<NW> contrib = cmul(T, cmul(f, cscl(Le, kw)));
                                if (cnonzero(contrib)) {
                                    storeCol<NW>(c.paths.neeEmis, c.paths.neeEmisS, cap, i, contrib, 0.0f);
                                    const uint32_t s = warpPush(&c.q.counts[2]);
                                    c.q.shadowPath[s] = i | 0x80000000u;
                                    c.q.shadowOrig[s] = make_float4(so.x, so.y, so.z, 0.0f);
                                    c.q.shadowDir[s] = make_float4(wi.x, wi.y, wi.z, shadowTMax);
                                    pendEmis = true;
                                }
                            }
                        }
                    }
                }
            }
        }
        __syncthreads();
        if (live) {
            // BSDF sample (PathIntegratorRandCore.h:280-321)
            cx.debug = debugFlags;
            const float u1 = curand_uniform(&st);
            const float u2 = curand_uniform(&st);
            const BsdfSample smp = bsdfSample(cx, u1, u2);
            if (smp.valid && !(smp.pdf <= kMinPdf)) {
                const Col<NW> f = evalCol<NW>(cx, smp.dir, rho, scatterCoef, wv);
                T = throughCol<NW>(T, cx, smp, f, rho);
                if (smp.sss && smp.sssSteps > 0) {
                    // subsurface tier B (PathIntegratorRandCore.h:169-204)
                    const float maxR = maxScatter(cx.m);
                    if (maxR > kMinRadius) {
                        for (int stp = 0; stp < smp.sssSteps; ++stp) {
                            (void)curand_uniform(&st);
                            (void)curand_uniform(&st);
                            const float u3 = curand_uniform(&st);
                            const float mfp = maxR * (-logf(fmax2(1.0e-8f, u3)));
                            const float surv = expf(-mfp / maxR);
                            T = cmul(T, cscl(rho, surv));
                        }
                        const float ed = sqrtf(dot3(smp.exitOffset, smp.exitOffset));
                        if (ed > 0.0f) {
                            T = cscl(T, expf(-ed / maxR));
                        }
                    }
                }
                if constexpr (NW == 0) {
                    // debug tint of glass paths (RGB display aid; not applied to spectra)
                    if (debugFlags & kDbgTintGlass) {
                        T.c = smp.transmitted ? mul3(T.c, f3(0.2f, 1.0f, 0.2f)) : mul3(T.c, f3(1.0f, 0.2f, 0.2f));
                    }
                }
                const float tl = pathWeight<NW>(T);
                if (isfinite(tl) && !(tl <= 0.0f) && !(tl > 1.0e8f)) {
                    bool survive = true;
                    if (depth >= c.rrMinDepth) {
                        const float surv = fmin2(0.95f, fmax2(tl, 0.05f));
                        if (curand_uniform(&st) > surv) {
                            survive = false;
                        } else {
                            T = cscl(T, 1.0f / surv);
                        }
                    }
                    if (survive) {
                        eta = smp.nextEta;
                        const float bias = fmax2(1.0e-4f, 1.0e-3f * t);
                        const float sign = dot3(n, smp.dir) >= 0.0f ? 1.0f : -1.0f;
                        const float3 no = xadd(pos, xscl(n, __fmul_rn(sign, bias)));
                        c.paths.orig[i] = make_float4(no.x, no.y, no.z, bias);
                        // emitter MIS mode: a negative pdf marks a vertex that does not
                        // take part (the next hit's emission keeps weight 1)
                        const bool misSample = misVertex && !smp.transmitted && !smp.sss &&
                            dot3(n, smp.dir) > 0.0f && !inTransmitCones(cx, smp.dir);
                        c.paths.dir[i] = make_float4(smp.dir.x, smp.dir.y, smp.dir.z,
                            (emitterMis && !misSample) ? -smp.pdf : smp.pdf);
                        storeCol<NW>(NW == 0 ? c.paths.thr : nullptr, c.paths.thrS, cap, i, T, eta);
                        cont = true;
                    }
                }
            }
            rngStore(c.paths, i, st);
        }
        if (valid) {
            if constexpr (NW == 0) {
                c.paths.visEnv[i] = 0;
                c.paths.visEmis[i] = 0;
                if (cont) {
                    storeCol<NW>(c.paths.rad, c.paths.radS, cap, i, L, __int_as_float(depth + 1));
                    queueNext(c, i, nextCount, nextQueue);
                } else if (pendEnv || pendEmis) {
                    storeCol<NW>(c.paths.rad, c.paths.radS, cap, i, L, __int_as_float(depth));
                    const uint32_t s = warpPush(&c.q.counts[3]);
                    c.q.finish[s] = i;
                } else {
                    writeSample<NW>(c, i, L, wv);
                }
            } else {
                if (live) {
                    L = loadCol<NW>(r4, &sRad[0][threadIdx.x], kShadeThreads, 0u);
                } else {
                    L = loadCol<NW>(r4, c.paths.radS, cap, i);
                    if (visEnv) {
                        L = cadd(L, pendingEnv<NW>(c, i));
                    }
                    if (visEmis) {
                        L = cadd(L, pendingEmis<NW>(c, i));
                    }
                }
                if (cont || pendEnv || pendEmis) {
                    storeCol<NW>(nullptr, c.paths.radS, cap, i, L, 0.0f);
                    depthEta(c)[i] = make_float2(__int_as_float(cont ? depth + 1 : depth), eta);
                    if (cont) {
                        queueNext(c, i, nextCount, nextQueue);
                    } else {
                        const uint32_t s = warpPush(&c.q.counts[3]);
                        c.q.finish[s] = i;
                    }
                } else {
                    writeSample<NW>(c, i, L, wv);
                }
                c.paths.visEnv[i] = 0;
                c.paths.visEmis[i] = 0;
            }
        }
    }
    const unsigned int misses = c.q.counts[4 + 2 * (iter & 1)];
    for (unsigned int k = (gridDim.x - 1u - blockIdx.x) * blockDim.x + threadIdx.x; k < misses;
         k += gridDim.x * blockDim.x) {
        shadeMiss<NW>(c, c.q.missQueue[k], fresh);
    }
}

// Occlusion of the queued shadow rays (LightSamplingCore.h:187-197, 360-369).
template <bool Count, bool Inst>
__global__ void __launch_bounds__(256, 4) k_shadow(const LaunchCtx* __restrict__ cp, int iter)
{
    const LaunchCtx& c = *cp;
    extern __shared__ uint2 smemStack[];
    const unsigned int count = c.q.counts[2];
    const int par = iter & 1;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(&c.q.rays[1], static_cast<unsigned long long>(count));
        c.q.counts[10 + (par ^ 1)] = 0u; // next shadow stage's fetch counter
    }
    unsigned int* fetch = &c.q.counts[10 + par];
    for (;;) {
        const unsigned int k = warpFetch(fetch);
        if (__shfl_sync(0xffffffffu, k, 0) >= count) {
            break;
        }
        if (k >= count) {
            continue;
        }
        const uint32_t e = c.q.shadowPath[k];
        const float4 o4 = c.q.shadowOrig[k];
        const float4 d4 = c.q.shadowDir[k];
        const float3 dn = xnormalize(f3(d4.x, d4.y, d4.z));
        HitRec h;
        const float tMax = d4.w > 0.0f ? d4.w : kRayTMax; // emitter MIS rays end short of the light
        const bool occluded = traceRay<true, Count, Inst>(sceneOf(c, e & 0x7FFFFFFFu), f3(o4.x, o4.y, o4.z), dn, kShadowBias, tMax, h,
            c.q.overflow, c.q.visits + 2, smemStack + threadIdx.x, blockDim.x);
        if (!occluded) {
            const uint32_t i = e & 0x7FFFFFFFu;
            if (e & 0x80000000u) {
                c.paths.visEmis[i] = 1;
            } else {
                c.paths.visEnv[i] = 1;
            }
        }
    }
}

// Paths that terminated while their NEE shadow rays were in flight; in
// slot-ordered mode also the next bounce's extend queue (List; nothing here
// marks a slot).
template <int NW, bool List>
__global__ void __launch_bounds__(kListThreads) k_finalize(const LaunchCtx* __restrict__ cp, int sel)
{
    const LaunchCtx& c = *cp;
    const unsigned int count = c.q.counts[3];
    for (unsigned int k = blockIdx.x * blockDim.x + threadIdx.x; k < count; k += gridDim.x * blockDim.x) {
        const uint32_t i = c.q.finish[k];
        const Waves<NW> wv = pathWaves<NW>(c, i);
        Col<NW> L = loadCol<NW>(c.paths.rad[i], c.paths.radS, c.paths.capacity, i);
        if (c.paths.visEnv[i]) {
            L = cadd(L, pendingEnv<NW>(c, i));
        }
        if (c.paths.visEmis[i]) {
            L = cadd(L, pendingEmis<NW>(c, i));
        }
        writeSample<NW>(c, i, L, wv);
    }
    if constexpr (List) {
        listMarked(c, sel);
    }
}

// Per pixel: fold the batch's samples in sample order (PathTracer.cu:232-272).
// activeCount[1] counts the pixels that go on (KeepActive), so that the list is
// compacted only when some pixels stopped and some did not: three launches less
// for a wave in which none stops and for a render's last batch.
constexpr int kAccumulateThreads = 256;
__global__ void __launch_bounds__(kAccumulateThreads) k_accumulate(const LaunchCtx* __restrict__ cp, int activeCount, int batch)
{
    const LaunchCtx& c = *cp;
    const int* active = c.acc.active[c.activeSel];
    const int maxSpp = c.params.max_samples_per_pixel;
    const int minSpp = c.params.min_samples;
    const float thr = c.params.relative_error_threshold;
    const bool stdErr = c.params.adaptive_criterion == 1 || c.params.adaptive_criterion == 2;
    // criterion 2: a pixel all of whose samples are black stops after max(min spp, 64) samples
    const bool blackStops = c.params.adaptive_criterion == 2;
    const uint32_t blackSpp = static_cast<uint32_t>(minSpp > 64 ? minSpp : 64);
    unsigned int kept = 0;
    for (int li = blockIdx.x * blockDim.x + threadIdx.x; li < activeCount; li += gridDim.x * blockDim.x) {
        const int p = active[li];
        uint8_t conv = c.acc.converged[p];
        if (conv) {
            continue;
        }
        uint32_t n = c.acc.counts[p];
        float mean = c.acc.lumMean[p];
        float m2 = c.acc.m2[p];
        float4 a = c.acc.acc[p];
        for (int s = 0; s < batch && !conv; ++s) {
            const float4 smp = c.acc.samples[static_cast<size_t>(s) * activeCount + li];
            const float sl =
                __fadd_rn(__fadd_rn(__fmul_rn(smp.x, 0.2126f), __fmul_rn(smp.y, 0.7152f)), __fmul_rn(smp.z, 0.0722f));
            const float fn1 = static_cast<float>(n + 1);
            const float delta = __fsub_rn(sl, mean);
            const float nm = __fadd_rn(mean, __fdiv_rn(delta, fn1));
            m2 = __fadd_rn(m2, __fmul_rn(delta, __fsub_rn(sl, nm)));
            mean = nm;
            const float invN = __fdiv_rn(1.0f, fn1);
            const float fn = static_cast<float>(n);
            a.x = __fmul_rn(__fadd_rn(__fmul_rn(a.x, fn), smp.x), invN);
            a.y = __fmul_rn(__fadd_rn(__fmul_rn(a.y, fn), smp.y), invN);
            a.z = __fmul_rn(__fadd_rn(__fmul_rn(a.z, fn), smp.z), invN);
            a.w = 1.0f;
            ++n;
            if (maxSpp > 0 && n >= static_cast<uint32_t>(maxSpp)) {
                conv = 1;
                break;
            }
            if ((n % 4u) != 0u) {
                continue;
            }
            // isAdaptivePixelConverged (PathTracerAdaptiveSampling.h:16-40)
            if (n >= static_cast<uint32_t>(minSpp) && n > 0 && mean >= 1.0e-5f) {
                const float var = __fdiv_rn(m2, static_cast<float>(n));
                float rel = __fdiv_rn(__fsqrt_rn(var), fmaxf(mean, 1.0e-4f));
                if (stdErr) {
                    rel = __fdiv_rn(rel, __fsqrt_rn(static_cast<float>(n)));
                }
                if (rel < thr) {
                    conv = 1;
                }
            } else if (blackStops && n >= blackSpp && mean == 0.0f && m2 == 0.0f) {
                conv = 1;
            }
        }
        c.acc.counts[p] = n;
        c.acc.lumMean[p] = mean;
        c.acc.m2[p] = m2;
        c.acc.acc[p] = a;
        c.acc.converged[p] = conv;
        kept += conv == 0 && !(maxSpp > 0 && n >= static_cast<uint32_t>(maxSpp)) ? 1u : 0u;
    }
    __shared__ unsigned int sKept[kAccumulateThreads / 32];
    kept = __reduce_add_sync(0xffffffffu, kept);
    if ((threadIdx.x & 31) == 0) {
        sKept[threadIdx.x >> 5] = kept;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < kAccumulateThreads / 32; ++w) {
            kept += sKept[w];
        }
        if (kept != 0u) {
            atomicAdd(&c.acc.activeCount[1], static_cast<int>(kept));
        }
    }
}

// Per-scene active ranges (the active list is sorted by pixel) and job
// offsets of the current batch: scene s owns active entries
// [sceneActiveStart[s], sceneActiveStart[s + 1]) and jobs
// [sceneJobStart[s], sceneJobStart[s + 1]).
__global__ void k_scene_jobs(const LaunchCtx* __restrict__ cp, int sceneCount, int waves)
{
    const LaunchCtx& c = *cp;
    const int n = c.q.batch->activeCount;
    const int* active = c.acc.active[c.activeSel];
    for (int s = threadIdx.x; s <= sceneCount; s += blockDim.x) {
        uint32_t pos = static_cast<uint32_t>(n);
        if (s < sceneCount) {
            const int key = static_cast<int>(c.views[s].pixelBase);
            int lo = 0, hi = n; // first entry >= key
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (active[mid] < key) {
                    lo = mid + 1;
                } else {
                    hi = mid;
                }
            }
            pos = static_cast<uint32_t>(lo);
        }
        c.sceneActiveStart[s] = pos;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        unsigned long long acc = 0;
        for (int s = 0; s < sceneCount; ++s) {
            c.sceneJobStart[s] = acc;
            acc += static_cast<unsigned long long>(c.sceneActiveStart[s + 1] - c.sceneActiveStart[s]) *
                static_cast<unsigned long long>(waves);
        }
        c.sceneJobStart[sceneCount] = acc;
    }
}

// A pixel stays on the active list until it converged or reached the sample
// cap (the tests of compactActiveListKernel, PathTracer.cu:385-391).
struct KeepActive {
    const uint8_t* converged;
    const uint32_t* counts;
    int maxSpp;
    __device__ __forceinline__ bool operator()(int p) const
    {
        return converged[p] == 0 && !(maxSpp > 0 && counts[p] >= static_cast<uint32_t>(maxSpp));
    }
};
// Select predicate / value over the entries of an active list.
struct KeepListed {
    const int* list;
    KeepActive keep;
    __device__ __forceinline__ bool operator()(long long i) const { return keep(list[i]); }
};
struct ListedPixel {
    const int* list;
    __device__ __forceinline__ int operator()(long long i) const { return list[i]; }
};

__global__ void k_reset(const LaunchCtx* __restrict__ cp, int pixels)
{
    const LaunchCtx& c = *cp;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < pixels; i += gridDim.x * blockDim.x) {
        c.acc.acc[i] = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
        c.acc.counts[i] = 0;
        c.acc.lumMean[i] = 0.0f;
        c.acc.m2[i] = 0.0f;
        c.acc.converged[i] = 0;
        c.acc.active[0][i] = i;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        c.acc.activeCount[0] = pixels;
        c.acc.activeCount[1] = 0;
    }
}

__global__ void __launch_bounds__(256) k_trace_rays(DevScene S, int n, const float* o, const float* d, const float* tmin,
    const float* tmax, uint8_t* hit, float* t, uint32_t* tri, float* normal, float* uv, unsigned int* overflow)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float3 ro = f3(o[3 * i], o[3 * i + 1], o[3 * i + 2]);
        const float3 dn = xnormalize(f3(d[3 * i], d[3 * i + 1], d[3 * i + 2]));
        HitRec h;
        const bool ok = traceRay<false, false, true>(S, ro, dn, tmin[i], tmax[i], h, overflow);
        hit[i] = ok ? 1 : 0;
        float3 nn = f3(0.0f, 0.0f, 0.0f);
        float tu = 0.0f, tv = 0.0f;
        if (ok) {
            hitShadingAt(S, S.shade[h.tri], h.inst, dn, h.u, h.v, nn, tu, tv);
        }
        if (t) {
            t[i] = ok ? h.t : 0.0f;
        }
        if (tri) {
            tri[i] = ok ? h.tri : 0u;
        }
        if (normal) {
            normal[3 * i] = nn.x;
            normal[3 * i + 1] = nn.y;
            normal[3 * i + 2] = nn.z;
        }
        if (uv) {
            uv[2 * i] = tu;
            uv[2 * i + 1] = tv;
        }
    }
}

// Region render (clearRegionAccumulatorKernel, PathTracer.cu:305-344): clears
// the accumulators of the pixels in [minX, maxX] x [minY, maxY] when `clear`
// and makes them the active list, row by row (so it stays sorted).
__global__ void k_region(const LaunchCtx* __restrict__ cp, int width, int minX, int minY, int maxX, int maxY, bool clear)
{
    const LaunchCtx& c = *cp;
    const int rw = maxX - minX + 1, rh = maxY - minY + 1;
    const int n = rw * rh;
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const int idx = (minY + t / rw) * width + minX + t % rw;
        if (clear) {
            c.acc.acc[idx] = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
            c.acc.counts[idx] = 0;
            c.acc.lumMean[idx] = 0.0f;
            c.acc.m2[idx] = 0.0f;
            c.acc.converged[idx] = 0;
        }
        c.acc.active[0][t] = idx;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        c.acc.activeCount[0] = n;
        c.acc.activeCount[1] = 0;
    }
}

__global__ void k_rng_tape(int width, int height, int firstWave, int waves, int stride, int seedOffset, float* out)
{
    const long long P = static_cast<long long>(width) * height;
    const long long total = P * waves;
    for (long long k = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; k < total;
         k += static_cast<long long>(gridDim.x) * blockDim.x) {
        const uint32_t w = static_cast<uint32_t>(k / P);
        const uint32_t p = static_cast<uint32_t>(k % P);
        const uint32_t wave = static_cast<uint32_t>(firstWave) + w;
        const uint32_t seed = p * 747796405u + wave + (wave + 1u + static_cast<uint32_t>(seedOffset)) * 2891336453u;
        curandStateXORWOW st;
        curand_init(seed, 0ull, 0ull, &st);
        float* row = out + k * stride;
        for (int j = 0; j < stride; ++j) {
            row[j] = curand_uniform(&st);
        }
    }
}

inline int gridFor(long long n, int block = 256, int cap = 148 * 16)
{
    long long g = (n + block - 1) / block;
    if (g < 1) {
        g = 1;
    }
    return static_cast<int>(g < cap ? g : cap);
}

} // namespace

void launchGenerate(const LaunchCtx* d, int count, int extendSel, int nw, cudaStream_t s, unsigned long long jobOffset)
{
    if (nw == 8) {
        k_generate<8><<<gridFor(count), 256, 0, s>>>(d, count, extendSel, jobOffset);
    } else if (nw == 4) {
        k_generate<4><<<gridFor(count), 256, 0, s>>>(d, count, extendSel, jobOffset);
    } else {
        k_generate<0><<<gridFor(count), 256, 0, s>>>(d, count, extendSel, jobOffset);
    }
}
namespace {
template <bool Inst> constexpr size_t traceSmemBytes() { return sizeof(WarpTrace<Inst>) * (kTraceThreads / 32); }
static_assert(traceSmemBytes<true>() <= 48 * 1024, "dynamic shared memory without opting in");
template <class F> int blocksPerSm(F kernel, int threads, size_t smem)
{
    int blocks = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, kernel, threads, smem);
    return blocks > 0 ? blocks : 1;
}
} // namespace
void launchExtend(const LaunchCtx* c, int sel, bool identity, int iter, int grid, bool count, bool inst, bool lane,
    bool multi, cudaStream_t s)
{
    const size_t smem = sizeof(uint2) * kSharedStack * 256;
    if (lane && !count) {
        if (inst && multi) {
            k_extend_lane<true, true><<<grid, kTraceThreads, traceSmemBytes<true>(), s>>>(c, sel, identity, iter);
        } else if (inst) {
            k_extend_lane<true, false><<<grid, kTraceThreads, traceSmemBytes<true>(), s>>>(c, sel, identity, iter);
        } else if (multi) {
            k_extend_lane<false, true><<<grid, kTraceThreads, traceSmemBytes<false>(), s>>>(c, sel, identity, iter);
        } else {
            k_extend_lane<false, false><<<grid, kTraceThreads, traceSmemBytes<false>(), s>>>(c, sel, identity, iter);
        }
        k_route<<<grid, kListThreads, 0, s>>>(c, sel, iter);
    } else if (inst) {
        if (count) {
            k_extend<true, true><<<grid, 256, smem, s>>>(c, sel, identity, iter);
        } else {
            k_extend<false, true><<<grid, 256, smem, s>>>(c, sel, identity, iter);
        }
    } else if (count) {
        k_extend<true, false><<<grid, 256, smem, s>>>(c, sel, identity, iter);
    } else {
        k_extend<false, false><<<grid, 256, smem, s>>>(c, sel, identity, iter);
    }
}
int extendKernels(bool count, bool inst, bool lane)
{
    return (!count && lane) ? 2 : 1;
}
int extendLaneOccupancy()
{
    return blocksPerSm(k_extend_lane<false, false>, kTraceThreads, traceSmemBytes<false>());
}
int extendLaneInstOccupancy()
{
    return blocksPerSm(k_extend_lane<true, false>, kTraceThreads, traceSmemBytes<true>());
}
int shadowLaneOccupancy()
{
    return blocksPerSm(k_shadow_lane<false, false>, kTraceThreads, traceSmemBytes<false>());
}
int shadowLaneInstOccupancy()
{
    return blocksPerSm(k_shadow_lane<true, false>, kTraceThreads, traceSmemBytes<true>());
}
void launchShade(const LaunchCtx* c, int sel, int iter, bool first, int grid, int nw, cudaStream_t s)
{
    if (nw == 8) {
        k_shade<8><<<grid, kShadeThreads, 0, s>>>(c, sel, iter, first);
    } else if (nw == 4) {
        k_shade<4><<<grid, kShadeThreads, 0, s>>>(c, sel, iter, first);
    } else {
        k_shade<0><<<grid, kShadeThreads, 0, s>>>(c, sel, iter, first);
    }
}
void launchShadow(const LaunchCtx* c, int iter, int grid, bool count, bool inst, bool lane, bool multi, cudaStream_t s)
{
    const size_t smem = sizeof(uint2) * kSharedStack * 256;
    if (lane && !count) {
        if (inst && multi) {
            k_shadow_lane<true, true><<<grid, kTraceThreads, traceSmemBytes<true>(), s>>>(c, iter);
        } else if (inst) {
            k_shadow_lane<true, false><<<grid, kTraceThreads, traceSmemBytes<true>(), s>>>(c, iter);
        } else if (multi) {
            k_shadow_lane<false, true><<<grid, kTraceThreads, traceSmemBytes<false>(), s>>>(c, iter);
        } else {
            k_shadow_lane<false, false><<<grid, kTraceThreads, traceSmemBytes<false>(), s>>>(c, iter);
        }
    } else if (inst) {
        if (count) {
            k_shadow<true, true><<<grid, 256, smem, s>>>(c, iter);
        } else {
            k_shadow<false, true><<<grid, 256, smem, s>>>(c, iter);
        }
    } else if (count) {
        k_shadow<true, false><<<grid, 256, smem, s>>>(c, iter);
    } else {
        k_shadow<false, false><<<grid, 256, smem, s>>>(c, iter);
    }
}
int shadeOccupancy(int nw)
{
    // (one value per instantiation, computed once per process; renderers on
    // several host threads may race to fill it, with the same value)
    static std::atomic<int> occ[3] = {{0}, {0}, {0}};
    const int k = nw == 8 ? 2 : (nw == 4 ? 1 : 0);
    if (occ[k].load(std::memory_order_relaxed) == 0) {
        int b = 1;
        if (nw == 8) {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_shade<8>, kShadeThreads, 0);
        } else if (nw == 4) {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_shade<4>, kShadeThreads, 0);
        } else {
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_shade<0>, kShadeThreads, 0);
        }
        occ[k].store(b > 0 ? b : 1, std::memory_order_relaxed);
    }
    return occ[k].load(std::memory_order_relaxed);
}
void stageOccupancy(int& extendBlocks, int& shadeBlocks, int& shadowBlocks)
{
    extendBlocks = shadeBlocks = shadowBlocks = 1;
    const size_t smem = sizeof(uint2) * kSharedStack * 256;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&extendBlocks, k_extend<false, false>, 256, smem);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&shadeBlocks, k_shade<0>, kShadeThreads, 0);
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&shadowBlocks, k_shadow<false, false>, 256, smem);
}
namespace {
template <int NW> void finalize(const LaunchCtx* c, int sel, int grid, bool list, cudaStream_t s)
{
    if (list) {
        k_finalize<NW, true><<<grid, kListThreads, 0, s>>>(c, sel);
    } else {
        k_finalize<NW, false><<<grid, kListThreads, 0, s>>>(c, sel);
    }
}
} // namespace
void launchFinalize(const LaunchCtx* c, int sel, int grid, int nw, bool list, cudaStream_t s)
{
    if (nw == 8) {
        finalize<8>(c, sel, grid, list, s);
    } else if (nw == 4) {
        finalize<4>(c, sel, grid, list, s);
    } else {
        finalize<0>(c, sel, grid, list, s);
    }
}
void launchAccumulate(const LaunchCtx* c, int activeCount, int batch, cudaStream_t s)
{
    k_accumulate<<<gridFor(activeCount, kAccumulateThreads), kAccumulateThreads, 0, s>>>(c, activeCount, batch);
}
size_t compactTempBytes(int n)
{
    return selectTempBytes(n);
}
cudaError_t launchCompactStable(const int* in, int* out, int* outCount, int n, const uint8_t* converged,
    const uint32_t* counts, int maxSpp, void* temp, size_t tempBytes, cudaStream_t s)
{
    return launchSelect(static_cast<long long>(n), KeepListed{in, KeepActive{converged, counts, maxSpp}},
        ListedPixel{in}, out, outCount, temp, tempBytes, s);
}
void launchSceneJobs(const LaunchCtx* c, int sceneCount, int waves, cudaStream_t s)
{
    k_scene_jobs<<<1, 1024, 0, s>>>(c, sceneCount, waves);
}
void launchResetAccum(const LaunchCtx* c, int pixels, cudaStream_t s) { k_reset<<<gridFor(pixels), 256, 0, s>>>(c, pixels); }
void launchTraceRays(const DevScene& S, int n, const float* o, const float* d, const float* tmin, const float* tmax,
    uint8_t* hit, float* t, uint32_t* tri, float* normal, float* uv, cudaStream_t s, unsigned int* overflow)
{
    k_trace_rays<<<gridFor(n), 256, 0, s>>>(S, n, o, d, tmin, tmax, hit, t, tri, normal, uv, overflow);
}
void launchRngTape(int width, int height, int firstWave, int waves, int stride, int seedOffset, float* out,
    cudaStream_t s)
{
    k_rng_tape<<<gridFor(static_cast<long long>(width) * height * waves), 256, 0, s>>>(width, height, firstWave, waves,
        stride, seedOffset, out);
}
void launchRegion(const LaunchCtx* c, int width, int minX, int minY, int maxX, int maxY, bool clear, cudaStream_t s)
{
    const long long n = static_cast<long long>(maxX - minX + 1) * (maxY - minY + 1);
    k_region<<<gridFor(n), 256, 0, s>>>(c, width, minX, minY, maxX, maxY, clear);
}

} // namespace pt
