// Device-side building blocks of the spectral path tracer for sm_100a:
// samplers, hero wavelengths, compressed BVH8 traversal, surface interaction,
// area-light sampling, BSDFs and the per-path integrator loop.
//
// Each function cites the reference routine whose semantics it restates.
#pragma once

#include "vs_math.h"
#include "vs_scene.h"
#include "vs_spectral.h"
#include "vs_devscene.h"
#include <cuda_runtime.h>

// Large device functions called from several places.  They are inlined:
// on B200 that measured 10-17% faster than calls in the path-tracing
// megakernel and 4% faster in the ReSTIR kernels, whose out-of-line stack
// frames spilled through L2 to HBM.  Define VS_OUTLINE as __noinline__ to
// build them out of line.
#ifndef VS_OUTLINE
#define VS_OUTLINE __forceinline__
#endif

namespace vs {

// ---------------------------------------------------------------------------
// CIE X/Y/Z and D65 downsampled to every 5th nm (94 entries,
// src/base/color/spd.cpp:31-38,96-110) and the CIE Y integral (:14-23).
// The tables are read at a different wavelength by every lane, so they live
// in global memory as one (x, y, z, d65) record per entry and come through L1
// (1.5 KB): constant memory serves one address per cycle and serialised each
// of the 24 reads of a four-wavelength linear_srgb over the warp's lanes.
// Measured against constant memory: 1024 x 1024 at 8 spp of the 2.3 M-triangle
// scene 40.2 -> 37.3 ms, the box room's 256 x 256 at 16 spp 2.62 -> 2.32 ms.
// ---------------------------------------------------------------------------
// Internal linkage: every translation unit that launches kernels reading them
// fills its own copy with upload_spectral_consts_tu().
static __constant__ float c_inv_cie_y_integral;
static __device__ float4 d_cie[kSpd5Count];

static inline cudaError_t upload_spectral_consts_tu(const float *x, const float *y, const float *z, const float *d65,
                                                    float y_integral) {
    float4 t[kSpd5Count];
    for (int i = 0; i < kSpd5Count; ++i) t[i] = make_float4(x[i], y[i], z[i], d65[i]);
    const float inv = 1.0f / y_integral;
    cudaError_t e = cudaMemcpyToSymbol(c_inv_cie_y_integral, &inv, sizeof(inv));
    return e == cudaSuccess ? cudaMemcpyToSymbol(d_cie, t, sizeof(t)) : e;
}

// ---------------------------------------------------------------------------
// Samplers.  IndependentSampler (src/render_core/samplers/independent.cpp:24-42)
// seeds with tea(tea(px, py), tea(sample, dim)) (src/math/util.h:13-24, 4
// rounds) and draws with a 24-bit LCG (:27-33).  The PCG option draws from
// PCG32 (O'Neill 2014, XSH-RR output) seeded from the same TEA hash and a seed.
// ---------------------------------------------------------------------------
VS_HD uint32_t tea4(uint32_t v0, uint32_t v1) {
    uint32_t s0 = 0;
#pragma unroll
    for (int n = 0; n < 4; ++n) {
        s0 += 0x9e3779b9u;
        v0 += ((v1 << 4) + 0xa341316cu) ^ (v1 + s0) ^ ((v1 >> 5) + 0xc8013ea4u);
        v1 += ((v0 << 4) + 0xad90777du) ^ (v0 + s0) ^ ((v0 >> 5) + 0x7e95761eu);
    }
    return v0;
}

struct Sampler {
    uint64_t state;  // LCG state (low 32 bits) or the 64-bit PCG32 state
    uint32_t kind;
    uint32_t seed;   // PCG32 stream selector: increment (seed << 1) | 1
    VS_HD void start(uint32_t px, uint32_t py, uint32_t sample, uint32_t dim, uint32_t k, uint32_t sd) {
        kind = k;
        seed = sd;
        uint32_t s = tea4(tea4(px, py), tea4(sample, dim));
        if (kind == kSamplerIndependent) {
            state = s;
        } else {
            // PCG32 seeding (pcg32_srandom_r): state 0, one step, add the
            // initial state (the TEA hash), one more step.
            const uint64_t inc = (static_cast<uint64_t>(seed) << 1u) | 1u;
            state = inc;
            state += s;
            state = state * 6364136223846793005ull + inc;
        }
    }
    VS_HD float next() {
        if (kind == kSamplerIndependent) {
            uint32_t s = static_cast<uint32_t>(state);
            s = 1664525u * s + 1013904223u;
            state = s;
            return static_cast<float>(s & 0x00ffffffu) * (1.0f / 16777216.0f);
        }
        // PCG32 step and XSH-RR output; the top 24 bits make the float.
        const uint64_t old = state;
        state = old * 6364136223846793005ull + ((static_cast<uint64_t>(seed) << 1u) | 1u);
        const uint32_t xorshifted = static_cast<uint32_t>(((old >> 18u) ^ old) >> 27u);
        const uint32_t rot = static_cast<uint32_t>(old >> 59u);
        const uint32_t r = (xorshifted >> rot) | (xorshifted << ((32u - rot) & 31u));
        return static_cast<float>(r >> 8) * (1.0f / 16777216.0f);
    }
    VS_HD f2 next2() {
        float a = next();
        float b = next();
        return {a, b};
    }
};

// ---------------------------------------------------------------------------
// Spectra: N hero wavelengths per path.
// ---------------------------------------------------------------------------
template <int N>
struct Spec {
    float v[N];
    __device__ __forceinline__ static Spec fill(float s) {
        Spec r;
#pragma unroll
        for (int i = 0; i < N; ++i) r.v[i] = s;
        return r;
    }
    __device__ __forceinline__ float max() const {
        float m = v[0];
#pragma unroll
        for (int i = 1; i < N; ++i) m = fmaxf(m, v[i]);
        return m;
    }
    __device__ __forceinline__ bool all_zero() const {
        bool z = true;
#pragma unroll
        for (int i = 0; i < N; ++i) z = z && (v[i] == 0.0f);
        return z;
    }
};
template <int N>
__device__ __forceinline__ Spec<N> operator*(const Spec<N> &a, const Spec<N> &b) {
    Spec<N> r;
#pragma unroll
    for (int i = 0; i < N; ++i) r.v[i] = a.v[i] * b.v[i];
    return r;
}
template <int N>
__device__ __forceinline__ Spec<N> operator+(const Spec<N> &a, const Spec<N> &b) {
    Spec<N> r;
#pragma unroll
    for (int i = 0; i < N; ++i) r.v[i] = a.v[i] + b.v[i];
    return r;
}
template <int N>
__device__ __forceinline__ Spec<N> operator*(const Spec<N> &a, float s) {
    Spec<N> r;
#pragma unroll
    for (int i = 0; i < N; ++i) r.v[i] = a.v[i] * s;
    return r;
}

template <int N>
struct Wavelengths {
    float lambda[N];
    float pdf[N];
};

// SRGBSpectrum (spectra/srgb.cpp:16-24): three channels at the peak
// wavelengths of the sRGB primaries (the published constant of the ocarina
// module the reference builds on, absent from its tree: unpinned), pdf 1.
// The wavelengths are stored negated: the sign marks RGB transport, so that
// colour decodes pass RGB through and spectral data (conductor and glass
// IOR curves) is read at |lambda|.
template <int N>
__device__ __forceinline__ Wavelengths<N> rgb_wavelengths() {
    Wavelengths<N> w;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        w.lambda[i] = i == 0 ? -602.785f : (i == 1 ? -539.285f : -445.772f);
        w.pdf[i] = 1.0f;
    }
    return w;
}
// RGB transport always has three channels (the loader sets the dimension),
// so the test compiles away for the other widths.
template <int N>
__device__ __forceinline__ bool is_rgb(const Wavelengths<N> &w) {
    if constexpr (N != 3) return false;
    return w.lambda[0] < 0.0f;
}

// The table records around a wavelength and the weight of the upper one:
// spd_eval's lookup in the 94-entry tables.
struct CieLookup {
    uint32_t i;
    float fr;
};
__device__ __forceinline__ CieLookup cie_lookup(float lambda) {
    const float interval = static_cast<float>(kCieSamples) / static_cast<float>(kSpd5Count);
    const float t = (clampf(lambda, kLambdaMin, kLambdaMax) - kLambdaMin) / interval;
    const uint32_t sample_count = static_cast<uint32_t>((kLambdaMax - kLambdaMin) / interval) + 1u;
    return {static_cast<uint32_t>(fminf(t, static_cast<float>(sample_count - 2u))), t - floorf(t)};
}
__device__ __forceinline__ f3 cie_xyz(float lambda) {
    const CieLookup k = cie_lookup(lambda);
    const float4 l = __ldg(&d_cie[k.i]), r = __ldg(&d_cie[k.i + 1]);
    return {l.x + k.fr * (r.x - l.x), l.y + k.fr * (r.y - l.y), l.z + k.fr * (r.z - l.z)};
}
__device__ __forceinline__ float cie_d65(float lambda) {
    const CieLookup k = cie_lookup(lambda);
    const float l = __ldg(&d_cie[k.i].w), r = __ldg(&d_cie[k.i + 1].w);
    return l + k.fr * (r - l);
}

// HeroWavelengthSpectrum::sample_wavelength (hero.cpp:286-299).
template <int N>
__device__ __forceinline__ Wavelengths<N> sample_wavelengths(float u) {
    Wavelengths<N> w;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float offset = static_cast<float>(static_cast<uint32_t>(i) * (1.0f / N));
        float up = u + offset;
        up = up - floorf(up);
        float l = sample_visible_wavelength(up);
        w.lambda[i] = l;
        w.pdf[i] = visible_wavelength_pdf(l);
    }
    return w;
}

// HeroWavelengthSpectrum::cie_xyz + xyz_to_linear_srgb (hero.cpp:261-285).
template <int N>
__device__ VS_OUTLINE f3 linear_srgb(const Spec<N> &s, const Wavelengths<N> &w) {
    // SRGBSpectrum::linear_srgb: the channels themselves.
    if (is_rgb(w)) return make3(s.v[0], s.v[N > 1 ? 1 : 0], s.v[N > 2 ? 2 : 0]);
    f3 sum = make3(0.0f);
    int valid = 0;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float l = w.lambda[i];
        float p = w.pdf[i];
        valid += p > 0.0f ? 1 : 0;
        const f3 c = cie_xyz(l);
        sum.x += safe_div(c.x * s.v[i], p);
        sum.y += safe_div(c.y * s.v[i], p);
        sum.z += safe_div(c.z * s.v[i], p);
    }
    float factor = 1.0f / (static_cast<float>(valid) * (1.0f / c_inv_cie_y_integral));
    return xyz_to_linear_srgb(sum * factor);
}

// Albedo spectrum of sigmoid coefficients (RGBAlbedoSpectrum, hero.cpp:177-184).
template <int N>
__device__ __forceinline__ Spec<N> albedo_spectrum(const float *c, const Wavelengths<N> &w) {
    Spec<N> r;
    if (is_rgb(w)) {
        // SRGBSpectrum::decode_to_albedo: the colour itself (c holds RGB).
#pragma unroll
        for (int i = 0; i < N; ++i) r.v[i] = c[i < 3 ? i : 2];
        return r;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) r.v[i] = sigmoid_poly(c[0], c[1], c[2], w.lambda[i]);
    return r;
}

// Radiance of an area light (AreaLight::L, area.cpp:91-95; colour decode
// RGBIlluminationSpectrum, hero.cpp:204-219; blackbody emitter is new).
template <int N>
__device__ __forceinline__ Spec<N> emitter_spectrum(const AreaLight &L, const Wavelengths<N> &w) {
    Spec<N> r;
    if (is_rgb(w)) {
        // SRGBSpectrum::decode_to_illumination: the colour times the scale.
#pragma unroll
        for (int i = 0; i < N; ++i) r.v[i] = L.rgb_avg[i < 3 ? i : 2];
        return r;
    }
#pragma unroll
    for (int i = 0; i < N; ++i) {
        float l = w.lambda[i];
        float e;
        if (L.kind == kEmitRGB) {
            e = sigmoid_poly(L.coef[0], L.coef[1], L.coef[2], l) * L.coef[3] * cie_d65(l);
        } else {
            e = planck(l, L.coef[0]) * L.coef[1];
        }
        r.v[i] = e * L.scale;
    }
    return r;
}

// ---------------------------------------------------------------------------
// Ray origin offset (Waechter & Binder, "A Fast and Robust Method for Avoiding
// Self-Intersection", Ray Tracing Gems ch. 6): integer ulp nudge along the
// normal away from the origin, plain float nudge near zero.
// ---------------------------------------------------------------------------
VS_HD float offset_component(float p, float n) {
    const float kOrigin = 1.0f / 32.0f;
    const float kFloatScale = 1.0f / 65536.0f;
    const float kIntScale = 256.0f;
    int of = static_cast<int>(kIntScale * n);
    int pi = static_cast<int>(float_bits(p));
    float pn = bits_float(static_cast<uint32_t>(pi + (p < 0.0f ? -of : of)));
    return fabsf(p) < kOrigin ? p + kFloatScale * n : pn;
}
VS_HD f3 offset_ray_origin(f3 p, f3 n) {
    return {offset_component(p.x, n.x), offset_component(p.y, n.y), offset_component(p.z, n.z)};
}

// spawn_ray / spawn_ray_to (src/base/scattering/interaction.h:272-291).
struct Ray {
    f3 o;
    f3 d;
    float tmax;
};
VS_HD Ray spawn_ray(f3 pos, f3 ng, f3 dir) {
    f3 n = dot(ng, dir) > 0.0f ? ng : -ng;
    return {offset_ray_origin(pos, n), dir, 3.402823466e+38f};
}
VS_HD Ray spawn_ray_to(f3 pos, f3 ng, f3 target) {
    f3 dir = target - pos;
    f3 n = dot(ng, dir) > 0.0f ? ng : -ng;
    return {offset_ray_origin(pos, n), dir, 1.0f - kShadowEpsilon};
}

// ---------------------------------------------------------------------------
// Watertight ray/triangle test (Woop, Benthin, Wald, JCGT 2013) written with
// explicitly rounded operations so that it gives bit-identical results on the
// GPU and in the CPU oracle.  Barycentrics: u weights vertex 1, v vertex 2.
// ---------------------------------------------------------------------------
struct RayPre {
    // Triangle test: origin and shear in the ray's axis order (kz: dominant
    // direction component, then kx = kz + 1, ky = kz + 2 modulo 3).
    f3 o;
    float sx, sy, sz;
    int kz;
    // Box test, in world axes: reciprocal direction, and -o / d less (near
    // planes) and plus (far planes) the bound below on its rounding errors.
    f3 inv_d;
    f3 cn, cf;
    uint32_t oct;  // bit i set when inv_d[i] < 0
    f3 wo, wd;     // the ray in world axes (for instance transforms)
};

// `bound`: the largest coordinate magnitude, per axis, of the BVH's boxes.
//
// The box distances of intersect_children are q * (2^e / d) + ((p - o) / d),
// the second term as p / d + (-o / d).  In units of 2^-24 (|o| + |plane|) / |d|
// the reciprocal (good to 2 ulp) costs them up to 4, their own roundings up to
// 6 and the triangle test's vertex differences and shear up to 4.  cn and cf
// move every near plane down and every far plane up by 16 of these units, so a
// box is entered whenever the float triangle test can accept one of its
// triangles.  Measured against rays aimed at the corners of axis-aligned
// triangles, with the reciprocal off by 2 ulp: 4 units lose 0.8 % of the hits,
// 6 units 2 in a million, 8 units none of 47 million.
// The margin is taken of |o / d| as it was computed, so that it is infinite
// wherever that overflows (a zero direction component, |o| above 3.4e8): the
// planes of the axis are then infinite or NaN on the side that keeps the box
// (a NaN is dropped by the minima and maxima).
__device__ __forceinline__ RayPre precompute_ray(f3 o, f3 d, f3 bound) {
    RayPre r;
    r.wo = o;
    r.wd = d;
    const float tiny = 1e-30f;
    r.inv_d = {__fdividef(1.0f, fabsf(d.x) > tiny ? d.x : copysignf(tiny, d.x)),
               __fdividef(1.0f, fabsf(d.y) > tiny ? d.y : copysignf(tiny, d.y)),
               __fdividef(1.0f, fabsf(d.z) > tiny ? d.z : copysignf(tiny, d.z))};
    const float k = 1.0f / 1048576.0f;
    const f3 b = {-o.x * r.inv_d.x, -o.y * r.inv_d.y, -o.z * r.inv_d.z};
    const f3 e = {k * fmaf(bound.x, fabsf(r.inv_d.x), fabsf(b.x)), k * fmaf(bound.y, fabsf(r.inv_d.y), fabsf(b.y)),
                  k * fmaf(bound.z, fabsf(r.inv_d.z), fabsf(b.z))};
    r.cn = b - e;
    r.cf = b + e;
    float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    r.kz = (ax > ay) ? (ax > az ? 0 : 2) : (ay > az ? 1 : 2);
    const int kx = r.kz == 2 ? 0 : r.kz + 1;
    const int ky = kx == 2 ? 0 : kx + 1;
    r.o = {comp(o, kx), comp(o, ky), comp(o, r.kz)};
    const float dz = comp(d, r.kz);
    r.sx = __fdiv_rn(comp(d, kx), dz);
    r.sy = __fdiv_rn(comp(d, ky), dz);
    r.sz = __fdiv_rn(1.0f, dz);
    r.oct = (r.inv_d.x < 0.0f ? 1u : 0u) | (r.inv_d.y < 0.0f ? 2u : 0u) | (r.inv_d.z < 0.0f ? 4u : 0u);
    return r;
}

// A vertex relative to the ray's origin, in its axis order.
__device__ __forceinline__ f3 ray_axes(const RayPre &r, const float4 &v) {
    const bool k0 = r.kz == 0, k1 = r.kz == 1;
    return {__fsub_rn(k0 ? v.y : (k1 ? v.z : v.x), r.o.x), __fsub_rn(k0 ? v.z : (k1 ? v.x : v.y), r.o.y),
            __fsub_rn(k0 ? v.x : (k1 ? v.y : v.z), r.o.z)};
}

// Returns true and fills (t, u, v) when the ray hits the triangle with
// tmin < t < tmax.  The published test swaps kx and ky for a negative dominant
// component to keep the winding; the swap negates U, V, W, their sum and T
// exactly, so t, u and v and every comparison below are the same without it
// (up to the sign of a zero u or v, which is set at the end).
__device__ __forceinline__ bool intersect_triangle(const RayPre &r, const float4 &v0, const float4 &v1,
                                                   const float4 &v2, float tmin, float tmax,
                                                   float &t_out, float &u_out, float &v_out) {
    const f3 a = ray_axes(r, v0), b = ray_axes(r, v1), c = ray_axes(r, v2);
    float Ax = __fsub_rn(a.x, __fmul_rn(r.sx, a.z));
    float Ay = __fsub_rn(a.y, __fmul_rn(r.sy, a.z));
    float Bx = __fsub_rn(b.x, __fmul_rn(r.sx, b.z));
    float By = __fsub_rn(b.y, __fmul_rn(r.sy, b.z));
    float Cx = __fsub_rn(c.x, __fmul_rn(r.sx, c.z));
    float Cy = __fsub_rn(c.y, __fmul_rn(r.sy, c.z));
    float U = __fsub_rn(__fmul_rn(Cx, By), __fmul_rn(Cy, Bx));
    float V = __fsub_rn(__fmul_rn(Ax, Cy), __fmul_rn(Ay, Cx));
    float W = __fsub_rn(__fmul_rn(Bx, Ay), __fmul_rn(By, Ax));
    if (U == 0.0f || V == 0.0f || W == 0.0f) {
        double CxBy = static_cast<double>(Cx) * static_cast<double>(By);
        double CyBx = static_cast<double>(Cy) * static_cast<double>(Bx);
        U = static_cast<float>(CxBy - CyBx);
        double AxCy = static_cast<double>(Ax) * static_cast<double>(Cy);
        double AyCx = static_cast<double>(Ay) * static_cast<double>(Cx);
        V = static_cast<float>(AxCy - AyCx);
        double BxAy = static_cast<double>(Bx) * static_cast<double>(Ay);
        double ByAx = static_cast<double>(By) * static_cast<double>(Ax);
        W = static_cast<float>(BxAy - ByAx);
    }
    if ((U < 0.0f || V < 0.0f || W < 0.0f) && (U > 0.0f || V > 0.0f || W > 0.0f)) return false;
    float det = __fadd_rn(__fadd_rn(U, V), W);
    if (det == 0.0f) return false;
    float Az = __fmul_rn(r.sz, a.z);
    float Bz = __fmul_rn(r.sz, b.z);
    float Cz = __fmul_rn(r.sz, c.z);
    float T = __fadd_rn(__fadd_rn(__fmul_rn(U, Az), __fmul_rn(V, Bz)), __fmul_rn(W, Cz));
    float t = __fdiv_rn(T, det);
    if (!(t > tmin && t < tmax)) return false;
    t_out = t;
    u_out = __fdiv_rn(V, det);
    v_out = __fdiv_rn(W, det);
    if (r.sz < 0.0f) {
        // A zero V or W came from the products above; swapped, its sign is
        // that of their difference the other way round.
        if (V == 0.0f)
            u_out = __fdiv_rn(static_cast<float>(static_cast<double>(Ay) * static_cast<double>(Cx) -
                                                 static_cast<double>(Ax) * static_cast<double>(Cy)), -det);
        if (W == 0.0f)
            v_out = __fdiv_rn(static_cast<float>(static_cast<double>(By) * static_cast<double>(Ax) -
                                                 static_cast<double>(Bx) * static_cast<double>(Ay)), -det);
    }
    return true;
}

// ---------------------------------------------------------------------------
// Compressed BVH8 traversal (node groups / triangle groups with an ordered hit
// mask, after Ylitie, Karras, Laine, HPG 2017).  Closest hit breaks exact ties
// in t by the lower primitive index, so the result does not depend on the
// traversal order.
// ---------------------------------------------------------------------------
constexpr int kStackSize = 32;
// Relative slack applied to box distances so that box culling is conservative
// with respect to the float triangle test.
constexpr float kBoxSlack = 1.000001f;

// A bound on the float triangle test's error in t for a hit on the triangle
// (a, b, c): 2^-16 of the vertices' largest coordinate distance from the ray
// origin, in units of t (over the ray's dominant direction component).  The
// test's error is absolute, of the order of the vertices' distances, so a
// relative slack alone does not cover hits at tiny t.  Closest-hit culling
// compares boxes against best_t plus this bound, so a box entered within the
// error of the best hit (another triangle at the same t, as on an edge shared
// next to the origin) is still opened.
__device__ __forceinline__ float tri_t_error(const RayPre &r, const float4 &v0, const float4 &v1, const float4 &v2) {
    const f3 a = ray_axes(r, v0), b = ray_axes(r, v1), c = ray_axes(r, v2);
    const float m = fmaxf(fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fmaxf(fabsf(a.z), fabsf(b.x))),
                          fmaxf(fmaxf(fabsf(b.y), fabsf(b.z)), fmaxf(fmaxf(fabsf(c.x), fabsf(c.y)), fabsf(c.z))));
    return m * fabsf(r.sz) * (1.0f / 65536.0f);
}

// Byte i of w, q, as the float 1 + q 2^-15: one byte permute.
__device__ __forceinline__ float ubyte_biased(uint32_t w, uint32_t i) {
    return __uint_as_float(__byte_perm(w, 0x3f800000u, 0x7604u | (i << 4)));
}
__device__ __forceinline__ float max3(float a, float b, float c) {
    float r;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
    float r;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(r) : "f"(a), "f"(b), "f"(c));
    return r;
}

// Tests the 8 children of one node; returns the new node and triangle groups.
//
// Traversal is bound by instruction issue (the nodes hit L1 and L2), so the
// test is written for few instructions per child: the near and far plane of
// each axis are picked once per node by the ray's octant (no minimum and
// maximum per axis and child), a plane distance is one byte permute and one
// multiply-add, U * (1 + q 2^-15) + (base - U) with U = 2^15 2^e / d, and the
// slab test is two three-input and two two-input minima and maxima.  Rounding
// base - U costs at most 2^-9 grid steps, which 2^-7 steps of slack on each
// side cover, besides cn and cf.  Empty slots hold zero boxes and zero meta
// bytes and contribute no bits, so they are not skipped.
// Measured, 2.1 M camera rays against 2.3 M triangles: 0.57 -> 0.41 ms; bounce
// rays 0.54 -> 0.37 ms, shadow rays 0.43 -> 0.31 ms; 10,000 emitters in a room,
// bounce rays 1.29 -> 0.87 ms (per-child reconstruction of both planes in
// floats, minima and maxima per axis before; ray replacement on both sides).
// Slower: both planes of an axis in one packed fma.rn.f32x2 (more registers),
// byte-to-float conversions in place of the permute, 96-byte nodes fetched
// with 32-byte loads, testing triangles only once 8 lanes have one.
__device__ __forceinline__ void intersect_children(const uint4 *nodes, uint32_t node_index, const RayPre &r,
                                                   float tmax, uint2 &node_group, uint2 &tri_group) {
    const uint4 *np = nodes + static_cast<size_t>(node_index) * 5u;
    const uint4 w0 = __ldg(np + 0);
    const uint4 w1 = __ldg(np + 1);
    const uint4 w2 = __ldg(np + 2);
    const uint4 w3 = __ldg(np + 3);
    const uint4 w4 = __ldg(np + 4);
    const float Ux = __uint_as_float((w0.w & 0xffu) << 23) * (r.inv_d.x * 32768.0f);
    const float Uy = __uint_as_float(((w0.w >> 8) & 0xffu) << 23) * (r.inv_d.y * 32768.0f);
    const float Uz = __uint_as_float(((w0.w >> 16) & 0xffu) << 23) * (r.inv_d.z * 32768.0f);
    const uint32_t imask = w0.w >> 24;
    const float px = __uint_as_float(w0.x), py = __uint_as_float(w0.y), pz = __uint_as_float(w0.z);
    const float g = 1.0f / 4194304.0f;
    const float bnx = fmaf(fabsf(Ux), -g, fmaf(px, r.inv_d.x, r.cn.x) - Ux);
    const float bny = fmaf(fabsf(Uy), -g, fmaf(py, r.inv_d.y, r.cn.y) - Uy);
    const float bnz = fmaf(fabsf(Uz), -g, fmaf(pz, r.inv_d.z, r.cn.z) - Uz);
    const float bfx = fmaf(fabsf(Ux), g, fmaf(px, r.inv_d.x, r.cf.x) - Ux);
    const float bfy = fmaf(fabsf(Uy), g, fmaf(py, r.inv_d.y, r.cf.y) - Uy);
    const float bfz = fmaf(fabsf(Uz), g, fmaf(pz, r.inv_d.z, r.cf.z) - Uz);
    const bool nx = r.oct & 1u, ny = r.oct & 2u, nz = r.oct & 4u;
    const uint32_t near_x[2] = {nx ? w3.z : w2.x, nx ? w3.w : w2.y}, far_x[2] = {nx ? w2.x : w3.z, nx ? w2.y : w3.w};
    const uint32_t near_y[2] = {ny ? w4.x : w2.z, ny ? w4.y : w2.w}, far_y[2] = {ny ? w2.z : w4.x, ny ? w2.w : w4.y};
    const uint32_t near_z[2] = {nz ? w4.z : w3.x, nz ? w4.w : w3.y}, far_z[2] = {nz ? w3.x : w4.z, nz ? w3.y : w4.w};
    uint32_t hits = 0;
#pragma unroll
    for (uint32_t c = 0; c < 8; ++c) {
        const uint32_t h = c >> 2, b = c & 3u;
        const float tn = fmaxf(max3(fmaf(ubyte_biased(near_x[h], b), Ux, bnx), fmaf(ubyte_biased(near_y[h], b), Uy, bny),
                                    fmaf(ubyte_biased(near_z[h], b), Uz, bnz)), 0.0f);
        const float tf = fminf(min3(fmaf(ubyte_biased(far_x[h], b), Ux, bfx), fmaf(ubyte_biased(far_y[h], b), Uy, bfy),
                                    fmaf(ubyte_biased(far_z[h], b), Uz, bfz)), tmax);
        if (tn <= tf) hits |= 1u << c;
    }
    // Internal children in traversal order: bit c moves to c ^ oct.
    uint32_t ihits = hits & imask;
    if (nx) ihits = ((ihits << 1) & 0xaau) | ((ihits >> 1) & 0x55u);
    if (ny) ihits = ((ihits << 2) & 0xccu) | ((ihits >> 2) & 0x33u);
    if (nz) ihits = ((ihits << 4) & 0xf0u) | (ihits >> 4);
    // Leaf children: their triangles (most nodes have few or none hit).
    uint32_t lhits = hits & ~imask, thits = 0;
    while (lhits) {
        const uint32_t c = __ffs(lhits) - 1u;
        lhits &= lhits - 1u;
        const uint32_t m = __byte_perm(w1.z, w1.w, c) & 0xffu;
        thits |= (m >> 5) << (m & 31u);
    }
    node_group = make_uint2(w1.x, (ihits << 24) | imask);
    tri_group = make_uint2(w1.y, thits);
}

__device__ __forceinline__ void count_traversal(const DeviceScene &s, uint32_t nodes, uint32_t tris) {
    if (s.stats) {
        atomicAdd(&s.stats[0], 1ull);
        atomicAdd(&s.stats[1], static_cast<unsigned long long>(nodes));
        atomicAdd(&s.stats[2], static_cast<unsigned long long>(tris));
    }
}

// ---------------------------------------------------------------------------
// Two-level traversal (instancing): the top level is the same BVH8 walk over
// instance boxes; a leaf entry's instance takes the ray into object space
// (world-to-object rows, explicitly rounded so that the oracle gets the same
// bits) and walks its mesh's BVH8.  Hits report global primitive ids (the
// instance's first primitive + the triangle's index in its mesh), and exact t
// ties go to the lower global id as in the one-level walk.
// ---------------------------------------------------------------------------
__device__ __forceinline__ f3 xf_point(const float4 &r0, const float4 &r1, const float4 &r2, f3 p) {
    return {__fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(r0.x, p.x), __fmul_rn(r0.y, p.y)), __fmul_rn(r0.z, p.z)), r0.w),
            __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(r1.x, p.x), __fmul_rn(r1.y, p.y)), __fmul_rn(r1.z, p.z)), r1.w),
            __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(r2.x, p.x), __fmul_rn(r2.y, p.y)), __fmul_rn(r2.z, p.z)), r2.w)};
}
__device__ __forceinline__ f3 xf_vector(const float4 &r0, const float4 &r1, const float4 &r2, f3 v) {
    return {__fadd_rn(__fadd_rn(__fmul_rn(r0.x, v.x), __fmul_rn(r0.y, v.y)), __fmul_rn(r0.z, v.z)),
            __fadd_rn(__fadd_rn(__fmul_rn(r1.x, v.x), __fmul_rn(r1.y, v.y)), __fmul_rn(r1.z, v.z)),
            __fadd_rn(__fadd_rn(__fmul_rn(r2.x, v.x), __fmul_rn(r2.y, v.y)), __fmul_rn(r2.z, v.z))};
}

// The largest coordinate magnitudes of the boxes below a node: its grid's.
VS_HD f3 node_bound(const uint4 &w0) {
    return {fabsf(bits_float(w0.x)) + 256.0f * bits_float((w0.w & 0xffu) << 23),
            fabsf(bits_float(w0.y)) + 256.0f * bits_float(((w0.w >> 8) & 0xffu) << 23),
            fabsf(bits_float(w0.z)) + 256.0f * bits_float(((w0.w >> 16) & 0xffu) << 23)};
}

// The closest hit inside instance `inst` with t below the current best.
static __device__ __noinline__ void instance_closest(const DeviceScene &s, const RayPre &rw, uint32_t inst,
                                                      float tmax, float &best_t, float &best_err, uint32_t &best_prim,
                                                      float &best_u, float &best_v, uint32_t &visits) {
    const float4 *x = s.inst_xf + 4u * inst;
    const float4 r0 = __ldg(x), r1 = __ldg(x + 1), r2 = __ldg(x + 2), meta = __ldg(x + 3);
    const uint32_t first = __float_as_uint(meta.y);
    const RayPre r = precompute_ray(xf_point(r0, r1, r2, rw.wo), xf_vector(r0, r1, r2, rw.wd),
                                    node_bound(__ldg(s.nodes + 5u * static_cast<size_t>(__float_as_uint(meta.x)))));
    uint2 stack[kStackSize];
    int sp = 0;
    uint2 ng = make_uint2(__float_as_uint(meta.x), (1u << (24u + (0u ^ r.oct))) | 1u);
    uint2 tg;
    while (true) {
        {
            uint32_t bit = __ffs(ng.y & 0xff000000u) - 1u;
            ng.y &= ~(1u << bit);
            uint32_t slot = (bit - 24u) ^ r.oct;
            uint32_t child = ng.x + __popc(ng.y & 0xffu & ((1u << slot) - 1u));
            if ((ng.y & 0xff000000u) != 0u && sp < kStackSize) stack[sp++] = ng;
            intersect_children(s.nodes, child, r, (best_t + best_err) * kBoxSlack, ng, tg);
            ++visits;
        }
        while (tg.y & 0x00ffffffu) {
            uint32_t bit = __ffs(tg.y & 0x00ffffffu) - 1u;
            tg.y &= ~(1u << bit);
            const float4 *tp = s.tri_v + static_cast<size_t>(tg.x + bit) * 3u;
            float4 a = __ldg(tp + 0), b = __ldg(tp + 1), c = __ldg(tp + 2);
            float t, u, v;
            float tri_tmax = best_prim == kInvalid ? tmax : best_t * kBoxSlack;
            if (intersect_triangle(r, a, b, c, 0.0f, tri_tmax, t, u, v)) {
                uint32_t prim = first + __float_as_uint(a.w);
                if (t < best_t || (t == best_t && prim < best_prim)) {
                    best_t = t; best_prim = prim; best_u = u; best_v = v;
                    best_err = tri_t_error(r, a, b, c);
                }
            }
        }
        if (ng.y <= 0x00ffffffu) {
            if (sp == 0) break;
            ng = stack[--sp];
        }
    }
}

// Whether the ray hits anything inside instance `inst` with t in (0, tmax).
static __device__ __noinline__ bool instance_any(const DeviceScene &s, const RayPre &rw, uint32_t inst, float tmax,
                                                 uint32_t &visits) {
    const float4 *x = s.inst_xf + 4u * inst;
    const float4 r0 = __ldg(x), r1 = __ldg(x + 1), r2 = __ldg(x + 2), meta = __ldg(x + 3);
    const RayPre r = precompute_ray(xf_point(r0, r1, r2, rw.wo), xf_vector(r0, r1, r2, rw.wd),
                                    node_bound(__ldg(s.nodes + 5u * static_cast<size_t>(__float_as_uint(meta.x)))));
    uint2 stack[kStackSize];
    int sp = 0;
    uint2 ng = make_uint2(__float_as_uint(meta.x), (1u << (24u + (0u ^ r.oct))) | 1u);
    uint2 tg;
    while (true) {
        {
            uint32_t bit = __ffs(ng.y & 0xff000000u) - 1u;
            ng.y &= ~(1u << bit);
            uint32_t slot = (bit - 24u) ^ r.oct;
            uint32_t child = ng.x + __popc(ng.y & 0xffu & ((1u << slot) - 1u));
            if ((ng.y & 0xff000000u) != 0u && sp < kStackSize) stack[sp++] = ng;
            intersect_children(s.nodes, child, r, tmax * kBoxSlack, ng, tg);
            ++visits;
        }
        while (tg.y & 0x00ffffffu) {
            uint32_t bit = __ffs(tg.y & 0x00ffffffu) - 1u;
            tg.y &= ~(1u << bit);
            const float4 *tp = s.tri_v + static_cast<size_t>(tg.x + bit) * 3u;
            float4 a = __ldg(tp + 0), b = __ldg(tp + 1), c = __ldg(tp + 2);
            float t, u, v;
            if (intersect_triangle(r, a, b, c, 0.0f, tmax, t, u, v)) return true;
        }
        if (ng.y <= 0x00ffffffu) {
            if (sp == 0) return false;
            ng = stack[--sp];
        }
    }
}

// Closest hit with t in (0, tmax).  Returns false on a miss.
static __device__ __noinline__ bool trace_closest(const DeviceScene &s, const RayPre &r, float tmax, Hit &hit,
                                           float &t_hit) {
    uint2 stack[kStackSize];
    int sp = 0;
    uint32_t nodes_visited = 0, tris_tested = 0;
    float best_t = tmax, best_err = 0.0f;
    uint32_t best_prim = kInvalid;
    float best_u = 0.0f, best_v = 0.0f;
    // Root as the only internal child (slot 0) of a virtual parent at index 0.
    uint2 ng = make_uint2(0u, (1u << (24u + (0u ^ r.oct))) | 1u);
    uint2 tg;
    // Invariant at the top of the loop: ng holds at least one internal hit.
    while (true) {
        {
            uint32_t bit = __ffs(ng.y & 0xff000000u) - 1u;
            ng.y &= ~(1u << bit);
            uint32_t slot = (bit - 24u) ^ r.oct;
            uint32_t child = ng.x + __popc(ng.y & 0xffu & ((1u << slot) - 1u));
            if ((ng.y & 0xff000000u) != 0u && sp < kStackSize) stack[sp++] = ng;
            intersect_children(s.nodes, child, r, (best_t + best_err) * kBoxSlack, ng, tg);
            ++nodes_visited;
        }
        if (s.two_level) {
            while (tg.y & 0x00ffffffu) {
                uint32_t bit = __ffs(tg.y & 0x00ffffffu) - 1u;
                tg.y &= ~(1u << bit);
                instance_closest(s, r, __ldg(s.tlas_inst + tg.x + bit), tmax, best_t, best_err, best_prim, best_u,
                                 best_v, nodes_visited);
            }
        }
        while (tg.y & 0x00ffffffu) {
            uint32_t bit = __ffs(tg.y & 0x00ffffffu) - 1u;
            tg.y &= ~(1u << bit);
            uint32_t ti = tg.x + bit;
            const float4 *tp = s.tri_v + static_cast<size_t>(ti) * 3u;
            float4 a = __ldg(tp + 0), b = __ldg(tp + 1), c = __ldg(tp + 2);
            float t, u, v;
            ++tris_tested;
            float tri_tmax = best_prim == kInvalid ? tmax : best_t * kBoxSlack;
            if (intersect_triangle(r, a, b, c, 0.0f, tri_tmax, t, u, v)) {
                uint32_t prim = __float_as_uint(a.w);
                if (t < best_t || (t == best_t && prim < best_prim)) {
                    best_t = t; best_prim = prim; best_u = u; best_v = v;
                    best_err = tri_t_error(r, a, b, c);
                }
            }
        }
        if (ng.y <= 0x00ffffffu) {
            if (sp == 0) break;
            ng = stack[--sp];
        }
    }
    count_traversal(s, nodes_visited, tris_tested);
    if (best_prim == kInvalid) return false;
    hit.prim_id = best_prim;
    hit.inst_id = __ldg(&s.prims[best_prim].w);
    hit.u = best_u;
    hit.v = best_v;
    t_hit = best_t;
    return true;
}

// Any hit with t in (0, tmax).
static __device__ __noinline__ bool trace_any(const DeviceScene &s, const RayPre &r, float tmax) {
    uint2 stack[kStackSize];
    int sp = 0;
    uint32_t nodes_visited = 0, tris_tested = 0;
    uint2 ng = make_uint2(0u, (1u << (24u + (0u ^ r.oct))) | 1u);
    uint2 tg;
    // Invariant at the top of the loop: ng holds at least one internal hit.
    while (true) {
        {
            uint32_t bit = __ffs(ng.y & 0xff000000u) - 1u;
            ng.y &= ~(1u << bit);
            uint32_t slot = (bit - 24u) ^ r.oct;
            uint32_t child = ng.x + __popc(ng.y & 0xffu & ((1u << slot) - 1u));
            if ((ng.y & 0xff000000u) != 0u && sp < kStackSize) stack[sp++] = ng;
            intersect_children(s.nodes, child, r, tmax * kBoxSlack, ng, tg);
            ++nodes_visited;
        }
        if (s.two_level) {
            while (tg.y & 0x00ffffffu) {
                uint32_t bit = __ffs(tg.y & 0x00ffffffu) - 1u;
                tg.y &= ~(1u << bit);
                if (instance_any(s, r, __ldg(s.tlas_inst + tg.x + bit), tmax, nodes_visited)) {
                    count_traversal(s, nodes_visited, tris_tested);
                    return true;
                }
            }
        }
        while (tg.y & 0x00ffffffu) {
            uint32_t bit = __ffs(tg.y & 0x00ffffffu) - 1u;
            tg.y &= ~(1u << bit);
            uint32_t ti = tg.x + bit;
            const float4 *tp = s.tri_v + static_cast<size_t>(ti) * 3u;
            float4 a = __ldg(tp + 0), b = __ldg(tp + 1), c = __ldg(tp + 2);
            float t, u, v;
            ++tris_tested;
            if (intersect_triangle(r, a, b, c, 0.0f, tmax, t, u, v)) {
                count_traversal(s, nodes_visited, tris_tested);
                return true;
            }
        }
        if (ng.y <= 0x00ffffffu) {
            if (sp == 0) break;
            ng = stack[--sp];
        }
    }
    count_traversal(s, nodes_visited, tris_tested);
    return false;
}

// Resumable traversal: the node and triangle visits of trace_closest /
// trace_any, one node (with the triangles it hit) per step, so that a warp can
// give a lane whose ray has finished a new ray while the others continue (ray
// replacement).  A ray visits the same nodes and triangles in the same order,
// so it gets the same result.
struct TravState {
    uint2 ng, tg;
    int sp;
    float tmax;
    float best_t;
    float best_err;  // tri_t_error of the best hit
    uint32_t best_prim;
    float best_u, best_v;
};

__device__ __forceinline__ void trav_init(TravState &t, const RayPre &r, float tmax) {
    t.ng = make_uint2(0u, (1u << (24u + (0u ^ r.oct))) | 1u);
    t.tg = make_uint2(0u, 0u);
    t.sp = 0;
    t.tmax = tmax;
    t.best_t = tmax;
    t.best_err = 0.0f;
    t.best_prim = kInvalid;
    t.best_u = 0.0f;
    t.best_v = 0.0f;
}

// Which traversal code a kernel compiles: kLevelsFlat (one world-space BVH8
// only), kLevelsTwo (instanced scenes only) or kLevelsAny (decided per ray
// from the scene: kernels that serve several scenes at once).  Kernels of one
// scene pick their instantiation on the host, so the flat traversal keeps its
// registers.
constexpr int kLevelsFlat = 0, kLevelsTwo = 1, kLevelsAny = 2;

// Resident blocks of 128 threads per SM asked of the flat traversal kernels:
// 64 registers a thread.  Left alone the compiler takes 96 to 128 of them for
// the unrolled child test, and with 4 or 5 blocks the passes take 20 % longer
// (2.1 M camera rays, 2.3 M triangles: 0.50 ms; 8 blocks 0.41, 9 blocks 0.43,
// 10 blocks 0.47).  The two-level kernels call their instance traversals out of
// line and are asked for 6 (80 registers instead of 146).
constexpr int kTraverseBlocks = 8;
constexpr int traverse_blocks(int levels) { return levels == kLevelsFlat ? kTraverseBlocks : 6; }

// One step of the closest-hit traversal; true when the traversal has ended
// (the result is in t.best_*).
template <int Levels = kLevelsFlat>
__device__ __forceinline__ bool closest_step(const DeviceScene &s, const RayPre &r, TravState &t, uint2 *stack) {
    {
        uint32_t bit = __ffs(t.ng.y & 0xff000000u) - 1u;
        t.ng.y &= ~(1u << bit);
        uint32_t slot = (bit - 24u) ^ r.oct;
        uint32_t child = t.ng.x + __popc(t.ng.y & 0xffu & ((1u << slot) - 1u));
        if ((t.ng.y & 0xff000000u) != 0u && t.sp < kStackSize) stack[t.sp++] = t.ng;
        intersect_children(s.nodes, child, r, (t.best_t + t.best_err) * kBoxSlack, t.ng, t.tg);
    }
    if (Levels == kLevelsTwo || (Levels == kLevelsAny && s.two_level)) {
        uint32_t visits = 0;
        while (t.tg.y & 0x00ffffffu) {
            uint32_t bit = __ffs(t.tg.y & 0x00ffffffu) - 1u;
            t.tg.y &= ~(1u << bit);
            instance_closest(s, r, __ldg(s.tlas_inst + t.tg.x + bit), t.tmax, t.best_t, t.best_err, t.best_prim,
                             t.best_u, t.best_v, visits);
        }
    }
    while (t.tg.y & 0x00ffffffu) {
        uint32_t bit = __ffs(t.tg.y & 0x00ffffffu) - 1u;
        t.tg.y &= ~(1u << bit);
        uint32_t ti = t.tg.x + bit;
        const float4 *tp = s.tri_v + static_cast<size_t>(ti) * 3u;
        float4 a = __ldg(tp + 0), b = __ldg(tp + 1), c = __ldg(tp + 2);
        float th, u, v;
        float tri_tmax = t.best_prim == kInvalid ? t.tmax : t.best_t * kBoxSlack;
        if (intersect_triangle(r, a, b, c, 0.0f, tri_tmax, th, u, v)) {
            uint32_t prim = __float_as_uint(a.w);
            if (th < t.best_t || (th == t.best_t && prim < t.best_prim)) {
                t.best_t = th;
                t.best_err = tri_t_error(r, a, b, c);
                t.best_prim = prim;
                t.best_u = u;
                t.best_v = v;
            }
        }
    }
    if (t.ng.y <= 0x00ffffffu) {
        if (t.sp == 0) return true;
        t.ng = stack[--t.sp];
    }
    return false;
}

// The hit of a finished closest-hit traversal (inst_id kInvalid: miss).
__device__ __forceinline__ Hit trav_hit(const DeviceScene &s, const TravState &t) {
    if (t.best_prim == kInvalid) return Hit{kInvalid, kInvalid, 0.0f, 0.0f};
    return Hit{__ldg(&s.prims[t.best_prim].w), t.best_prim, t.best_u, t.best_v};
}

// One step of the any-hit traversal; true when it has ended, with `hit` set
// when an intersection was found.
template <int Levels = kLevelsFlat>
__device__ __forceinline__ bool any_step(const DeviceScene &s, const RayPre &r, TravState &t, uint2 *stack,
                                         bool &hit) {
    {
        uint32_t bit = __ffs(t.ng.y & 0xff000000u) - 1u;
        t.ng.y &= ~(1u << bit);
        uint32_t slot = (bit - 24u) ^ r.oct;
        uint32_t child = t.ng.x + __popc(t.ng.y & 0xffu & ((1u << slot) - 1u));
        if ((t.ng.y & 0xff000000u) != 0u && t.sp < kStackSize) stack[t.sp++] = t.ng;
        intersect_children(s.nodes, child, r, t.tmax * kBoxSlack, t.ng, t.tg);
    }
    if (Levels == kLevelsTwo || (Levels == kLevelsAny && s.two_level)) {
        uint32_t visits = 0;
        while (t.tg.y & 0x00ffffffu) {
            uint32_t bit = __ffs(t.tg.y & 0x00ffffffu) - 1u;
            t.tg.y &= ~(1u << bit);
            if (instance_any(s, r, __ldg(s.tlas_inst + t.tg.x + bit), t.tmax, visits)) {
                hit = true;
                return true;
            }
        }
    }
    while (t.tg.y & 0x00ffffffu) {
        uint32_t bit = __ffs(t.tg.y & 0x00ffffffu) - 1u;
        t.tg.y &= ~(1u << bit);
        uint32_t ti = t.tg.x + bit;
        const float4 *tp = s.tri_v + static_cast<size_t>(ti) * 3u;
        float4 a = __ldg(tp + 0), b = __ldg(tp + 1), c = __ldg(tp + 2);
        float th, u, v;
        if (intersect_triangle(r, a, b, c, 0.0f, t.tmax, th, u, v)) {
            hit = true;
            return true;
        }
    }
    if (t.ng.y <= 0x00ffffffu) {
        if (t.sp == 0) {
            hit = false;
            return true;
        }
        t.ng = stack[--t.sp];
    }
    return false;
}

}  // namespace vs
