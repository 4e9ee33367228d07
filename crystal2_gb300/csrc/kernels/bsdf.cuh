// BSDFs of the reference's materials, evaluated in the local frame (x = dpdu, y = N, z = dpdv).
//
// Every material of the reference builds exactly one BxDF per hit (Materials/*.cpp), so the
// BSDF container (BSDFs/BSDF.cpp:25-130) reduces to: world->local by the transposed TNB frame
// and fixVector, the reflect/transmit selection of Pdf and DistributionFunction (with the
// operator-precedence behaviour of BSDF.cpp:39-40), and one sampled BxDF.
#pragma once
#include "dev_common.cuh"

namespace c2g {

struct Frame {
    float3 T, N, B;  // dpdu, shading normal (facing the incoming ray), dpdv
};

__device__ __forceinline__ float3 to_local(const Frame& f, float3 w) {
    return clamp1(f3(dot(f.T, w), dot(f.N, w), dot(f.B, w)));
}
__device__ __forceinline__ float3 to_world(const Frame& f, float3 w) {
    return clamp1(f.T * w.x + f.N * w.y + f.B * w.z);
}

struct BxDF {
    int mtype;
    int flags;          // BxDFType of the material's BxDF
    float3 R;           // color / kd
    float3 R_pi;        // R / pi (diffuse, Oren-Nayar)
    float3 S;           // ks (plastic)
    float ax, ay;
    float etaA, etaB;
    float eta_ab, eta_ba;  // etaA / etaB, etaB / etaA
    float term_o;       // what f takes from wo alone (bsdf_prepare)
};

__device__ __forceinline__ int material_flags(int mtype) {
    switch (mtype) {
        case MAT_DIFFUSE: return BXDF_DIFFUSE | BXDF_REFLECTION;
        case MAT_MIRROR: return BXDF_SPECULAR | BXDF_REFLECTION;
        case MAT_GLASS_ROUGH: return BXDF_TRANSMISSION | BXDF_REFLECTION | BXDF_GLOSSY;
        case MAT_GLASS_SMOOTH: return BXDF_TRANSMISSION | BXDF_REFLECTION | BXDF_SPECULAR;
        case MAT_MICRO_GGX:
        case MAT_MICRO_BECKMANN: return BXDF_REFLECTION | BXDF_GLOSSY;
        case MAT_PLASTIC_GGX:
        case MAT_PLASTIC_BECKMANN: return BXDF_REFLECTION | BXDF_GLOSSY;
        case MAT_ORENNAYAR: return BXDF_DIFFUSE | BXDF_REFLECTION;
        case MAT_BLINNPHONG: return BXDF_GLOSSY | BXDF_REFLECTION;
    }
    return 0;
}

__device__ __forceinline__ BxDF make_bxdf(const Material& m, bool front_face) {
    BxDF b;
    b.mtype = m.type;
    b.flags = material_flags(m.type);
    b.R = f3(m.color[0], m.color[1], m.color[2]);
    b.R_pi = f3(m.color_pi[0], m.color_pi[1], m.color_pi[2]);
    b.S = f3(m.ks[0], m.ks[1], m.ks[2]);
    b.ax = m.ax;
    b.ay = m.ay;
    // Glass / Micro swap the IORs on back faces (Glass.cpp:19-20, MicrofacetMaterial.cpp:20-21);
    // Mirror uses 1, 1 (MirrorMaterial.cpp:11-13).
    b.etaA = 1.f;
    const bool dielectric = m.type != MAT_MIRROR && m.type != MAT_DIFFUSE && m.type != MAT_ORENNAYAR && m.type != MAT_BLINNPHONG;
    b.etaB = dielectric ? m.ior : 1.f;
    if (!front_face && dielectric) { float t = b.etaA; b.etaA = b.etaB; b.etaB = t; }
    b.eta_ab = b.etaA / b.etaB;
    b.eta_ba = b.etaB / b.etaA;
    if (m.type == MAT_BLINNPHONG) b.ax = m.ior;  // the exponent K
    return b;
}

__device__ __forceinline__ float sq(float x) { return x * x; }

// x / pi, correctly rounded, for x in [0, 1].  The quotient's remainder is exact in an FMA, so one
// correction of x * (1 / pi) rounds it right (Markstein 1990); checked against the division for every
// mantissa.  Below 2^-100, where the remainder could lose bits, the division itself.  A rounded division
// is some ten instructions and a diffuse vertex with two lights made 42, 16 of them by pi; with R / pi
// ready in the material and this, shading of the Cornell box takes 2.15 ms instead of 2.39.
__device__ __forceinline__ float over_pi(float x) {
    const float inv = 1.0f / kPiF, q = __fmul_rn(x, inv);
    return x > 0x1p-100f ? __fmaf_rn(__fmaf_rn(-kPiF, q, x), inv, q) : x / kPiF;
}

// ---- Fresnel (BSDFs/Models/Fresnel.cpp) -------------------------------------------------
__device__ __forceinline__ float fresnel_dielectric(const BxDF& b, float cosI) {
    const float etaA = b.etaA, etaB = b.etaB;
    float sinI = sqrtf(fmaxf(0.f, 1.f - cosI * cosI));
    float sinT = b.eta_ab * sinI;
    if (sinT >= 1.f) return 1.f;
    float cosT = sqrtf(fmaxf(0.f, 1.f - sinT * sinT));
    float rparl = ((etaB * cosI) - (etaA * cosT)) / ((etaB * cosI) + (etaA * cosT));
    float rperp = ((etaA * cosI) - (etaB * cosT)) / ((etaA * cosI) + (etaB * cosT));
    return (rparl * rparl + rperp * rperp) / 2;
}
__device__ __forceinline__ float fresnel_schlick(float r0, const BxDF& b, float cosI) {
    float sinI = sqrtf(fmaxf(0.f, 1.f - cosI * cosI));
    float sinT = b.eta_ab * sinI;
    if (sinT >= 1.f) return 1.f;
    return r0 + (1.f - r0) * powf(1.f - cosI, 5.f);
}
// Micro uses Schlick with R0 = 0.99 (MicrofacetMaterial.cpp:23); glass uses the dielectric.
__device__ __forceinline__ float bxdf_fresnel(const BxDF& b, float cosI) {
    if (b.mtype == MAT_MICRO_GGX || b.mtype == MAT_MICRO_BECKMANN) return fresnel_schlick(0.99f, b, cosI);
    return fresnel_dielectric(b, cosI);
}

// ---- microfacet distributions (BSDFs/Models/MicrofacetDistribution.cpp) -------------------
__device__ __forceinline__ bool is_beckmann(int mtype) { return mtype == MAT_MICRO_BECKMANN || mtype == MAT_PLASTIC_BECKMANN; }

__device__ __forceinline__ float2 cos_sin_phi(float3 w, float sinT) {
    if (sinT == 0.f) return make_float2(1.f, 0.f);
    return make_float2(fminf(fmaxf(w.x / sinT, -1.f), 1.f), fminf(fmaxf(-w.z / sinT, -1.f), 1.f));
}

__device__ __forceinline__ float ndf_D(const BxDF& b, float3 wh, Rounding r) {
    if (!is_beckmann(b.mtype)) {
        float cos2 = wh.y * wh.y;
        float sin2 = fmaxf(0.f, r == Rounding::FREE ? 1.f - cos2 : r == Rounding::SAMPLED ? one_minus_rounded_sq(wh.y) : one_minus_sq(wh.y));
        float2 p = cos_sin_phi(wh, sqrtf(sin2));
        float A = sq(p.x) / sq(b.ax) + sq(p.y) / sq(b.ay);
        return 1.f / (kPiF * b.ax * b.ay * sq(r == Rounding::FREE ? A - cos2 * (A - 1) : __fmaf_rn(-cos2, A - 1, A)));
    }
    float cos2 = wh.y * wh.y;
    float sin2 = r == Rounding::FREE ? 1.f - cos2 : one_minus_rounded_sq(wh.y);
    float tan2 = sin2 / cos2;
    if (isinf(tan2)) return 0.f;
    float cos4 = cos2 * cos2;
    float2 v = cos_sin_phi(wh, sqrtf(r == Rounding::LIGHT ? one_minus_sq(wh.y) : sin2));
    float bot = kPiF * b.ax * b.ay * cos4;
    float top = expf(-tan2 * (sq(v.x) / sq(b.ax) + sq(v.y) / sq(b.ay)));
    return top / bot;
}

__device__ __forceinline__ float ndf_lambda(const BxDF& b, float3 w, Rounding r) {
    if (!is_beckmann(b.mtype)) {
        float cos2 = w.y * w.y;
        float sin2 = r == Rounding::FREE ? 1.f - cos2 : one_minus_rounded_sq(w.y);
        float tan2 = sin2 / cos2;
        if (isinf(tan2)) return 0.f;
        float2 p = cos_sin_phi(w, sqrtf(r == Rounding::LIGHT ? one_minus_sq(w.y) : sin2));
        float a2 = sq(p.x) * sq(b.ax) + sq(p.y) * sq(b.ay);
        return (-1 + sqrtf(1 + a2 * tan2)) / 2;
    }
    float cosT = w.y;
    float sinT = sqrtf(1.f - cosT * cosT);
    float tanT = fabsf(sinT / cosT);
    if (isinf(tanT)) return 0.f;
    float2 v = cos_sin_phi(w, sinT);
    float alpha = sqrtf(sq(v.x) * sq(b.ax) + sq(v.y) * sq(b.ay));
    float a = 1.f / (tanT * alpha);
    if (a >= 1.6f) return 0.f;
    return (1 - 1.259f * a + 0.396f * a * a) / (3.535f * a + 2.181f * a * a);
}

// Smith's G of the prepared wo (b.term_o is its Lambda) and wi.
__device__ __forceinline__ float ndf_G(const BxDF& b, float3 wi, Rounding r) { return 1.f / (1.f + b.term_o + ndf_lambda(b, wi, r)); }

// GetUnitVectorUsingCos (Utils.h:79-83)
__device__ __forceinline__ float3 unit_from_cos(float cosT, float phi) {
    float r = sqrtf(1 - cosT * cosT);
    float s, c;
    sincosf(phi, &s, &c);
    return f3(r * c, cosT, -r * s);
}

__device__ __forceinline__ float3 ndf_sample(const BxDF& b, float2 u) {
    float cosT, phi;
    if (!is_beckmann(b.mtype)) {
        if (b.ax == b.ay) {
            cosT = sqrtf((1 - u.x) / (u.x * (b.ax * b.ax - 1) + 1));
            phi = kTwoPiF * u.y;
        } else {
            phi = atanf(b.ay / b.ax * tanf(kTwoPiF * u.y + kHalfPiF));
            if (u.y > 0.5f) phi += kPiF;
            float s, c;
            sincosf(phi, &s, &c);
            float A = sq(c) / sq(b.ax) + sq(s) / sq(b.ay);
            float cos2 = A * (u.x - 1) / (u.x * (A - 1) - A);
            cosT = sqrtf(cos2);
        }
        return unit_from_cos(cosT, phi);
    }
    float logS = logf(1.f - u.x);
    if (isinf(logS)) logS = 0;
    float tan2;
    if (b.ax == b.ay) {
        tan2 = -sq(b.ax) * logS;
        phi = u.y * kTwoPiF;
    } else {
        phi = atanf(b.ay / b.ax * tanf(kTwoPiF * u.y + kHalfPiF));
        if (u.y > 0.5f) phi += kPiF;
        float s, c;
        sincosf(phi, &s, &c);
        tan2 = -logS / (c * c / sq(b.ax) + s * s / sq(b.ay));
    }
    cosT = 1.f / sqrtf(1.f + tan2);
    return unit_from_cos(cosT, phi);
}

__device__ __forceinline__ float3 reflect(float3 I, float3 N) { return I - N * dot(N, I) * 2.f; }

// refract(wo, wh, eta, wt) (Utils.h:102-112)
__device__ __forceinline__ bool refract(float3 wo, float3 wh, float eta, float3& wt) {
    float cosO = fminf(fmaxf(dot(wo, wh), -1.f), 1.f);
    float sin2O = fmaxf(0.f, 1.f - cosO * cosO);
    float sin2I = eta * eta * sin2O;
    if (sin2I > 1.f) return false;
    float cosI = sqrtf(1.f - sin2I);
    wt = eta * (-wo) + (eta * cosO - cosI) * wh;
    return true;
}

// ---- microfacet BxDFs (BSDFs/Microfacet.cpp) --------------------------------------------
// The density of a direction and the value of the BxDF share the half vector H and D(H); a vertex
// evaluates them for every light and for two samples of its own, and a GGX evaluation is some twenty
// divisions and square roots.  So Lambda(wo), and the Fresnel blend's power of wo, are kept for the vertex
// (bsdf_prepare), and a sampled direction uses its H and D twice, unless the clamp that follows the
// density changed it.  Shading of the slit room (most of it GGX): 4.65 -> 4.30 ms, of the many-material frame 12.7 -> 11.3.
__device__ __forceinline__ float mf_refl_pdf(float3 wo, float3 H, float D) { return D * fabsf(H.y) / (4 * dot(wo, H)); }
__device__ __forceinline__ float3 mf_refl_f(const BxDF& b, float3 wo, float3 wi, float3 H, float D, Rounding r) {
    if (wo.y * wi.y < 0) return f3(0.f, 0.f, 0.f);
    float F = bxdf_fresnel(b, fmaxf(0.f, dot(wo, H)));
    float G = ndf_G(b, wi, r);
    return b.R * D * G * F / (4 * fmaxf(0.f, wi.y) * fmaxf(0.f, wo.y));
}
__device__ __forceinline__ float mf_trans_pdf(const BxDF& b, float3 wo, float3 wi, float3 H, float D) {
    if (wo.y * wi.y > 0) return 0.f;
    float eta = b.eta_ba;
    float s = dot(wo, H) + eta * dot(wi, H);
    return D * fabsf(H.y) * (eta * eta * fabsf(dot(H, wi)) / sq(s));
}
__device__ __forceinline__ float3 mf_trans_f(const BxDF& b, float3 wo, float3 wi, float3 H, float D, Rounding r) {
    if (wi.y * wo.y > 0) return f3(0.f, 0.f, 0.f);
    if (wo.y == 0.f) return f3(0.f, 0.f, 0.f);
    float eta = b.eta_ba;
    if (H.y < 0) H = -H;  // D is even in H
    float bot = sq(dot(wo, H) + eta * dot(wi, H));
    float F = 1.f - bxdf_fresnel(b, fmaxf(0.f, dot(wo, H)));
    float G = ndf_G(b, wi, r);
    return b.R * D * G * F * fabsf(dot(H, wo)) * fabsf(dot(H, wi)) / (bot * fmaxf(0.f, -wi.y) * fmaxf(0.f, wo.y));
}
// Half vector of a reflection, or of a transmission.
__device__ __forceinline__ float3 mf_half(const BxDF& b, bool trans, float3 wo, float3 wi) {
    return normalize(wo + wi * (trans ? b.eta_ba : 1.f));
}
// f and pdf of one (wo, wi) pair.
__device__ __forceinline__ float3 mf_f_pdf(const BxDF& b, bool trans, float3 wo, float3 wi, float& pdf, Rounding r) {
    const float3 H = mf_half(b, trans, wo, wi);
    const float D = ndf_D(b, H, r);
    pdf = trans ? mf_trans_pdf(b, wo, wi, H, D) : mf_refl_pdf(wo, H, D);
    return trans ? mf_trans_f(b, wo, wi, H, D, r) : mf_refl_f(b, wo, wi, H, D, r);
}
// f and pdf of a sampled direction: the density of wi as drawn, then f of wi clamped to [-1, 1].  The
// density takes the technique from wi's side (glass), f from the technique that drew it.
__device__ __forceinline__ float3 mf_sampled(const BxDF& b, bool trans, float3 wo, float3& wi, float& pdf, Rounding r) {
    const bool across = b.mtype == MAT_GLASS_ROUGH && wo.y * wi.y < 0;
    float3 H = mf_half(b, across, wo, wi);
    float D = ndf_D(b, H, r);
    pdf = across ? mf_trans_pdf(b, wo, wi, H, D) : mf_refl_pdf(wo, H, D);
    const float3 c = clamp1(wi);
    if (c.x != wi.x || c.y != wi.y || c.z != wi.z || trans != across) {
        H = mf_half(b, trans, wo, c);
        D = ndf_D(b, H, r);
    }
    wi = c;
    return trans ? mf_trans_f(b, wo, wi, H, D, r) : mf_refl_f(b, wo, wi, H, D, r);
}

// ---- FresnelBlend (BSDFs/FresnelBlend.cpp) ----------------------------------------------
__device__ __forceinline__ float fb_power(float cosT) { return 1.f - powf(1.f - 0.5f * cosT, 5.f); }
__device__ __forceinline__ float3 fb_f_pdf(const BxDF& b, float3 wo, float3 wi, float& pdf, Rounding r) {
    float3 H = normalize(wo + wi);
    float D = ndf_D(b, H, r);
    pdf = 0.5f * (over_pi(fmaxf(0.f, wi.y)) + D * fabsf(H.y) / (4 * dot(wo, H)));
    float cosI = fmaxf(0.f, wi.y), cosO = fmaxf(0.f, wo.y);
    float k = (28.f / (23.f * kPiF));
    float3 diffuse = k * b.R * (f3(1.f, 1.f, 1.f) - b.S) * b.term_o;  // times fb_power(cosI)
    float cwh = dot(wi, H);
    float sp = D / (4 * cwh * fmaxf(cosI, cosO));
    float3 schlick = b.S + (f3(1.f, 1.f, 1.f) - b.S) * powf(1.f - cwh, 5.f);
    const float pw = fb_power(cosI);
    if (r == Rounding::FREE) return diffuse * pw + sp * schlick;
    return f3(__fmaf_rn(diffuse.x, pw, __fmul_rn(sp, schlick.x)), __fmaf_rn(diffuse.y, pw, __fmul_rn(sp, schlick.y)),
              __fmaf_rn(diffuse.z, pw, __fmul_rn(sp, schlick.z)));
}

// ---- Oren-Nayar (BSDFs/Reflections.cpp:7-66); A, B in ax, ay -----------------------------
__device__ __forceinline__ float3 on_f(const BxDF& b, float3 wo, float3 wi) {
    const float sinO = sqrtf(fmaxf(0.f, 1.f - wo.y * wo.y)), sinI = sqrtf(fmaxf(0.f, 1.f - wi.y * wi.y));
    float sinA, tanB;
    if (wo.y < wi.y) { sinA = sinI; tanB = sinO / wo.y; }
    else { sinA = sinO; tanB = sinI / wi.y; }
    float dcos = 0.f;
    if (sinI > 1e-5f && sinO > 1e-5f) {
        const float2 dI = cos_sin_phi(wi, sinI), dO = cos_sin_phi(wo, sinO);
        dcos = fmaxf(0.f, dI.x * dO.x + dI.y * dO.y);
    }
    return b.R_pi * (b.ax + b.ay * (dcos * sinA * tanB));
}

// ---- Blinn-Phong (BSDFs/BlinnPhongReflection.cpp:14-58); exponent K in ax -------------------
// The reference raises float to int powers with std::pow, i.e. in double: so does this.
__device__ __forceinline__ float bp_pdf(const BxDF& b, float3 wo, float3 wi) {
    const float3 wh = normalize(wo + wi);
    const float k = b.ax;
    return (float)((double)((k + 2.f) / kTwoPiF) * pow((double)fmaxf(0.f, wh.y), (double)(k + 1.f)));
}
__device__ __forceinline__ float3 bp_f(const BxDF& b, float3 wo, float3 wi) {
    const float3 wh = normalize(wo + wi);
    const float k = b.ax;
    const float s = (float)pow((double)fmaxf(0.f, wh.y), (double)k) * (k + 2.f) / kTwoPiF;
    return b.R * s / (4.f * fmaxf(0.f, wi.y) * fmaxf(0.f, wo.y));
}
// A rejected half vector is redrawn.  The reference redraws from a static std::mt19937 shared by
// all render threads (BlinnPhongReflection.cpp:33-56), which no other run can reproduce; here the
// next pair is a hash of the rejected pair and the attempt number, and the loop stops after
// kPhongAttempts draws (the sample then fails) instead of looping without bound.
constexpr int kPhongAttempts = 64;
__device__ __forceinline__ float2 phong_redraw(float2 u, int attempt) {
    const uint32_t h = hash32(__float_as_uint(u.x) ^ hash32(__float_as_uint(u.y) + 0x9E3779B9u * (uint32_t)(attempt + 1)));
    const uint32_t g = hash32(h ^ 0x85EBCA6Bu);
    return make_float2((float)(h >> 8) * 0x1p-24f, (float)(g >> 8) * 0x1p-24f);
}

// ---- per-BxDF dispatch (local frame) ------------------------------------------------------
// f and pdf of the BxDF at one (wo, wi) pair.
__device__ __forceinline__ float3 bxdf_f_pdf(const BxDF& b, float3 wo, float3 wi, float& pdf, Rounding r) {
    switch (b.mtype) {
        case MAT_DIFFUSE: pdf = over_pi(fmaxf(0.f, wi.y)); return b.R_pi;
        case MAT_MICRO_GGX:
        case MAT_MICRO_BECKMANN: return mf_f_pdf(b, false, wo, wi, pdf, r);
        case MAT_GLASS_ROUGH: return mf_f_pdf(b, wo.y * wi.y < 0, wo, wi, pdf, r);
        case MAT_PLASTIC_GGX:
        case MAT_PLASTIC_BECKMANN: return fb_f_pdf(b, wo, wi, pdf, r);
        case MAT_ORENNAYAR: pdf = over_pi(fmaxf(0.f, wi.y)); return on_f(b, wo, wi);
        case MAT_BLINNPHONG: pdf = bp_pdf(b, wo, wi); return bp_f(b, wo, wi);
    }
    pdf = 0.f;
    return f3(0.f, 0.f, 0.f);
}

// NextCosineUnitHemiSphere (Utils.h:114-123)
__device__ __forceinline__ float3 cosine_hemisphere(float2 u, float& pdf) {
    float r = sqrtf(u.x);
    float phi = u.y * kTwoPiF;
    float s, c;
    sincosf(phi, &s, &c);
    float x = r * c, z = r * s;
    float y = sqrtf(1.0f - r * r);
    pdf = over_pi(y);
    return f3(x, y, z);
}

// BxDF::SampleDirection.  Returns f; writes wi (local), pdf and the sampled type.  A zero return
// leaves pdf as it was, like the reference.
__device__ __forceinline__ float3 bxdf_sample(const BxDF& b, float2 u, float3 wo, float3& wi, float& pdf, int& stype, Rounding r) {
    const float3 zero = f3(0.f, 0.f, 0.f);
    switch (b.mtype) {
        case MAT_DIFFUSE: {
            wi = cosine_hemisphere(u, pdf);
            return b.R_pi;
        }
        case MAT_MIRROR: {
            wi = f3(-wo.x, wo.y, -wo.z);
            pdf = 1.0f;
            return b.R;  // FresnelNoOp
        }
        case MAT_GLASS_SMOOTH: {  // SpecularFresnel (SpecularFresnel.cpp:28-46)
            float fr = fresnel_dielectric(b, wo.y);
            if (u.x < fr) {
                stype = BXDF_REFLECTION | BXDF_SPECULAR;
                wi = f3(-wo.x, wo.y, -wo.z);
                pdf = fr;
                return fr * b.R;
            }
            stype = BXDF_TRANSMISSION | BXDF_SPECULAR;
            refract(wo, f3(0.f, 1.f, 0.f), b.eta_ab, wi);
            pdf = 1.f - fr;
            return (1.f - fr) * b.R;
        }
        case MAT_MICRO_GGX:
        case MAT_MICRO_BECKMANN: {
            float3 wh = ndf_sample(b, u);
            if (dot(wo, wh) <= 0) return zero;
            wi = reflect(-wo, wh);
            return mf_sampled(b, false, wo, wi, pdf, r);
        }
        case MAT_GLASS_ROUGH: {  // MicrofacetBlend (Microfacet.cpp:164-199)
            float3 wh = ndf_sample(b, u);
            if (dot(wo, wh) <= 0) return zero;
            float fr = fresnel_dielectric(b, dot(wo, wh));
            const bool refl = u.x < fr;
            float3 t;
            const bool trans = !refl && refract(wo, wh, b.eta_ab, t);  // else total reflection
            stype = (trans ? BXDF_TRANSMISSION : BXDF_REFLECTION) | BXDF_GLOSSY;
            wi = trans ? t : reflect(-wo, wh);
            const float3 f = mf_sampled(b, trans, wo, wi, pdf, r);
            pdf = pdf * (refl ? fr : 1 - fr);
            return f;
        }
        case MAT_PLASTIC_GGX:
        case MAT_PLASTIC_BECKMANN: {  // FresnelBlend::SampleDirection
            float2 s = u;
            if (s.x < 0.5f) {
                s.x = s.x * 2.f;
                wi = cosine_hemisphere(s, pdf);
            } else {
                s.x = (s.x - 0.5f) * 2.f;
                float3 wh = ndf_sample(b, s);
                float3 L = reflect(-wo, wh);
                if (L.y * wo.y <= 0) return zero;
                wi = clamp1(L);
            }
            return fb_f_pdf(b, wo, wi, pdf, r);
        }
        case MAT_ORENNAYAR: {
            wi = cosine_hemisphere(u, pdf);
            return on_f(b, wo, wi);
        }
        case MAT_BLINNPHONG: {
            float2 s = u;
            for (int attempt = 0; attempt < kPhongAttempts; attempt++) {
                const float cosT = (float)pow((double)s.x, 1.0 / (double)(b.ax + 2.f));
                const float phi = kTwoPiF * s.y;
                const float3 N = unit_from_cos(cosT, phi);
                if (dot(N, wo) < 0.f) { s = phong_redraw(s, attempt); continue; }
                const float3 w = reflect(-wo, N);
                if (w.y < 0.f) { s = phong_redraw(s, attempt); continue; }
                wi = w;
                pdf = bp_pdf(b, wo, wi);
                return bp_f(b, wo, wi);
            }
            return zero;
        }
    }
    return zero;
}

// ---- BSDF container (BSDF.cpp) --------------------------------------------------------------
__device__ __forceinline__ bool matches(int bxdf_flags, int flags) { return (bxdf_flags & flags) == bxdf_flags; }

// The terms of f that depend on wo alone, once per vertex; before the calls below.
__device__ __forceinline__ void bsdf_prepare(BxDF& b, const Frame& fr, float3 wo_w, bool guided) {
    const float3 wo = to_local(fr, wo_w);
    switch (b.mtype) {
        case MAT_MICRO_GGX:
        case MAT_MICRO_BECKMANN:
        case MAT_GLASS_ROUGH: b.term_o = ndf_lambda(b, wo, guided ? Rounding::FREE : Rounding::SAMPLED); break;
        case MAT_PLASTIC_GGX:
        case MAT_PLASTIC_BECKMANN: b.term_o = fb_power(fmaxf(0.f, wo.y)); break;
        default: b.term_o = 0.f;
    }
}

// BSDF::DistributionFunction and BSDF::Pdf(flags) of one direction pair in one pass.
__device__ __forceinline__ float3 bsdf_f_pdf(const BxDF& b, const Frame& fr, float3 wo_w, float3 wi_w, int flags, float& pdf, bool guided) {
    float3 wo = to_local(fr, wo_w), wi = to_local(fr, wi_w);
    bool refl = wi.y * wo.y > 0;
    bool fcond = (refl && (b.flags & BXDF_REFLECTION)) || (!refl && (b.flags & BXDF_TRANSMISSION));
    bool pcond = (matches(b.flags, flags) && refl && (b.flags & BXDF_REFLECTION)) || (!refl && (b.flags & BXDF_TRANSMISSION));
    pdf = 0.f;
    float3 f = f3(0.f, 0.f, 0.f);
    if (fcond || pcond) {
        float p;
        float3 v = bxdf_f_pdf(b, wo, wi, p, guided ? Rounding::FREE : Rounding::LIGHT);
        if (fcond) f = v;
        if (pcond) pdf = p;
    }
    return f;
}

// Returns f; wi_w, pdf, stype written when the BxDF matches `flags`.  ok = false when the BSDF
// returned zero (no matching BxDF, or the sampled value/pdf is zero).
__device__ __forceinline__ float3 bsdf_sample(const BxDF& b, const Frame& fr, float u1, float2 u2, float3 wo_w,
                                              float3& wi_w, float& pdf, int flags, int& stype, bool& ok, bool guided) {
    ok = false;
    const float3 zero = f3(0.f, 0.f, 0.f);
    if (!matches(b.flags, flags)) return zero;
    (void)u1;  // one BxDF: (int)(min(0.9999999404f, u1) * 1) == 0
    stype = b.flags;
    float3 wo = to_local(fr, wo_w);
    float3 wi = zero;
    float3 L = bxdf_sample(b, u2, wo, wi, pdf, stype, guided ? Rounding::FREE : Rounding::SAMPLED);
    if (is_zero(L) || pdf == 0.f) return zero;
    wi_w = to_world(fr, wi);
    ok = true;
    return L;
}

}  // namespace c2g
