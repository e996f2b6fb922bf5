// sb_math.cuh — small float3 helpers and the per-probe geometry shared by the
// trace and blend kernels (gi_probes.js:1692-1726, gi_oct.js:61-85).
#pragma once
#include "sb_internal.cuh"

namespace sb {

__device__ __forceinline__ float3 mk(float x, float y, float z) { return make_float3(x, y, z); }
__device__ __forceinline__ float3 xyz(float4 v) { return make_float3(v.x, v.y, v.z); }
__device__ __forceinline__ float3 operator+(float3 a, float3 b) { return mk(a.x + b.x, a.y + b.y, a.z + b.z); }
__device__ __forceinline__ float3 operator-(float3 a, float3 b) { return mk(a.x - b.x, a.y - b.y, a.z - b.z); }
__device__ __forceinline__ float3 operator*(float3 a, float s) { return mk(a.x * s, a.y * s, a.z * s); }
__device__ __forceinline__ float3 mul3(float3 a, float3 b) { return mk(a.x * b.x, a.y * b.y, a.z * b.z); }
__device__ __forceinline__ float dot3(float3 a, float3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ float3 cross3(float3 a, float3 b) {
    return mk(a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x);
}
__device__ __forceinline__ float3 normalize3(float3 a) {
    float l = sqrtf(dot3(a, a));
    return a * (1.0f / l);
}
__device__ __forceinline__ float luma3(float3 c) { return c.x * 0.2126f + c.y * 0.7152f + c.z * 0.0722f; }
__device__ __forceinline__ float clampf(float v, float lo, float hi) { return fminf(fmaxf(v, lo), hi); }
__device__ __forceinline__ float mixf(float a, float b, float t) { return a * (1.0f - t) + b * t; }

// Two FP32 lanes per operation (PTX ISA 8.6), each rounded as the single one is.
__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ unsigned long long pack2(float2 v) { return pack2(v.x, v.y); }
__device__ __forceinline__ float2 unpack2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ unsigned long long mul2(unsigned long long a, unsigned long long b) {
    unsigned long long r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// Compensated (Kahan) accumulation s += w * x: the product enters through one
// FMA with the running compensation c, and c keeps the low part that the
// addition to s loses. The compiler does not reassociate these (no fast-math).
__device__ __forceinline__ void kahan_fma(float& s, float& c, float w, float x) {
    const float y = fmaf(w, x, -c);
    const float t = s + y;
    c = (t - s) - y;
    s = t;
}

// The probe of an update slot (both less than probeTotal).
__device__ __forceinline__ uint32_t probe_of(const DevCascade& C, uint32_t slot) {
    const uint32_t p = C.probeOffset + slot;
    return p < C.probeTotal ? p : p - C.probeTotal;
}

// Probe position, gi_probes.js:1714-1726 (relocation x classifyStrength = 0).
__device__ __forceinline__ float3 probe_world_pos(const DevCascade& C, uint32_t p) {
    uint32_t ix = p % C.res[0], iy = (p / C.res[0]) % C.res[1], iz = p / (C.res[0] * C.res[1]);
    float fx = float(ix) / fmaxf(1.0f, float(C.res[0]) - 1.0f);
    float fy = float(iy) / fmaxf(1.0f, float(C.res[1]) - 1.0f);
    float fz = float(iz) / fmaxf(1.0f, float(C.res[2]) - 1.0f);
    return mk(C.gridMin[0] + fx * C.gridSize[0], C.gridMin[1] + fy * C.gridSize[1], C.gridMin[2] + fz * C.gridSize[2]);
}

// Spherical-Fibonacci ray k of N with Cranley-Patterson rotation by the frame
// jitter, normalized (gi_probes.js:1692-1704, 1984, 2331):
//   z = 1 - 2 frac((k + 0.5)/N + j),  phi = k * pi (3 - sqrt 5) + 2 pi j.
// phi reaches hundreds of radians; evaluated naively in FP32 its rounding tilts
// the ray by ~1e-5 rad, and u = (k + 0.5)/N + j rounded to FP32 moves z by ~1e-7,
// which near the poles (small r) tilts the ray by ~1e-6 rad. So phi / pi, reduced
// mod 2, and u, z and r = sqrt(1 - z^2) = 2 sqrt(u (1 - u)) are formed in FP64
// (here it runs at half the FP32 rate, a tenth of what FP32 pairs cost); sincospif
// takes the rounded angle with a first-order correction for the rest, the square
// root one Newton step. The direction keeps ~1e-7 rad of error for every jitter.
__device__ __forceinline__ float3 ray_dir(uint32_t k, uint32_t N, float jitter) {
    const double G = (double)0.7639320492744446f + (double)-2.6774234385129603e-08f;  // 3 - sqrt(5)
    const double u = ((double)k + 0.5) / (double)N + (double)jitter;
    const double uw = u - floor(u);  // in [0, 1)
    const float z = (float)(1.0 - 2.0 * uw);
    const double s4 = uw * (1.0 - uw);  // (1 - z^2) / 4
    float r = 0.0f;
    if (s4 > 0.0) {
        const float r0 = sqrtf((float)s4);
        r = 2.0f * (r0 + (float)(s4 - (double)r0 * (double)r0) / (2.0f * r0));
    }
    double x = (double)k * G + 2.0 * (double)jitter;
    x -= 2.0 * floor(x * 0.5);
    const float hi = (float)x;
    float s, c;
    sincospif(hi, &s, &c);
    const float d = 3.141592653589793f * (float)(x - (double)hi);
    const float s1 = fmaf(c, d, s), c1 = fmaf(-s, d, c);
    return normalize3(mk(r * c1, r * s1, z));
}

// octEncodeNode / octDecodeNode, gi_oct.js:61-85
__device__ __forceinline__ float2 oct_encode(float3 n) {
    float inv = 1.0f / fmaxf(fabsf(n.x) + fabsf(n.y) + fabsf(n.z), 1e-20f);
    float ox = n.x * inv, oy = n.y * inv;
    float fx = (1.0f - fabsf(oy)) * (ox >= 0.0f ? 1.0f : -1.0f);
    float fy = (1.0f - fabsf(ox)) * (oy >= 0.0f ? 1.0f : -1.0f);
    bool lower = n.z < 0.0f;
    float ex = lower ? fx : ox, ey = lower ? fy : oy;
    return make_float2(ex * 0.5f + 0.5f, ey * 0.5f + 0.5f);
}
__device__ __forceinline__ float3 oct_decode(float u, float v) {
    float fx = u * 2.0f - 1.0f, fy = v * 2.0f - 1.0f;
    float nz = 1.0f - fabsf(fx) - fabsf(fy);
    float t = fmaxf(-nz, 0.0f);
    float nx = fx + (fx >= 0.0f ? -t : t);
    float ny = fy + (fy >= 0.0f ? -t : t);
    return normalize3(mk(nx, ny, nz));
}

__device__ __forceinline__ float4 half4_to_float4(uint2 h) {
    __half2 a = *reinterpret_cast<__half2*>(&h.x), b = *reinterpret_cast<__half2*>(&h.y);
    float2 fa = __half22float2(a), fb = __half22float2(b);
    return make_float4(fa.x, fa.y, fb.x, fb.y);
}
__device__ __forceinline__ uint2 float4_to_half4(float4 v) {
    __half2 a = __floats2half2_rn(v.x, v.y), b = __floats2half2_rn(v.z, v.w);
    uint2 r;
    r.x = *reinterpret_cast<uint32_t*>(&a);
    r.y = *reinterpret_cast<uint32_t*>(&b);
    return r;
}

// Footprints: what a bilinear read inside a probe's 8 x 8 tile needs, side by side.
// The tile-local coordinate 0.5 + uv * 6 lies in [0.5, 6.5], so a read starts at one
// of 7 x 7 texels; footprint (x, y) of probe p, at p * 49 + y * 7 + x, holds texels
// (x, y), (x + 1, y), (x, y + 1), (x + 1, y + 1) as binary16: the colours' (r, g)
// pairs, then b and the alphas of the rows (32 bytes); the depth moments' pairs (16
// bytes). The atlases hold the same texels for the host; the readers here take one
// load per tap instead of four, in one to two cache lines per probe instead of one
// per texel row.
constexpr uint32_t FOOT = 7u * 7u;
constexpr uint32_t FOOT_U4 = 2u;  // uint4 per colour footprint

struct FootTap {
    uint32_t at;  // y * 7 + x
    float fx, fy;
};
__device__ __forceinline__ FootTap foot_tap(float2 o) {
    const float xl = fmaf(o.x, 6.0f, 0.5f), yl = fmaf(o.y, 6.0f, 0.5f);
    const float x0 = floorf(xl), y0 = floorf(yl);
    return {(uint32_t)y0 * 7u + (uint32_t)x0, xl - x0, yl - y0};
}
// The bilinear weights of texels 00, 10, 01, 11.
__device__ __forceinline__ float4 foot_weights(const FootTap& t) {
    return make_float4((1.0f - t.fx) * (1.0f - t.fy), t.fx * (1.0f - t.fy), (1.0f - t.fx) * t.fy, t.fx * t.fy);
}
__device__ __forceinline__ float2 half2_at(uint32_t w) { return __half22float2(*reinterpret_cast<const __half2*>(&w)); }
// Two float4 as one 32-byte operation (p 32-byte aligned).
__device__ __forceinline__ void store32(float4* p, float4 a, float4 b) {
    asm volatile("st.global.v8.f32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "f"(a.x), "f"(a.y), "f"(a.z),
                 "f"(a.w), "f"(b.x), "f"(b.y), "f"(b.z), "f"(b.w)
                 : "memory");
}
__device__ __forceinline__ void load_foot(const uint4* p, uint32_t w[8]) {
    asm("ld.global.nc.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
        : "l"(p));
}
__device__ __forceinline__ float bilerp(float a, float b, float c, float d, float4 w) {
    return a * w.x + b * w.y + c * w.z + d * w.w;
}
__device__ __forceinline__ float3 foot_rgb(const uint4* foot, uint32_t at, float4 w) {
    uint32_t u[8];
    load_foot(foot + FOOT_U4 * at, u);
    const float2 a = half2_at(u[0]), b = half2_at(u[1]), c = half2_at(u[2]), d = half2_at(u[3]);
    const float2 b0 = half2_at(u[4]), b1 = half2_at(u[5]);
    return mk(bilerp(a.x, b.x, c.x, d.x, w), bilerp(a.y, b.y, c.y, d.y, w), bilerp(b0.x, b0.y, b1.x, b1.y, w));
}
__device__ __forceinline__ float4 foot_rgba(const uint4* foot, uint32_t at, float4 w) {
    uint32_t u[8];
    load_foot(foot + FOOT_U4 * at, u);
    const float2 a = half2_at(u[0]), b = half2_at(u[1]), c = half2_at(u[2]), d = half2_at(u[3]);
    const float2 b0 = half2_at(u[4]), b1 = half2_at(u[5]), a0 = half2_at(u[6]), a1 = half2_at(u[7]);
    return make_float4(bilerp(a.x, b.x, c.x, d.x, w), bilerp(a.y, b.y, c.y, d.y, w), bilerp(b0.x, b0.y, b1.x, b1.y, w),
                       bilerp(a0.x, a0.y, a1.x, a1.y, w));
}
__device__ __forceinline__ float2 foot_depth(const uint4* foot, uint32_t at, float4 w) {
    const uint4 u = __ldg(foot + at);
    const float2 a = half2_at(u.x), b = half2_at(u.y), c = half2_at(u.z), d = half2_at(u.w);
    return make_float2(bilerp(a.x, b.x, c.x, d.x, w), bilerp(a.y, b.y, c.y, d.y, w));
}
// A footprint from its four texels (RGBA16F: rg | ba).
__device__ __forceinline__ void store_foot(uint4* foot, uint32_t at, uint2 t00, uint2 t10, uint2 t01, uint2 t11) {
    foot[FOOT_U4 * at] = make_uint4(t00.x, t10.x, t01.x, t11.x);
    foot[FOOT_U4 * at + 1u] = make_uint4(__byte_perm(t00.y, t10.y, 0x5410u), __byte_perm(t01.y, t11.y, 0x5410u),
                                         __byte_perm(t00.y, t10.y, 0x7632u), __byte_perm(t01.y, t11.y, 0x7632u));
}

}  // namespace sb
