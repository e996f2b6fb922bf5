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

// Compensated (Kahan) accumulation s += w * x: the product enters through one
// FMA with the running compensation c, and c keeps the low part that the
// addition to s loses. The compiler does not reassociate these (no fast-math).
__device__ __forceinline__ void kahan_fma(float& s, float& c, float w, float x) {
    const float y = fmaf(w, x, -c);
    const float t = s + y;
    c = (t - s) - y;
    s = t;
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

}  // namespace sb
