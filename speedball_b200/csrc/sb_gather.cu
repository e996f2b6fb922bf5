// sb_gather.cu — the receiver gather: the irradiance the probe field gives a
// surface point, the consumer of the atlases this library updates. The
// reference evaluates it per fragment in GiProbeNode (gi_probes.js:530-657,
// 816-850, 884-928); here one thread evaluates one G-buffer sample.
//
// Per sample: P = position * samplePositionScale + Nvis * normalBias[0] *
// sampleBiasScale; with one cascade, _sampleCascade at P; with two, the coarse
// and fine looped gathers blended by the fine box's border band, each choosing
// its cage at the unbiased surface position (the looped gather's stated intent,
// gi_probes.js:628-631). Each of the 8 cage taps reads the RGBA16F atlas
// bilinearly (exact weights; the footprint stays inside the probe's tile, so the
// sampler's edge clamp never applies) in the detail normal's octahedral
// direction; with chebyStrength > 0 it also fetches the depth moments toward
// the surface for the Chebyshev visibility weight and applies the wrap weight.
// Output E = max(sample, 0) * intensity * enabled as float4 (rgb, 1).
//
// Work is one probe field's worth of tiny atlases (L1/L2-resident) against a
// streamed G-buffer: 48 bytes in and 16 bytes out per sample are the HBM traffic.
// What bounds it: the default receiver the L1's wavefronts (78%; 32 8-byte reads of
// the atlas rows took 91% of them for 57 us at 1080p, 8 32-byte reads of the
// footprints take 40 us), the others issue slots (about 100 instructions a tap with
// the Chebyshev weight: 77 -> 51 us at 1366 x 768 in two cascades; 325 with both
// lobes: 242 -> 200 us at 1080p, tier high). So texels are widened and summed two at
// a time (f32x2), nothing that is the same for the taps is formed per tap, and no
// index goes through a float-to-integer conversion. Classification is inert
// (classifyStrength 0): no state atlas is read.
#include "sb_kernels.cuh"
#include "sb_math.cuh"

namespace sb {

namespace {

// Reciprocals and square roots of normal numbers, one instruction each (1 ulp, and
// 2 ulp for the inverse square root); denormal arguments count as 0.
__device__ __forceinline__ float rcp_fast(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_fast(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float sqrt_fast(float x) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ float3 fast_normalize(float3 a) { return a * rsqrt_fast(dot3(a, a)); }

// The cage of a point: its first probe, the point's fractions, and per tap i (bits
// x, y, z) the trilinear weight and the probe's index.
struct Cage {
    float base[3], frac[3];
    uint32_t first, dy, dz;  // probe index of tap 0; steps along y and z
};
__device__ __forceinline__ Cage cage_of(const GatherCascade& C, float3 p) {
    Cage g;
    const float cp[3] = {p.x, p.y, p.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float gf = (cp[a] - C.gridMin[a]) * C.perCell[a];
        g.base[a] = clampf(floorf(gf), 0.0f, C.lastBase[a]);
        g.frac[a] = clampf(gf - g.base[a], 0.0f, 1.0f);
    }
    g.dy = C.resX;
    g.dz = C.resX * C.resY;
    g.first = (uint32_t)g.base[2] * g.dz + (uint32_t)g.base[1] * g.dy + (uint32_t)g.base[0];
    return g;
}
__device__ __forceinline__ float cage_weight(const Cage& g, int i) {
    const float wx = i & 1 ? g.frac[0] : 1.0f - g.frac[0], wy = i & 2 ? g.frac[1] : 1.0f - g.frac[1],
                wz = i & 4 ? g.frac[2] : 1.0f - g.frac[2];
    return wx * wy * wz + 1e-4f;
}
__device__ __forceinline__ uint32_t cage_probe(const Cage& g, int i) {
    return g.first + (i & 1 ? 1u : 0u) + (i & 2 ? g.dy : 0u) + (i & 4 ? g.dz : 0u);
}

// octEncodeNode of a direction of any length (the encoding divides by the L1 norm).
// A zero or infinite one gives NaN weights, and those an output of 0; with `safe` a
// zero one encodes as octEncodeNode's floor makes it.
__device__ __forceinline__ float2 oct_any(float3 n, bool safe = false) {
    const float l1 = fabsf(n.x) + fabsf(n.y) + fabsf(n.z);
    const float inv = rcp_fast(safe ? fmaxf(l1, 1e-20f) : l1);
    const float ox = n.x * inv, oy = n.y * inv;
    // (+ 0: the side of a zero is the positive one, whatever its sign)
    const float fx = copysignf(1.0f - fabsf(oy), ox + 0.0f), fy = copysignf(1.0f - fabsf(ox), oy + 0.0f);
    const bool lower = n.z < 0.0f;
    return make_float2((lower ? fx : ox) * 0.5f + 0.5f, (lower ? fy : oy) * 0.5f + 0.5f);
}

// foot_tap without conversions: adding 2^23 rounds uv * 6, which lies half a texel
// below the tile-local coordinate, to the footprint's index. (Where the coordinate
// is a whole number it may take the one before, with weight 1 on the same texel.)
__device__ __forceinline__ FootTap tap_of(float2 o) {
    const float mx = fmaf(__saturatef(o.x), 6.0f, 8388608.0f), my = fmaf(__saturatef(o.y), 6.0f, 8388608.0f);
    FootTap t;
    t.at = (__float_as_uint(my) & 7u) * 7u + (__float_as_uint(mx) & 7u);
    t.fx = fmaf(o.x, 6.0f, 0.5f - (mx - 8388608.0f));
    t.fy = fmaf(o.y, 6.0f, 0.5f - (my - 8388608.0f));
    return t;
}

// A colour summed as (r, g) and as the two columns' b, two lanes per operation.
struct Sum2 {
    unsigned long long rg, b;
};
// Bilinear weights, each twice and by column.
struct Weights2 {
    unsigned long long w[4], row0, row1;
};
__device__ __forceinline__ Weights2 weights2(const FootTap& t) {
    const float4 w = foot_weights(t);
    Weights2 r;
    r.w[0] = pack2(w.x, w.x);
    r.w[1] = pack2(w.y, w.y);
    r.w[2] = pack2(w.z, w.z);
    r.w[3] = pack2(w.w, w.w);
    r.row0 = pack2(w.x, w.y);
    r.row1 = pack2(w.z, w.w);
    return r;
}
__device__ __forceinline__ Sum2 foot_rgb2(const uint4* foot, uint32_t at, const Weights2& w) {
    uint32_t u[8];
    load_foot(foot + FOOT_U4 * at, u);
    Sum2 s;
    s.rg = mul2(pack2(half2_at(u[0])), w.w[0]);
    s.rg = fma2(pack2(half2_at(u[1])), w.w[1], s.rg);
    s.rg = fma2(pack2(half2_at(u[2])), w.w[2], s.rg);
    s.rg = fma2(pack2(half2_at(u[3])), w.w[3], s.rg);
    s.b = fma2(pack2(half2_at(u[5])), w.row1, mul2(pack2(half2_at(u[4])), w.row0));
    return s;
}
__device__ __forceinline__ void add_scaled(Sum2& acc, const Sum2& s, float w) {
    const unsigned long long w2 = pack2(w, w);
    acc.rg = fma2(s.rg, w2, acc.rg);
    acc.b = fma2(s.b, w2, acc.b);
}
__device__ __forceinline__ float3 sum_of(const Sum2& s, float scale) {
    const float2 rg = unpack2(s.rg), b = unpack2(s.b);
    return mk(rg.x * scale, rg.y * scale, (b.x + b.y) * scale);
}
// An rgba footprint read: (r, g) and, over the columns, b and a.
struct Sum4 {
    unsigned long long rg, b, a;
};
__device__ __forceinline__ Sum4 foot_rgba2(const uint4* foot, uint32_t at, const Weights2& w) {
    uint32_t u[8];
    load_foot(foot + FOOT_U4 * at, u);
    Sum4 s;
    s.rg = mul2(pack2(half2_at(u[0])), w.w[0]);
    s.rg = fma2(pack2(half2_at(u[1])), w.w[1], s.rg);
    s.rg = fma2(pack2(half2_at(u[2])), w.w[2], s.rg);
    s.rg = fma2(pack2(half2_at(u[3])), w.w[3], s.rg);
    s.b = fma2(pack2(half2_at(u[5])), w.row1, mul2(pack2(half2_at(u[4])), w.row0));
    s.a = fma2(pack2(half2_at(u[7])), w.row1, mul2(pack2(half2_at(u[6])), w.row0));
    return s;
}

// The taps' offsets to a point, per axis and side: tap i lies at base + bits(i).
struct Offsets {
    float x0, x1, y0, y1, z0, z1;  // point - probe
};
__device__ __forceinline__ Offsets offsets_to(const GatherCascade& C, const Cage& g, float3 p) {
    // the probe at grid index k: gridMin + k * cell (within an ulp of the reference's
    // gridMin + k / (res - 1) * gridSize)
    return {p.x - fmaf(g.base[0], C.cell[0], C.gridMin[0]), p.x - fmaf(g.base[0] + 1.0f, C.cell[0], C.gridMin[0]),
            p.y - fmaf(g.base[1], C.cell[1], C.gridMin[1]), p.y - fmaf(g.base[1] + 1.0f, C.cell[1], C.gridMin[1]),
            p.z - fmaf(g.base[2], C.cell[2], C.gridMin[2]), p.z - fmaf(g.base[2] + 1.0f, C.cell[2], C.gridMin[2])};
}
__device__ __forceinline__ float3 offset_at(const Offsets& o, int i) {
    return mk(i & 1 ? o.x1 : o.x0, i & 2 ? o.y1 : o.y0, i & 4 ? o.z1 : o.z0);
}

// A tap's weight under the Chebyshev visibility and the wrap weight.
__device__ __forceinline__ float visible_weight(const GatherCascade& C, float cs, float chebyBias, uint32_t foot,
                                                float3 toSurf, float3 Nn, float wTri) {
    const float d2 = dot3(toSurf, toSurf), inv = rsqrt_fast(fmaxf(d2, 1e-12f)), dist = d2 * inv;
    const FootTap tD = tap_of(oct_any(toSurf, true));
    const float2 m = foot_depth(C.footDepth, foot + tD.at, foot_weights(tD));
    const float variance = fabsf(m.y - m.x * m.x);
    const float dm = fmaxf(dist - m.x - chebyBias, 0.0f);
    const float chebyRaw = variance * rcp_fast(fmaxf(variance + dm * dm, 1e-6f));
    const float cheby = dist <= m.x + chebyBias ? 1.0f : chebyRaw;
    const float visW = (1.0f - cs) + fmaxf(cheby * cheby * cheby, 0.05f) * cs;
    const float wrap = dot3(toSurf, Nn) * (inv * -0.5f) + 0.5f;
    const float wrapW = (1.0f - cs) + fmaxf(wrap * wrap, 0.05f) * cs;
    return wTri * wrapW * visW;
}

// FULL = false compiles the default receiver alone (chebyStrength 0, no dual
// detail): no depth fetch and no second fetch direction.
template <bool FULL>
__device__ __forceinline__ float3 gather_cascade(const GatherCascade& C, const GatherArgs& A, float chebyBias,
                                                 float3 cageP, float3 P, float3 Nvis, float3 Ndir, bool dual) {
    const Cage g = cage_of(C, cageP);
    const FootTap tN = tap_of(oct_any(Ndir));
    const Weights2 wN = weights2(tN);
    Sum2 acc = {0ull, 0ull};
    float wsum = 0.0f;
    if (!FULL) {
#pragma unroll 4
        for (int i = 0; i < 8; ++i) {
            const float w = cage_weight(g, i);
            add_scaled(acc, foot_rgb2(C.foot, cage_probe(g, i) * FOOT + tN.at, wN), w);
            wsum += w;
        }
        return sum_of(acc, 1.0f / fmaxf(wsum, 1e-4f));
    }
    const float cs = A.chebyStrength;
    const float3 Nn = fast_normalize(Nvis);
    const FootTap tS = dual ? tap_of(oct_any(Nvis)) : tN;
    const Weights2 wS = weights2(tS);
    const Offsets o = offsets_to(C, g, P);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t foot = cage_probe(g, i) * FOOT;
        float w = cage_weight(g, i);
        if (cs != 0.0f) w = visible_weight(C, cs, chebyBias, foot, offset_at(o, i), Nn, w);
        const float detail = dual ? A.detailStrength : 1.0f;
        add_scaled(acc, foot_rgb2(C.foot, foot + tN.at, wN), w * detail);
        if (dual) add_scaled(acc, foot_rgb2(C.foot, foot + tS.at, wS), w * (1.0f - detail));
        wsum += w;
    }
    return sum_of(acc, 1.0f / fmaxf(wsum, 1e-4f));
}

// Five blocks per SM and four taps in flight: 40 us against 42 with four blocks and
// eight taps (1080p).
template <bool FULL>
__global__ void __launch_bounds__(256, FULL ? 4 : 5) k_gather(const GatherArgs A) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.count) return;
    const float4 p4 = __ldcs(A.position + i), n4 = __ldcs(A.stableNormal + i), d4 = __ldcs(A.detailNormal + i);
    const float3 Nvis = xyz(n4), Ndir = xyz(d4);
    const float3 reflP = xyz(p4) * A.samplePositionScale;
    const float3 P = reflP + Nvis * A.normalBias0 * A.sampleBiasScale;
    float3 E;
    if (A.cascades < 2) {
        E = gather_cascade<FULL>(A.c[0], A, A.chebyBias[0], P, P, Nvis, Ndir, A.dualDetail != 0);
    } else {
        const GatherCascade& F = A.c[1];
        const float f0 = (P.x - F.gridMin[0]) / fmaxf(F.gridSize[0], 1e-6f);
        const float f1 = (P.y - F.gridMin[1]) / fmaxf(F.gridSize[1], 1e-6f);
        const float f2 = (P.z - F.gridMin[2]) / fmaxf(F.gridSize[2], 1e-6f);
        const float fLo = fminf(fminf(f0, f1), f2);
        const float fHi = fminf(fminf(1.0f - f0, 1.0f - f1), 1.0f - f2);
        const float wIn = clampf(fminf(fLo, fHi) / fmaxf(A.borderBand, 1e-4f), 0.0f, 1.0f);
        const float wFine = wIn * clampf(float(A.cascades) - 1.0f, 0.0f, 1.0f);
        E = mk(0.0f, 0.0f, 0.0f);
        if (wFine < 1.0f) E = gather_cascade<FULL>(A.c[0], A, A.chebyBias[0], reflP, P, Nvis, Ndir, false);
        if (wFine > 0.0f) {
            const float3 Ef = gather_cascade<FULL>(A.c[1], A, A.chebyBias[1], reflP, P, Nvis, Ndir, false);
            E = E * (1.0f - wFine) + Ef * wFine;
        }
    }
    const float k = A.intensity * A.enabled;
    __stcs(A.out + i, make_float4(fmaxf(E.x, 0.0f) * k, fmaxf(E.y, 0.0f) * k, fmaxf(E.z, 0.0f) * k, 1.0f));
}


// smoothstep with the reciprocal of its (constant) edge span supplied
__device__ __forceinline__ float smoothstepf(float e0, float invSpan, float x) {
    const float t = clampf((x - e0) * invSpan, 0.0f, 1.0f);
    return t * t * (3.0f - 2.0f * t);
}

// One cascade of the combined receiver (_sampleCombinedCascadeLooped,
// gi_probes.js:662-771): the irradiance taps with the cage at the biased point
// P, and per tap with a live lobe the parallax-corrected rough / glossy fetch.
// FULL = false: one cascade, chebyStrength 0, no dual detail.
template <bool FULL>
__device__ __forceinline__ void combined_cascade(const GatherCascade& C, const GatherArgs& A, float chebyBias, float3 P, float3 reflP,
                                 float3 Nvis, float3 Ndir, float3 Rn, bool dual, float rw, float lobeMix,
                                 float3& irr, float4& refl) {
    if (!FULL) dual = false;
    const Cage g = cage_of(C, P);
    const float3 Nn = fast_normalize(Nvis);
    const FootTap tN = tap_of(oct_any(Ndir)), tS = dual ? tap_of(oct_any(Nvis)) : tN;
    const FootTap tR = tap_of(oct_any(Rn, true));
    const Weights2 wN = weights2(tN), wS = weights2(tS);
    const float4 bR = foot_weights(tR);
    const float cs = FULL ? A.chebyStrength : 0.0f;
    const bool glossyOn = C.glossy != nullptr;
    const bool wantsRough = lobeMix > 0.0f, wantsGlossy = glossyOn && lobeMix < 1.0f;
    const bool wantsTap = rw > 0.0f && (wantsRough || wantsGlossy);
    const Offsets oP = offsets_to(C, g, P), oR = offsets_to(C, g, reflP);
    Sum2 acc = {0ull, 0ull};
    Sum4 rough = {0ull, 0ull, 0ull};
    float wsum = 0.0f, roughW = 0.0f, glossyW = 0.0f;
    unsigned long long glossyRg = 0ull, glossyBa = 0ull;
#pragma unroll 2
    for (int i = 0; i < 8; ++i) {
        const uint32_t probe = cage_probe(g, i), foot = probe * FOOT;
        float w = cage_weight(g, i);
        if (cs != 0.0f) w = visible_weight(C, cs, chebyBias, foot, offset_at(oP, i), Nn, w);
        const float detail = dual ? A.detailStrength : 1.0f;
        add_scaled(acc, foot_rgb2(C.foot, foot + tN.at, wN), w * detail);
        if (dual) add_scaled(acc, foot_rgb2(C.foot, foot + tS.at, wS), w * (1.0f - detail));
        wsum += w;
        if (!wantsTap) continue;
        // the reflection ray against the sphere of the probe's mean depth toward R
        const float2 dR = foot_depth(C.footDepth, foot + tR.at, bR);
        const float radius = fmaxf(dR.x, 1e-4f), radius2 = radius * radius;
        const float3 q = offset_at(oR, i);
        const float q2 = dot3(q, q), qDotR = dot3(q, Rn);
        // radius^2 - q^2 + (q.R)^2 with |R| = 1 is radius^2 - |q x R|^2: the cross
        // product keeps the two nearly equal squares from cancelling in FP32
        const float3 qxR = cross3(q, Rn);
        const float disc = radius2 - dot3(qxR, qxR);
        const float sqrtDisc = sqrt_fast(fmaxf(disc, 0.0f));
        const float nearT = -qDotR - sqrtDisc, farT = -qDotR + sqrtDisc;
        const float rayT = nearT > 1e-4f ? nearT : farT;
        const float invR2 = rcp_fast(fmaxf(radius2, 1e-4f));
        const float relVar = fmaxf(dR.y - radius2, 0.0f) * invR2;
        const float stableDepth = 1.0f - smoothstepf(0.02f, 1.0f / 0.18f, relVar);
        const float validHit = (disc > 1e-6f && rayT > 1e-4f) ? 1.0f : 0.0f;
        const float insideWeight = smoothstepf(0.0f, 1.0f / 0.12f, (radius2 - q2) * invR2);
        const float pw = stableDepth * validHit * insideWeight;
        const float3 corrected = fast_normalize(q + Rn * fmaxf(rayT, 0.0f));
        const float2 oSR = oct_any(Rn * (1.0f - pw) + corrected * pw, true);
        const float probeW = w * w;
        if (wantsGlossy) {
            // the probe's glossy tile (row and column exact: the index has 15 bits), and the
            // bilinear read inside it, as in tap_of (glossyOct texels and a gutter)
            const uint32_t row = (uint32_t)((float(probe) + 0.5f) * C.perGlossyRow);
            const float oct = C.glossyOct;
            const float mx = fmaf(__saturatef(oSR.x), oct, 8388608.0f), my = fmaf(__saturatef(oSR.y), oct, 8388608.0f);
            const uint32_t x = __float_as_uint(mx) & 31u, y = __float_as_uint(my) & 31u;
            const float fx = fmaf(oSR.x, oct, 0.5f - (mx - 8388608.0f)), fy = fmaf(oSR.y, oct, 0.5f - (my - 8388608.0f));
            const uint2* p = C.glossy + (row * C.glossyTile + y) * C.glossyW +
                             (probe - row * C.glossyTilesX) * C.glossyTile + x;
            const uint2 t[4] = {__ldg(p), __ldg(p + 1), __ldg(p + C.glossyW), __ldg(p + C.glossyW + 1)};
            const float gw = probeW * (0.2f * (1.0f - pw) + pw);
            const float bw[4] = {(1.0f - fx) * (1.0f - fy) * gw, fx * (1.0f - fy) * gw, (1.0f - fx) * fy * gw, fx * fy * gw};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const unsigned long long w2 = pack2(bw[c], bw[c]);
                glossyRg = fma2(pack2(half2_at(t[c].x)), w2, glossyRg);
                glossyBa = fma2(pack2(half2_at(t[c].y)), w2, glossyBa);
            }
            glossyW += gw;
        }
        if (wantsRough) {
            const FootTap tB = tap_of(oSR);
            const Sum4 br = foot_rgba2(C.footRough, foot + tB.at, weights2(tB));
            const unsigned long long w2 = pack2(probeW, probeW);
            rough.rg = fma2(br.rg, w2, rough.rg);
            rough.b = fma2(br.b, w2, rough.b);
            rough.a = fma2(br.a, w2, rough.a);
            roughW += probeW;
        }
    }
    irr = sum_of(acc, 1.0f / fmaxf(wsum, 1e-4f));
    const float2 rrg = unpack2(rough.rg), rb = unpack2(rough.b), ra = unpack2(rough.a);
    const float4 roughAcc = make_float4(rrg.x, rrg.y, rb.x + rb.y, ra.x + ra.y);
    const float ri = 1.0f / fmaxf(roughW, 1e-4f);
    refl = make_float4(roughAcc.x * ri, roughAcc.y * ri, roughAcc.z * ri, roughAcc.w * ri);
    if (glossyOn) {
        const float gi = 1.0f / fmaxf(glossyW, 1e-4f);
        const float2 grg = unpack2(glossyRg), gba = unpack2(glossyBa);
        const float4 glossyAcc = make_float4(grg.x, grg.y, gba.x, gba.y);
        refl = make_float4(glossyAcc.x * gi * (1.0f - lobeMix) + refl.x * lobeMix,
                           glossyAcc.y * gi * (1.0f - lobeMix) + refl.y * lobeMix,
                           glossyAcc.z * gi * (1.0f - lobeMix) + refl.z * lobeMix,
                           glossyAcc.w * gi * (1.0f - lobeMix) + refl.w * lobeMix);
    }
}

template <bool FULL>
__global__ void __launch_bounds__(256, FULL ? 3 : 4) k_gather_combined(const GatherArgs A) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= A.count) return;
    const float4 p4 = __ldcs(A.position + i), n4 = __ldcs(A.stableNormal + i), d4 = __ldcs(A.detailNormal + i);
    const float4 r4 = __ldcs(A.reflection + i);
    const float3 Nvis = xyz(n4), Ndir = xyz(d4), Rn = normalize3(xyz(r4));
    const float roughness = r4.w;
    const float3 reflP = xyz(p4) * A.samplePositionScale;
    const float3 P = reflP + Nvis * A.normalBias0 * A.sampleBiasScale;
    const float part = roughness <= A.roughnessLimit ? 1.0f : 0.0f;
    const float rw = clampf(A.reflectionIntensity * A.enabled * part, 0.0f, 1.0f);
    const float lobeMix = A.c[0].glossy ? smoothstepf(0.22f, 1.0f / 0.36f, roughness) : 1.0f;
    float3 E;
    float4 S;
    if (!FULL || A.cascades < 2) {
        combined_cascade<FULL>(A.c[0], A, A.chebyBias[0], P, reflP, Nvis, Ndir, Rn, A.dualDetail != 0, rw, lobeMix, E, S);
    } else {
        // cascade ownership at the surface position (gi_probes.js:787-792)
        const GatherCascade& F = A.c[1];
        const float f0 = (reflP.x - F.gridMin[0]) / fmaxf(F.gridSize[0], 1e-6f);
        const float f1 = (reflP.y - F.gridMin[1]) / fmaxf(F.gridSize[1], 1e-6f);
        const float f2 = (reflP.z - F.gridMin[2]) / fmaxf(F.gridSize[2], 1e-6f);
        const float fLo = fminf(fminf(f0, f1), f2);
        const float fHi = fminf(fminf(1.0f - f0, 1.0f - f1), 1.0f - f2);
        const float wIn = clampf(fminf(fLo, fHi) / fmaxf(A.borderBand, 1e-4f), 0.0f, 1.0f);
        const float wFine = wIn * clampf(float(A.cascades) - 1.0f, 0.0f, 1.0f);
        E = mk(0.0f, 0.0f, 0.0f);
        S = make_float4(0.f, 0.f, 0.f, 0.f);
        if (wFine < 1.0f) combined_cascade<FULL>(A.c[0], A, A.chebyBias[0], P, reflP, Nvis, Ndir, Rn, false, rw, lobeMix, E, S);
        if (wFine > 0.0f) {
            float3 Ef;
            float4 Sf;
            combined_cascade<FULL>(A.c[1], A, A.chebyBias[1], P, reflP, Nvis, Ndir, Rn, false, rw, lobeMix, Ef, Sf);
            E = E * (1.0f - wFine) + Ef * wFine;
            S = make_float4(S.x * (1.0f - wFine) + Sf.x * wFine, S.y * (1.0f - wFine) + Sf.y * wFine,
                            S.z * (1.0f - wFine) + Sf.z * wFine, S.w * (1.0f - wFine) + Sf.w * wFine);
        }
    }
    const float k = A.intensity * A.enabled;
    __stcs(A.out + i, make_float4(fmaxf(E.x, 0.0f) * k, fmaxf(E.y, 0.0f) * k, fmaxf(E.z, 0.0f) * k, 1.0f));
    const float4 o = rw > 0.0f ? make_float4(fmaxf(S.x, 0.0f) * rw, fmaxf(S.y, 0.0f) * rw, fmaxf(S.z, 0.0f) * rw,
                                             clampf(fmaxf(S.w, 0.0f), 0.0f, 1.0f) * rw)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
    __stcs(A.outReflection + i, o);
}

}  // namespace

cudaError_t launch_gather_combined(const GatherArgs& A, cudaStream_t st) {
    if (A.count == 0) return cudaSuccess;
    const bool full = A.cascades > 1 || A.chebyStrength != 0.0f || A.dualDetail;
    if (full) k_gather_combined<true><<<(A.count + 255) / 256, 256, 0, st>>>(A);
    else k_gather_combined<false><<<(A.count + 255) / 256, 256, 0, st>>>(A);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_gather(const GatherArgs& A, cudaStream_t st) {
    if (A.count == 0) return cudaSuccess;
    const bool full = A.cascades > 1 || A.chebyStrength != 0.0f || A.dualDetail;
    if (full) k_gather<true><<<(A.count + 255) / 256, 256, 0, st>>>(A);
    else k_gather<false><<<(A.count + 255) / 256, 256, 0, st>>>(A);
    note_launch();
    return cudaGetLastError();
}

}  // namespace sb
