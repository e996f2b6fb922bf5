// sb_trace.cu — the probe trace as a three-stage wavefront (traceKernel,
// gi_probes.js:1977-2214, split where its per-ray work diverges):
//
//   A  k_trace_primary  closest hit per probe ray (traverseClosest) -> raw
//                       16-byte hit record.
//      k_emit           per ray: hit t in FP64, hit frame, and the NEE
//                       pre-tests per candidate light (the reference's
//                       ndl * peak > 0 and range gates); passing candidates
//                       become shadow-ray jobs, one atomic per warp.
//   B  k_trace_shadow   any hit per job (traverseAny); blocked lights are
//                       cleared from the ray's visibility mask.
//   C  k_shade          emissive + unblocked NEE terms (ascending light index,
//                       the reference's summation order) + one-bounce atlas
//                       read, or the SH-9 sky on a miss -> rayData.
//
// A and B are persistent and work-stealing. On the 8-wide tree (*_walk8, *_batch) a
// lane whose ray has ended takes the next one (sb_walk8.cuh, sb_walk2.cuh); on the
// other layouts warps pull 32 items per atomic. A issues rays direction-major: a
// warp holds ray k of 32 neighbouring probes, i.e. 32 parallel rays, which keeps
// the BVH walks of a warp together.
#include <algorithm>

#include "sb_walk2.cuh"
#include "sb_wave.cuh"

namespace sb {

// Resident 256-thread blocks per SM the register allocation must allow
// (4 x 256 threads: 64 registers; measured best for both traversal stages).
#ifndef SB_PRIMARY_MIN_BLOCKS
#define SB_PRIMARY_MIN_BLOCKS 4
#endif
#ifndef SB_SHADOW_MIN_BLOCKS
#define SB_SHADOW_MIN_BLOCKS 4
#endif
// The same for the walks of the 8-wide tree: 80 registers. Four blocks (64 registers,
// spills, less L1 beside the shared memory) measured 59 against 48 us on the room's
// primary rays, 122 against 98 us on the atrium's and 966 against 932 us for 2.07M
// bounce rays with a shadow ray each.
#ifndef SB_WALK8_MIN_BLOCKS
#define SB_WALK8_MIN_BLOCKS 3
#endif

// ---------------------------------------------------------------- bodies
// Each stage's per-item work is a device function over `const WaveCtx&`; the
// per-solve kernels pass their parameter, the batched kernels an item of the
// __grid_constant__ BatchArgs (indexed in the parameter space, warp-uniform).

__device__ __forceinline__ void add_visits(unsigned long long* c, int at, uint32_t rays, const Visits& v) {
    if (!c) return;
    if (rays) atomicAdd(&c[0], (unsigned long long)rays);
    atomicAdd(&c[at], (unsigned long long)v.tlas);
    atomicAdd(&c[at + 1], (unsigned long long)v.inst);
    atomicAdd(&c[at + 2], (unsigned long long)v.blas);
    atomicAdd(&c[at + 3], (unsigned long long)v.tri);
}

// The raw record of ray rayIdx's closest hit (FP32 t, no facing bit): k_emit finishes it.
__device__ __forceinline__ void write_hit(const DevCascade& C, uint32_t rayIdx, int tri, int inst, float t,
                                          uint32_t uv) {
    C.hits[rayIdx] = tri >= 0 ? make_uint4((uint32_t)tri, (uint32_t)inst, __float_as_uint(t), uv)
                              : make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, __float_as_uint(-1.0f), 0u);
}

// Stage A: the closest hit of one probe ray (item-local issue index g).
__device__ __forceinline__ void primary_ray(const WaveCtx& W, const uint4* tl, bool pairs, uint32_t g, Visits& vis) {
    const DevCascade& C = W.C;
    uint32_t slot, k;
    ray_of(W, g, W.order != 0, slot, k);
    const float3 ro = slot_origin(C, slot);
    const float3 rd = ray_dir(k, C.rays, W.P.frameJitter);
    float bestT, bu, bv;
    int tri, inst;
    trace_closest(W.S, tl, ro, rd, bestT, tri, inst, bu, bv, vis, W.err, pairs);
    write_hit(C, slot * C.rays + k, tri, inst, bestT, pack_uv(bu, bv));
}

// The CTA's shared memory: the tables (filled here), then each warp's, used by the
// moved slots' walk first and by the 8-wide one after it.
struct WalkSmem {
    Walk8Tables* tables;
    Walk2Shared* w2;
    Walk8Shared* w8;
    uint2* stk;
};
__host__ __device__ __forceinline__ uint32_t walk_stride(uint32_t depth, bool moved) {
    const uint32_t w8 = (uint32_t)(sizeof(Walk8Shared) + depth * 32u * sizeof(uint2));
    return moved && sizeof(Walk2Shared) > w8 ? (uint32_t)sizeof(Walk2Shared) : w8;
}
static uint32_t walk_smem(uint32_t depth, bool moved, uint32_t threads) {
    return (uint32_t)sizeof(Walk8Tables) + threads / 32u * walk_stride(depth, moved);
}
__device__ __forceinline__ WalkSmem walk_shared(void* smem, uint32_t depth, bool moved) {
    WalkSmem m;
    m.tables = reinterpret_cast<Walk8Tables*>(smem);
    walk8_tables(*m.tables);
    char* p = reinterpret_cast<char*>(smem) + sizeof(Walk8Tables) + (threadIdx.x / 32u) * walk_stride(depth, moved);
    m.w2 = reinterpret_cast<Walk2Shared*>(p);
    m.w8 = reinterpret_cast<Walk8Shared*>(p);
    m.stk = reinterpret_cast<uint2*>(p + sizeof(Walk8Shared));
    return m;
}

// A walk's next items for the lanes in `want`: positions of the shared cursor; whether
// it has more (before it is asked in vain, so that the walk knows its last rays).
__device__ __forceinline__ uint32_t take(uint32_t* cursor, uint32_t total, uint32_t want, bool& more) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t base = 0;
    if (lane == 0) base = atomicAdd(cursor, (uint32_t)__popc(want));
    base = __shfl_sync(ALL_LANES, base, 0);
    more = base < total && total - base > (uint32_t)__popc(want);
    return base + (uint32_t)__popc(want & ((1u << lane) - 1u));
}

// Stage A on the 8-wide tree. next(want, g) gives the lanes in `want` their
// item-local issue positions (ok: this lane has one) and returns false when none
// are left; dir(k, inv) is ray direction k with its inverse.
//
// The moved slots' hits go to the ray records (free until the shading), the tree's
// to the hit records; emission takes the nearer one.
template <class Next, class Dir>
__device__ __forceinline__ void primary_moved(const WaveCtx& W, Walk2Shared& sm, Next next, Dir dir, Visits& vis) {
    const DevCascade& C = W.C;
    const uint32_t lane = threadIdx.x & 31u;
    uint4* out = reinterpret_cast<uint4*>(C.rayData);
    auto gen = [&](bool& more, uint32_t want, float3& o, float3& d, float3& winv, float& tmax, uint32_t& tag) {
        uint32_t g;
        bool ok;
        more = next(want, g, ok);
        if (!ok || !(want >> lane & 1u)) return false;
        uint32_t slot, k;
        ray_of(W, g, W.order != 0, slot, k);
        o = slot_origin(C, slot);
        d = dir(k, winv);
        tmax = T_MAX;
        tag = slot * C.rays + k;
        return true;
    };
    if (walk2_usable(W.S)) {
        walk2<false>(W.S, sm, gen, [&](uint32_t tag, float t, uint4 hit, bool) {
            out[tag] = make_uint4(hit.x, hit.y, __float_as_uint(t), hit.z);
        }, vis, W.err);
        return;
    }
    for (bool more = true; more;) {  // a BLAS too deep for it: one ray per lane
        float3 o, d, winv;
        float t, bu = 0.0f, bv = 0.0f;
        uint32_t tag;
        if (!gen(more, ALL_LANES, o, d, winv, t, tag)) continue;
        int tri = -1, inst = -1;
        dyn_walk<false>(W.S, o, d, winv, t, tri, inst, bu, bv, vis, W.err);
        out[tag] = make_uint4((uint32_t)tri, (uint32_t)inst, __float_as_uint(t), pack_uv(bu, bv));
    }
}

template <class Next, class Dir>
__device__ __forceinline__ uint32_t primary_walk8(const WaveCtx& W, const WalkSmem& m, Next next, Dir dir,
                                                  Visits& vis) {
    const DevCascade& C = W.C;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t nRays = 0;
    auto gen = [&](bool& more, uint32_t want, float3& o, float3& d, float3& winv, float& tmax, uint32_t& tag,
                   uint4& hit) {
        uint32_t g;
        bool ok;
        more = next(want, g, ok);
        if (!ok || !(want >> lane & 1u)) return false;
        uint32_t slot, k;
        ray_of(W, g, W.order != 0, slot, k);
        o = slot_origin(C, slot);
        d = dir(k, winv);
        tag = slot * C.rays + k;
        tmax = T_MAX;
        hit = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u);
        ++nRays;
        return true;
    };
    auto fin = [&](uint32_t tag, float t, uint4 hit, bool) { write_hit(C, tag, (int)hit.x, (int)hit.y, t, hit.z); };
    walk8<false>(W.S, *m.tables, *m.w8, m.stk, W.S.wideDepth + 1u, gen, fin, vis, W.err);
    return nRays;
}

// A blocked light leaves its ray's mask.
__device__ __forceinline__ void clear_light(const WaveCtx& W, uint32_t tag) {
    const uint32_t li = tag & 63u;
    uint4* v = W.C.vis + (tag >> 6);
    if (li < 32) atomicAnd(&v->z, ~(1u << li));
    else atomicAnd(&v->w, ~(1u << (li - 32)));
}

// Stage B on the 8-wide tree, next(want, j) as for stage A, with jobs. A job that
// the moved slots block loses its length: the tree's walk skips it when it comes to
// it later (it may not see that yet, and then clears the same light again).
template <class Next>
__device__ __forceinline__ void shadow_moved(const WaveCtx& W, Walk2Shared& sm, Next next, Visits& vis) {
    const uint32_t lane = threadIdx.x & 31u;
    auto gen = [&](bool& more, uint32_t want, float3& o, float3& d, float3& winv, float& tmax, uint32_t& tag) {
        uint32_t j;
        bool ok;
        more = next(want, j, ok);
        if (!ok || !(want >> lane & 1u)) return false;
        const float4 a = W.jobs[2 * j], b = W.jobs[2 * j + 1];
        o = xyz(a);
        d = xyz(b);
        winv = mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
        tmax = a.w;
        tag = j;
        return true;
    };
    auto fin = [&](uint32_t j, float, uint4, bool blocked) {
        if (!blocked) return;
        clear_light(W, __float_as_uint(W.jobs[2 * j + 1].w));
        W.jobs[2 * j].w = 0.0f;
    };
    if (walk2_usable(W.S)) {
        walk2<true>(W.S, sm, gen, fin, vis, W.err);
        return;
    }
    for (bool more = true; more;) {
        float3 o, d, winv;
        float t, u = 0.0f, v = 0.0f;
        uint32_t tag;
        if (!gen(more, ALL_LANES, o, d, winv, t, tag)) continue;
        int tri = -1, inst = -1;
        if (dyn_walk<true>(W.S, o, d, winv, t, tri, inst, u, v, vis, W.err))
            fin(tag, t, make_uint4(0u, 0u, 0u, 0u), true);
    }
}

template <class Next>
__device__ __forceinline__ void shadow_walk8(const WaveCtx& W, const WalkSmem& m, Next next, Visits& vis) {
    const uint32_t lane = threadIdx.x & 31u;
    auto gen = [&](bool& more, uint32_t want, float3& o, float3& d, float3& winv, float& tmax, uint32_t& tag, uint4&) {
        uint32_t j;
        bool ok;
        more = next(want, j, ok);
        if (!ok || !(want >> lane & 1u)) return false;
        const float4 a = W.jobs[2 * j], b = W.jobs[2 * j + 1];
        o = xyz(a);
        d = xyz(b);
        winv = mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
        tmax = a.w;
        tag = __float_as_uint(b.w);
        return tmax > RAY_EPS;  // no hit lies nearer than that
    };
    auto fin = [&](uint32_t tag, float, uint4, bool blocked) {
        if (blocked) clear_light(W, tag);
    };
    walk8<true>(W.S, *m.tables, *m.w8, m.stk, W.S.wideDepth + 1u, gen, fin, vis, W.err);
}

// Stage A2, warp-collective (all 32 lanes call it; `active` lanes hold ray g):
// the hit parameter re-evaluated in FP64, the hit frame, and the NEE
// gates of every candidate light. Each lane runs the gates with no warp sync;
// one warp scan and one atomicAdd then reserve the warp's shadow-ray jobs, and
// each ray's passing candidates are written together in list order, so a shadow
// warp mostly holds rays that share an origin. Jobs carry the ray's record index.
// `gates`: GATE_LIGHTS entries of shared memory, the warp's own.
__device__ __forceinline__ uint32_t emit_ray(const WaveCtx& W, bool active, uint32_t g, float4* gates) {
    const DevCascade& C = W.C;
    const GateTable T = gate_table(W, gates);
    const uint32_t N = C.rays;
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t rayIdx = 0;
    int tri = -1;
    HitFrame fr;
    fr.hitPos = mk(0.f, 0.f, 0.f);
    fr.ng = mk(0.f, 0.f, 1.f);
    fr.faceFwd = true;
    fr.traceBias = 0.f;
    uint4 h = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u);
    if (active) {
        uint32_t slot, k;
        ray_of(W, g, W.order != 0, slot, k);
        rayIdx = slot * N + k;
        h = C.hits[rayIdx];
        if (W.S.wideNodes && W.S.dynCount) {  // the moved slots' hit, when it is no farther
            const uint4 d = reinterpret_cast<const uint4*>(C.rayData)[rayIdx];
            if (d.x != 0xFFFFFFFFu && (h.x == 0xFFFFFFFFu || __uint_as_float(d.z) <= __uint_as_float(h.z))) h = d;
        }
        if (h.x != 0xFFFFFFFFu) {
            tri = (int)h.x;
            const uint32_t inst = h.y;
            const float3 ro = slot_origin(C, slot), rd = wave_dir(W, k);
            const float t = refine_t(W.S, (uint32_t)tri, inst, ro, rd);
            fr = hit_frame(W, (uint32_t)tri, inst, ro, rd, t, -1);
            h.y = inst | (fr.faceFwd ? 0x80000000u : 0u);
            h.z = __float_as_uint(t);
        }
    }
    LightList L{nullptr, 0u};
    if (tri >= 0) L = light_list(W, fr.hitPos);
    unsigned long long pass = 0ull;
    for (uint32_t i = 0; i < L.count; ++i)
        if (table_gate(W, T, light_at(L, i), fr.hitPos, fr.ng)) pass |= 1ull << i;
    const uint32_t mine = (uint32_t)__popcll(pass);
    uint32_t incl = mine;
#pragma unroll
    for (uint32_t d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xFFFFFFFFu, incl, d);
        if (lane >= d) incl += v;
    }
    const uint32_t warpJobs = __shfl_sync(0xFFFFFFFFu, incl, 31);
    uint32_t jb = 0;
    if (warpJobs) {
        if (lane == 0) jb = atomicAdd(&W.work[2], warpJobs);
        jb = __shfl_sync(0xFFFFFFFFu, jb, 0);
    }
    uint32_t j = jb + incl - mine, tested0 = 0u, tested1 = 0u, nJobs = 0;
    const uint32_t tag = rayIdx << 6;
    while (pass) {
        const uint32_t i = (uint32_t)(__ffsll((long long)pass) - 1);
        pass &= pass - 1ull;
        const uint32_t li = light_at(L, i);
        if (j < W.jobCap) {
            float3 wi;
            float dist;
            light_ray(T, li, fr.hitPos, wi, dist);
            store32(W.jobs + 2 * j, make_float4(fr.hitPos.x, fr.hitPos.y, fr.hitPos.z, dist - fr.traceBias),
                    make_float4(wi.x, wi.y, wi.z, __uint_as_float(tag | li)));
            if (li < 32) tested0 |= 1u << li;
            else tested1 |= 1u << (li - 32);
            ++nJobs;
        } else {
            latch(W.err, ERR_CAPACITY);
        }
        ++j;
    }
    if (active) {
        if (tri >= 0) C.hits[rayIdx] = h;
        C.vis[rayIdx] = make_uint4(tested0, tested1, tested0, tested1);
    }
    return nJobs;
}

// Stage B: one shadow job; a blocked light is cleared from the ray's mask.
__device__ __forceinline__ void shadow_job(const WaveCtx& W, const uint4* tl, bool pairs, float4 a, float4 b,
                                           Visits& vis) {
    if (trace_any(W.S, tl, xyz(a), xyz(b), a.w, vis, W.err, pairs)) clear_light(W, __float_as_uint(b.w));
}

// Stage C: emissive + unblocked NEE terms + bounce, or the sky, of one ray
// (item-local probe-major index g).
__device__ __forceinline__ void shade_ray(const WaveCtx& W, uint32_t g) {
    const DevCascade& C = W.C;
    const uint32_t N = C.rays;
    uint32_t slot, k;
    ray_of(W, g, false, slot, k);
    const uint32_t rayIdx = slot * N + k;
    const float3 ro = slot_origin(C, slot), rd = wave_dir(W, k);
    uint4 h = C.hits[rayIdx];
    float3 outRgb;
    float hitT = -1.0f;
    if (h.x != 0xFFFFFFFFu) {
        uint32_t tri = h.x, inst = h.y & 0x7FFFFFFFu;
        float t = __uint_as_float(h.z);
        hitT = t;
        HitFrame fr = hit_frame(W, tri, inst, ro, rd, t, (int)(h.y >> 31));
        uint32_t m = __ldg(W.S.triMaterial + tri);
        const float* M = W.S.materials + (size_t)m * 28u;
        float3 baseColor = mk(__ldg(M), __ldg(M + 1), __ldg(M + 2));
        float3 emissive = mk(__ldg(M + 7), __ldg(M + 8), __ldg(M + 9));
        float3 radiance = emissive * W.P.debugEmissiveScale;
        float metal = __ldg(M + 4), transm = __ldg(M + 5);
        float3 kdr = baseColor * W.P.debugAlbedoScale * (1.0f - metal) * (1.0f - transm);
        float3 kd = mk(clampf(kdr.x, 0.f, 0.95f), clampf(kdr.y, 0.f, 0.95f), clampf(kdr.z, 0.f, 0.95f));
        if (C.reflect) {
            // with the reflection lobes on, a hit on a surface with no diffuse energy
            // and no emission is stored as -(t + 2): the blend keeps its depth, the
            // lobes ignore it (gi_probes.js:2055-2062)
            const float diffuseEnergy = (1.0f - metal) * (1.0f - transm);
            const float emissivePeak = fmaxf(fmaxf(emissive.x, emissive.y), emissive.z);
            if (!(diffuseEnergy > 0.02f || emissivePeak > 1e-6f)) hitT = -(t + ROUGH_UNSHADED_T_BIAS);
        }
        uint4 v = C.vis[rayIdx];
        unsigned long long ok = (unsigned long long)v.z | (unsigned long long)v.w << 32;
        while (ok) {
            uint32_t li = (uint32_t)(__ffsll((long long)ok) - 1);
            ok &= ok - 1ull;
            LightEval e = light_eval(W, li, fr.hitPos, fr.ng);
            radiance = radiance + light_term(W, e, kd);
        }
        float3 bounce = mul3(sample_atlas(C, fr.hitPos, fr.ng), kd) * (1.0f / PI_F);
        float bl = luma3(bounce);
        float roll = W.P.radianceClamp / fmaxf(fmaxf(W.P.radianceClamp, bl), 1e-6f);
        outRgb = radiance + bounce * roll * W.P.debugBounceScale;
    } else {
        outRgb = sky_sh(W.P, rd);
    }
    C.rayData[rayIdx] = make_float4(outRgb.x, outRgb.y, outRgb.z, hitT);
}

// ---------------------------------------------------------------- per solve

// Positions from a cursor up to `total`. Neighbouring rays are alike, and a warp whose 32
// are all long ones ends late where warps take only a few; `mix` then gives it eight
// from each quarter of the positions: 48 -> 42 us for the room's 32,768 closest hits,
// 79 -> 76 for 210,912 (59 a warp). Larger launches and the shadow jobs, whose
// neighbours share their first nodes, measured the same to 4% slower mixed.
__device__ __forceinline__ auto from_cursor(uint32_t* cursor, uint32_t total, bool mix = false) {
    mix = mix && total <= 64u * gridDim.x * (blockDim.x / 32u);
    const uint32_t row = mix ? ((total + 7u) / 8u + 3u) / 4u : 0u, end = mix ? row * 32u : total;
    return [cursor, total, row, end](uint32_t want, uint32_t& g, bool& ok) {
        bool more;
        const uint32_t p = take(cursor, end, want, more), b = p / 8u;
        g = row ? ((b % 4u) * row + b / 4u) * 8u + p % 8u : p;
        ok = p < end && g < total;
        return more;
    };
}

// Stages A and B of one solve on the 8-wide tree, by a warp, until its cursors are
// drained. A returns the rays it walked.
template <class Dir>
__device__ __forceinline__ uint32_t primary_stage(const WaveCtx& W, const WalkSmem& m, Dir dir, Visits& vis) {
    const uint32_t total = W.slotCount * W.C.rays;
    if (W.S.dynCount) primary_moved(W, *m.w2, from_cursor(&W.work[4], total), dir, vis);
    __syncwarp();
    const uint32_t n = primary_walk8(W, m, from_cursor(&W.work[0], total, true), dir, vis);
    __syncwarp();
    return n;
}
__device__ __forceinline__ void shadow_stage(const WaveCtx& W, const WalkSmem& m, uint32_t total, Visits& vis) {
    if (W.S.dynCount) shadow_moved(W, *m.w2, from_cursor(&W.work[5], total), vis);
    __syncwarp();
    shadow_walk8(W, m, from_cursor(&W.work[1], total), vis);
    __syncwarp();
}
__device__ __forceinline__ uint32_t job_count(const WaveCtx& W) {
    return min(*(volatile uint32_t*)&W.work[2], W.jobCap);
}

// The ray directions of a solve, by a CTA: for the later stages, and with their
// inverses for this CTA's walks (walk_shared synchronizes).
__device__ __forceinline__ void write_dirs(const WaveCtx& W) {
    for (uint32_t k = threadIdx.x; k < W.C.rays; k += blockDim.x) {
        const float3 d = ray_dir(k, W.C.rays, W.P.frameJitter);
        W.dirs[k] = make_float4(d.x, d.y, d.z, 0.0f);
    }
}
__device__ __forceinline__ void stage_dirs(const WaveCtx& W, float4* sm) {
    for (uint32_t k = threadIdx.x; k < W.C.rays; k += blockDim.x) {
        const float3 d = ray_dir(k, W.C.rays, W.P.frameJitter);
        sm[2 * k] = make_float4(d.x, d.y, d.z, 0.0f);
        sm[2 * k + 1] = make_float4(1.0f / d.x, 1.0f / d.y, 1.0f / d.z, 0.0f);
    }
}
__device__ __forceinline__ float3 staged_dir(const float4* sm, uint32_t k, float3& winv) {
    winv = xyz(sm[2 * k + 1]);
    return xyz(sm[2 * k]);
}

// The 8-wide tree (bvhKind 1).
__global__ void __launch_bounds__(256, SB_WALK8_MIN_BLOCKS) k_trace_primary_walk8(WaveCtx W) {
    extern __shared__ float4 smem[];
    stage_begin(W.slotBegin ? nullptr : W.C.stamps, 0);  // (a later chunk of the same solve)
    if (!*W.S.valid) return;
    if (blockIdx.x == 0) write_dirs(W);
    stage_dirs(W, smem);
    const WalkSmem m = walk_shared(smem + 2 * W.C.rays, W.S.wideDepth + 1u, W.S.dynCount != 0u);
    Visits vis = {0, 0, 0, 0};
    const uint32_t nRays = primary_stage(
        W, m, [&](uint32_t k, float3& winv) { return staged_dir(smem, k, winv); }, vis);
    add_visits(W.counters, 2, nRays, vis);
}

__global__ void __launch_bounds__(256, SB_WALK8_MIN_BLOCKS) k_trace_shadow_walk8(WaveCtx W) {
    extern __shared__ float4 smem[];
    stage_begin(W.C.stamps, 2);
    if (!*W.S.valid) return;
    const WalkSmem m = walk_shared(smem, W.S.wideDepth + 1u, W.S.dynCount != 0u);
    Visits vis = {0, 0, 0, 0};
    shadow_stage(W, m, job_count(W), vis);
    add_visits(W.counters, 6, 0u, vis);
}

// The binary scene BVH and the two-level walk (bvhKind 2 and 0).
__global__ void __launch_bounds__(256, SB_PRIMARY_MIN_BLOCKS) k_trace_primary(WaveCtx W) {
    extern __shared__ uint4 sTlas[];
    stage_begin(W.slotBegin ? nullptr : W.C.stamps, 0);  // (a later chunk of the same solve)
    const bool pairs = closest_pairs(W.S);
    const uint4* tl = stage_tlas(W, sTlas, pairs);
    if (!*W.S.valid) return;
    if (blockIdx.x == 0) write_dirs(W);
    const uint32_t total = W.slotCount * W.C.rays;
    const uint32_t lane = threadIdx.x & 31u;
    Visits vis = {0, 0, 0, 0};
    uint32_t nRays = 0;
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&W.work[0], 32u);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= total) break;
        // the batch at this issue position: costliest first when an order is given
        // (a permutation of the (total + 31) / 32 batches; clamped all the same)
        const uint32_t batch =
            W.C.batchOrder ? min(__ldg(W.C.batchOrder + (base >> 5)), (total - 1u) >> 5) : base >> 5;
        const uint32_t g = batch * 32u + lane;
        const long long t0 = W.C.batchCost ? clock64() : 0;
        if (g < total) {
            primary_ray(W, tl, pairs, g, vis);
            ++nRays;
        }
        if (W.C.batchCost) {
            __syncwarp();
            if (lane == 0) W.C.batchCost[batch] = (uint32_t)min(clock64() - t0, 0xFFFFFFFFll);
        }
    }
    add_visits(W.counters, 2, nRays, vis);
}

// The closest-hit batch order for the next full solve, by one CTA (all its
// threads call it; blockDim a multiple of 32): batches by descending recorded
// cycles, a counting sort over 128 log-spaced bins (4 per octave), so the
// persistent kernel starts the long batches first and its last warps hold
// short ones. Order within a bin is arbitrary; results do not depend on it.
__device__ __forceinline__ uint32_t cost_bin(uint32_t c) {
    if (c < 4u) return 0u;
    const uint32_t msb = 31u - __clz(c);
    return min(127u, msb * 4u + ((c >> (msb - 2u)) & 3u));
}
__device__ void order_batches(const uint32_t* cost, uint32_t* order, uint32_t n, uint32_t* at /* shared, 128 */) {
    for (uint32_t i = threadIdx.x; i < 128u; i += blockDim.x) at[i] = 0u;
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) atomicAdd(&at[cost_bin(__ldcg(cost + i))], 1u);
    __syncthreads();
    if (threadIdx.x < 32) {  // exclusive scan from the costliest bin down: 4 bins per lane
        const uint32_t l = threadIdx.x;
        uint32_t v[4], sum = 0;
        for (uint32_t j = 0; j < 4; ++j) {
            v[j] = at[127u - (4u * l + j)];
            sum += v[j];
        }
        uint32_t incl = sum;
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t u = __shfl_up_sync(0xFFFFFFFFu, incl, d);
            if (l >= d) incl += u;
        }
        uint32_t run = incl - sum;
        for (uint32_t j = 0; j < 4; ++j) {
            at[127u - (4u * l + j)] = run;
            run += v[j];
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) order[atomicAdd(&at[cost_bin(__ldcg(cost + i))], 1u)] = i;
}

// 64 registers: left to itself the compiler takes 84, and the atrium's emission 48 us
// instead of 41 (40 registers: 46).
constexpr int EMIT_MIN_BLOCKS = 8;
__global__ void __launch_bounds__(128, EMIT_MIN_BLOCKS) k_emit(WaveCtx W) {
    __shared__ float4 gates[4][GATE_LIGHTS];
    stage_begin(W.C.stamps, 1);
    if (!*W.S.valid) return;
    const uint32_t total = W.slotCount * W.C.rays;
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t nJobs = emit_ray(W, g < total, g, gates[threadIdx.x / 32u]);
    if (W.counters) {
        const uint32_t warpDone = __reduce_add_sync(0xFFFFFFFFu, nJobs);
        if ((threadIdx.x & 31u) == 0 && warpDone) atomicAdd(&W.counters[1], (unsigned long long)warpDone);
    }
}

__global__ void __launch_bounds__(256, SB_SHADOW_MIN_BLOCKS) k_trace_shadow(WaveCtx W) {
    extern __shared__ uint4 sTlas[];
    stage_begin(W.C.stamps, 2);
    const bool pairs = any_pairs(W.S);
    const uint4* tl = stage_tlas(W, sTlas, pairs);
    if (!*W.S.valid) return;
    const uint32_t total = min(*(volatile uint32_t*)&W.work[2], W.jobCap);
    const uint32_t lane = threadIdx.x & 31u;
    Visits vis = {0, 0, 0, 0};
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(&W.work[1], 32u);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= total) break;
        uint32_t j = base + lane;
        if (j >= total) continue;
        const float4 a = W.jobs[2 * j], b = W.jobs[2 * j + 1];
        shadow_job(W, tl, pairs, a, b, vis);
    }
    add_visits(W.counters, 6, 0u, vis);
    if (W.C.batchOrderOut) {
        // the queue is drained: the first CTA whose warps are all done orders the
        // closest-hit batches for the next solve while the others finish their jobs
        __shared__ uint32_t at[128];
        __shared__ uint32_t first;
        __syncthreads();
        if (threadIdx.x == 0) first = atomicAdd(&W.work[3], 1u) == 0u ? 1u : 0u;
        __syncthreads();
        if (first) order_batches(W.C.batchCost, W.C.batchOrderOut, (W.slotCount * W.C.rays + 31u) / 32u, at);
    }
}

// The cursors of the stages ahead, for the next solve (128 threads).
static_assert(SB_BATCH_MAX * WORK_WORDS <= 128, "one word per thread of a CTA");
__device__ __forceinline__ void clear_work(uint32_t* work, uint32_t words) {
    if (work && blockIdx.x == 0 && threadIdx.x < words) work[threadIdx.x] = 0u;
}

__global__ void __launch_bounds__(128) k_shade(WaveCtx W) {
    stage_begin(W.C.stamps, 3);
    clear_work(W.work, WORK_WORDS);
    if (!*W.S.valid) return;
    const uint32_t g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= W.slotCount * W.C.rays) return;
    shade_ray(W, g);
}

// emitterVisKernel (gi_probes.js:2216-2260): per (updated probe, emitter) a
// shadow ray from the probe to a point of the emitter's disk, chosen by a sin
// hash of (probe, emitter, epoch seed) evaluated in separately rounded FP32,
// folded into the emitter's visibility history with retention 0.8.
//
// The rays join stage B's jobs. By themselves they are too few to fill the chip (2,197
// probes and 3 emitters: 206 warps) and take as long as their longest walk, 72 us,
// while stage B walks ninety times as many in 155: there they cost 9 us, the jobs' and
// the fold's launches included. The outcomes of a probe's rays are the emitters' bits of an
// unblocked mask behind the rays' own.
__global__ void __launch_bounds__(128) k_emitter_jobs(WaveCtx W) {
    stage_wait();
    if (!*W.S.valid) return;
    const DevCascade& C = W.C;
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31u;
    const bool active = i < W.slotCount;
    const uint32_t slot = W.slotBegin + (active ? i : 0u), probeIndex = probe_of(C, slot);
    const uint32_t ray = C.probeTotal * C.rays + slot;
    const float3 ro = slot_origin(C, slot);
    uint32_t open = 0u;
    for (uint32_t e = 0; e < C.emitterCount; ++e) {
        const uint32_t li = C.emitterBase + e;
        const float* L = C.lights + (size_t)li * 17u;
        const float3 center = mk(L[1], L[2], L[3]);
        const float sourceRadius = fmaxf(L[14], 0.0f);
        const float3 axis = center - ro;
        const float dist = sqrtf(dot3(axis, axis));
        const bool far = active && dist > fmaxf(sourceRadius, 1e-3f);
        const uint32_t jobs = __ballot_sync(ALL_LANES, far);
        if (!jobs) continue;
        uint32_t j = 0;
        if (lane == 0) j = atomicAdd(&W.work[2], (uint32_t)__popc(jobs));
        j = __shfl_sync(ALL_LANES, j, 0) + (uint32_t)__popc(jobs & ((1u << lane) - 1u));
        if (!far) continue;
        if (j >= W.jobCap) {
            latch(W.err, ERR_CAPACITY);  // (unreachable: the queue has a job per probe and emitter too)
            continue;
        }
        const float3 d = axis * (1.0f / dist);
        const float3 up = fabsf(d.y) < 0.999f ? mk(0.0f, 1.0f, 0.0f) : mk(1.0f, 0.0f, 0.0f);
        const float3 tangent = normalize3(cross3(up, d));
        const float3 bitangent = cross3(d, tangent);
        const float seed = __fadd_rn(__fadd_rn(__fmul_rn(float(probeIndex), 12.9898f), __fmul_rn(float(e), 78.233f)),
                                     __fmul_rn(W.P.emitterVisSeed, 37.719f));
        const float h0 = __fmul_rn(sinf(seed), 43758.5453f);
        const float h1 = __fmul_rn(sinf(__fadd_rn(seed, 19.19f)), 24634.6345f);
        const float u = h0 - floorf(h0), v = h1 - floorf(h1);
        const float diskRadius = sqrtf(u) * sourceRadius;
        const float diskAngle = v * 6.283185307179586f;
        const float3 target = center + (tangent * (cosf(diskAngle) * diskRadius) + bitangent * (sinf(diskAngle) * diskRadius));
        const float3 sdir = normalize3(target - ro);
        const float traceBias = fmaxf(C.cellMin * 0.005f * W.P.debugTraceBiasScale, RAY_EPS * W.P.debugRayEpsScale);
        store32(W.jobs + 2 * j, make_float4(ro.x, ro.y, ro.z, fmaxf(dist - sourceRadius - traceBias, 1e-4f)),
                make_float4(sdir.x, sdir.y, sdir.z, __uint_as_float(ray << 6 | e)));
        open |= 1u << e;
    }
    if (active) C.vis[ray] = make_uint4(open, 0u, open, 0u);
}

__global__ void __launch_bounds__(128) k_emitter_vis(DevScene S, DevCascade C) {
    stage_wait();
    const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= C.updatedCount || !*S.valid) return;
    const uint32_t open = C.vis[C.probeTotal * C.rays + slot].z;
    float* vp = C.emitterVis + (size_t)probe_of(C, slot) * EMITTER_CAP;
    for (uint32_t e = 0; e < C.emitterCount; ++e) {
        const float sample = open >> e & 1u ? 1.0f : 0.0f;
        vp[e] = sample * (1.0f - EMITTER_VIS_RETENTION) + vp[e] * EMITTER_VIS_RETENTION;
    }
}

cudaError_t launch_emitter_vis(const DevScene& S, const DevCascade& C, cudaStream_t st) {
    if (C.updatedCount == 0 || C.emitterCount == 0) return cudaSuccess;
    return launch_stage(k_emitter_vis, (C.updatedCount + 127) / 128, 128, 0, st, S, C);
}

// Stage C alone over probe slots [0, slotCount) from the records already in
// C.hits / C.vis (the adjoint re-evaluates shading this way).
cudaError_t launch_shade(const DevScene& S, const DevCascade& C, const DevParams& P, const float4* dirs,
                         uint32_t slotCount, cudaStream_t st) {
    if (slotCount == 0) return cudaSuccess;
    WaveCtx W{};
    W.S = S;
    W.C = C;
    W.P = P;
    W.slotBegin = 0;
    W.slotCount = slotCount;
    W.rayMagic = div_magic(C.rays);
    W.dirs = const_cast<float4*>(dirs);
    const uint32_t rays = slotCount * C.rays;
    k_shade<<<(rays + 127) / 128, 128, 0, st>>>(W);
    note_launch();
    return cudaGetLastError();
}

static int persistent_grid(const void* kernel, int block, size_t smem, const TraceTuning& tune, uint32_t items) {
    int perSm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&perSm, kernel, block, smem);
    if (perSm < 1) perSm = 1;
    int grid = tune.numSms * perSm;
    uint32_t needed = (items + block - 1) / block;
    if ((uint32_t)grid > needed) grid = (int)needed;
    return grid < 1 ? 1 : grid;
}

static int walk8_grid(const void* kernel, int block, size_t smem, const TraceTuning& tune, uint32_t items) {
    if (smem > 48u * 1024u) cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return persistent_grid(kernel, block, smem, tune, items);
}

cudaError_t launch_trace(const DevScene& S, const DevCascade& C, const DevParams& P, uint32_t* err,
                         unsigned long long* counters, uint32_t* work, float4* dirs, const TraceTuning& tune,
                         cudaStream_t st, float4* jobs, uint32_t jobCap, uint32_t slotBegin, uint32_t slotCount) {
    if (slotCount == 0) return cudaSuccess;
    WaveCtx W;
    W.S = S;
    W.C = C;
    W.P = P;
    W.err = err;
    W.counters = counters;
    W.work = work;
    W.jobs = jobs;
    W.jobCap = jobCap;
    W.dirs = dirs;
    W.slotBegin = slotBegin;
    W.slotCount = slotCount;
    W.slotMagic = div_magic(slotCount);
    W.rayMagic = div_magic(C.rays);
    W.order = tune.sortKey == 1 ? 0u : 1u;  // direction-major (sortKey 0, and 2 over probe tiles); 1 = probe-major
    // the scene-BVH walk reads no TLAS
    uint32_t smemNodes = !S.flatOn && S.tlasNodeCount <= tune.smemTlasNodes ? S.tlasNodeCount : 0u;
    W.smemTlas = smemNodes;
    const size_t smem = (size_t)smemNodes * 64u;  // room for the child-pair TLAS (the 32-byte nodes need half)
    if (smem > 48u * 1024u) {
        cudaFuncSetAttribute(k_trace_primary, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaFuncSetAttribute(k_trace_shadow, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    }
    const uint32_t rays = slotCount * C.rays, perRay = (rays + 127) / 128;
    const int block = (int)tune.block;
    const size_t smem8 = walk_smem(S.wideDepth + 1u, S.dynCount != 0u, tune.block);
    const size_t smemP = smem8 + 2u * C.rays * sizeof(float4);
    cudaError_t e;
    if (S.wideNodes)
        k_trace_primary_walk8<<<walk8_grid((const void*)k_trace_primary_walk8, block, smemP, tune, rays), block, smemP,
                                st>>>(W);
    else
        k_trace_primary<<<persistent_grid((const void*)k_trace_primary, block, smem, tune, rays), block, smem, st>>>(W);
    note_launch();
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    if ((e = launch_stage(k_emit, perRay, 128, 0, st, W)) != cudaSuccess) return e;
    if (C.emitterCount && (e = launch_stage(k_emitter_jobs, (slotCount + 127) / 128, 128, 0, st, W)) != cudaSuccess)
        return e;
    // shadow jobs: at most lightCount per ray (the queue is sized for it)
    if (S.wideNodes)
        e = launch_stage(k_trace_shadow_walk8,
                         (uint32_t)walk8_grid((const void*)k_trace_shadow_walk8, block, smem8, tune, rays * 4u),
                         (uint32_t)block, smem8, st, W);
    else
        e = launch_stage(k_trace_shadow,
                         (uint32_t)persistent_grid((const void*)k_trace_shadow, block, smem, tune, rays * 4u),
                         (uint32_t)block, smem, st, W);
    return e != cudaSuccess ? e : launch_stage(k_shade, perRay, 128, 0, st, W);
}

// ---------------------------------------------------------------- batched
// The same four stages over every item of a BatchArgs: one launch per stage
// for all scenes and cascades, each item with its own cursors and job queue.
//
// The CTAs of a walk start on the items in proportion to their rays (stage B: jobs),
// and a warp whose item is drained goes on with the next. So the context a warp
// reads is uniform and most warps run dry once. One cursor over all items, a chunk of
// 32 at a time with the walk ended where the item changed, measured 145 + 155 us
// against 142 + 140 for four fields of 512 to 1,331 probes x 80 rays.
__device__ __forceinline__ uint32_t next_item(const BatchArgs& B, uint32_t i) { return i + 1 < B.n ? i + 1 : 0u; }

__global__ void __launch_bounds__(256, SB_WALK8_MIN_BLOCKS) k_trace_primary_batch(const __grid_constant__ BatchArgs B) {
    extern __shared__ float4 smem[];
    stage_begin(B.it[0].W.C.stamps, 0);
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t first = batch_item(B, (uint32_t)((uint64_t)blockIdx.x * B.totalRays / gridDim.x));
    for (uint32_t j = blockIdx.x; j < B.n; j += gridDim.x) write_dirs(B.it[j].W);
    stage_dirs(B.it[first].W, smem);
    const WalkSmem m = walk_shared(smem + 2 * B.maxRays, B.wideDepth + 1u, B.moved != 0u);
    Visits vis = {0, 0, 0, 0};
    uint32_t nRays = 0;
    uint32_t i = first;
    for (uint32_t visited = 0; visited < B.n; ++visited, i = next_item(B, i)) {
        const WaveCtx& W = B.it[i].W;
        if (!*W.S.valid) continue;
        if (W.S.wideNodes) {
            nRays += primary_stage(W, m, [&](uint32_t k, float3& winv) {
                if (i == first) return staged_dir(smem, k, winv);
                const float3 d = ray_dir(k, W.C.rays, W.P.frameJitter);
                winv = mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
                return d;
            }, vis);
            continue;
        }
        const bool pairs = closest_pairs(W.S);
        for (;;) {  // the other layouts: 32 rays at a time, one per lane
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&W.work[0], 32u);
            base = __shfl_sync(ALL_LANES, base, 0);
            if (base >= B.it[i].rays) break;
            if (base + lane < B.it[i].rays) {
                primary_ray(W, pairs ? W.S.tlasPairs : W.S.tlas, pairs, base + lane, vis);
                ++nRays;
            }
            __syncwarp();
        }
    }
    add_visits(B.counters, 2, nRays, vis);
}

__global__ void __launch_bounds__(128, EMIT_MIN_BLOCKS) k_emit_batch(const __grid_constant__ BatchArgs B) {
    __shared__ float4 gates[4][GATE_LIGHTS];
    stage_begin(B.it[0].W.C.stamps, 1);
    const uint32_t gg = blockIdx.x * blockDim.x + threadIdx.x;
    if (gg - (threadIdx.x & 31u) >= B.totalRays) return;  // whole warps only
    const BatchItem& I = B.it[batch_item(B, gg & ~31u)];
    if (!*I.W.S.valid) return;
    const uint32_t g = gg - I.rayBase;
    const uint32_t nJobs = emit_ray(I.W, g < I.rays, g, gates[threadIdx.x / 32u]);
    if (B.counters) {
        const uint32_t warpDone = __reduce_add_sync(0xFFFFFFFFu, nJobs);
        if ((threadIdx.x & 31u) == 0 && warpDone) atomicAdd(&B.counters[1], (unsigned long long)warpDone);
    }
}

__global__ void __launch_bounds__(256, SB_WALK8_MIN_BLOCKS) k_trace_shadow_batch(const __grid_constant__ BatchArgs B) {
    extern __shared__ float4 smem[];
    stage_begin(B.it[0].W.C.stamps, 2);
    const uint32_t lane = threadIdx.x & 31u;
    const WalkSmem m = walk_shared(smem, B.wideDepth + 1u, B.moved != 0u);
    Visits vis = {0, 0, 0, 0};
    uint32_t i = 0;
    {  // the item this CTA starts on
        const uint32_t own = lane < B.n ? job_count(B.it[lane].W) : 0u;
        uint32_t all = own;
#pragma unroll
        for (uint32_t d = 1; d < SB_BATCH_MAX; d <<= 1) {
            const uint32_t v = __shfl_up_sync(ALL_LANES, all, d);
            if (lane >= d) all += v;
        }
        const uint32_t jobs = __shfl_sync(ALL_LANES, all, SB_BATCH_MAX - 1u);
        const uint32_t at = (uint32_t)((uint64_t)blockIdx.x * jobs / gridDim.x);
        const uint32_t ahead = __ballot_sync(ALL_LANES, lane < B.n && all <= at);  // items wholly ahead of it
        i = min((uint32_t)__popc(ahead), B.n - 1u);
    }
    for (uint32_t visited = 0; visited < B.n; ++visited, i = next_item(B, i)) {
        const WaveCtx& W = B.it[i].W;
        const uint32_t total = job_count(W);
        if (!total || !*W.S.valid) continue;
        if (W.S.wideNodes) {
            shadow_stage(W, m, total, vis);
            continue;
        }
        const bool pairs = any_pairs(W.S);
        for (;;) {
            uint32_t base = 0;
            if (lane == 0) base = atomicAdd(&W.work[1], 32u);
            base = __shfl_sync(ALL_LANES, base, 0);
            if (base >= total) break;
            if (base + lane < total)
                shadow_job(W, pairs ? W.S.tlasPairs : W.S.tlas, pairs, W.jobs[2 * (base + lane)],
                           W.jobs[2 * (base + lane) + 1], vis);
            __syncwarp();
        }
    }
    add_visits(B.counters, 6, 0u, vis);
}

__global__ void __launch_bounds__(128) k_shade_batch(const __grid_constant__ BatchArgs B) {
    stage_begin(B.it[0].W.C.stamps, 3);
    clear_work(B.work, SB_BATCH_MAX * WORK_WORDS);
    const uint32_t gg = blockIdx.x * blockDim.x + threadIdx.x;
    if (gg >= B.totalRays) return;
    const BatchItem& I = B.it[batch_item(B, gg & ~31u)];
    const uint32_t g = gg - I.rayBase;
    if (g >= I.rays || !*I.W.S.valid) return;
    shade_ray(I.W, g);
}

const void* trace_batch_kernel(int stage) {
    switch (stage) {
        case 0: return (const void*)k_trace_primary_batch;
        case 1: return (const void*)k_emit_batch;
        case 2: return (const void*)k_trace_shadow_batch;
        case 3: return (const void*)k_shade_batch;
        default: return nullptr;
    }
}

uint32_t trace_batch_smem(const BatchArgs& B, uint32_t threads) {
    const uint32_t smem =
        walk_smem(B.wideDepth + 1u, B.moved != 0u, threads) + 2u * B.maxRays * (uint32_t)sizeof(float4);
    if (smem > 48u * 1024u)
        for (int stage = 0; stage <= 2; stage += 2)
            cudaFuncSetAttribute(trace_batch_kernel(stage), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    return smem;
}

cudaError_t launch_trace_batch(const BatchArgs& B, const TraceTuning& tune, cudaStream_t st) {
    if (B.n == 0 || B.totalRays == 0) return cudaSuccess;
    const int block = (int)tune.block;
    const uint32_t rays = B.totalRays;
    const size_t smem = trace_batch_smem(B, tune.block);
    k_trace_primary_batch<<<walk8_grid((const void*)k_trace_primary_batch, block, smem, tune, rays), block, smem,
                            st>>>(B);
    note_launch();
    k_emit_batch<<<(rays + 127) / 128, 128, 0, st>>>(B);
    note_launch();
    k_trace_shadow_batch<<<walk8_grid((const void*)k_trace_shadow_batch, block, smem, tune, rays * 4u), block, smem,
                           st>>>(B);
    note_launch();
    k_shade_batch<<<(rays + 127) / 128, 128, 0, st>>>(B);
    note_launch();
    return cudaGetLastError();
}

// Arbitrary rays through traverseClosest / traverseAny (global TLAS reads).
__global__ void k_raycast(DevScene S, const float* ro, const float* rd, uint32_t n, float* tOut, int32_t* triOut,
                          int32_t* instOut, uint32_t* err) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !*S.valid) return;
    Visits vis = {0, 0, 0, 0};
    float t, bu, bv;
    int tri, inst;
    float3 o = mk(ro[3 * i], ro[3 * i + 1], ro[3 * i + 2]), d = mk(rd[3 * i], rd[3 * i + 1], rd[3 * i + 2]);
    const bool pairs = closest_pairs(S);
    trace_closest(S, pairs ? S.tlasPairs : S.tlas, o, d, t, tri, inst, bu, bv, vis, err, pairs);
    if (tri >= 0) t = refine_t(S, (uint32_t)tri, (uint32_t)inst, o, d);
    tOut[i] = t;
    triOut[i] = tri;
    instOut[i] = inst;
}

__global__ void k_occluded(DevScene S, const float* ro, const float* rd, const float* maxDist, uint32_t n, uint8_t* out,
                           uint32_t* err) {
    uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !*S.valid) return;
    Visits vis = {0, 0, 0, 0};
    const bool pairs = any_pairs(S);
    out[i] = trace_any(S, pairs ? S.tlasPairs : S.tlas, mk(ro[3 * i], ro[3 * i + 1], ro[3 * i + 2]),
                       mk(rd[3 * i], rd[3 * i + 1], rd[3 * i + 2]), maxDist[i], vis, err, pairs)
                 ? 1
                 : 0;
}

// The rays of a query for the walks: the next ones of the lanes in `want` (all lanes call
// it), by a cursor: the query's, or (OWN) one of the CTA's two, 0 the tree's walk, 1 the moved
// slots'.
template <bool ANY, bool OWN> struct QueryRays {
    const float *ro, *rd, *maxDist;
    uint32_t n, end;  // end: of the cursor's positions
    uint32_t* cursor;
    // (OWN: the CTA synchronizes before the first call)
    __device__ QueryRays(const float* ro, const float* rd, const float* maxDist, uint32_t n, uint32_t* cursor)
        : ro(ro), rd(rd), maxDist(maxDist), n(n), end(n), cursor(cursor) {
        if (OWN) {
            __shared__ uint32_t own[2];
            if (threadIdx.x < 2u) own[threadIdx.x] = 0u;
            this->cursor = own;
            end = ((n + 31u) / 32u + gridDim.x - 1u - blockIdx.x) / gridDim.x * 32u;
        }
    }
    __device__ QueryRays moved() const {  // (OWN) the same rays by the other cursor
        QueryRays r = *this;
        ++r.cursor;
        return r;
    }
    __device__ __forceinline__ bool operator()(bool& more, uint32_t want, float3& o, float3& d, float3& winv,
                                               float& tmax, uint32_t& tag) const {
        const uint32_t p = take(cursor, end, want, more);
        const uint32_t i = OWN ? (p / 32u * gridDim.x + blockIdx.x) * 32u + p % 32u : p;
        if (!(p < end && i < n && (want >> (threadIdx.x & 31u) & 1u))) return false;
        const size_t i3 = 3 * (size_t)i;
        o = mk(ro[i3], ro[i3 + 1], ro[i3 + 2]);
        d = mk(rd[i3], rd[i3 + 1], rd[i3 + 2]);
        winv = mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
        tmax = ANY ? maxDist[i] : T_MAX;
        tag = i;
        return true;
    }
};

// A warp's rays through the moved slots, by walk2 (a BLAS too deep for it: one ray per lane).
template <bool ANY, class Rays, class Fin>
__device__ __forceinline__ void walk2_rays(const DevScene& S, Walk2Shared& sm, Rays rays, Fin fin, Visits& vis,
                                           uint32_t* err) {
    if (walk2_usable(S)) {
        walk2<ANY>(S, sm, rays, fin, vis, err);
        return;
    }
    for (bool more = true; more;) {
        float3 o, d, winv;
        float t, u = 0.0f, v = 0.0f;
        uint32_t i;
        int tri = -1, inst = -1;
        if (rays(more, ALL_LANES, o, d, winv, t, i)) {
            const bool blocked = dyn_walk<ANY, !ANY>(S, o, d, winv, t, tri, inst, u, v, vis, err);
            fin(i, t, make_uint4((uint32_t)tri, (uint32_t)inst, 0u, 0u), blocked);
        }
        __syncwarp();
    }
}

// Queries of fewer rays are one launch that needs nothing ahead of it and nothing after.
constexpr uint32_t FEW_RAYS = 1u << 18;

// The same on the 8-wide tree. The warps share the rays by a cursor, a word of the stream's
// own: queries on several streams run side by side. OWN, without one, for few rays and for
// captured queries (which may be replayed beside any other): each CTA takes every
// gridDim.x-th 32 rays, its warps share those, and the hits' parameters are formed here
// (refine_t). With a clear of the cursor ahead and a launch for the parameters behind, closest
// hits of 1 / 100 / 10,000 / 131,072 rays take 16.6 / 27.3 / 35.1 / 53.5 us in the atrium
// instead of 11.0 / 21.6 / 29.0 / 47.0; from 2^19 rays the cursor spreads them better (2.07M:
// 417 against 437). MOVED: the scene has moved slots, and what they gave
// is in the outputs; `here` (OWN): these warps walk them first (any hits: a ray is blocked by
// either, and `out` is 0 before; in a launch of their own closest hits of 1 / 100 /
// 200,000 rays took 15.5 / 41.3 / 109.8 us in the atrium with three slots moved, so 12.5 /
// 39.2 / 103.5).
template <bool ANY, bool MOVED, bool OWN>
__global__ void __launch_bounds__(256, SB_WALK8_MIN_BLOCKS) k_query_walk8(DevScene S, const float* ro, const float* rd,
                                                                          const float* maxDist, uint32_t n,
                                                                          float* tOut, int32_t* triOut,
                                                                          int32_t* instOut, uint8_t* out,
                                                                          uint32_t here, uint32_t* cursor,
                                                                          uint32_t* err) {
    extern __shared__ float4 smem[];
    if (!*S.valid) return;
    const QueryRays<ANY, OWN> rays(ro, rd, maxDist, n, cursor);
    const WalkSmem m = walk_shared(smem, S.wideDepth + 1u, MOVED && OWN && here);  // (synchronizes)
    Visits vis = {0, 0, 0, 0};
    if (MOVED && OWN && here) {
        walk2_rays<ANY>(S, *m.w2, rays.moved(), [&](uint32_t i, float t, uint4 hit, bool blocked) {
            if (ANY) {
                if (blocked) out[i] = 1;
            } else {
                tOut[i] = t;
                triOut[i] = (int32_t)hit.x;
                instOut[i] = (int32_t)hit.y;
            }
        }, vis, err);
        if (ANY) __syncwarp();
        else __syncthreads();  // the tree's walk takes the CTA's rays anew, each with its hit
    }
    auto gen = [&](bool& more, uint32_t idle, float3& o, float3& d, float3& winv, float& tmax, uint32_t& tag,
                   uint4& hit) {
        if (!rays(more, idle, o, d, winv, tmax, tag)) return false;
        hit = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u);
        if (MOVED && ANY) return out[tag] == 0;  // (not seen yet: walked in vain)
        if (MOVED) {
            tmax = tOut[tag];
            hit.x = (uint32_t)triOut[tag];
            hit.y = (uint32_t)instOut[tag];
        }
        return true;
    };
    auto fin = [&](uint32_t i, float t, uint4 hit, bool blocked) {
        if (ANY) {
            if (!MOVED || blocked) out[i] = blocked ? 1 : 0;
        } else {
            if (OWN && hit.x != 0xFFFFFFFFu) {
                const size_t i3 = 3 * (size_t)i;
                t = refine_t(S, hit.x, hit.y, mk(ro[i3], ro[i3 + 1], ro[i3 + 2]), mk(rd[i3], rd[i3 + 1], rd[i3 + 2]));
            }
            tOut[i] = t;
            triOut[i] = (int32_t)hit.x;
            instOut[i] = (int32_t)hit.y;
        }
    };
    walk8<ANY>(S, *m.tables, *m.w8, m.stk, S.wideDepth + 1u, gen, fin, vis, err);
}

// The moved slots ahead of the tree, into the outputs, for queries of FEW_RAYS rays or
// more one thread per ray: rays that neighbour one another walk the slots together, and there
// are enough of them. Fewer go by walk2, whose launch does not last as long as its longest
// ray. (Walked by each lane of the tree's walk as it took a ray, 8 lanes or so together, as
// they were, three slots cost 400,000 rays in the atrium 182 and 89 us (closest, any) and 29
// of them 776 and 352; so 149 and 75, 567 and 274. 65,536 rays by thread / by walk2, closest:
// 103 / 82 us with three slots, 254 / 160 with 29; 10^6 of a camera's 306 / 341, 426 / 677.)
template <bool ANY>
__global__ void __launch_bounds__(128) k_query_moved(DevScene S, const float* ro, const float* rd,
                                                     const float* maxDist, uint32_t n, float* tOut, int32_t* triOut,
                                                     int32_t* instOut, uint8_t* out, uint32_t* err) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !*S.valid) return;
    const size_t i3 = 3 * (size_t)i;
    const float3 o = mk(ro[i3], ro[i3 + 1], ro[i3 + 2]), d = mk(rd[i3], rd[i3 + 1], rd[i3 + 2]);
    float t = ANY ? maxDist[i] : T_MAX, bu = 0.0f, bv = 0.0f;
    int tri = -1, inst = -1;
    Visits vis = {0, 0, 0, 0};
    const bool blocked =
        dyn_walk<ANY, !ANY>(S, o, d, mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z), t, tri, inst, bu, bv, vis, err);
    if (ANY) {
        out[i] = blocked ? 1 : 0;
    } else {
        tOut[i] = t;
        triOut[i] = tri;
        instOut[i] = inst;
    }
}
// The hits' parameters in FP64 (refine_t), one thread per ray.
__global__ void k_refine_hits(DevScene S, const float* ro, const float* rd, uint32_t n, float* t, const int32_t* tri,
                              const int32_t* inst) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || !*S.valid || tri[i] < 0) return;
    const size_t i3 = 3 * (size_t)i;
    t[i] = refine_t(S, (uint32_t)tri[i], (uint32_t)inst[i], mk(ro[i3], ro[i3 + 1], ro[i3 + 2]),
                    mk(rd[i3], rd[i3 + 1], rd[i3 + 2]));
}

// A query on the 8-wide tree.
template <bool ANY>
static cudaError_t launch_query(const DevScene& S, const float* ro, const float* rd, const float* maxDist, uint32_t n,
                                float* tOut, int32_t* triOut, int32_t* instOut, uint8_t* out, uint32_t* cursor,
                                int numSms, uint32_t* err, cudaStream_t st) {
    const TraceTuning tune{256u, 0u, 0u, numSms, 0u};
    const bool moved = S.dynCount != 0u, few = n < FEW_RAYS, here = moved && few;
    if (few) cursor = nullptr;
    cudaError_t e = cursor ? cudaMemsetAsync(cursor, 0, 4u, st) : cudaSuccess;
    if (e == cudaSuccess && ANY && here) e = cudaMemsetAsync(out, 0, n, st);
    if (e != cudaSuccess) return e;
    if (moved && !here) {
        k_query_moved<ANY><<<(n + 127) / 128, 128, 0, st>>>(S, ro, rd, maxDist, n, tOut, triOut, instOut, out, err);
        note_launch();
    }
    const auto kernel = cursor ? moved ? k_query_walk8<ANY, true, false> : k_query_walk8<ANY, false, false>
                               : moved ? k_query_walk8<ANY, true, true> : k_query_walk8<ANY, false, true>;
    const size_t smem = walk_smem(S.wideDepth + 1u, here, 256u);
    kernel<<<walk8_grid((const void*)kernel, 256, smem, tune, n), 256, smem, st>>>(
        S, ro, rd, maxDist, n, tOut, triOut, instOut, out, here ? 1u : 0u, cursor, err);
    note_launch();
    if (!ANY && cursor) {
        k_refine_hits<<<(n + 127) / 128, 128, 0, st>>>(S, ro, rd, n, tOut, triOut, instOut);
        note_launch();
    }
    return cudaGetLastError();
}

cudaError_t launch_raycast(const DevScene& S, const float* ro, const float* rd, uint32_t n, float* tOut,
                           int32_t* triOut, int32_t* instOut, uint32_t* cursor, int numSms, uint32_t* err,
                           cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    if (S.wideNodes)
        return launch_query<false>(S, ro, rd, nullptr, n, tOut, triOut, instOut, nullptr, cursor, numSms, err, st);
    k_raycast<<<(n + 127) / 128, 128, 0, st>>>(S, ro, rd, n, tOut, triOut, instOut, err);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_occluded(const DevScene& S, const float* ro, const float* rd, const float* maxDist, uint32_t n,
                            uint8_t* out, uint32_t* cursor, int numSms, uint32_t* err, cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    if (S.wideNodes)
        return launch_query<true>(S, ro, rd, maxDist, n, nullptr, nullptr, nullptr, out, cursor, numSms, err, st);
    k_occluded<<<(n + 127) / 128, 128, 0, st>>>(S, ro, rd, maxDist, n, out, err);
    note_launch();
    return cudaGetLastError();
}

}  // namespace sb

namespace sb {
// The probe rays of a solve exactly as the trace stage forms them (probe
// origin and ray_dir with the current frame jitter): ray slot * rays + k.
__global__ void k_probe_rays(const DevCascade C, float jitter, float* ro, float* rd) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= C.updatedCount * C.rays) return;
    const uint32_t slot = i / C.rays, k = i % C.rays;
    const float3 o = slot_origin(C, slot);
    const float3 d = ray_dir(k, C.rays, jitter);
    ro[3 * i] = o.x; ro[3 * i + 1] = o.y; ro[3 * i + 2] = o.z;
    rd[3 * i] = d.x; rd[3 * i + 1] = d.y; rd[3 * i + 2] = d.z;
}
// The tables of slot_origin (with a cascade's grid) and wave_dir.
__global__ void k_probe_positions(DevCascade C, float4* pos) {
    const uint32_t p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= C.probeTotal) return;
    const float3 v = probe_world_pos(C, p);
    pos[p] = make_float4(v.x, v.y, v.z, 0.0f);
}
cudaError_t launch_probe_positions(const DevCascade& C, float4* pos, cudaStream_t st) {
    if (C.probeTotal == 0) return cudaSuccess;
    k_probe_positions<<<(C.probeTotal + 255) / 256, 256, 0, st>>>(C, pos);
    note_launch();
    return cudaGetLastError();
}
__global__ void k_ray_dirs(uint32_t rays, float jitter, float4* dirs) {
    const uint32_t k = threadIdx.x;
    if (k >= rays) return;
    const float3 d = ray_dir(k, rays, jitter);
    dirs[k] = make_float4(d.x, d.y, d.z, 0.0f);
}
cudaError_t launch_ray_dirs(uint32_t rays, float jitter, float4* dirs, cudaStream_t st) {
    k_ray_dirs<<<1, MAX_RAYS, 0, st>>>(rays, jitter, dirs);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_probe_rays(const DevCascade& C, float jitter, float* ro, float* rd, cudaStream_t st) {
    const uint32_t n = C.updatedCount * C.rays;
    if (n == 0) return cudaSuccess;
    k_probe_rays<<<(n + 255) / 256, 256, 0, st>>>(C, jitter, ro, rd);
    note_launch();
    return cudaGetLastError();
}
}  // namespace sb

extern "C" uint32_t sb_triangle_test(void) { return SB_WATERTIGHT ? 1u : 0u; }
