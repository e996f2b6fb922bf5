// sb_walk8.cuh — the 8-wide scene-BVH walk of a persistent warp: one ray per lane,
// one node visit per step in every lane, item tests collected across the lanes.
//
// A warp whose lanes walk their rays to the end (or to the next leaf) leaves two
// thirds of its lanes idle: the rays need different numbers of visits, and a
// lane that holds items waits for those that do not. Here nothing waits for
// another lane's ray. Every step visits one node per walking lane; the items of
// the leaves it hits go to a queue in shared memory, and when 32 have gathered
// each lane tests one, whoever's ray it belongs to. A lane whose ray has ended
// takes a new one. The price is that a ray's limit shrinks up to one queue later
// than it could, which costs some visits.
//
// The visiting order per ray is that of a walk that tests a node's items at once:
// children in increasing (slot XOR octant), a node's items before its children.
// The queue keeps each ray's items in that order, and of equal t the first wins,
// so the hit is the same one. (An item that only the later limit lets through
// starts at or behind the hit found and is not accepted.)
//
// Node (5 x uint4, 80 bytes, from sb_flat.h's): origin xyz, the axes' scales in
// bfloat16 (they are powers of two) x | y << 16; first child, first item, interior
// mask << 24 | item mask, scale z << 16; then the child boxes' bytes lo x, y, z,
// hi x, y, z (two words each). Bit 3 s + j of the item mask: slot s holds a j-th
// item; items lie in the order of their bits.
//
// What bounds it (ncu, 1080p diffuse bounce in the 262k-triangle atrium, 2.07M rays):
// issue slots (65%) and the L1's wavefronts (52%: every lane reads a node of its
// own); a visit is about 190 of a step's instructions, half of them on the integer
// pipe, which takes one every second cycle. So what is not a plane distance is kept
// short: the box tests end in subtractions whose signs one three-input logic
// operation and one funnel shift per child collect, and the masks of hit children
// go through small tables in shared memory. Measured against one walk per lane (for
// any hits on a binary tree), the last rays shared: closest hits 1431 -> 507 us there,
// 194 -> 92 us for the atrium's probe rays with its moved slots, 119 -> 42 us for the
// room's 32,768; any hits 438 -> 360, 163 -> 95 and 102 -> 49 us. Four lanes per ray, two
// children each, measured 1359 us on the bounce: item tests found too few lanes.
#pragma once
#include "sb_traverse.cuh"

namespace sb {

constexpr uint32_t ALL_LANES = 0xFFFFFFFFu;
constexpr uint32_t WALK8_QUEUE = 64;

// One warp's shared memory; the stacks (depth x 32 entries, one column per lane) follow it.
struct Walk8Shared {
    float4 o[32];                  // the lanes' rays: origin; direction, tag
    float4 d[32];
    unsigned long long best[32];   // bits of the ray's limit << 32 | order of its hit in its round
    uint4 hit[32];                 // closest hits: tri, inst, packed (u, v), 0
    uint2 item[WALK8_QUEUE];       // item index, lane of its ray
    uint2 give[32];                // groups on their way to idle lanes; low half of y: donor, lane of its ray
};


// Lanes that wait (for a ray, or for their last items) before a round is made for
// them. 4 to 12 measured within 2% of one another.
constexpr int WALK8_IDLE = 8, WALK8_WAIT = 6;
// With no rays left: lanes without a node before others give them theirs (1 to 8: the
// same), and before fewer than 32 items are tested (12 to 31: 2% on small launches).
constexpr int WALK8_GIVE = 4, WALK8_TAIL = 31;

// Box-test instruction forms of sm_100, each exact: three-input min / max (PTX ISA
// 8.8) and two children's plane distances per packed f32x2 add + fma (PTX ISA 8.6).
__device__ __forceinline__ float max3f(float a, float b, float c) {
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}
__device__ __forceinline__ float min3f(float a, float b, float c) {
    float d;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// Plane distances of bytes b and b + 1 of w: q * s + o for both, where
// s2 = (s, s) and o2 = (o, o). A byte becomes the float 2^23 + q with one permute,
// and q with one subtraction.
__device__ __forceinline__ void q_pair(uint32_t w, uint32_t b, unsigned long long s2, unsigned long long o2, float& t0,
                                       float& t1) {
    const uint32_t a0 = __byte_perm(w, 0x4B000000u, 0x7540u | b);
    const uint32_t a1 = __byte_perm(w, 0x4B000000u, 0x7540u | (b + 1u));
    const unsigned long long bias = 0xCB000000CB000000ull;  // (-2^23, -2^23)
    unsigned long long r;
    asm("{\n\t.reg .b64 a;\n\tmov.b64 a, {%1, %2};\n\tadd.rn.f32x2 a, a, %3;\n\tfma.rn.f32x2 %0, a, %4, %5;\n\t}"
        : "=l"(r)
        : "r"(a0), "r"(a1), "l"(bias), "l"(s2), "l"(o2));
    asm("mov.b64 {%0, %1}, %2;" : "=f"(t0), "=f"(t1) : "l"(r));
}

// A hit's barycentrics in 16 bits each, as the hit records hold them.
__device__ __forceinline__ uint32_t pack_uv(float u, float v) {
    return (uint32_t)__float2uint_rn(clampf(u, 0.f, 1.f) * 65535.0f) |
           (uint32_t)__float2uint_rn(clampf(v, 0.f, 1.f) * 65535.0f) << 16;
}

// Tables of a CTA, ahead of its warps' shared memory: for an octant and a mask of
// slots the bits 7 - (slot XOR octant), so that taking the highest first visits
// them roughly near to far; and for a mask of slots its item bits.
struct alignas(16) Walk8Tables {
    uint8_t order[8][256];
    uint32_t items[256];
};
constexpr Walk8Tables make_walk8_tables() {
    Walk8Tables T{};
    for (uint32_t i = 0; i < 256u; ++i)
        for (uint32_t s = 0; s < 8u; ++s) {
            if (!(i >> s & 1u)) continue;
            for (uint32_t oct = 0; oct < 8u; ++oct) T.order[oct][i] |= (uint8_t)(1u << (7u - (s ^ oct)));
            T.items[i] |= 7u << (3u * s);
        }
    return T;
}
static __device__ const Walk8Tables kWalk8Tables = make_walk8_tables();
__device__ __forceinline__ void walk8_tables(Walk8Tables& T) {
    for (uint32_t i = threadIdx.x; i < sizeof(Walk8Tables) / 16u; i += blockDim.x)
        reinterpret_cast<uint4*>(&T)[i] = __ldg(reinterpret_cast<const uint4*>(&kWalk8Tables) + i);
    __syncthreads();
}

// The slots of the hit children of a node (nearer than tmax).
__device__ __forceinline__ uint32_t walk8_visit(const uint4& h0, uint32_t scaleZ, const uint4& qa, const uint4& qb,
                                                const uint4& qc, float3 o, float3 inv, uint32_t oct, float tmax) {
    const float sx = __uint_as_float(h0.w << 16) * inv.x, sy = __uint_as_float(h0.w & 0xFFFF0000u) * inv.y,
                sz = __uint_as_float(scaleZ) * inv.z;
    const float ox = (__uint_as_float(h0.x) - o.x) * inv.x;
    const float oy = (__uint_as_float(h0.y) - o.y) * inv.y;
    const float oz = (__uint_as_float(h0.z) - o.z) * inv.z;
    const bool nx = oct & 1u, ny = oct & 2u, nz = oct & 4u;
    const unsigned long long sx2 = pack2(sx, sx), sy2 = pack2(sy, sy), sz2 = pack2(sz, sz);
    const unsigned long long ox2 = pack2(ox, ox), oy2 = pack2(oy, oy), oz2 = pack2(oz, oz);
    uint32_t miss = 0;
#pragma unroll
    for (int k = 1; k >= 0; --k) {  // slots 4 k .. 4 k + 3
        float tnx[4], tny[4], tnz[4], tfx[4], tfy[4], tfz[4];
        const uint32_t lx = k ? qa.y : qa.x, hx = k ? qb.w : qb.z, ly = k ? qa.w : qa.z, hy = k ? qc.y : qc.x,
                       lz = k ? qb.y : qb.x, hz = k ? qc.w : qc.z;
        auto q_quad = [](uint32_t w, unsigned long long s2, unsigned long long o2, float t[4]) {
            q_pair(w, 0u, s2, o2, t[0], t[1]);
            q_pair(w, 2u, s2, o2, t[2], t[3]);
        };
        q_quad(nx ? hx : lx, sx2, ox2, tnx);
        q_quad(ny ? hy : ly, sy2, oy2, tny);
        q_quad(nz ? hz : lz, sz2, oz2, tnz);
        q_quad(nx ? lx : hx, sx2, ox2, tfx);
        q_quad(ny ? ly : hy, sy2, oy2, tfy);
        q_quad(nz ? lz : hz, sz2, oz2, tfz);
#pragma unroll
        for (int s = 3; s >= 0; --s) {
            const float tNear = max3f(tnx[s], tny[s], tnz[s]), tFar = min3f(tfx[s], tfy[s], tfz[s]);
            // missed: tFar < tNear, tFar < 0 or tNear >= tmax, by sign bits
            const uint32_t m = __float_as_uint(tFar - tNear) | __float_as_uint(tFar) | ~__float_as_uint(tNear - tmax);
            miss = __funnelshift_l(m, miss, 1);
        }
    }
    return ~miss & 0xFFu;
}

// The walks of a persistent warp. gen (all lanes call it): gives each lane that
// asks for one a new ray (origin, direction, inverse direction, tmax, tag and,
// closest, the best hit ahead of the tree) and returns whether it got one; `more`
// turns false when there are none left. fin (in the lane of an ended walk): tag,
// limit, best hit, blocked.
//
// When no rays are left, the lanes share those in hand. A few rays make ten times
// the average's visits, and a launch lasted as long as they did in one lane each: of the
// 79 us of 210,912 closest-hit walks the last rays were taken after 28. So a lane that
// has no node takes another's lowest stacked group, or what is in its group beside the
// child in turn, with the ray (`home`: the lane that holds its limit and its hit), and
// the rays are written when the warp has ended. The order in which a ray's items are
// met is then no longer that of one walk, which matters only between items of equal t:
// where a tie for the nearest shows up, the ray is walked again by itself, up to that t.
// Measured (primary, shadow): the room's 32,768 rays and 95,728 jobs 59 -> 42, 67 -> 49
// us; the atrium's 113 -> 98, 112 -> 98; four batched fields 136 -> 116, 139 -> 128; a
// diffuse bounce with shadow rays of 9,216 rays 84 -> 73 us, 921,600 473 -> 444, 2.07M
// 966 -> 932 (the first figures with the sharing at 64 registers, where it spills).
template <bool ANY, class Gen, class Fin>
__device__ __forceinline__ void walk8(const DevScene& S, const Walk8Tables& T, Walk8Shared& sm, uint2* stk,
                                      uint32_t depth, Gen gen, Fin fin, Visits& vis, uint32_t* err) {
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    stk += lane;
    vis.inst -= vis.tri;  // every item test of this walk reads its instance's rows: with the end, one each
    enum : uint32_t { FREE, WALK, ENDED };  // ENDED: no node left, items perhaps
    uint32_t state = FREE;
    float3 o = mk(0.f, 0.f, 0.f), inv = o;
    float tmax = 0.0f;
    uint32_t oct = 0, gBase = 0, gBits = 0, sp = 0, iter = 0;
    uint32_t last = 0;              // queue position after this ray's last item
    uint32_t head = 0, tail = 0;    // the queue: items tested, items queued
    uint32_t home = lane;           // the lane whose ray this one walks
    uint32_t base = 0;              // the stack's lowest entry (those below were given away)
    bool more = true, own = false;  // own: this lane's ray is not written yet
    bool share = S.iterCap >= SB_WALK_STEPS_DEFAULT;  // (a lower step limit is meant for one lane's walk)
    uint32_t ties = 0;
    auto root = [&]() {
        gBase = 0;  // the root alone: node 0
        gBits = 1u << (31u ^ oct) | 1u << 16;
        sp = base = 0;
        home = lane;
        state = WALK;
    };
    auto aim = [&](float3 winv) {
        inv = mk(fminf(fmaxf(winv.x, -1e30f), 1e30f), fminf(fmaxf(winv.y, -1e30f), 1e30f),
                 fminf(fmaxf(winv.z, -1e30f), 1e30f));
        oct = (inv.x < 0.0f ? 1u : 0u) | (inv.y < 0.0f ? 2u : 0u) | (inv.z < 0.0f ? 4u : 0u);
    };
    for (;;) {
        if (more) {
            // ended walks whose items are all tested are written and their lanes take new
            // rays, several at a time
            const bool done = state == FREE || (state == ENDED && (int32_t)(last - head) <= 0);
            const uint32_t idle = __ballot_sync(ALL_LANES, done);
            if (__popc(idle) >= WALK8_IDLE || !__any_sync(ALL_LANES, state == WALK)) {
                if (done && own) {
                    const bool blocked = ANY && (uint32_t)sm.best[lane] == 0u;
                    fin(__float_as_uint(sm.d[lane].w), tmax, ANY ? make_uint4(0u, 0u, 0u, 0u) : sm.hit[lane], blocked);
                    vis.blas += 8u * iter;  // box tests
                    iter = 0;
                    state = FREE;
                    own = false;
                }
                if (idle) {
                    float3 d, winv;
                    uint32_t tag;
                    uint4 hit;
                    if (gen(more, idle, o, d, winv, tmax, tag, hit)) {
                        aim(winv);
                        sm.o[lane] = make_float4(o.x, o.y, o.z, 0.0f);
                        sm.d[lane] = make_float4(d.x, d.y, d.z, __uint_as_float(tag));
                        sm.best[lane] = (unsigned long long)__float_as_uint(tmax) << 32 | 0xFFFFFFFFull;
                        if (!ANY) sm.hit[lane] = hit;
                        root();
                        last = head;
                        own = true;
                    }
                    __syncwarp();
                }
            }
        } else {
            const uint32_t walking = __ballot_sync(ALL_LANES, state == WALK);
            if (!walking && tail == head) {
                if (ties == 0u) break;
                // (see below) these rays again, in order, up to the t found
                if (own && ties >> lane & 1u) {
                    const unsigned long long b = sm.best[lane];
                    o = xyz(sm.o[lane]);
                    const float4 d = sm.d[lane];
                    aim(mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z));
                    tmax = __uint_as_float((uint32_t)(b >> 32) + 1u);
                    sm.best[lane] = (unsigned long long)__float_as_uint(tmax) << 32 | 0xFFFFFFFFull;
                    sm.o[lane].w = 1.0f;
                    root();
                }
                share = false;
                ties = 0u;
                __syncwarp();
            } else if (share && __popc(~walking) >= WALK8_GIVE) {
                // no rays are left to take: lanes without a node take what waits in others
                const bool spare = state == WALK && (sp > base || __popc(gBits >> 24) > 1);
                const uint32_t donors = __ballot_sync(ALL_LANES, spare);
                if (donors) {
                    const uint32_t n = min(__popc(donors), __popc(~walking)), r = __popc(donors & below);
                    if (spare && r < n) {
                        uint2 e = make_uint2(gBase, 0u);
                        if (sp > base) {
                            e = stk[base * 32u];
                            ++base;
                        } else {  // all of the group but the child in turn
                            const uint32_t next = 1u << (31u - __clz(gBits));
                            e.y = gBits ^ next;
                            gBits = (gBits & 0x00FFFFFFu) | next;
                        }
                        sm.give[r] = make_uint2(e.x, e.y | lane << 8 | home);
                    }
                    __syncwarp();
                    const uint32_t q = __popc(~walking & below);
                    const bool take = state != WALK && q < n;
                    const uint2 e = take ? sm.give[q] : make_uint2(gBase, gBits | lane << 8 | home);
                    const uint32_t from = e.y >> 8 & 31u;
                    o.x = __shfl_sync(ALL_LANES, o.x, from);
                    o.y = __shfl_sync(ALL_LANES, o.y, from);
                    o.z = __shfl_sync(ALL_LANES, o.z, from);
                    inv.x = __shfl_sync(ALL_LANES, inv.x, from);
                    inv.y = __shfl_sync(ALL_LANES, inv.y, from);
                    inv.z = __shfl_sync(ALL_LANES, inv.z, from);
                    oct = __shfl_sync(ALL_LANES, oct, from);
                    tmax = __shfl_sync(ALL_LANES, tmax, from);
                    if (take) {
                        gBase = e.x;
                        gBits = e.y & 0xFFFF0000u;
                        home = e.y & 31u;
                        sp = base = 0;
                        state = WALK;
                    }
                }
            }
        }
        // one node in every walking lane
        uint32_t tBits = 0, tBase = 0, tMask = 0;
        if (state == WALK) {
            const uint32_t pos = 31u - __clz(gBits);
            gBits ^= 1u << pos;
            const uint32_t before = (1u << (16u + (pos ^ 31u ^ oct))) - 0x10000u;  // interior slots ahead of it
            const uint4* p = S.wideNodes + 5u * (gBase + __popc(gBits & before));
            const uint4 h0 = __ldg(p), h1 = __ldg(p + 1), qa = __ldg(p + 2), qb = __ldg(p + 3), qc = __ldg(p + 4);
            const uint32_t hits = walk8_visit(h0, h1.w, qa, qb, qc, o, inv, oct, tmax);
            const uint32_t ih = hits & h1.z >> 24;
            tMask = h1.z & 0x00FFFFFFu;
            tBits = T.items[hits] & tMask;
            tBase = h1.y;
            // the hit children become the group in hand; what is left of the last one waits
            const bool rest = gBits >= 1u << 24;
            if (ih && rest) stk[min(sp, depth - 1u) * 32u] = make_uint2(gBase, gBits);
            sp += ih && rest ? 1u : 0u;
            const bool pop = !ih && !rest && sp > base;
            sp -= pop ? 1u : 0u;
            const uint2 e = pop ? stk[sp * 32u] : make_uint2(gBase, gBits);
            const uint32_t order = T.order[oct][ih];
            gBase = ih ? h1.x : e.x;
            gBits = ih ? __byte_perm(h1.z, order, 0x4377u) : e.y;  // order << 24 | interior mask << 16
            ++iter;
            if (iter > S.iterCap || sp > depth) {
                latch(err, sp > depth ? ERR_CAPACITY : ERR_WATCHDOG);  // (one entry per level: sp stays within)
                gBits = 0;
            }
            if (gBits < 1u << 24) state = ENDED;
        }
        // its items to the queue: positions from the counts' bits, or one per lane and
        // pass where they do not fit
        const uint32_t cnt = __popc(tBits);
        const uint32_t c0 = __ballot_sync(ALL_LANES, cnt & 1u), c1 = __ballot_sync(ALL_LANES, cnt & 2u),
                       c2 = __ballot_sync(ALL_LANES, cnt & 4u), c3 = __ballot_sync(ALL_LANES, cnt >= 8u);
        bool fits = false;
        {
            const uint32_t sum = __popc(c0) + 2u * __popc(c1) + 4u * __popc(c2);
            fits = !c3 && tail - head + sum <= WALK8_QUEUE;
            if (fits) {
                uint32_t at = tail + __popc(c0 & below) + 2u * __popc(c1 & below) + 4u * __popc(c2 & below);
                if (tBits) {
                    last = at + cnt;
                    do {
                        const uint32_t b = __ffs(tBits) - 1u;
                        sm.item[at % WALK8_QUEUE] = make_uint2(tBase + __popc(tMask & ((1u << b) - 1u)), home);
                        tBits &= tBits - 1u;
                        ++at;
                    } while (tBits);
                }
                tail += sum;
            }
        }
        // a round of tests when 32 have gathered, or when lanes wait for theirs
        for (;;) {
            const uint32_t has = fits ? 0u : __ballot_sync(ALL_LANES, tBits != 0u);
            if (has && tail - head < 32u) {
                if (tBits) {
                    const uint32_t b = __ffs(tBits) - 1u, at = tail + __popc(has & below);
                    tBits &= tBits - 1u;
                    sm.item[at % WALK8_QUEUE] = make_uint2(tBase + __popc(tMask & ((1u << b) - 1u)), home);
                    last = at + 1u;
                }
                tail += __popc(has);
                continue;
            }
            if (tail - head < 32u) {
                if (tail == head) break;
                const uint32_t wait =
                    __ballot_sync(ALL_LANES, more ? state == ENDED && (int32_t)(last - head) > 0 : state != WALK);
                if (__popc(wait) < (more ? WALK8_WAIT : WALK8_TAIL) && (!wait || __any_sync(ALL_LANES, state == WALK))) break;
            }
            __syncwarp();
            const uint32_t n = min(32u, tail - head);
            bool ok = false;
            float t = 0.0f, u, v;
            bool tie = false;  // (as near as the hit in hand)
            uint2 e = make_uint2(0u, 0u), it = e;
            if (lane < n) {
                e = sm.item[(head + lane) % WALK8_QUEUE];
                it = __ldg(S.wideItems + e.x);
                const float4 r0 = __ldg(S.inst + 4 * it.y), r1 = __ldg(S.inst + 4 * it.y + 1),
                             r2 = __ldg(S.inst + 4 * it.y + 2);
                const float dSign = __ldg(&S.inst[4 * it.y + 3].z);
                const bool skip = __ldg(S.slotSkip + it.y) != 0;
                const float3 ro = xyz(sm.o[e.y]), rd = xyz(sm.d[e.y]);
                const float limit = __uint_as_float((uint32_t)(sm.best[e.y] >> 32));
                const float3 lro = mk(dot3(xyz(r0), ro) + r0.w, dot3(xyz(r1), ro) + r1.w, dot3(xyz(r2), ro) + r2.w);
                const float3 lrd = mk(dot3(xyz(r0), rd), dot3(xyz(r1), rd), dot3(xyz(r2), rd));
                float det;
                uint32_t hb;
                const float upTo = ANY || more ? limit : __uint_as_float(__float_as_uint(limit) + 1u);
                ok = tri_hit(S, it.x, lro, lrd, upTo, t, det, u, v, hb) && !skip &&
                     (hb & (ANY ? TB_SHADOW_OK : TB_CLOSEST_OK)) && side_ok(hb, det * dSign);
                tie = ok;
                ok = ok && t < limit;
                ++vis.tri;
            }
            if (__any_sync(ALL_LANES, ok || tie)) {
                const unsigned long long mine = ANY ? 0ull : (unsigned long long)__float_as_uint(t) << 32 | lane;
                if (ok) {
                    if (ANY) sm.best[e.y] = 0ull;  // blocked
                    else atomicMin(&sm.best[e.y], mine);
                }
                __syncwarp();
                if (!ANY && ok && sm.best[e.y] == mine) sm.hit[e.y] = make_uint4(it.x, it.y, pack_uv(u, v), 0u);
                if (!ANY && share && !more) {
                    const unsigned long long b = sm.best[e.y];
                    tie = tie && (uint32_t)(b >> 32) == __float_as_uint(t) && !(ok && b == mine) && (uint32_t)b != 0xFFFFFFFFu;
                    ties |= __reduce_or_sync(ALL_LANES, tie ? 1u << e.y : 0u);
                }
                __syncwarp();
                if (state != FREE) {
                    const unsigned long long b = sm.best[home];
                    if (!ANY) tmax = __uint_as_float((uint32_t)(b >> 32));
                    else if ((uint32_t)b == 0u) state = ENDED;
                }
            }
            head += n;
        }
    }
    if (own) {
        const unsigned long long b = sm.best[lane];
        // (a second walk that found nothing: the first one's hit stands)
        const uint32_t t = (uint32_t)(b >> 32) - (sm.o[lane].w != 0.0f && (uint32_t)b == 0xFFFFFFFFu ? 1u : 0u);
        fin(__float_as_uint(sm.d[lane].w), __uint_as_float(t), ANY ? make_uint4(0u, 0u, 0u, 0u) : sm.hit[lane],
            ANY && (uint32_t)b == 0u);
    }
    vis.blas += 8u * iter;
    vis.inst += vis.tri;  // (see the start)
}

}  // namespace sb
