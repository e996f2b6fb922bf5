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
// go through small tables in shared memory. Measured against one walk per lane:
// closest hits 1431 -> 542 us there, 194 -> 118 us for the atrium's probe rays with
// its moved slots, 119 -> 61 us for the room's 32,768; any hits (which had a binary
// tree) 438 -> 362, 163 -> 110 and 102 -> 66 us. Four lanes per ray, two children
// each, measured 1359 us on the bounce: item tests found too few lanes.
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
};


// Lanes that wait (for a ray, or for their last items) before a round is made for
// them. 4 to 12 measured within 2% of one another.
constexpr int WALK8_IDLE = 8, WALK8_WAIT = 6;

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

__device__ __forceinline__ unsigned long long pack2(float lo, float hi) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
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
struct Walk8Tables {
    uint8_t order[8][256];
    uint32_t items[256];
};
__device__ __forceinline__ void walk8_tables(Walk8Tables& T) {
    for (uint32_t i = threadIdx.x; i < 8u * 256u; i += blockDim.x) {
        const uint32_t oct = i >> 8;
        uint32_t r = 0;
        for (uint32_t s = 0; s < 8; ++s) r |= (i >> s & 1u) << (7u - (s ^ oct));
        T.order[oct][i & 255u] = (uint8_t)r;
    }
    for (uint32_t i = threadIdx.x; i < 256u; i += blockDim.x) {
        uint32_t r = 0;
        for (uint32_t s = 0; s < 8; ++s) r |= (i >> s & 1u) * (7u << (3u * s));
        T.items[i] = r;
    }
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
template <bool ANY, class Gen, class Fin>
__device__ __forceinline__ void walk8(const DevScene& S, const Walk8Tables& T, Walk8Shared& sm, uint2* stk,
                                      uint32_t depth, Gen gen, Fin fin, Visits& vis, uint32_t* err) {
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    stk += lane;
    enum : uint32_t { FREE, WALK, ENDED };  // ENDED: no node left, items perhaps
    uint32_t state = FREE;
    float3 o = mk(0.f, 0.f, 0.f), inv = o;
    float tmax = 0.0f;
    uint32_t oct = 0, gBase = 0, gBits = 0, sp = 0, iter = 0;
    uint32_t last = 0;              // queue position after this ray's last item
    uint32_t head = 0, tail = 0;    // the queue: items tested, items queued
    bool more = true;
    for (;;) {
        // ended walks whose items are all tested are written and their lanes take new
        // rays, several at a time
        const bool done = state == FREE || (state == ENDED && (int32_t)(last - head) <= 0);
        const uint32_t idle = __ballot_sync(ALL_LANES, done);
        if (__popc(idle) >= WALK8_IDLE || !__any_sync(ALL_LANES, state == WALK)) {
            if (done && state == ENDED) {
                const bool blocked = ANY && (uint32_t)sm.best[lane] == 0u;
                fin(__float_as_uint(sm.d[lane].w), tmax, ANY ? make_uint4(0u, 0u, 0u, 0u) : sm.hit[lane], blocked);
                vis.blas += 8u * iter;  // box tests
                state = FREE;
            }
            if (more && idle) {
                float3 d, winv;
                uint32_t tag;
                uint4 hit;
                if (gen(more, idle, o, d, winv, tmax, tag, hit)) {
                    inv = mk(fminf(fmaxf(winv.x, -1e30f), 1e30f), fminf(fmaxf(winv.y, -1e30f), 1e30f),
                             fminf(fmaxf(winv.z, -1e30f), 1e30f));
                    oct = (inv.x < 0.0f ? 1u : 0u) | (inv.y < 0.0f ? 2u : 0u) | (inv.z < 0.0f ? 4u : 0u);
                    sm.o[lane] = make_float4(o.x, o.y, o.z, 0.0f);
                    sm.d[lane] = make_float4(d.x, d.y, d.z, __uint_as_float(tag));
                    sm.best[lane] = (unsigned long long)__float_as_uint(tmax) << 32 | 0xFFFFFFFFull;
                    if (!ANY) sm.hit[lane] = hit;
                    gBase = 0;  // the root alone: node 0
                    gBits = 1u << (31u ^ oct) | 1u << 16;
                    sp = iter = 0;
                    last = head;
                    state = WALK;
                }
                __syncwarp();
            } else if (idle == ALL_LANES) {
                break;
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
            const bool pop = !ih && !rest && sp;
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
                        sm.item[at % WALK8_QUEUE] = make_uint2(tBase + __popc(tMask & ((1u << b) - 1u)), lane);
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
                    sm.item[at % WALK8_QUEUE] = make_uint2(tBase + __popc(tMask & ((1u << b) - 1u)), lane);
                    last = at + 1u;
                }
                tail += __popc(has);
                continue;
            }
            if (tail - head < 32u) {
                if (tail == head) break;
                const uint32_t wait = __ballot_sync(ALL_LANES, state == ENDED && (int32_t)(last - head) > 0);
                if (__popc(wait) < WALK8_WAIT && (!wait || __any_sync(ALL_LANES, state == WALK))) break;
            }
            __syncwarp();
            const uint32_t n = min(32u, tail - head);
            bool ok = false;
            float t, u, v;
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
                ok = tri_hit(S, it.x, lro, lrd, limit, t, det, u, v, hb) && !skip &&
                     (hb & (ANY ? TB_SHADOW_OK : TB_CLOSEST_OK)) && side_ok(hb, det * dSign);
                ++vis.tri;
            }
            if (__any_sync(ALL_LANES, ok)) {
                const unsigned long long mine = ANY ? 0ull : (unsigned long long)__float_as_uint(t) << 32 | lane;
                if (ok) {
                    if (ANY) sm.best[e.y] = 0ull;  // blocked
                    else atomicMin(&sm.best[e.y], mine);
                }
                __syncwarp();
                if (!ANY && ok && sm.best[e.y] == mine) sm.hit[e.y] = make_uint4(it.x, it.y, pack_uv(u, v), 0u);
                __syncwarp();
                if (state != FREE) {
                    const unsigned long long b = sm.best[lane];
                    if (!ANY) tmax = __uint_as_float((uint32_t)(b >> 32));
                    else if ((uint32_t)b == 0u) state = ENDED;
                }
            }
            head += n;
        }
    }
    vis.inst += vis.tri;
}

}  // namespace sb
