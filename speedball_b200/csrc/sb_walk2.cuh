// sb_walk2.cuh — the moved and deformed instance slots of a ray (DevScene's
// dynList), walked by a persistent warp: per slot its world bounds (the reference's TLAS leaf test), then its BLAS as the child-pair
// nodes the refits keep current, near child first.
//
// One thread that walks its ray's slots alone makes a chain of some hundred
// dependent loads, and the few rays that graze a dense mesh set the kernel's end
// while the chip is idle. So the triangles of the leaves a ray hits go to a queue
// and are tested by 32 lanes at once, two leaves hit in one step are opened
// together, and lanes whose rays meet no slot take new rays (as in sb_walk8.cuh).
// The results meet the scene-BVH walk's only in the next stage, so a warp that has
// no rays left here goes on with that walk while others finish theirs. Its last rays
// its lanes share, as in walk8: one that grazes a dense mesh in each of its slots had
// kept its warp here to the end of the launch. The atrium's three movers and one
// deformer cost 99 + 72 us in kernels of one thread per ray (two rays in three meet
// none of them), 72 + 63 us in such kernels of this walk, and 21 + 21 us ahead of the
// tree's walk in the same launch; shared, the launches took 96 -> 92 and 101 -> 95 us,
// of 1,536 probes' rays 66 -> 56 and 57 -> 40.
#pragma once
#include "sb_walk8.cuh"

namespace sb {

constexpr uint32_t WALK2_QUEUE = 256;  // at most 31 waiting, then 4 of every lane a pass
constexpr uint32_t WALK2_DEPTH = 24;   // stacked far children; deeper BLASes: dyn_walk

struct Walk2Shared {
    float4 o[32];                 // local origin, determinant sign
    float4 d[32];                 // local direction, slot
    unsigned long long best[32];  // bits of the ray's limit << 32 | its hit's place in the order
    uint32_t place[32];           // of the slot the ray is in: number in dynList << 24
    uint4 hit[32];                // triangle, slot, packed (u, v), the slack of reach
    uint32_t item[WALK2_QUEUE];   // lane of its ray << 24 | triangle
    uint32_t stk[WALK2_DEPTH][32];  // far children
    uint2 give[32];               // far children on their way to idle lanes; donor, lane of its ray
};

// True when every slot's BLAS can be walked by walk2.
__device__ __forceinline__ bool walk2_usable(const DevScene& S) {
    if (!S.depth || !S.pairs) return false;
    const uint32_t db = __ldg(S.depth);
    return db != DEPTH_UNKNOWN && db <= WALK2_DEPTH;
}

// gen and fin as for walk8; the best hit starts as none within tmax. Of several hits of the
// nearest t it is the first slot's lowest triangle, the one that the reference's order meets
// first: the lanes' items meet in no fixed order, so the place in that order is the low
// half of what they take the minimum of.
//
// Closest hits pass over a box only where it starts behind the hit in hand by more than
// the rounding of both (`reach`). A BLAS's boxes are exact: a triangle in the plane of its
// box starts, by the box, at or a few ulp behind its own t, so with the plain limit a
// triangle as near as the hit in hand is tested or not as the one or the other is met
// first, and the lanes that share a ray meet them in no fixed order (17 to 51 of 12,288
// probe rays at planes of two sizes of triangles named another one than walks that share
// nothing). Moeller-Trumbore's t is off by some 1e-7 of the triangle's size and distance over
// the cosine to its normal: 1e-4 of the limit and of the BLAS's size cover all but rays
// within a milliradian of the plane, and are less than a triangle of the meshes here.
template <bool ANY, class Gen, class Fin>
__device__ __forceinline__ void walk2(const DevScene& S, Walk2Shared& sm, Gen gen, Fin fin, Visits& vis,
                                      uint32_t* err) {
    const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
    enum : uint32_t { FREE, WALK, ENDED };  // ENDED: this slot's nodes are done, items perhaps
    uint32_t state = FREE;
    float3 wo = mk(0.f, 0.f, 0.f), wd = wo, winv = wo, o = wo, inv = wo;
    float tmax = 0.0f, lim = 0.0f;  // lim: reach(tmax)
    uint32_t tag = 0, k = 0, cur = PE_NONE, sp = 0, iter = 0, last = 0, head = 0, tail = 0;
    bool more = true;
    uint32_t home = lane, base = 0;  // as in walk8
    bool own = false;
    const bool share = S.iterCapRef >= SB_WALK_STEPS_REF_DEFAULT;  // as in walk8
    // the lane's ray into its next slot; false: none left
    auto next_slot = [&]() {
        for (; k < S.dynCount; ) {
            const uint32_t slot = __ldg(S.dynList + k++);
            if (S.slotBounds) {
                const float* b = S.slotBounds + 6u * slot;
                const float3 lo = mk(__ldg(b), __ldg(b + 1), __ldg(b + 2)),
                             hi = mk(__ldg(b + 3), __ldg(b + 4), __ldg(b + 5));
                if (!slab(lo, hi, wo, winv, ANY ? tmax : reach(tmax, slot_slack(lo, hi, winv)))) continue;
            }
            ++vis.inst;
            const float4 m = __ldg(S.inst + 4 * slot + 3);
            if (!(m.w > 0.5f)) continue;
            const float4 r0 = __ldg(S.inst + 4 * slot), r1 = __ldg(S.inst + 4 * slot + 1),
                         r2 = __ldg(S.inst + 4 * slot + 2);
            o = mk(dot3(xyz(r0), wo) + r0.w, dot3(xyz(r1), wo) + r1.w, dot3(xyz(r2), wo) + r2.w);
            const float3 d = mk(dot3(xyz(r0), wd), dot3(xyz(r1), wd), dot3(xyz(r2), wd));
            inv = mk(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
            const uint32_t root = __float_as_uint(m.x);
            if (root >= __float_as_uint(m.y) || root >= S.nodeCount) continue;
            const uint4 a = __ldg(S.nodes + 2 * root), b = __ldg(S.nodes + 2 * root + 1);
            ++vis.blas;
            const float3 lo = mk(__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z)),
                         hi = mk(__uint_as_float(a.w), __uint_as_float(b.x), __uint_as_float(b.y));
            const float slack = blas_slack(lo, hi, inv);
            lim = ANY ? tmax : reach(tmax, slack);
            if (!slab(lo, hi, o, inv, lim)) continue;
            if (!ANY) sm.hit[lane].w = __float_as_uint(slack);
            cur = b.w == INTERIOR ? PE_BLAS | root : ((b.w >> 24) ? b.w : PE_NONE);
            if (cur == PE_NONE) continue;
            sm.o[lane] = make_float4(o.x, o.y, o.z, m.z);
            sm.d[lane] = make_float4(d.x, d.y, d.z, __uint_as_float(slot));
            sm.place[lane] = (k - 1u) << 24;
            sp = base = iter = 0;  // (a step limit holds for each slot, as in dyn_walk)
            home = lane;
            last = head;
            state = WALK;
            return true;
        }
        return false;
    };
    for (;;) {
        bool flush = false;
        if (more) {
            const bool done = state == FREE || (state == ENDED && (int32_t)(last - head) <= 0);
            const uint32_t idle = __ballot_sync(ALL_LANES, done);
            if (__popc(idle) >= WALK8_IDLE || !__any_sync(ALL_LANES, state == WALK)) {
                const bool blocked = ANY && done && own && (uint32_t)sm.best[lane] == 0u;
                if (blocked) {
                    fin(tag, tmax, make_uint4(0u, 0u, 0u, 0u), true);
                    own = false;
                }
                const uint32_t want = __ballot_sync(ALL_LANES, done && !own);
                if (want && gen(more, want, wo, wd, winv, tmax, tag)) {
                    sm.best[lane] = (unsigned long long)__float_as_uint(tmax) << 32 | 0xFFFFFFFFull;
                    if (!ANY) sm.hit[lane] = make_uint4(0xFFFFFFFFu, 0xFFFFFFFFu, 0u, 0u);
                    k = 0;
                    own = true;
                }
                if (done) {
                    state = FREE;
                    if (own && !next_slot()) {
                        fin(tag, tmax, ANY ? make_uint4(0u, 0u, 0u, 0u) : sm.hit[lane], false);
                        own = false;
                    }
                }
                __syncwarp();
            }
        } else {
            // no rays are left to take: the lanes share those in hand, as in walk8. A ray goes
            // on to its next slot when no lane is in this one and the queue is empty (its
            // local ray is the lanes' and the items').
            const uint32_t busy = __reduce_or_sync(ALL_LANES, state == WALK ? 1u << home : 0u);
            const bool ready = own && state != WALK && !(busy >> lane & 1u);
            flush = __any_sync(ALL_LANES, ready);
            if (!flush && !busy && tail == head) break;
            if (flush && tail == head) {
                if (ready) {
                    const unsigned long long b = sm.best[lane];
                    const bool blocked = ANY && (uint32_t)b == 0u;
                    tmax = __uint_as_float((uint32_t)(b >> 32));
                    state = FREE;
                    if (blocked || !next_slot()) {
                        fin(tag, tmax, ANY ? make_uint4(0u, 0u, 0u, 0u) : sm.hit[lane], blocked);
                        own = false;
                    }
                }
                __syncwarp();
            }
            // (a lane whose own ray waits for the queue takes nothing)
            const uint32_t walking =
                __ballot_sync(ALL_LANES, state == WALK || (ready && tail != head));
            const bool spare = share && state == WALK && sp > base;
            const uint32_t donors = __popc(~walking) >= WALK8_GIVE ? __ballot_sync(ALL_LANES, spare) : 0u;
            if (donors) {
                const uint32_t n = min(__popc(donors), __popc(~walking)), r = __popc(donors & below);
                if (spare && r < n) sm.give[r] = make_uint2(sm.stk[base++][lane], lane << 8 | home);
                __syncwarp();
                const uint32_t q = __popc(~walking & below);
                const bool take = !(walking >> lane & 1u) && q < n;
                const uint2 e = take ? sm.give[q] : make_uint2(0u, lane << 8);
                const uint32_t from = e.y >> 8;
                o.x = __shfl_sync(ALL_LANES, o.x, from);
                o.y = __shfl_sync(ALL_LANES, o.y, from);
                o.z = __shfl_sync(ALL_LANES, o.z, from);
                inv.x = __shfl_sync(ALL_LANES, inv.x, from);
                inv.y = __shfl_sync(ALL_LANES, inv.y, from);
                inv.z = __shfl_sync(ALL_LANES, inv.z, from);
                lim = __shfl_sync(ALL_LANES, lim, from);
                if (take) {
                    cur = e.x;
                    home = e.y & 31u;
                    sp = base = 0;
                    state = WALK;
                }
            }
        }
        // one node in every walking lane
        uint32_t off0 = 0, n0 = 0, off1 = 0, n1 = 0;  // the hit leaves' triangles, nearer leaf first
        if (state == WALK) {
            if (cur >> 24) {  // a root that is a leaf
                off0 = cur & 0x00FFFFFFu;
                n0 = cur >> 24;
                cur = PE_NONE;
            } else {
                const uint4* p = S.pairs + 4u * (cur & (PE_BLAS - 1u));
                const uint4 q0 = __ldg(p), q1 = __ldg(p + 1), q2 = __ldg(p + 2), q3 = __ldg(p + 3);
                vis.blas += 2;
                float t0 = 0.f, t1 = 0.f;
                const bool h0 = slab_near(__uint_as_float(q0.x), __uint_as_float(q0.z), __uint_as_float(q2.x),
                                          __uint_as_float(q0.y), __uint_as_float(q0.w), __uint_as_float(q2.y), o, inv,
                                          lim, t0) && q3.x != PE_NONE;
                const bool h1 = slab_near(__uint_as_float(q1.x), __uint_as_float(q1.z), __uint_as_float(q2.z),
                                          __uint_as_float(q1.y), __uint_as_float(q1.w), __uint_as_float(q2.w), o, inv,
                                          lim, t1) && q3.y != PE_NONE;
                const bool swap = h0 && h1 && t1 < t0;
                uint32_t a = h0 ? q3.x : PE_NONE, b = h1 ? q3.y : PE_NONE;
                if (swap) {
                    const uint32_t x = a;
                    a = b;
                    b = x;
                }
                cur = PE_NONE;
                if (a != PE_NONE) {
                    if (a >> 24) { off0 = a & 0x00FFFFFFu; n0 = a >> 24; }
                    else cur = a;
                }
                if (b != PE_NONE) {
                    if (b >> 24) { off1 = b & 0x00FFFFFFu; n1 = b >> 24; }
                    else if (cur == PE_NONE) cur = b;
                    else if (sp < WALK2_DEPTH) sm.stk[sp++][lane] = b;
                    else latch(err, ERR_CAPACITY);  // unreachable: walk2_usable bounds the depth
                }
                if (++iter > S.iterCapRef) {
                    latch(err, ERR_WATCHDOG);
                    cur = PE_NONE;
                    sp = base;
                }
            }
            if (cur == PE_NONE && sp > base) cur = sm.stk[--sp][lane];
            if (cur == PE_NONE) state = ENDED;
        }
        // the triangles to the queue, four of each lane a pass, and rounds of tests
        for (;;) {
            const uint32_t mine = min(n0 + n1, 4u);
            const uint32_t c0 = __ballot_sync(ALL_LANES, mine & 1u), c1 = __ballot_sync(ALL_LANES, mine & 2u),
                           c2 = __ballot_sync(ALL_LANES, mine & 4u);
            uint32_t at = tail + __popc(c0 & below) + 2u * __popc(c1 & below) + 4u * __popc(c2 & below);
            for (uint32_t i = 0; i < mine; ++i, ++at) {
                if (!n0) {
                    off0 = off1;
                    n0 = n1;
                    n1 = 0;
                }
                sm.item[at % WALK2_QUEUE] = home << 24 | off0++;
                --n0;
            }
            if (mine) last = at;
            const bool any = (c0 | c1 | c2) != 0u;
            tail += __popc(c0) + 2u * __popc(c1) + 4u * __popc(c2);
            for (;;) {
                if (tail - head < 32u) {
                    if (tail == head) break;
                    if (any) break;  // more may come
                    const uint32_t wait =
                        __ballot_sync(ALL_LANES, more ? state == ENDED && (int32_t)(last - head) > 0 : state != WALK);
                    if (!flush && __popc(wait) < (more ? WALK8_WAIT : WALK8_TAIL) &&
                        (!wait || __any_sync(ALL_LANES, state == WALK)))
                        break;
                }
                __syncwarp();
                const uint32_t n = min(32u, tail - head);
                bool ok = false;
                float t = 0.0f, u, v;
                uint32_t tri = 0, of = 0, slot = 0;  // of: the lane whose ray it is
                unsigned long long key = 0ull;       // (any hits: blocked)
                if (lane < n) {
                    tri = sm.item[(head + lane) % WALK2_QUEUE];
                    of = tri >> 24;
                    tri &= 0x00FFFFFFu;
                    const float4 ro = sm.o[of], rd = sm.d[of];
                    const unsigned long long best = sm.best[of];
                    const uint32_t limit = (uint32_t)(best >> 32);
                    slot = __float_as_uint(rd.w);
                    float det;
                    uint32_t hb;
                    const float upTo = __uint_as_float(ANY ? limit : limit + 1u);  // as near counts too
                    ok = tri_hit(S, tri, xyz(ro), xyz(rd), upTo, t, det, u, v, hb) &&
                         (hb & (ANY ? TB_SHADOW_OK : TB_CLOSEST_OK)) && side_ok(hb, det * ro.w);
                    if (!ANY) {
                        key = (unsigned long long)__float_as_uint(t) << 32 | sm.place[of] | tri;
                        ok = ok && key < best;
                    }
                    ++vis.tri;
                }
                if (__any_sync(ALL_LANES, ok)) {
                    if (ok) {
                        if (ANY) sm.best[of] = 0ull;
                        else atomicMin(&sm.best[of], key);
                    }
                    __syncwarp();
                    if (!ANY && ok && sm.best[of] == key)
                        sm.hit[of] = make_uint4(tri, slot, pack_uv(u, v), sm.hit[of].w);
                    __syncwarp();
                    if (state != FREE) {
                        const unsigned long long b = sm.best[home];
                        if (!ANY) lim = reach(tmax = __uint_as_float((uint32_t)(b >> 32)), __uint_as_float(sm.hit[home].w));
                        else if ((uint32_t)b == 0u) state = ENDED;
                    }
                }
                head += n;
            }
            if (!any) break;
        }
    }
}

}  // namespace sb
