// sb_build.cu — BLAS build on the GPU in the reference's threaded layout.
//
// The reference builds each BLAS on the CPU with three-mesh-bvh
// (spectral_scene.js:898-966, ~200 ms for a large mesh, the cost its refit
// lane exists to avoid, gi_refit.js:7-8) and re-flattens it into 8 x u32
// nodes (flattenBVHRoot, 658-721). This builder is a linear BVH (Karras,
// "Maximizing Parallelism in the Construction of BVHs, Octrees, and k-d
// Trees", HPG 2012) emitting that layout directly:
//   1. per triangle the centre of its vertex bounds; the bounds of the centres;
//   2. a 30-bit Morton code of each centre within those;
//   3. a stable LSD radix sort of (code, triangle), 3 passes of 10 bits, with
//      warp-level ranking (match.any) so equal digits keep their order;
//   4. the binary radix tree over the sorted codes, equal codes ordered by
//      position (Karras' tie rule). It is the Cartesian tree of the common prefix
//      lengths of neighbours: the node that splits between g and g + 1 reaches to
//      the next shorter prefix on either side, which masks of 32 prefix bytes and
//      the minima of 32, 1024, ... of them find in a few steps. A node of more than
//      `leafSize` triangles is an interior node of the output; a child of one with
//      at most that many is an output leaf;
//   5. the output places without a climb: the tree below a node of K output leaves
//      has 2 K - 1 nodes, and in pre-order a node comes after every output leaf and
//      interior node that starts left of it and after its ancestors that start with
//      it. So prefix sums over the positions, of leaves and of interior nodes by
//      their first position, give every node its index and its miss link;
//   6. the bounds: an output leaf's as the refit computes them (its triangles in
//      order, strict < and >); an interior node's as the minimum and maximum of its
//      range of output leaves, one warp per node, from the leaves' boxes and those
//      of 32, 1024, ... positions. (The refit's unions order -0 below +0 and no
//      leaf's bound is a NaN, so they are the minima and maxima of order-preserving
//      integers, which the warp reduces in hardware.)
// The output triangle order is the sorted order (triangle at each position).
//
// What bounds it is the chain of dependent phases, not their work: a mesh of a few
// thousand triangles fills a few SMs. Up to BUILD_CLUSTER_TRIS triangles one launch
// of a thread-block cluster of at most 8 CTAs runs all phases with hardware cluster
// barriers between them; above that each phase is a launch over more SMs, placed
// ahead of the end of the one before it (at 20,000 triangles 98 us by a cluster,
// 69 us by launches; at 8,192 54 us by a cluster, at 10,000 67 us by launches). No loop waits on another thread; every
// walk is bounded by the tree depth (at most 64 levels: each adds a bit of the
// 62-bit key + position). A build of 1,024 / 8,192 / 65,537 / 600,000 triangles
// takes 36 / 54 / 76 / 203 us; as 19 launches and copies with a bottom-up climb
// over arrival counters (41 us on a mesh of 9k by itself) and a scan by one CTA it
// took 142 / 168 / 195 / 627 us.
#include <cooperative_groups.h>

#include <algorithm>
#include <cstddef>
#include <type_traits>

#include "sb_kernels.cuh"

namespace sb {

namespace {

constexpr uint32_t kThreads = 1024;             // of every CTA
constexpr uint32_t kWarps = kThreads / 32;
constexpr uint32_t kBits = 10, kDigits = 1u << kBits;
constexpr uint32_t kSortCtas = 148;             // of a sort pass: each reads the others' digit counts
constexpr uint32_t kMaxCtas = 1024;             // of the other phases
constexpr uint32_t BUILD_CLUSTER_TRIS = 8192;   // at most this many by one cluster

__device__ __forceinline__ uint32_t f2o(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float o2f(uint32_t u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

__device__ __forceinline__ uint32_t expand10(uint32_t v) {
    v &= 0x3FFu;
    v = (v | (v << 16)) & 0x030000FFu;
    v = (v | (v << 8)) & 0x0300F00Fu;
    v = (v | (v << 4)) & 0x030C30C3u;
    v = (v | (v << 2)) & 0x09249249u;
    return v;
}

// One build's inputs, scratch and outputs.
struct Build {
    const float* pos;
    const uint32_t* idx;
    uint32_t V, T, leafSize, chunk;  // chunk: positions per CTA and phase, a multiple of kThreads
    uint32_t levels;                 // prefix and box levels above the positions (32 per step)
    float4* centre;                  // T
    uint32_t* part;                  // per CTA 8: centre bounds; then leaf and node sums
    uint32_t *keyA, *keyB, *valA;    // T each; the sorted triangles lie in `order`
    uint32_t* hist;                  // per CTA of a sort pass kDigits
    uint8_t* prefix;                 // per position and level: common prefix with the next, minima above
    uint32_t *first, *last;          // T: range of the interior node of the output that splits after a position
    uint32_t *starts, *leafCount;    // T: interior nodes that start here; triangles of the output leaf that does
    uint2* before;                   // T + 1: output leaves, and all output nodes, that start left of a position
    uint4 *boxLo, *boxHi;            // per position and level: box of 32^level positions' output leaves (f2o)
    uint32_t levelAt[6];             // offset of each level in them and in prefix (a multiple of 32)
    uint32_t *order, *nodes, *nodeCount;
    uint32_t* err;
};

struct BuildShared {
    uint2 sum2[kWarps];
    uint32_t sum[kWarps];
    uint32_t box[6];
    uint32_t lo[kWarps][3], hi[kWarps][3];
    union {
        float tri[6][kThreads];            // bounds of the triangles of a tile
        uint32_t far[kThreads + 1];        // splits of a tile whose range leaves their 32; their number
    } u;
    uint32_t cnt[kWarps][kDigits];         // a sort pass' digits per warp (launches of other phases end above)
};

__device__ __forceinline__ uint32_t warp_scan(uint32_t v) {  // inclusive
    const uint32_t lane = threadIdx.x & 31u;
#pragma unroll
    for (int s = 1; s < 32; s <<= 1) {
        const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, v, s);
        if (lane >= (uint32_t)s) v += y;
    }
    return v;
}
// Exclusive scan over the CTA's threads; `total` of all. Synchronizes.
__device__ __forceinline__ uint32_t block_scan(uint32_t v, uint32_t* tmp, uint32_t& total) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5, x = warp_scan(v);
    if (lane == 31) tmp[w] = x;
    __syncthreads();
    const uint32_t sums = warp_scan(tmp[lane]);
    total = __shfl_sync(0xFFFFFFFFu, sums, 31);
    const uint32_t ahead = __shfl_sync(0xFFFFFFFFu, sums, (w + 31u) & 31u);
    __syncthreads();
    return (w ? ahead : 0u) + x - v;
}

// 1. centres (source order) and this CTA's part of their bounds
__device__ __forceinline__ void build_centres(const Build& B, BuildShared& sm, uint32_t cta, uint32_t ctas) {
    if (threadIdx.x < 6) sm.box[threadIdx.x] = threadIdx.x < 3 ? 0xFFFFFFFFu : 0u;
    __syncthreads();
    uint32_t omn[3] = {0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, omx[3] = {0u, 0u, 0u};
    for (uint32_t t = cta * kThreads + threadIdx.x; t < B.T; t += ctas * kThreads) {
        const uint32_t id[3] = {B.idx[3 * (size_t)t], B.idx[3 * (size_t)t + 1], B.idx[3 * (size_t)t + 2]};
        float c[3] = {0.f, 0.f, 0.f};
        if (id[0] < B.V && id[1] < B.V && id[2] < B.V) {
            float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
            for (int k = 0; k < 3; ++k)
                for (int a = 0; a < 3; ++a) {
                    const float v = B.pos[3 * (size_t)id[k] + a];
                    if (v < mn[a]) mn[a] = v;
                    if (v > mx[a]) mx[a] = v;
                }
            for (int a = 0; a < 3; ++a) c[a] = mn[a] + (mx[a] - mn[a]) * 0.5f;
            if (isfinite(c[0]) && isfinite(c[1]) && isfinite(c[2]))
                for (int a = 0; a < 3; ++a) {
                    omn[a] = min(omn[a], f2o(c[a]));
                    omx[a] = max(omx[a], f2o(c[a]));
                }
        } else {
            latch(B.err, ERR_LAYOUT);
        }
        B.centre[t] = make_float4(c[0], c[1], c[2], 0.0f);
    }
    for (int a = 0; a < 3; ++a) {
        const uint32_t mn = __reduce_min_sync(0xFFFFFFFFu, omn[a]), mx = __reduce_max_sync(0xFFFFFFFFu, omx[a]);
        if ((threadIdx.x & 31u) == 0) {
            atomicMin(&sm.box[a], mn);
            atomicMax(&sm.box[3 + a], mx);
        }
    }
    __syncthreads();
    if (threadIdx.x < 6) B.part[cta * 8u + threadIdx.x] = sm.box[threadIdx.x];
}

// 2. Morton codes; the tree's counters cleared
__device__ __forceinline__ void build_codes(const Build& B, BuildShared& sm, uint32_t cta, uint32_t ctas) {
    if (threadIdx.x < 32) {
        for (uint32_t a = 0; a < 6; ++a) {
            uint32_t v = a < 3 ? 0xFFFFFFFFu : 0u;
            for (uint32_t c = threadIdx.x; c < ctas; c += 32) {
                const uint32_t x = B.part[c * 8u + a];
                v = a < 3 ? min(v, x) : max(v, x);
            }
            v = a < 3 ? __reduce_min_sync(0xFFFFFFFFu, v) : __reduce_max_sync(0xFFFFFFFFu, v);
            if (threadIdx.x == 0) sm.box[a] = v;
        }
    }
    __syncthreads();
    const uint32_t end = min(B.T, (cta + 1u) * B.chunk);
    for (uint32_t t = cta * B.chunk + threadIdx.x; t < end; t += kThreads) {
        const float4 c4 = B.centre[t];
        const float c[3] = {c4.x, c4.y, c4.z};
        uint32_t q[3];
        for (int a = 0; a < 3; ++a) {
            const float mn = o2f(sm.box[a]), mx = o2f(sm.box[3 + a]);
            const float ext = mx - mn;
            float x = ext > 0.0f ? (c[a] - mn) / ext : 0.0f;
            x = isfinite(x) ? fminf(fmaxf(x, 0.0f), 1.0f) : 0.0f;
            q[a] = min((uint32_t)(x * 1024.0f), 1023u);
        }
        B.keyA[t] = (expand10(q[0]) << 2) | (expand10(q[1]) << 1) | expand10(q[2]);
        B.starts[t] = 0u;
        B.leafCount[t] = 0u;
    }
}

// 3. stable LSD radix sort, one digit per pass: the digits of this CTA's chunk per
// warp (each warp a contiguous part) and their sums, then, with all CTAs' sums
// written, the keys and triangles to their places. Pass 0 reads triangle t at t.
__device__ __forceinline__ uint32_t warp_part(const Build& B) { return B.chunk / kWarps; }  // a multiple of 32

__device__ __forceinline__ void build_count(const Build& B, BuildShared& sm, uint32_t cta, const uint32_t* keys,
                                            uint32_t shift) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    for (uint32_t d = lane; d < kDigits; d += 32) sm.cnt[w][d] = 0u;
    __syncwarp();
    const uint32_t from = cta * B.chunk + w * warp_part(B), to = min(B.T, from + warp_part(B));
    for (uint32_t p = from; p < to; p += 32) {
        const bool valid = p + lane < to;
        const uint32_t digit = valid ? keys[p + lane] >> shift & (kDigits - 1u) : kDigits;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, digit);
        if (valid && lane == (uint32_t)(__ffs(peers) - 1)) sm.cnt[w][digit] += __popc(peers);
        __syncwarp();
    }
    __syncthreads();
    uint32_t n = 0;
    for (uint32_t x = 0; x < kWarps; ++x) n += sm.cnt[x][threadIdx.x];
    B.hist[cta * kDigits + threadIdx.x] = n;
}

__device__ __forceinline__ void build_place(const Build& B, BuildShared& sm, uint32_t cta, uint32_t ctas,
                                            const uint32_t* keys, const uint32_t* vals, uint32_t shift,
                                            uint32_t* keysOut, uint32_t* valsOut) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5, d = threadIdx.x;  // one digit per thread
    uint32_t ahead = 0, all = 0;
#pragma unroll 8
    for (uint32_t c = 0; c < ctas; ++c) {
        const uint32_t x = B.hist[c * kDigits + d];
        if (c < cta) ahead += x;
        all += x;
    }
    uint32_t total;
    uint32_t run = block_scan(all, sm.sum, total) + ahead;
    for (uint32_t x = 0; x < kWarps; ++x) {
        const uint32_t n = sm.cnt[x][d];
        sm.cnt[x][d] = run;
        run += n;
    }
    __syncthreads();
    const uint32_t from = cta * B.chunk + w * warp_part(B), to = min(B.T, from + warp_part(B));
    for (uint32_t p = from; p < to; p += 32) {
        const bool valid = p + lane < to;
        const uint32_t key = valid ? keys[p + lane] : 0u;
        const uint32_t digit = valid ? key >> shift & (kDigits - 1u) : kDigits;
        const uint32_t peers = __match_any_sync(0xFFFFFFFFu, digit);
        const uint32_t at = valid ? sm.cnt[w][digit] + __popc(peers & ((1u << lane) - 1u)) : 0u;
        __syncwarp();
        if (valid && lane == (uint32_t)(__ffs(peers) - 1)) sm.cnt[w][digit] += __popc(peers);
        __syncwarp();
        if (valid && at < B.T) {
            keysOut[at] = key;
            valsOut[at] = vals ? vals[p + lane] : p + lane;
        }
    }
}

// 4. common prefixes of neighbours in this CTA's chunk, and their minima over 32 and
// 1024 positions. 0 (shorter than any) stands after the last position.
__device__ __forceinline__ void build_prefixes(const Build& B, BuildShared& sm, const uint32_t* keys, uint32_t cta) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    const uint32_t end = min((B.T + 31u) & ~31u, (cta + 1u) * B.chunk);
    for (uint32_t base = cta * B.chunk; base < end; base += kThreads) {
        const uint32_t j = base + threadIdx.x;
        uint32_t d = 0;
        if (j + 1u < B.T) {
            const uint32_t x = keys[j] ^ keys[j + 1u];
            d = x ? __clz(x) : 32u + __clz(j ^ (j + 1u));  // keys have 30 bits: at least 2
        }
        if (j < end) B.prefix[j] = (uint8_t)d;
        const uint32_t m = __reduce_min_sync(0xFFFFFFFFu, d);
        if (lane == 0) {
            if (j < end) B.prefix[B.levelAt[1] + (j >> 5)] = (uint8_t)m;
            sm.sum[w] = m;
        }
        __syncthreads();
        if (w == 0) {
            const uint32_t n = __reduce_min_sync(0xFFFFFFFFu, sm.sum[lane]);
            if (lane == 0) B.prefix[B.levelAt[2] + (base >> 10)] = (uint8_t)n;
        }
        __syncthreads();
    }
}

// The entries shorter than v among the 32 of a level from `at` (a multiple of 32).
__device__ __forceinline__ uint32_t shorter(const Build& B, uint32_t at, uint32_t v) {
    const uint4* p = reinterpret_cast<const uint4*>(B.prefix + at);
    const uint4 a = p[0], b = p[1];
    const uint32_t vv = v * 0x01010101u, word[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    uint32_t m = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) m |= ((__vcmpltu4(word[k], vv) & 0x01010101u) * 0x01020408u >> 24) << (4 * k);
    return m;
}
// The nearest position right of g (left, or -1) with a prefix shorter than v, when
// its own 32 hold none. n[k]: entries of level k.
__device__ __forceinline__ int64_t shorter_far(const Build& B, uint32_t g, uint32_t v, bool right) {
    uint32_t i = g >> 5;  // entry of level k
    for (uint32_t k = 1;; ++k) {
        const uint32_t top = k == B.levels, in = i & 31u;
        for (uint32_t b = i >> 5;;) {
            const uint32_t n = (k == 1 ? (B.T + 31u) >> 5 : k == 2 ? (B.T + 1023u) >> 10
                                : k == 3 ? (B.T + 32767u) >> 15 : (B.T + 1048575u) >> 20);  // entries of this level
            uint32_t m = shorter(B, B.levelAt[k] + 32u * b, v);
            const uint32_t left = n - 32u * b;
            if (left < 32u) m &= (1u << left) - 1u;
            if (b == i >> 5) m &= right ? (in == 31u ? 0u : 0xFFFFFFFFu << (in + 1u)) : (1u << in) - 1u;
            if (m) {  // down to the position
                uint32_t e = 32u * b + (right ? __ffs(m) - 1u : 31u - __clz(m));
                for (uint32_t l = k; l-- > 0;) {
                    uint32_t q = shorter(B, (l ? B.levelAt[l] : 0u) + 32u * e, v);
                    if (!q) return -2;  // unreachable: the minimum above said otherwise
                    e = 32u * e + (right ? __ffs(q) - 1u : 31u - __clz(q));
                }
                return e;
            }
            if (!top) break;
            if (right ? 32u * (b + 1u) >= n : b == 0u) return right ? (int64_t)B.T - 1 : -1;
            b = right ? b + 1u : b - 1u;
        }
        i >>= 5;
    }
}

// The tree: the output's interior nodes and where its leaves start.
__device__ __forceinline__ void build_tree(const Build& B, BuildShared& sm, uint32_t cta, uint32_t ctas) {
    if (B.T <= B.leafSize) {  // the root is a leaf
        if (cta == 0 && threadIdx.x == 0) B.leafCount[0] = B.T;
        return;
    }
    auto emit = [&](uint32_t g, int64_t l, int64_t r) {  // the split between g and g + 1; l, r: the shorter prefixes
        const int64_t lo = l + 1, hi = r;
        uint32_t last = 0u;  // not an interior node of the output
        if (!(l >= -1 && lo <= (int64_t)g && (int64_t)g < hi && hi < (int64_t)B.T)) {
            latch(B.err, ERR_LAYOUT);
        } else if (hi - lo + 1 > (int64_t)B.leafSize) {
            last = (uint32_t)hi;
            B.first[g] = (uint32_t)lo;
            atomicAdd(B.starts + lo, 1u);
            const uint32_t nl = g - (uint32_t)lo + 1u, nr = (uint32_t)hi - g;
            if (nl <= B.leafSize) B.leafCount[lo] = nl;
            if (nr <= B.leafSize) B.leafCount[g + 1u] = nr;
        }
        B.last[g] = last;
    };
    for (uint32_t g0 = cta * kThreads; g0 + 1u < B.T; g0 += ctas * kThreads) {
        if (threadIdx.x == 0) sm.u.far[kThreads] = 0u;
        __syncthreads();
        const uint32_t g = g0 + threadIdx.x;
        if (g + 1u < B.T) {
            const uint32_t in = g & 31u, base = g & ~31u, m = shorter(B, base, B.prefix[g]);
            const uint32_t mr = m & (in == 31u ? 0u : 0xFFFFFFFFu << (in + 1u)), ml = m & ((1u << in) - 1u);
            if ((ml || base == 0u) && mr)
                emit(g, ml ? (int64_t)base + 31 - __clz(ml) : -1, base + __ffs(mr) - 1u);
            else
                sm.u.far[atomicAdd(&sm.u.far[kThreads], 1u)] = g;
        }
        __syncthreads();
        // the others, by full warps
        for (uint32_t i = threadIdx.x; i < sm.u.far[kThreads]; i += kThreads) {
            const uint32_t f = sm.u.far[i], in = f & 31u, base = f & ~31u, v = B.prefix[f], m = shorter(B, base, v);
            const uint32_t mr = m & (in == 31u ? 0u : 0xFFFFFFFFu << (in + 1u)), ml = m & ((1u << in) - 1u);
            emit(f, ml ? (int64_t)base + 31 - __clz(ml) : shorter_far(B, f, v, false),
                 mr ? base + __ffs(mr) - 1u : shorter_far(B, f, v, true));
        }
        __syncthreads();
    }
}

// 5. output leaves and nodes that start in this CTA's chunk
__device__ __forceinline__ void build_sums(const Build& B, BuildShared& sm, uint32_t cta) {
    const uint32_t end = min(B.T, (cta + 1u) * B.chunk);
    uint32_t leaves = 0, all = 0;
    for (uint32_t j = cta * B.chunk + threadIdx.x; j < end; j += kThreads) {
        const uint32_t leaf = B.leafCount[j] ? 1u : 0u;
        leaves += leaf;
        all += leaf + B.starts[j];
    }
    leaves = __reduce_add_sync(0xFFFFFFFFu, leaves);
    all = __reduce_add_sync(0xFFFFFFFFu, all);
    if ((threadIdx.x & 31u) == 0) sm.sum2[threadIdx.x >> 5] = make_uint2(leaves, all);
    __syncthreads();
    if (threadIdx.x < 32) {
        const uint2 x = sm.sum2[threadIdx.x];
        const uint32_t a = __reduce_add_sync(0xFFFFFFFFu, x.x), b = __reduce_add_sync(0xFFFFFFFFu, x.y);
        if (threadIdx.x == 0) {
            B.part[cta * 8u + 6u] = a;
            B.part[cta * 8u + 7u] = b;
        }
    }
}

struct BuildBox {
    uint32_t lo[3], hi[3];  // f2o
};
__device__ __forceinline__ BuildBox empty_box() {
    return {{0xFFFFFFFFu, 0xFFFFFFFFu, 0xFFFFFFFFu}, {0u, 0u, 0u}};
}
__device__ __forceinline__ void unite(BuildBox& a, uint4 lo, uint4 hi) {
    a.lo[0] = min(a.lo[0], lo.x); a.lo[1] = min(a.lo[1], lo.y); a.lo[2] = min(a.lo[2], lo.z);
    a.hi[0] = max(a.hi[0], hi.x); a.hi[1] = max(a.hi[1], hi.y); a.hi[2] = max(a.hi[2], hi.z);
}
__device__ __forceinline__ void unite_warp(BuildBox& a) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        a.lo[k] = __reduce_min_sync(0xFFFFFFFFu, a.lo[k]);
        a.hi[k] = __reduce_max_sync(0xFFFFFFFFu, a.hi[k]);
    }
}
__device__ __forceinline__ void store_box(const Build& B, uint32_t at, const BuildBox& b) {
    B.boxLo[at] = make_uint4(b.lo[0], b.lo[1], b.lo[2], 0u);
    B.boxHi[at] = make_uint4(b.hi[0], b.hi[1], b.hi[2], 0u);
}
__device__ __forceinline__ void store_node(const Build& B, uint32_t at, uint32_t size, const BuildBox& b,
                                           uint32_t payload) {
    if ((uint64_t)at + size > 2ull * B.T - 1ull) {  // sizes that do not add up: never write outside
        latch(B.err, ERR_LAYOUT);
        return;
    }
    uint32_t* n = B.nodes + 8ull * at;
    for (int a = 0; a < 3; ++a) {
        n[a] = __float_as_uint(o2f(b.lo[a]));
        n[3 + a] = __float_as_uint(o2f(b.hi[a]));
    }
    n[6] = at + size;
    n[7] = payload;
}

// The vertices of the triangle at position q into bounds, as the refit does it:
// in order, strict < and >.
__device__ __forceinline__ void grow_by_triangle(const Build& B, uint32_t q, float mn[3], float mx[3]) {
    const uint32_t t = B.order[q];
    if (t >= B.T) return;
    for (int k = 0; k < 3; ++k) {
        const uint32_t v = B.idx[3 * (size_t)t + k];
        if (v >= B.V) continue;
        for (int x = 0; x < 3; ++x) {
            const float y = B.pos[3 * (size_t)v + x];
            if (y < mn[x]) mn[x] = y;
            if (y > mx[x]) mx[x] = y;
        }
    }
}

// 5, 6. prefix sums of the chunk, its output leaves, and the box levels within it
__device__ __forceinline__ void build_leaves(const Build& B, BuildShared& sm, uint32_t cta, uint32_t ctas) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t leaves = 0, all = 0;  // ahead of the chunk
    for (uint32_t c = lane; c < cta; c += 32) {
        leaves += B.part[c * 8u + 6u];
        all += B.part[c * 8u + 7u];
    }
    leaves = __reduce_add_sync(0xFFFFFFFFu, leaves);
    all = __reduce_add_sync(0xFFFFFFFFu, all);
    const uint32_t end = min(B.T, (cta + 1u) * B.chunk);
    for (uint32_t base = cta * B.chunk; base < end; base += kThreads) {
        const uint32_t j = base + threadIdx.x;
        float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
        if (j < end) grow_by_triangle(B, j, mn, mx);
        for (int x = 0; x < 3; ++x) {
            sm.u.tri[x][threadIdx.x] = mn[x];
            sm.u.tri[3 + x][threadIdx.x] = mx[x];
        }
        const uint32_t cnt = j < end ? B.leafCount[j] : 0u, st = j < end ? B.starts[j] : 0u;
        const uint32_t leaf = cnt ? 1u : 0u;
        uint32_t nl, na;
        const uint32_t l = leaves + block_scan(leaf, sm.sum, nl), a = all + block_scan(leaf + st, sm.sum, na);
        leaves += nl;
        all += na;
        if (j < end) B.before[j] = make_uint2(l, a);
        if (j + 1u == B.T) {
            B.before[B.T] = make_uint2(l + leaf, a + leaf + st);
            *B.nodeCount = a + leaf + st;
        }
        BuildBox b = empty_box();
        if (leaf) {  // this position's triangle and the leaf's others; past the tile from their vertices
            for (uint32_t i = 1; i < cnt; ++i) {
                const uint32_t q = threadIdx.x + i;
                if (q >= kThreads) {
                    if (j + i < B.T) grow_by_triangle(B, j + i, mn, mx);
                    continue;
                }
                for (int x = 0; x < 3; ++x) {
                    const float lo = sm.u.tri[x][q], hi = sm.u.tri[3 + x][q];
                    if (lo < mn[x]) mn[x] = lo;
                    if (hi > mx[x]) mx[x] = hi;
                }
            }
            for (int x = 0; x < 3; ++x) {
                b.lo[x] = f2o(mn[x]);
                b.hi[x] = f2o(mx[x]);
            }
            store_node(B, a + st, 1u, b, cnt << 24 | j);
        }
        if (j < end) store_box(B, j, b);
        unite_warp(b);
        if (lane == 0) {
            if (j < end) store_box(B, B.levelAt[1] + (j >> 5), b);
            for (int x = 0; x < 3; ++x) {
                sm.lo[w][x] = b.lo[x];
                sm.hi[w][x] = b.hi[x];
            }
        }
        __syncthreads();
        if (w == 0) {
            for (int x = 0; x < 3; ++x) {
                b.lo[x] = sm.lo[lane][x];
                b.hi[x] = sm.hi[lane][x];
            }
            unite_warp(b);
            if (lane == 0) store_box(B, B.levelAt[2] + (base >> 10), b);
        }
        __syncthreads();
    }
}

// The prefix minima or the boxes of the levels above 1024 positions, one warp per
// entry (one CTA).
__device__ __forceinline__ void build_upper(const Build& B, bool boxes) {
    const uint32_t lane = threadIdx.x & 31u, w = threadIdx.x >> 5;
    uint32_t n = (B.T + 1023u) >> 10;
    for (uint32_t k = 3; k <= B.levels; ++k) {
        const uint32_t m = (n + 31u) >> 5;
        for (uint32_t i = w; i < m; i += kWarps) {
            const uint32_t c = 32u * i + lane, from = B.levelAt[k - 1] + c;
            if (boxes) {
                BuildBox b = empty_box();
                if (c < n) unite(b, B.boxLo[from], B.boxHi[from]);
                unite_warp(b);
                if (lane == 0) store_box(B, B.levelAt[k] + i, b);
            } else {
                const uint32_t v = __reduce_min_sync(0xFFFFFFFFu, c < n ? (uint32_t)B.prefix[from] : 255u);
                if (lane == 0) B.prefix[B.levelAt[k] + i] = (uint8_t)v;
            }
        }
        __syncthreads();
        n = m;
    }
}

// 6. interior nodes: found one per thread, their boxes by the whole warp
__device__ __forceinline__ void build_nodes(const Build& B, uint32_t cta, uint32_t ctas) {
    const uint32_t lane = threadIdx.x & 31u;
    if (B.T <= B.leafSize) return;  // the root is a leaf: no node was classified
    for (uint32_t i0 = cta * kThreads + (threadIdx.x & ~31u); i0 + 1u < B.T; i0 += ctas * kThreads) {
        const uint32_t i = i0 + lane;
        const uint32_t l = i + 1u < B.T ? B.last[i] : 0u, f = l ? B.first[i] : 0u;
        uint32_t at = 0, size = 0;
        if (l) {
            const uint2 from = B.before[f], to = B.before[l + 1u];
            size = 2u * (to.x - from.x) - 1u;
            at = from.y;
            // the ancestors that start here too: a node is its parent's left child when
            // the prefix after its range is longer than the one ahead of it
            const uint32_t ahead = f ? B.prefix[f - 1u] : 0u;
            for (uint32_t hi = l, level = 0; level < 80u && hi + 1u < B.T && B.prefix[hi] > ahead; ++level) {
                ++at;
                const uint32_t up = B.last[hi];
                if (up <= hi || up >= B.T) break;
                hi = up;
            }
        }
        BuildBox b = empty_box();
        uint32_t rest = __ballot_sync(0xFFFFFFFFu, l != 0u);
        while (rest) {
            const int src = __ffs(rest) - 1;
            rest &= rest - 1u;
            uint32_t p = __shfl_sync(0xFFFFFFFFu, f, src), q = __shfl_sync(0xFFFFFFFFu, l, src) + 1u;  // [p, q)
            BuildBox x = empty_box();
            for (uint32_t k = 0;; ++k) {  // the ends of the range that are not whole boxes of the next level
                const uint32_t lv = k ? B.levelAt[k] : 0u, p2 = (p + 31u) >> 5, q2 = q >> 5;
                if (k == B.levels || p2 >= q2) {
                    for (uint32_t j = p + lane; j < q; j += 32) unite(x, B.boxLo[lv + j], B.boxHi[lv + j]);
                    break;
                }
                if (p + lane < p2 << 5) unite(x, B.boxLo[lv + p + lane], B.boxHi[lv + p + lane]);
                if ((q2 << 5) + lane < q) unite(x, B.boxLo[lv + (q2 << 5) + lane], B.boxHi[lv + (q2 << 5) + lane]);
                p = p2;
                q = q2;
            }
            unite_warp(x);
            if ((int)lane == src) b = x;
        }
        if (l) store_node(B, at, size, b, 0xFFFFFFFFu);
    }
}

__device__ __forceinline__ const uint32_t* pass_keys(const Build& B, uint32_t pass) { return pass & 1u ? B.keyB : B.keyA; }
__device__ __forceinline__ uint32_t* pass_keys_out(const Build& B, uint32_t pass) { return pass & 1u ? B.keyA : B.keyB; }
// the triangles go to `order`, to valA and to `order` again
__device__ __forceinline__ const uint32_t* pass_vals(const Build& B, uint32_t pass) {
    return pass == 0 ? nullptr : pass == 1 ? B.order : B.valA;
}
__device__ __forceinline__ uint32_t* pass_vals_out(const Build& B, uint32_t pass) { return pass == 1 ? B.valA : B.order; }

// All phases by one cluster.
__global__ void __launch_bounds__(kThreads) k_build_cluster(const __grid_constant__ Build B) {
    extern __shared__ uint4 smem[];
    BuildShared& sm = *reinterpret_cast<BuildShared*>(smem);
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    const uint32_t cta = cluster.block_rank(), ctas = cluster.num_blocks();
    cudaTriggerProgrammaticLaunchCompletion();  // as in k_build_phase
    cudaGridDependencySynchronize();
    auto sync = [&] {
        if (ctas > 1) cluster.sync();
        else __syncthreads();
    };
    build_centres(B, sm, cta, ctas);
    sync();
    build_codes(B, sm, cta, ctas);
    __syncthreads();
    for (uint32_t pass = 0; pass < 3; ++pass) {
        build_count(B, sm, cta, pass_keys(B, pass), pass * kBits);
        sync();
        build_place(B, sm, cta, ctas, pass_keys(B, pass), pass_vals(B, pass), pass * kBits, pass_keys_out(B, pass),
                    pass_vals_out(B, pass));
        sync();
    }
    build_prefixes(B, sm, pass_keys(B, 3), cta);
    sync();
    build_tree(B, sm, cta, ctas);
    sync();
    build_sums(B, sm, cta);
    sync();
    build_leaves(B, sm, cta, ctas);
    sync();
    build_nodes(B, cta, ctas);
}

// One phase per launch.
enum : uint32_t { PHASE_CENTRES, PHASE_SORT, PHASE_PREFIXES = PHASE_SORT + 6, PHASE_UPPER, PHASE_TREE, PHASE_SUMS,
                  PHASE_LEAVES, PHASE_UPPER_BOXES, PHASE_NODES, PHASES };
__global__ void __launch_bounds__(kThreads) k_build_phase(const __grid_constant__ Build B, uint32_t phase) {
    extern __shared__ uint4 smem[];
    BuildShared& sm = *reinterpret_cast<BuildShared*>(smem);
    const uint32_t cta = blockIdx.x, ctas = gridDim.x;
    // the next phase's CTAs may be placed while this one's run; each waits here until
    // the launches ahead of it are complete
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
    if (phase == PHASE_CENTRES) {
        build_centres(B, sm, cta, ctas);
    } else if (phase < PHASE_PREFIXES) {  // count, then count and place, of the three passes
        const uint32_t pass = (phase - PHASE_SORT) / 2u;
        if (phase == PHASE_SORT) {
            build_codes(B, sm, cta, ctas);
            __syncthreads();
        }
        build_count(B, sm, cta, pass_keys(B, pass), pass * kBits);
        if (phase - PHASE_SORT & 1u) {
            __syncthreads();
            build_place(B, sm, cta, ctas, pass_keys(B, pass), pass_vals(B, pass), pass * kBits,
                        pass_keys_out(B, pass), pass_vals_out(B, pass));
        }
    } else if (phase == PHASE_PREFIXES) {
        build_prefixes(B, sm, pass_keys(B, 3), cta);
    } else if (phase == PHASE_TREE) {
        build_tree(B, sm, cta, ctas);
    } else if (phase == PHASE_SUMS) {
        build_sums(B, sm, cta);
    } else if (phase == PHASE_LEAVES) {
        build_leaves(B, sm, cta, ctas);
    } else if (phase == PHASE_UPPER || phase == PHASE_UPPER_BOXES) {
        build_upper(B, phase == PHASE_UPPER_BOXES);
    } else {
        build_nodes(B, cta, ctas);
    }
}

template <class Tp> cudaError_t grow(Tp*& p, size_t& cap, size_t n) {
    if (n <= cap) return cudaSuccess;
    if (p) cudaFree(p);
    p = nullptr;
    cap = 0;
    cudaError_t e = cudaMalloc(&p, n * sizeof(Tp));
    if (e == cudaSuccess) cap = n;
    return e;
}

}  // namespace

struct BlasBuilder {
    uint8_t* scratch = nullptr;  // grows to the largest mesh built
    size_t cap = 0;
    bool ready = false;          // kernel attributes set
    ~BlasBuilder() {
        if (scratch) cudaFree(scratch);
    }
};

BlasBuilder* blas_builder_create() { return new BlasBuilder(); }
void blas_builder_destroy(BlasBuilder* b) { delete b; }

cudaError_t blas_build(BlasBuilder* b, const float* pos, uint32_t V, const uint32_t* idx, uint32_t T,
                       uint32_t leafSize, uint32_t* nodes, uint32_t* order, uint32_t* nodeCount, uint32_t* err,
                       cudaStream_t st) {
    if (T == 0) return cudaSuccess;
    Build B{};
    B.pos = pos;
    B.idx = idx;
    B.V = V;
    B.T = T;
    B.leafSize = leafSize;
    B.order = order;
    B.nodes = nodes;
    B.nodeCount = nodeCount;
    B.err = err;
    // box levels: 1 per position, 32, 1024, ... positions until at most 32 boxes are left
    uint32_t boxes = (T + 31u) & ~31u, n = T;
    for (uint32_t k = 1; k < 5; ++k) {
        B.levelAt[k] = boxes;
        n = (n + 31u) / 32u;
        boxes += (n + 31u) & ~31u;
        B.levels = k;
        if (k >= 2 && n <= 32u) break;
    }
    const uint32_t tiles = (T + kThreads - 1u) / kThreads;
    uint32_t clusterCtas = 1;
    while (clusterCtas < 8 && clusterCtas * kThreads < T) clusterCtas *= 2;
    const bool byCluster = T <= BUILD_CLUSTER_TRIS;
    const uint32_t sortCtas = byCluster ? clusterCtas : std::min(kSortCtas, tiles);
    const uint32_t maxCtas = byCluster ? clusterCtas : std::min(kMaxCtas, tiles);
    // scratch, laid out 256-byte aligned; the first call sizes, the second places. The boxes
    // come after the last use of centres and keys, and take their place.
    uint8_t* base = nullptr;
    size_t at = 0;
    auto place = [&](auto*& p, size_t count) {
        p = reinterpret_cast<std::remove_reference_t<decltype(p)>>(base + at);
        at += (count * sizeof(*p) + 255) & ~size_t(255);
    };
    auto layout = [&] {
        at = 0;
        place(B.boxLo, boxes);
        place(B.boxHi, boxes);
        const size_t end = at;
        at = 0;
        place(B.centre, T);
        place(B.keyA, T);
        place(B.keyB, T);
        place(B.valA, T);
        at = std::max(at, end);
        place(B.part, maxCtas * 8);
        place(B.hist, sortCtas * kDigits);
        place(B.prefix, boxes);
        place(B.first, T);
        place(B.last, T);
        place(B.starts, T);
        place(B.leafCount, T);
        place(B.before, (size_t)T + 1);
    };
    layout();
    // Grown in powers of two, so that a pass over meshes of rising size frees and allocates
    // a few times, not for each; exactly where that much is not to be had. A block of up to
    // 1 MB is a part of the driver's 2 MB ones (3 us, or 350 when a new one has to be
    // mapped: so no more than the mesh needs, 58 bytes a triangle); larger ones are always
    // mapped, and unmapped again (350 + 280 us): powers of four.
    cudaError_t e = cudaSuccess;
    if (at > b->cap) {
        size_t want = 64u << 10;
        while (want < at) want *= want < 1u << 20 ? 2 : 4;
        if ((e = grow(b->scratch, b->cap, want)) != cudaSuccess) {
            cudaGetLastError();
            e = grow(b->scratch, b->cap, at);
        }
    }
    if (e != cudaSuccess) return e;
    base = b->scratch;
    layout();
    const int smem = (int)sizeof(BuildShared);
    if (!b->ready) {
        for (const void* f : {(const void*)k_build_cluster, (const void*)k_build_phase})
            if ((e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, smem)) != cudaSuccess) return e;
        b->ready = true;
    }
    if (byCluster) {
        const uint32_t ctas = clusterCtas;
        B.chunk = ((T + ctas - 1) / ctas + kThreads - 1) / kThreads * kThreads;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(ctas);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = (size_t)smem;
        cfg.stream = st;
        cudaLaunchAttribute attr[2] = {};
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = ctas;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        e = cudaLaunchKernelEx(&cfg, k_build_cluster, B);
        note_launch();
        return e != cudaSuccess ? e : cudaGetLastError();
    }
    cudaLaunchAttribute serial{};
    serial.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    serial.val.programmaticStreamSerializationAllowed = 1;
    for (uint32_t phase = 0; phase < PHASES; ++phase) {
        const bool upper = phase == PHASE_UPPER || phase == PHASE_UPPER_BOXES;
        const bool sort = phase >= PHASE_SORT && phase < PHASE_PREFIXES;
        if (upper && B.levels < 3) continue;
        const uint32_t ctas = phase < PHASE_PREFIXES ? sortCtas : maxCtas;
        B.chunk = ((T + ctas - 1) / ctas + kThreads - 1) / kThreads * kThreads;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(upper ? 1u : ctas);
        cfg.blockDim = dim3(kThreads);
        cfg.dynamicSmemBytes = sort ? (size_t)smem : offsetof(BuildShared, cnt);
        cfg.stream = st;
        cfg.attrs = &serial;
        cfg.numAttrs = phase == 0 ? 0 : 1;
        if ((e = cudaLaunchKernelEx(&cfg, k_build_phase, B, phase)) != cudaSuccess) return e;
        note_launch();
    }
    return cudaGetLastError();
}

}  // namespace sb
