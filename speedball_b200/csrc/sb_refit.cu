// sb_refit.cu — the refit and TLAS lanes on the GPU:
//   * BLAS refit (refitFlatBlasRange, gi_refit.js:34-165): exact leaf min/max in
//     the reference's visiting order, interiors as the JS Math.min/max union of
//     (i+1, miss(i+1)); run bottom-up in parallel with arrival counters, fused
//     with the re-gather of the pre-gathered triangles of the deformed leaves.
//   * per-instance transform math (computeDynamic, spectral_scene.js:1262-1294)
//     in FP64 with every operation separately rounded.
//   * TLAS build (buildTlasRecords, spectral_scene.js:973-1003): one CTA, level
//     by level; each level stable-sorts every interior segment by its FP64
//     centroid on the longest axis (a bitonic sort on (segment, key, position),
//     which equals a stable sort) and splits at the index midpoint.
//   * TLAS refit (refitFlatTlasRange, gi_refit.js:245-292): one CTA, deepest
//     level first.
// min/max are exact, so all bounds are bit-identical to the reference walk.
#include "sb_kernels.cuh"
#include "sb_pairs.cuh"

namespace sb {

constexpr uint32_t NONE = 0xFFFFFFFFu;

__device__ __forceinline__ void bad(uint32_t* gate, uint32_t* err) {
    if (gate) *gate = 0u;
    latch(err, ERR_LAYOUT);
}

// ------------------------------------------------------------- BLAS refit
// The words of a cached range: its verdict, its number of subtrees, the number of top
// nodes in its plan (NONE: no plan), the subtrees finished in a running refit.
constexpr uint32_t GATE = 0, GATE_SUBS = REFIT_RANGES, GATE_TOPS = 2 * REFIT_RANGES, GATE_DONE = 3 * REFIT_RANGES;

__global__ void k_refit_reset(uint32_t* parent, uint32_t* arrive, uint32_t root, uint32_t end, uint32_t* gate) {
    uint32_t i = root + blockIdx.x * blockDim.x + threadIdx.x;
    if (i == root) {
        gate[GATE] = 1u;  // valid until a check fails
        gate[GATE_SUBS] = gate[GATE_TOPS] = gate[GATE_DONE] = 0u;
    }
    if (i >= end) return;
    parent[i] = NONE;
    arrive[i] = 0u;
}

// The end of node i's subtree as its own miss word states it: miss(i) when it
// lies in (i, end], else the range end (the right spine of the range).
__device__ __forceinline__ uint32_t subtree_end(const uint32_t* nodes, uint32_t i, uint32_t end) {
    const uint32_t miss = nodes[8 * i + 6];
    return (miss > i && miss <= end) ? miss : end;
}

// A range's gate word: 0 = the layout check failed (the refit reports
// SB_ERR_LAYOUT_VIOLATION until the next upload); 1 = valid, and every node's
// own miss word ends its subtree (a leaf: i + 1; an interior node: where its
// right child's subtree ends), so subtrees can be cut out by index range;
// 2 = valid for the reference's refit, which reads only left children's miss
// words (gi_refit.js:96-139), while some other miss word is stale: the range is
// refit node by node without the subtree partition.
//
// Link children to parents and check the layout contract (gi_refit.js:96-139):
// right child = left child's miss, inside (left, end); leaves index inside the
// triangle and vertex pools. A node claimed twice, or an orphan, also fails.
__global__ void k_refit_link(const uint32_t* nodes, const uint32_t* triIndex, const uint32_t* triMaterial,
                             uint32_t triCount, uint32_t vertexCount, uint32_t materialCount, uint32_t* parent,
                             uint32_t root, uint32_t end, uint32_t* gate, uint32_t* err) {
    uint32_t i = root + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end) return;
    uint32_t info = nodes[8 * i + 7];
    if (info != INTERIOR) {
        uint32_t off = info & 0x00FFFFFFu, cnt = info >> 24;
        for (uint32_t t = off; t < off + cnt; ++t) {
            if (t >= triCount || triMaterial[t] >= materialCount) { bad(gate, err); return; }
            for (int k = 0; k < 3; ++k)
                if (triIndex[3 * t + k] >= vertexCount) { bad(gate, err); return; }
        }
        if (subtree_end(nodes, i, end) != i + 1u) atomicCAS(gate, 1u, 2u);
        return;
    }
    uint32_t l = i + 1;
    if (l >= end) { bad(gate, err); return; }
    uint32_t r = nodes[8 * l + 6];
    if (!(r > l && r < end)) { bad(gate, err); return; }
    if (atomicCAS(&parent[l], NONE, i) != NONE) bad(gate, err);
    if (atomicCAS(&parent[r], NONE, i) != NONE) bad(gate, err);
    if (subtree_end(nodes, i, end) != subtree_end(nodes, r, end)) atomicCAS(gate, 1u, 2u);
}

__global__ void k_refit_orphans(const uint32_t* parent, uint32_t root, uint32_t end, uint32_t* gate, uint32_t* err) {
    uint32_t i = root + 1 + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end) return;
    if (parent[i] == NONE) bad(gate, err);
}

__device__ __forceinline__ uint32_t arrive_at(uint32_t* counter) {
    uint32_t prev;
    asm volatile("atom.acq_rel.gpu.global.add.u32 %0, [%1], 1;" : "=r"(prev) : "l"(counter) : "memory");
    return prev;
}

// What a refit reads of the scene, and writes.
struct RefitArrays {
    uint32_t* nodes;
    const uint32_t* triIndex;
    const float4* vertices;  // two float4 per vertex, the position first
    const uint32_t *triMaterial, *matBits;
    float4* tris;
    const uint32_t* parent;
    uint32_t* arrive;
    uint4* pairs;
};

// A leaf's box over its triangles in order (cnt > 0), and its pre-gathered triangles
// from the deformed vertices. Four triangles' loads are in flight together.
__device__ __forceinline__ void refit_leaf(const RefitArrays& R, uint32_t off, uint32_t cnt, float box[6]) {
    for (int k = 0; k < 3; ++k) {
        box[k] = INFINITY;
        box[3 + k] = -INFINITY;
    }
    for (uint32_t at = 0; at < cnt; at += 4u) {
        float4 v[4][3];
        uint32_t bits[4];
#pragma unroll
        for (uint32_t j = 0; j < 4u; ++j) {
            const uint32_t t = off + min(at + j, cnt - 1u);
            bits[j] = __ldg(R.matBits + __ldg(R.triMaterial + t));
#pragma unroll
            for (int k = 0; k < 3; ++k) v[j][k] = __ldg(R.vertices + 2 * (size_t)__ldg(R.triIndex + 3 * t + k));
        }
#pragma unroll
        for (uint32_t j = 0; j < 4u; ++j) {
            if (at + j >= cnt) break;
            const uint32_t t = off + at + j;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float p[3] = {v[j][k].x, v[j][k].y, v[j][k].z};
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    if (p[a] < box[a]) box[a] = p[a];
                    if (p[a] > box[3 + a]) box[3 + a] = p[a];
                }
                R.tris[3 * t + k] = make_float4(p[0], p[1], p[2], k == 0 ? __uint_as_float(bits[j]) : 0.0f);
            }
        }
    }
}

// A node's box from its children's.
__device__ __forceinline__ void join_boxes(const uint32_t lb[6], const uint32_t rb[6], uint32_t box[6]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        box[k] = __float_as_uint(js_min(__uint_as_float(lb[k]), __uint_as_float(rb[k])));
        box[3 + k] = __float_as_uint(js_max(__uint_as_float(lb[3 + k]), __uint_as_float(rb[3 + k])));
    }
}
__device__ __forceinline__ void store_box(uint32_t* nodes, uint32_t i, const uint32_t b[6]) {
    *reinterpret_cast<uint4*>(nodes + 8 * (size_t)i) = make_uint4(b[0], b[1], b[2], b[3]);
    *reinterpret_cast<uint2*>(nodes + 8 * (size_t)i + 4) = make_uint2(b[4], b[5]);
}

// The climb through global memory: the second child to finish computes its parent.
__device__ __forceinline__ void refit_climb(const RefitArrays& R, uint32_t node) {
    for (;;) {
        const uint32_t p = R.parent[node];
        if (p == NONE) break;
        // arrival: release publishes this thread's box stores, acquire orders the
        // sibling's box reads below after the sibling's release (one acq_rel atomic)
        if (arrive_at(R.arrive + p) == 0u) break;
        R.arrive[p] = 0u;  // both children arrived: ready for the next refit of this range
        const uint32_t l = p + 1;
        const uint32_t r = *(const volatile uint32_t*)(R.nodes + 8 * l + 6);
        uint32_t lb[6], rb[6], box[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            lb[k] = *(const volatile uint32_t*)(R.nodes + 8 * l + k);
            rb[k] = *(const volatile uint32_t*)(R.nodes + 8 * r + k);
        }
        join_boxes(lb, rb, box);
        store_box(R.nodes, p, box);
        if (R.pairs) store_pair_boxes(R.pairs + 4u * p, lb, rb);  // the traversal's copy of both child boxes
        node = p;
    }
}

// Subtrees of at most REFIT_SUB nodes refit inside one CTA: the threaded layout stores
// a node's subtree as [i, miss(i)) (to the range end on the right spine), one node per
// thread. The partition (every node whose subtree fits while its parent's does not)
// is made once per validated range, next to the layout checks, and with it, when there
// are at most REFIT_SUB subtrees, a plan of the nodes above them, which the CTA that
// finishes last computes in the same way.
//
// What bounds it is the chain of dependent loads, not work: a deforming mesh of some
// thousand triangles is 0.4 MB. So a thread's node, triangle indices and vertices are
// loaded once, four triangles' at a time; the boxes climb in shared memory, one
// level per barrier (a counter per node and its fences cost more than the levels that
// nothing happens in); and what is above the subtrees costs one more load of their
// boxes. The atrium's deforming mesh refits in 15 us instead of 31 node by node.
constexpr uint32_t REFIT_SUB = 256;  // nodes per CTA subtree (= threads per CTA)

__device__ __forceinline__ uint32_t sub_size(const uint32_t* nodes, uint32_t i, uint32_t end) {
    const uint32_t miss = nodes[8 * i + 6];
    return (miss > i && miss <= end) ? miss - i : end - i;
}

// The subtrees' roots from the front of the range's words in subRoots, the nodes above
// them from the back (roots and top nodes are different nodes of the range).
__global__ void k_refit_partition(const uint32_t* nodes, const uint32_t* parent, uint32_t root, uint32_t end,
                                  uint32_t* gate, uint32_t* subRoots) {
    const uint32_t i = root + blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= end || gate[GATE] != 1u) return;
    if (sub_size(nodes, i, end) > REFIT_SUB) {
        subRoots[end - 1u - atomicAdd(gate + GATE_TOPS, 1u)] = i;
        return;
    }
    const uint32_t p = parent[i];
    if (p != NONE && sub_size(nodes, p, end) <= REFIT_SUB) return;
    subRoots[root + atomicAdd(gate + GATE_SUBS, 1u)] = i;
}

// The plan: behind the n roots, per top node (its index, left unit, right unit, 0),
// where units 0 .. n - 1 are the subtrees and n + t is top node t. One CTA.
__global__ void __launch_bounds__(REFIT_SUB) k_refit_plan(const uint32_t* nodes, uint32_t root, uint32_t end,
                                                          uint32_t* gate, uint32_t* subRoots) {
    __shared__ uint32_t unit[2 * REFIT_SUB];
    __shared__ uint32_t bad;
    const uint32_t n = gate[GATE_SUBS], tops = gate[GATE_TOPS], tid = threadIdx.x;
    const bool planned = gate[GATE] == 1u && n != 0u && n <= REFIT_SUB && tops + 1u == n &&
                         n + 4u * tops <= end - root;
    if (tid == 0) bad = 0u;
    if (planned) {
        if (tid < n) unit[tid] = subRoots[root + tid];
        if (tid < tops) unit[n + tid] = subRoots[end - 1u - tid];
    }
    __syncthreads();
    if (planned && tid < tops) {
        const uint32_t l = unit[n + tid] + 1u, r = nodes[8 * l + 6];
        uint32_t ul = NONE, ur = NONE;
        for (uint32_t u = 0; u < n + tops; ++u) {
            if (unit[u] == l) ul = u;
            if (unit[u] == r) ur = u;
        }
        if (ul == NONE || ur == NONE) bad = 1u;
        uint32_t* e = subRoots + root + n + 4u * tid;
        e[0] = unit[n + tid];
        e[1] = ul;
        e[2] = ur;
        e[3] = 0u;
    }
    __syncthreads();
    if (tid == 0 && (!planned || bad)) gate[GATE_TOPS] = NONE;
}

__global__ void __launch_bounds__(REFIT_SUB) k_refit_cta(const RefitArrays R, uint32_t root, uint32_t end,
                                                         uint32_t* gate, const uint32_t* subRoots, uint32_t* err) {
    __shared__ uint32_t sBox[6][2 * REFIT_SUB];
    __shared__ uint32_t sMiss[REFIT_SUB];
    __shared__ volatile uint32_t sDone[2 * REFIT_SUB];  // the round that computed a box
    __shared__ uint32_t sLast;
    const uint32_t tid = threadIdx.x;
    const uint32_t g = gate[GATE], nSub = gate[GATE_SUBS], tops = gate[GATE_TOPS];
    if (g == 0u) {
        if (blockIdx.x == 0 && tid == 0) latch(err, ERR_LAYOUT);  // the range's verdict stands
        return;
    }
    if (g != 1u) {  // no subtree partition for this layout: node by node, grid-stride
        for (uint32_t i = root + blockIdx.x * blockDim.x + tid; i < end; i += gridDim.x * blockDim.x) {
            const uint32_t info = R.nodes[8 * i + 7];
            if (info == INTERIOR) continue;
            if (info >> 24) {
                float b[6];
                refit_leaf(R, info & 0x00FFFFFFu, info >> 24, b);
                uint32_t w[6];
                for (int k = 0; k < 6; ++k) w[k] = __float_as_uint(b[k]);
                store_box(R.nodes, i, w);
            }
            refit_climb(R, i);
        }
        return;
    }
    // one level of boxes per round: unit u (children l, r) once both are done
    auto round = [&](uint32_t u, uint32_t l, uint32_t r, uint32_t now) {
        if (sDone[u] != NONE || sDone[l] >= now || sDone[r] >= now) return;
        uint32_t lb[6], rb[6], box[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            lb[k] = sBox[k][l];
            rb[k] = sBox[k][r];
        }
        join_boxes(lb, rb, box);
#pragma unroll
        for (int k = 0; k < 6; ++k) sBox[k][u] = box[k];
        sDone[u] = now;
    };
    auto store = [&](uint32_t node, uint32_t u, uint32_t l, uint32_t r, bool interior) {
        uint32_t b[6], lb[6], rb[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            b[k] = sBox[k][u];
            lb[k] = sBox[k][l];
            rb[k] = sBox[k][r];
        }
        store_box(R.nodes, node, b);
        if (interior && R.pairs) store_pair_boxes(R.pairs + 4u * node, lb, rb);
    };
    for (uint32_t t = blockIdx.x; t < nSub; t += gridDim.x) {
        const uint32_t r0 = subRoots[root + t];
        uint4 lo = make_uint4(0u, 0u, 0u, 0u), hi = lo;
        if (tid < end - r0) {
            lo = *reinterpret_cast<const uint4*>(R.nodes + 8 * (size_t)(r0 + tid));
            hi = *reinterpret_cast<const uint4*>(R.nodes + 8 * (size_t)(r0 + tid) + 4);
        }
        sMiss[tid] = hi.z;
        __syncthreads();
        const uint32_t m0 = sMiss[0], sz = min(m0 > r0 && m0 <= end ? m0 - r0 : end - r0, REFIT_SUB);
        const bool mine = tid < sz, interior = mine && hi.w == INTERIOR;
        uint32_t l = tid, r = tid;
        if (interior) {
            l = tid + 1u;
            r = l < sz ? sMiss[l] - r0 : NONE;
            if (r >= sz || r <= l) {  // a partition that does not match the layout
                latch(err, ERR_LAYOUT);
                l = r = tid;          // (never done: nothing above it is written)
            }
        }
        if (mine && !interior) {
            uint32_t box[6] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y};
            if (hi.w >> 24) {
                float b[6];
                refit_leaf(R, hi.w & 0x00FFFFFFu, hi.w >> 24, b);
#pragma unroll
                for (int k = 0; k < 6; ++k) box[k] = __float_as_uint(b[k]);
            }
#pragma unroll
            for (int k = 0; k < 6; ++k) sBox[k][tid] = box[k];
        }
        sDone[tid] = mine && !interior ? 0u : NONE;
        bool open = interior;
        for (uint32_t now = 1; now <= sz && __syncthreads_or(open); ++now) {
            if (interior) round(tid, l, r, now);
            open = interior && sDone[tid] == NONE;
        }
        __syncthreads();
        if (mine && sDone[tid] != NONE && (interior || hi.w >> 24)) store(r0 + tid, tid, l, r, interior);
        // above the subtree: through global memory, or by the CTA that finishes last
        if (tid == 0) {
            sLast = 0u;
            if (tops == NONE) refit_climb(R, r0);
            else if (tops) sLast = arrive_at(gate + GATE_DONE) + 1u == nSub ? 1u : 0u;
        }
        __syncthreads();
        if (sLast) {
            uint32_t node = 0, ul = 0, ur = 0;
            if (tid < tops) {
                const uint32_t* e = subRoots + root + nSub + 4u * tid;
                node = e[0];
                ul = e[1];
                ur = e[2];
                sDone[nSub + tid] = NONE;
            }
            if (tid < nSub) {
                const uint32_t* n = R.nodes + 8 * (size_t)subRoots[root + tid];
#pragma unroll
                for (int k = 0; k < 6; ++k) sBox[k][tid] = *(const volatile uint32_t*)(n + k);
                sDone[tid] = 0u;
            }
            open = true;
            for (uint32_t now = 1; now <= tops && __syncthreads_or(open); ++now) {
                if (tid < tops) round(nSub + tid, ul, ur, now);
                open = tid < tops && sDone[nSub + tid] == NONE;
            }
            __syncthreads();
            if (tid < tops && sDone[nSub + tid] != NONE) store(node, nSub + tid, ul, ur, true);
            if (tid == 0) gate[GATE_DONE] = 0u;
        }
        __syncthreads();  // the shared arrays serve the next subtree
    }
}

__global__ void k_scatter_vertices(float* v8, const float* p3, const float* n3, uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float* v = v8 + 8u * (size_t)i;
    v[0] = p3[3u * (size_t)i];
    v[1] = p3[3u * (size_t)i + 1u];
    v[2] = p3[3u * (size_t)i + 2u];
    if (n3) {
        v[3] = n3[3u * (size_t)i];
        v[4] = n3[3u * (size_t)i + 1u];
        v[5] = n3[3u * (size_t)i + 2u];
    }
}

cudaError_t launch_scatter_vertices(float* vertexData8, const float* positions, const float* normals, uint32_t n,
                                    cudaStream_t st) {
    if (n == 0) return cudaSuccess;
    k_scatter_vertices<<<(n + 255) / 256, 256, 0, st>>>(vertexData8, positions, normals, n);
    note_launch();
    return cudaGetLastError();
}

cudaError_t launch_refit_blas(const SceneBuffers& B, uint32_t root, uint32_t end, uint32_t* err, uint32_t* gate,
                              cudaStream_t st, bool validated) {
    if (end <= root) return cudaSuccess;
    uint32_t n = end - root;
    unsigned g = (n + 255) / 256;
    if (!validated) {
        k_refit_reset<<<g, 256, 0, st>>>(B.parent, B.arrive, root, end, gate); note_launch();
        k_refit_link<<<g, 256, 0, st>>>(B.nodes, B.triIndex, B.triMaterial, B.triCount, B.vertexCount,
                                        B.materialCount, B.parent, root, end, gate, err); note_launch();
        k_refit_orphans<<<g, 256, 0, st>>>(B.parent, root, end, gate, err); note_launch();
        k_refit_partition<<<g, 256, 0, st>>>(B.nodes, B.parent, root, end, gate, B.subRoots); note_launch();
        k_refit_plan<<<1, REFIT_SUB, 0, st>>>(B.nodes, root, end, gate, B.subRoots); note_launch();
    }
    // one CTA per subtree: how many there are is on the device (a subtree of a balanced
    // tree has 128 nodes or more; CTAs take further ones in turn)
    const RefitArrays R{B.nodes, B.triIndex, reinterpret_cast<const float4*>(B.vertexData), B.triMaterial, B.matBits,
                        B.tris, B.parent, B.arrive, B.pairs};
    const unsigned ctas = (n + 63u) / 64u;
    k_refit_cta<<<ctas < 1184u ? ctas : 1184u, REFIT_SUB, 0, st>>>(R, root, end, gate, B.subRoots, err);
    note_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------- instance math (FP64)
// Operation order is fixed and every product/sum separately rounded, so the
// results are reproducible bit-for-bit by a host evaluation in the same order.
#define DM(a, b) __dmul_rn((a), (b))
#define DA(a, b) __dadd_rn((a), (b))
#define DS(a, b) __dsub_rn((a), (b))

__device__ __forceinline__ double mat(const double* m, int r, int c) { return m[c * 4 + r]; }

__device__ double det4(const double* m) {
    double s01 = DS(DM(mat(m, 2, 0), mat(m, 3, 1)), DM(mat(m, 2, 1), mat(m, 3, 0)));
    double s02 = DS(DM(mat(m, 2, 0), mat(m, 3, 2)), DM(mat(m, 2, 2), mat(m, 3, 0)));
    double s03 = DS(DM(mat(m, 2, 0), mat(m, 3, 3)), DM(mat(m, 2, 3), mat(m, 3, 0)));
    double s12 = DS(DM(mat(m, 2, 1), mat(m, 3, 2)), DM(mat(m, 2, 2), mat(m, 3, 1)));
    double s13 = DS(DM(mat(m, 2, 1), mat(m, 3, 3)), DM(mat(m, 2, 3), mat(m, 3, 1)));
    double s23 = DS(DM(mat(m, 2, 2), mat(m, 3, 3)), DM(mat(m, 2, 3), mat(m, 3, 2)));
    double c0 = DA(DS(DM(mat(m, 1, 1), s23), DM(mat(m, 1, 2), s13)), DM(mat(m, 1, 3), s12));
    double c1 = DA(DS(DM(mat(m, 1, 0), s23), DM(mat(m, 1, 2), s03)), DM(mat(m, 1, 3), s02));
    double c2 = DA(DS(DM(mat(m, 1, 0), s13), DM(mat(m, 1, 1), s03)), DM(mat(m, 1, 3), s01));
    double c3 = DA(DS(DM(mat(m, 1, 0), s12), DM(mat(m, 1, 1), s02)), DM(mat(m, 1, 2), s01));
    return DS(DA(DS(DM(mat(m, 0, 0), c0), DM(mat(m, 0, 1), c1)), DM(mat(m, 0, 2), c2)), DM(mat(m, 0, 3), c3));
}

// Entry (r, c) of the adjugate.
__device__ __forceinline__ double cofactor(const double* m, int r, int c) {
    const int r0 = c == 0, r1 = 1 + (c <= 1), r2 = 2 + (c <= 2), c0 = r == 0, c1 = 1 + (r <= 1), c2 = 2 + (r <= 2);
    const double t0 = DM(mat(m, r0, c0), DS(DM(mat(m, r1, c1), mat(m, r2, c2)), DM(mat(m, r1, c2), mat(m, r2, c1))));
    const double t1 = DM(mat(m, r0, c1), DS(DM(mat(m, r1, c0), mat(m, r2, c2)), DM(mat(m, r1, c2), mat(m, r2, c0))));
    const double t2 = DM(mat(m, r0, c2), DS(DM(mat(m, r1, c0), mat(m, r2, c1)), DM(mat(m, r1, c1), mat(m, r2, c0))));
    const double m3 = DA(DS(t0, t1), t2);
    return ((r + c) & 1) ? -m3 : m3;
}

// First three rows of the inverse (adjugate / determinant), zeros if singular.
__device__ void inverse_rows(const double* m, double out[12]) {
    double det = det4(m);
    if (det == 0.0) {
        for (int i = 0; i < 12; ++i) out[i] = 0.0;
        return;
    }
    double inv = __ddiv_rn(1.0, det);
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 4; ++c) out[r * 4 + c] = DM(cofactor(m, r, c), inv);
}

__device__ __forceinline__ void transform_corner(const double* m, double x, double y, double z, double p[3]) {
    const double w = __ddiv_rn(1.0, DA(DA(DA(DM(m[3], x), DM(m[7], y)), DM(m[11], z)), m[15]));
    p[0] = DM(DA(DA(DA(DM(m[0], x), DM(m[4], y)), DM(m[8], z)), m[12]), w);
    p[1] = DM(DA(DA(DA(DM(m[1], x), DM(m[5], y)), DM(m[9], z)), m[13]), w);
    p[2] = DM(DA(DA(DA(DM(m[2], x), DM(m[6], y)), DM(m[10], z)), m[14]), w);
}

__device__ void transform_box(const double* m, const double lmin[3], const double lmax[3], double wmin[3],
                              double wmax[3]) {
    for (int a = 0; a < 3; ++a) { wmin[a] = INFINITY; wmax[a] = -INFINITY; }
    for (int i = 0; i < 8; ++i) {
        double p[3];
        transform_corner(m, (i & 1) ? lmax[0] : lmin[0], (i & 2) ? lmax[1] : lmin[1], (i & 4) ? lmax[2] : lmin[2], p);
        for (int a = 0; a < 3; ++a) {
            if (p[a] < wmin[a]) wmin[a] = p[a];
            if (p[a] > wmax[a]) wmax[a] = p[a];
        }
    }
}

// computeDynamic for one source instance: inverse rows, winding sign, FP64 AABB.
__device__ void compute_instance(const SceneBuffers& B, const InstanceTable& I, uint32_t src, uint32_t* err) {
    const double* m = I.world + (size_t)src * 16u;
    double inv[12];
    inverse_rows(m, inv);
    for (int k = 0; k < 12; ++k) I.invRows[(size_t)src * 12u + k] = __double2float_rn(inv[k]);
    I.detSign[src] = det4(m) < 0.0 ? -1.0f : 1.0f;
    double mn[3], mx[3];
    uint32_t root = I.blasRoot[src], end = I.blasEnd[src];
    if (I.active[src]) {
        if (!(root < end && end <= B.nodeCount)) {
            latch(err, ERR_LAYOUT);
            for (int a = 0; a < 3; ++a) mn[a] = mx[a] = 0.0;
        } else {
            const float* nb = reinterpret_cast<const float*>(B.nodes + (size_t)root * 8u);
            double lmin[3] = {nb[0], nb[1], nb[2]}, lmax[3] = {nb[3], nb[4], nb[5]};
            transform_box(m, lmin, lmax, mn, mx);
        }
    } else {
        for (int a = 0; a < 3; ++a) mn[a] = mx[a] = m[12 + a];
    }
    double* o = I.aabb + (size_t)src * 9u;
    for (int a = 0; a < 3; ++a) {
        o[a] = mn[a];
        o[3 + a] = mx[a];
        o[6 + a] = DM(DA(mn[a], mx[a]), 0.5);
        if (o[6 + a] != o[6 + a]) latch(err, ERR_NAN_KEY);
    }
}

// writeDynamic's instance record for one slot (spectral_scene.js:1340-1355),
// into both the reference tail and the derived instance rows.
__device__ void write_slot(const SceneBuffers& B, const InstanceTable& I, uint32_t slot, uint32_t src, bool rows) {
    const double* a = I.aabb + (size_t)src * 9u;
    float* lb = I.liveBounds + (size_t)slot * 6u;
    for (int k = 0; k < 6; ++k) lb[k] = __double2float_rn(a[k]);
    if (!rows) return;
    float* R = B.materials + B.instBase + (size_t)slot * 28u;
    const float* ir = I.invRows + (size_t)src * 12u;
    for (int k = 0; k < 12; ++k) R[k] = ir[k];
    R[12] = float(I.blasRoot[src]);
    R[13] = float(I.blasEnd[src]);
    R[14] = I.detSign[src];
    R[15] = I.active[src] ? 1.0f : 0.0f;
    for (int k = 16; k < 28; ++k) R[k] = 0.0f;
    B.inst[4 * slot] = make_float4(ir[0], ir[1], ir[2], ir[3]);
    B.inst[4 * slot + 1] = make_float4(ir[4], ir[5], ir[6], ir[7]);
    B.inst[4 * slot + 2] = make_float4(ir[8], ir[9], ir[10], ir[11]);
    B.inst[4 * slot + 3] = make_float4(__uint_as_float(I.blasRoot[src]), __uint_as_float(I.blasEnd[src]),
                                       I.detSign[src], I.active[src] ? 1.0f : 0.0f);
}

__device__ __forceinline__ void write_tlas_node(const SceneBuffers& B, uint32_t idx, const float bx[6], uint32_t miss,
                                                uint32_t off, uint32_t cnt) {
    float* N = B.materials + B.tlasBase + (size_t)idx * 12u;
    for (int k = 0; k < 6; ++k) N[k] = bx[k];
    N[6] = float(miss);
    N[7] = cnt ? float(off) : 0.0f;
    N[8] = float(cnt);
    N[9] = N[10] = N[11] = 0.0f;
    B.tlas[2 * idx] = make_uint4(__float_as_uint(bx[0]), __float_as_uint(bx[1]), __float_as_uint(bx[2]),
                                 __float_as_uint(bx[3]));
    B.tlas[2 * idx + 1] = make_uint4(__float_as_uint(bx[4]), __float_as_uint(bx[5]), miss, (cnt << 24) | (cnt ? off : 0u));
}

// ------------------------------------------------------------- TLAS build
// Order-preserving 64-bit key of a double (-0 folded onto +0, as the reference
// comparator c[a] - c[b] treats them as equal).
__device__ __forceinline__ unsigned long long sortable(double d) {
    if (d == 0.0) d = 0.0;
    unsigned long long b = (unsigned long long)__double_as_longlong(d);
    return (b & 0x8000000000000000ull) ? ~b : (b | 0x8000000000000000ull);
}

// Sort record: (group << 13 | position) and key; ordered by group, then key,
// then position, so ties keep the current order (a stable sort) and groups
// stay in place.
struct BuildRec {
    unsigned long long key;
    uint32_t segpos;
    uint32_t pad;
};
__device__ __forceinline__ bool rec_less(const BuildRec& a, const BuildRec& b) {
    uint32_t sa = a.segpos >> 13, sb = b.segpos >> 13;
    if (sa != sb) return sa < sb;
    if (a.key != b.key) return a.key < b.key;
    return (a.segpos & 0x1FFFu) < (b.segpos & 0x1FFFu);
}

// min with ties kept by the earlier position; NaN never selected (the strict
// `<` scan of buildTlasRecords from +Infinity)
__device__ __forceinline__ void red_min(double& v, uint32_t& p, double v2, uint32_t p2) {
    if (v2 != v2) return;
    if (v != v || v2 < v || (v2 == v && p2 < p)) { v = v2; p = p2; }
}
__device__ __forceinline__ void red_max(double& v, uint32_t& p, double v2, uint32_t p2) {
    if (v2 != v2) return;
    if (v != v || v2 > v || (v2 == v && p2 < p)) { v = v2; p = p2; }
}

struct Seg { uint16_t lo, hi, idx; };

// Up to this many instances a level orders its segments by rank (the summed
// squared segment lengths stay below n^2 / 2 per level); above it by one
// bitonic sort of all positions per level.
constexpr uint32_t TLAS_RANK_SORT_MAX = 512;

__host__ __device__ inline size_t tlas_build_smem(uint32_t n) {
    uint32_t P = 1;
    while (P < n) P <<= 1;
    size_t b = (size_t)P * sizeof(BuildRec) + (size_t)n * 4u * 3u + 4u + (size_t)n * sizeof(Seg) * 2u;
    return (b + 15u) & ~(size_t)15u;
}

__global__ void __launch_bounds__(1024) k_tlas_build(SceneBuffers B, InstanceTable I, uint32_t* err) {
    extern __shared__ unsigned char smem[];
    const uint32_t n = I.count;
    uint32_t P = 1;
    while (P < n) P <<= 1;
    BuildRec* rec = reinterpret_cast<BuildRec*>(smem);                       // P
    uint32_t* order = reinterpret_cast<uint32_t*>(rec + P);                  // n
    uint32_t* segOf = order + n;                                             // n (also a gather buffer)
    uint32_t* nodesTab = segOf + n;                                          // n+1
    Seg* segA = reinterpret_cast<Seg*>(nodesTab + n + 1);                    // n
    Seg* segB = segA + n;                                                    // n
    __shared__ uint32_t nSeg, nNext, level;
    __shared__ uint8_t axisOf[TLAS_BUILD_MAX];

    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) {
        compute_instance(B, I, i, err);
        order[i] = i;
    }
    if (threadIdx.x == 0) {
        // subtree node counts of the median split with leaf size 2
        nodesTab[0] = 1;
        for (uint32_t m = 1; m <= n; ++m) nodesTab[m] = m <= 2 ? 1u : 1u + nodesTab[m >> 1] + nodesTab[m - (m >> 1)];
        segA[0] = Seg{0, (uint16_t)n, 0};
        nSeg = 1;
        level = 0;
    }
    __syncthreads();
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, nWarps = blockDim.x >> 5;
    Seg* cur = segA;
    Seg* nxt = segB;
    while (nSeg > 0) {
        // positions whose leaf was emitted at an earlier level belong to no segment
        for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) segOf[j] = NONE;
        __syncthreads();
        // (a) bounds + node record per segment, one warp per segment
        for (uint32_t s = warp; s < nSeg; s += nWarps) {
            Seg sg = cur[s];
            double mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
            uint32_t pmn[3] = {NONE, NONE, NONE}, pmx[3] = {NONE, NONE, NONE};
            for (uint32_t j = sg.lo + lane; j < sg.hi; j += 32) {
                const double* a = I.aabb + (size_t)order[j] * 9u;
                for (int k = 0; k < 3; ++k) {
                    red_min(mn[k], pmn[k], a[k], j);
                    red_max(mx[k], pmx[k], a[3 + k], j);
                }
                segOf[j] = s;
            }
            for (int off = 16; off > 0; off >>= 1)
                for (int k = 0; k < 3; ++k) {
                    double v = __shfl_down_sync(0xFFFFFFFFu, mn[k], off);
                    uint32_t p = __shfl_down_sync(0xFFFFFFFFu, pmn[k], off);
                    if (p != NONE) red_min(mn[k], pmn[k], v, p);
                    v = __shfl_down_sync(0xFFFFFFFFu, mx[k], off);
                    p = __shfl_down_sync(0xFFFFFFFFu, pmx[k], off);
                    if (p != NONE) red_max(mx[k], pmx[k], v, p);
                }
            if (lane == 0) {
                float bx[6];
                for (int k = 0; k < 3; ++k) {
                    bx[k] = __double2float_rn(mn[k]);
                    bx[3 + k] = __double2float_rn(mx[k]);
                }
                uint32_t cnt = (uint32_t)sg.hi - sg.lo;
                uint32_t miss = sg.idx + nodesTab[cnt];
                if (cnt <= 2) {
                    write_tlas_node(B, sg.idx, bx, miss, sg.lo, cnt);
                    axisOf[s] = 255;
                } else {
                    write_tlas_node(B, sg.idx, bx, miss, 0, 0);
                    double ex = DS(mx[0], mn[0]), ey = DS(mx[1], mn[1]), ez = DS(mx[2], mn[2]);
                    axisOf[s] = (ex >= ey && ex >= ez) ? 0 : (ey >= ez ? 1 : 2);
                }
                I.nodeDepth[sg.idx] = level;
            }
        }
        __syncthreads();
        if (n <= TLAS_RANK_SORT_MAX) {
            // (b) the stable order of every interior segment by its split axis's FP64
            // centroid key: each position's rank among its segment's positions by
            // (key, position), one thread per position; leaf segments and finished
            // positions keep their place. The keys are staged once per level.
            unsigned long long* keys = reinterpret_cast<unsigned long long*>(rec);  // n keys, then n slots
            uint32_t* newOrder = reinterpret_cast<uint32_t*>(keys + n);
            for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) {
                const uint32_t s = segOf[j];
                const uint32_t ax = s == NONE ? 255u : axisOf[s];
                keys[j] = ax == 255u ? 0ull : sortable(I.aabb[(size_t)order[j] * 9u + 6u + ax]);
            }
            __syncthreads();
            for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) {
                const uint32_t s = segOf[j];
                uint32_t dest = j;
                if (s != NONE && axisOf[s] != 255u) {
                    const uint32_t lo = cur[s].lo, hi = cur[s].hi;
                    const unsigned long long kj = keys[j];
                    uint32_t r = 0;
                    for (uint32_t q = lo; q < hi; ++q) {
                        const unsigned long long kq = keys[q];
                        r += (kq < kj || (kq == kj && q < j)) ? 1u : 0u;
                    }
                    dest = lo + r;
                }
                newOrder[dest] = order[j];
            }
            __syncthreads();
            for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) order[j] = newOrder[j];
        } else {
            // (b) sort records grouped by the first position of their segment (or by their
            // own position when finished), so every group stays inside its range; leaf
            // segments and finished positions keep their order (constant key)
            for (uint32_t j = threadIdx.x; j < P; j += blockDim.x) {
                BuildRec r;
                if (j < n) {
                    uint32_t s = segOf[j];
                    uint32_t ax = s == NONE ? 255u : axisOf[s];
                    uint32_t group = s == NONE ? j : (uint32_t)cur[s].lo;
                    r.segpos = (group << 13) | j;
                    r.key = ax == 255 ? 0ull : sortable(I.aabb[(size_t)order[j] * 9u + 6u + ax]);
                } else {
                    r.segpos = 0xFFFFFFFFu;
                    r.key = ~0ull;
                }
                r.pad = 0;
                rec[j] = r;
            }
            __syncthreads();
            // (c) bitonic sort of P records
            for (uint32_t k = 2; k <= P; k <<= 1)
                for (uint32_t jj = k >> 1; jj > 0; jj >>= 1) {
                    for (uint32_t i = threadIdx.x; i < P; i += blockDim.x) {
                        uint32_t ixj = i ^ jj;
                        if (ixj > i) {
                            bool up = (i & k) == 0;
                            BuildRec a = rec[i], b = rec[ixj];
                            bool sw = up ? rec_less(b, a) : rec_less(a, b);
                            if (sw) { rec[i] = b; rec[ixj] = a; }
                        }
                    }
                    __syncthreads();
                }
            for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) segOf[j] = order[rec[j].segpos & 0x1FFFu];
            __syncthreads();
            for (uint32_t j = threadIdx.x; j < n; j += blockDim.x) order[j] = segOf[j];
        }
        // (d) children of interior segments, in order of lo
        if (threadIdx.x == 0) {
            uint32_t m = 0;
            for (uint32_t s = 0; s < nSeg; ++s) {
                Seg sg = cur[s];
                if ((uint32_t)sg.hi - sg.lo <= 2) continue;
                uint32_t mid = ((uint32_t)sg.lo + sg.hi) >> 1;
                nxt[m++] = Seg{sg.lo, (uint16_t)mid, (uint16_t)(sg.idx + 1)};
                nxt[m++] = Seg{(uint16_t)mid, sg.hi, (uint16_t)(sg.idx + 1 + nodesTab[mid - sg.lo])};
            }
            nNext = m;
            level = level + 1;
        }
        __syncthreads();
        Seg* t = cur; cur = nxt; nxt = t;
        if (threadIdx.x == 0) nSeg = nNext;
        __syncthreads();
    }
    if (threadIdx.x == 0) *I.scratch = level - 1;
    // (e) slots: order, inverse map, instance records, live bounds
    for (uint32_t s = threadIdx.x; s < n; s += blockDim.x) {
        uint32_t src = order[s];
        I.order[s] = src;
        I.slotOf[src] = s;
        write_slot(B, I, s, src, true);
    }
}

cudaError_t launch_tlas_build(const SceneBuffers& B, const InstanceTable& I, uint32_t* err, cudaStream_t st) {
    uint32_t n = I.count;
    if (n == 0 || n > TLAS_BUILD_MAX) return cudaErrorInvalidValue;
    size_t smem = tlas_build_smem(n);
    cudaError_t e = cudaFuncSetAttribute(k_tlas_build, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    k_tlas_build<<<1, 1024, smem, st>>>(B, I, err); note_launch();
    return cudaGetLastError();
}

// ------------------------------------------------------ transform lane
// updateTransforms (spectral_scene.js:1402-1514): recompute the listed source
// instances (all when srcList is null) and write their slots, then refit the TLAS.

// compute_instance and write_slot by a warp: every operation the same, an inverse
// entry per lane, then a box corner per lane. m: 16 doubles of shared memory, corner: 24.
// Returns the slot; bounds (of lane a < 3): its liveBounds entries a and 3 + a.
__device__ uint32_t update_instance_warp(const SceneBuffers& B, const InstanceTable& I, uint32_t src,
                                         const double* world, bool rows, double* m, double* corner, float& lo,
                                         float& hi, uint32_t* err) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t root = I.blasRoot[src], end = I.blasEnd[src], slot = I.slotOf[src];
    const bool active = I.active[src];
    if (lane < 16u) {
        const double v = world ? world[lane] : I.world[(size_t)src * 16u + lane];
        if (world) I.world[(size_t)src * 16u + lane] = v;
        m[lane] = v;
    }
    __syncwarp();
    // without new matrices or rows the inverses stand as they are
    const bool inside = root < end && end <= B.nodeCount, inverse = rows || world;
    const float* nb = reinterpret_cast<const float*>(B.nodes + (size_t)(inside ? root : 0u) * 8u);
    float b[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) b[k] = nb[k];
    float row = 0.0f, sign = 1.0f;
    if (inverse) {
        const double det = det4(m);
        const double inv = __ddiv_rn(1.0, det);
        if (lane < 12u) {
            row = __double2float_rn(det == 0.0 ? 0.0 : DM(cofactor(m, (int)(lane / 4u), (int)(lane % 4u)), inv));
            I.invRows[(size_t)src * 12u + lane] = row;
        }
        sign = det < 0.0 ? -1.0f : 1.0f;
    }
    if (lane < 8u) {
        double p[3];
        transform_corner(m, (lane & 1u) ? b[3] : b[0], (lane & 2u) ? b[4] : b[1], (lane & 4u) ? b[5] : b[2], p);
        for (int a = 0; a < 3; ++a) corner[3 * lane + a] = p[a];
    }
    __syncwarp();
    if (lane == 0) {
        if (inverse) I.detSign[src] = sign;
        if (active && !inside) latch(err, ERR_LAYOUT);
    }
    lo = hi = 0.0f;
    if (lane < 3u) {
        double mn = INFINITY, mx = -INFINITY;
        if (!active) mn = mx = m[12 + lane];
        else if (!inside) mn = mx = 0.0;
        else
            for (int i = 0; i < 8; ++i) {
                const double v = corner[3 * i + lane];
                if (v < mn) mn = v;
                if (v > mx) mx = v;
            }
        double* o = I.aabb + (size_t)src * 9u + lane;
        const double mid = DM(DA(mn, mx), 0.5);
        o[0] = mn;
        o[3] = mx;
        o[6] = mid;
        if (mid != mid) latch(err, ERR_NAN_KEY);
        lo = __double2float_rn(mn);
        hi = __double2float_rn(mx);
        I.liveBounds[(size_t)slot * 6u + lane] = lo;
        I.liveBounds[(size_t)slot * 6u + 3u + lane] = hi;
    }
    if (rows) {
        const float act = active ? 1.0f : 0.0f;
        float v = row;
        if (lane == 12u) v = float(root);
        if (lane == 13u) v = float(end);
        if (lane == 14u) v = sign;
        if (lane == 15u) v = act;
        if (lane >= 16u) v = 0.0f;
        if (lane < 28u) B.materials[B.instBase + (size_t)slot * 28u + lane] = v;
        if (lane == 12u) v = __uint_as_float(root);
        if (lane == 13u) v = __uint_as_float(end);
        if (lane < 16u) reinterpret_cast<float*>(B.inst)[16u * (size_t)slot + lane] = v;
    }
    __syncwarp();
    return slot;
}

// refitFlatTlasRange over the frozen partition, deepest level first (the
// body of one CTA; the caller's writes to liveBounds precede a barrier).
// The level pass on the records in global memory (larger TLASes).
__device__ __forceinline__ void tlas_refit_levels(const SceneBuffers& B, const InstanceTable& I, uint32_t nn,
                                                  int maxDepth) {
    for (int d = maxDepth; d >= 0; --d) {
        for (uint32_t i = threadIdx.x; i < nn; i += blockDim.x) {
            if (I.nodeDepth[i] != (uint32_t)d) continue;
            float* N = B.materials + B.tlasBase + (size_t)i * 12u;
            float bx[6];
            uint32_t miss = (uint32_t)N[6];
            float cf = N[8];
            if (cf > 0.0f) {
                uint32_t off = (uint32_t)N[7], cnt = (uint32_t)cf;
                float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
                for (uint32_t s = off; s < off + cnt; ++s) {
                    const float* b = I.liveBounds + (size_t)s * 6u;
                    for (int k = 0; k < 3; ++k) {
                        if (b[k] < mn[k]) mn[k] = b[k];
                        if (b[3 + k] > mx[k]) mx[k] = b[3 + k];
                    }
                }
                for (int k = 0; k < 3; ++k) { bx[k] = mn[k]; bx[3 + k] = mx[k]; }
                write_tlas_node(B, i, bx, miss, off, cnt);
            } else {
                const float* L = B.materials + B.tlasBase + (size_t)(i + 1) * 12u;
                const float* R = B.materials + B.tlasBase + (size_t)((uint32_t)L[6]) * 12u;
                for (int k = 0; k < 3; ++k) {
                    bx[k] = js_min(L[k], R[k]);
                    bx[3 + k] = js_max(L[3 + k], R[3 + k]);
                }
                write_tlas_node(B, i, bx, miss, 0, 0);
            }
        }
        __syncthreads();
    }
}

// The traversal's child-pair copy of the refit bounds (entries are structural).
__device__ __forceinline__ void tlas_refit_pairs(const SceneBuffers& B, uint32_t nn) {
    if (!B.tlasPairs) return;
    for (uint32_t i = threadIdx.x; i < nn; i += blockDim.x) {
        uint4 b = B.tlas[2 * i + 1];
        if ((b.w >> 24) != 0u || i + 1 >= nn) continue;
        uint32_t l = i + 1, r = B.tlas[2 * l + 1].z;
        if (!(r > l && r < nn)) continue;
        uint4 la = B.tlas[2 * l], lb = B.tlas[2 * l + 1], ra = B.tlas[2 * r], rb = B.tlas[2 * r + 1];
        const uint32_t b0[6] = {la.x, la.y, la.z, la.w, lb.x, lb.y};
        const uint32_t b1[6] = {ra.x, ra.y, ra.z, ra.w, rb.x, rb.y};
        store_pair_boxes(B.tlasPairs + 4u * i, b0, b1);
    }
}

// TLASes of up to this many nodes and slots refit in shared memory.
constexpr uint32_t TLAS_STAGE = 512;
// Up to this many listed instances are updated by a warp each, more by a thread each.
constexpr uint32_t TLAS_WARPS = 16, TLAS_WARP_UPDATES = 3 * TLAS_WARPS;

// The transform lane in one CTA: the listed (or every) source instance's rows and
// bounds, then the TLAS refit over them, deepest level first.
//
// One CTA's latency bounds it: loads, the FP64 chain of an inverse and the levels. So
// the TLAS's structure and slot bounds are staged while the instances are computed (a
// warp each: a determinant, then one cofactor and one corner per lane), the levels
// run on shared memory alone, and everything is written at the end. With
// three movers in the atrium's 34 instances 6.8 us instead of 13.5.
__global__ void __launch_bounds__(32 * TLAS_WARPS) k_update_refit_tlas(SceneBuffers B, InstanceTable I,
                                                                       const uint32_t* srcList, const double* world16,
                                                                       uint32_t count, int rewriteRows,
                                                                       uint32_t* err) {
    __shared__ uint32_t sBox[6][TLAS_STAGE];
    __shared__ float sBounds[6][TLAS_STAGE];
    __shared__ uint16_t sMiss[TLAS_STAGE], sOff[TLAS_STAGE], sCnt[TLAS_STAGE], sDepth[TLAS_STAGE];
    __shared__ double sM[TLAS_WARPS][16], sCorner[TLAS_WARPS][24];
    __shared__ float sNew[6][TLAS_WARP_UPDATES];
    __shared__ uint32_t sSlot[TLAS_WARP_UPDATES];
    const uint32_t total = srcList ? count : I.count, nn = B.tlasNodeCount, slots = B.instCount;
    const int maxDepth = (int)*(volatile uint32_t*)I.scratch;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const bool staged = nn <= TLAS_STAGE && slots <= TLAS_STAGE, byWarp = total <= TLAS_WARP_UPDATES;
    // with few instances their warps start on them at once and the others stage
    const uint32_t firstStage = byWarp && total <= TLAS_WARPS / 2 ? 32u * total : 0u;
    if (staged && threadIdx.x >= firstStage) {
        const float* T = B.materials + B.tlasBase;
        const uint32_t step = blockDim.x - firstStage;
        for (uint32_t i = threadIdx.x - firstStage; i < nn; i += step) {
            const float* N = T + (size_t)i * 12u;
            sMiss[i] = (uint16_t)N[6];
            sOff[i] = (uint16_t)N[7];
            sCnt[i] = N[8] > 0.0f ? (uint16_t)N[8] : 0u;
            sDepth[i] = (uint16_t)I.nodeDepth[i];
        }
        if (byWarp)  // (else they are all read anew below)
            for (uint32_t i = threadIdx.x - firstStage; i < 6u * slots; i += step) sBounds[i % 6u][i / 6u] = I.liveBounds[i];
    }
    if (byWarp) {
        for (uint32_t i = warp; i < total; i += TLAS_WARPS) {
            const uint32_t src = srcList ? srcList[i] : i;
            if (src >= I.count) {
                if (lane == 0) {
                    latch(err, ERR_LAYOUT);
                    sSlot[i] = NONE;
                }
                continue;
            }
            float lo, hi;
            const uint32_t slot =
                update_instance_warp(B, I, src, srcList && world16 ? world16 + (size_t)i * 16u : nullptr,
                                     rewriteRows != 0, sM[warp], sCorner[warp], lo, hi, err);
            if (lane == 0) sSlot[i] = slot;
            if (lane < 3u) {
                sNew[lane][i] = lo;
                sNew[3u + lane][i] = hi;
            }
        }
    } else {
        for (uint32_t i = threadIdx.x; i < total; i += blockDim.x) {
            const uint32_t src = srcList ? srcList[i] : i;
            if (src >= I.count) {
                latch(err, ERR_LAYOUT);
                continue;
            }
            if (srcList && world16)
                for (int k = 0; k < 16; ++k) I.world[(size_t)src * 16u + k] = world16[(size_t)i * 16u + k];
            compute_instance(B, I, src, err);
            write_slot(B, I, I.slotOf[src], src, rewriteRows != 0);
        }
    }
    __syncthreads();
    if (!staged) {
        tlas_refit_levels(B, I, nn, maxDepth);
        tlas_refit_pairs(B, nn);
        return;
    }
    if (byWarp) {
        if (threadIdx.x < 6u)
            for (uint32_t i = 0; i < total; ++i)
                if (sSlot[i] < slots) sBounds[threadIdx.x][sSlot[i]] = sNew[threadIdx.x][i];
    } else {
        for (uint32_t i = threadIdx.x; i < 6u * slots; i += blockDim.x) sBounds[i % 6u][i / 6u] = I.liveBounds[i];
    }
    __syncthreads();
    for (int d = maxDepth; d >= 0; --d) {
        for (uint32_t i = threadIdx.x; i < nn; i += blockDim.x) {
            if (sDepth[i] != (uint32_t)d) continue;
            uint32_t box[6];
            const uint32_t cnt = sCnt[i];
            if (cnt > 0u) {
                float mn[3] = {INFINITY, INFINITY, INFINITY}, mx[3] = {-INFINITY, -INFINITY, -INFINITY};
                for (uint32_t s = sOff[i]; s < sOff[i] + cnt; ++s)
                    for (int k = 0; k < 3; ++k) {
                        if (sBounds[k][s] < mn[k]) mn[k] = sBounds[k][s];
                        if (sBounds[3 + k][s] > mx[k]) mx[k] = sBounds[3 + k][s];
                    }
                for (int k = 0; k < 3; ++k) {
                    box[k] = __float_as_uint(mn[k]);
                    box[3 + k] = __float_as_uint(mx[k]);
                }
            } else {
                const uint32_t l = i + 1, r = sMiss[l];
                uint32_t lb[6], rb[6];
                for (int k = 0; k < 6; ++k) {
                    lb[k] = sBox[k][l];
                    rb[k] = sBox[k][r];
                }
                join_boxes(lb, rb, box);
            }
            for (int k = 0; k < 6; ++k) sBox[k][i] = box[k];
        }
        __syncthreads();
    }
    for (uint32_t i = threadIdx.x; i < nn; i += blockDim.x) {
        if ((int)sDepth[i] > maxDepth) continue;
        float b[6];
        for (int k = 0; k < 6; ++k) b[k] = __uint_as_float(sBox[k][i]);
        write_tlas_node(B, i, b, sMiss[i], sOff[i], sCnt[i]);
        // the traversal's child-pair copy of the bounds (entries are structural)
        const uint32_t l = i + 1u;
        if (!B.tlasPairs || sCnt[i] || l >= nn || !(sMiss[l] > l && sMiss[l] < nn)) continue;
        uint32_t lb[6], rb[6];
        for (int k = 0; k < 6; ++k) {
            lb[k] = sBox[k][l];
            rb[k] = sBox[k][sMiss[l]];
        }
        store_pair_boxes(B.tlasPairs + 4u * i, lb, rb);
    }
}

// Depth of every TLAS node and the refit-index checks of
// createFlatTlasRefitIndex (gi_refit.js:298-346); one thread, structural
// changes only.
__global__ void k_tlas_index(SceneBuffers B, InstanceTable I, uint32_t* owner, uint32_t* err) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    const uint32_t nn = B.tlasNodeCount, ic = B.instCount;
    for (uint32_t i = 0; i < nn; ++i) I.nodeDepth[i] = NONE;
    for (uint32_t s = 0; s < ic; ++s) owner[s] = NONE;
    uint32_t maxD = 0;
    if (nn) I.nodeDepth[0] = 0;
    for (uint32_t i = 0; i < nn; ++i) {
        const float* N = B.materials + B.tlasBase + (size_t)i * 12u;
        uint32_t d = I.nodeDepth[i];
        if (d == NONE) { latch(err, ERR_LAYOUT); return; }
        if (d > maxD) maxD = d;
        float cf = N[8];
        if (cf > 0.0f) {
            float off = N[7];
            if (!(off >= 0.0f) || floorf(off) != off || floorf(cf) != cf || off + cf > (float)ic) {
                latch(err, ERR_LAYOUT);
                return;
            }
            for (uint32_t s = (uint32_t)off; s < (uint32_t)(off + cf); ++s) {
                if (owner[s] != NONE) { latch(err, ERR_LAYOUT); return; }
                owner[s] = i;
            }
        } else {
            uint32_t l = i + 1;
            if (l >= nn) { latch(err, ERR_LAYOUT); return; }
            float rf = B.materials[B.tlasBase + (size_t)l * 12u + 6u];
            if (floorf(rf) != rf || !(rf > (float)l && rf < (float)nn)) { latch(err, ERR_LAYOUT); return; }
            uint32_t r = (uint32_t)rf;
            if (I.nodeDepth[l] != NONE || I.nodeDepth[r] != NONE) { latch(err, ERR_LAYOUT); return; }
            I.nodeDepth[l] = d + 1;
            I.nodeDepth[r] = d + 1;
        }
    }
    for (uint32_t s = 0; s < ic; ++s)
        if (owner[s] == NONE) { latch(err, ERR_LAYOUT); return; }
    *I.scratch = maxD;
}

cudaError_t launch_update_refit_tlas(const SceneBuffers& B, const InstanceTable& I, const uint32_t* srcList,
                                     const double* world16, uint32_t count, int rewriteRows, uint32_t* err,
                                     cudaStream_t st) {
    k_update_refit_tlas<<<1, 32 * TLAS_WARPS, 0, st>>>(B, I, srcList, world16, count, rewriteRows, err); note_launch();
    return cudaGetLastError();
}

cudaError_t launch_tlas_index(const SceneBuffers& B, const InstanceTable& I, uint32_t* owner, uint32_t* err,
                              cudaStream_t st) {
    k_tlas_index<<<1, 32, 0, st>>>(B, I, owner, err); note_launch();
    return cudaGetLastError();
}

}  // namespace sb
