// wf_bvh.cu — GPU binned-SAH BLAS builder, byte-identical to the reference's
// recursive CPU builder (bvh_builder.cpp:6-264) at equal options.
//
// Why the output matches:
//  * every float is computed with the reference's operations: centroid
//    ((p0 + p1) + p2) * 0.3333f, bin (int)((c - cmin) * (bins / (cmax - cmin)))
//    clamped to bins-1, and the SAH sweep's per-plane costs (half area,
//    count * area) with the first minimum over axis 0..2, then plane
//    0..bins-2, as the reference's strict "<" picks it (one thread per node in
//    the large phase, a warp scan over the bins in the small phase);
//  * bin and node bounds are min/max reductions, whose value does not depend
//    on the order (a -0.0/+0.0 tie is the one case where the reference keeps
//    the first operand it saw; a bound holding both zero signs may differ in
//    that bit only);
//  * the reference's in-place two-pointer partition (:121-137) is not stable,
//    but its permutation has a closed form that two scans reproduce in
//    parallel.  With nL left-going triangles, p = nL + [element nL goes
//    right], front = [0, p), back = [p, count):
//       front left-goer at i                 -> i
//       back right-goer at i                 -> i - 1
//       m-th front right-goer                -> g(m-1) - 1   (g(0) = count)
//       m-th back left-goer counted from the end, g(m) -> f(m), the position
//                                               of the m-th front right-goer
//    which also reproduces the left rotation the loop applies when no plane
//    exists and every triangle "goes right";
//  * nodes are created breadth-first or per warp, then renumbered: the
//    reference allocates each split node's child pair when it visits that node
//    in pre-order, so the pair of internal node X sits at
//    2 + 2 * (pre-order rank of X among internal nodes).
//
// Phases: nodes with more than kSmall triangles are processed level by level
// by the whole grid of one cooperative launch (chunked binning into
// shared-memory bins, side bits and chunked scans for the partition); subtrees
// of at most kSmall triangles are built by one CTA each, entirely in shared
// memory; the renumbering climbs from the leaves once and from every node once.
// Nothing is read back before the tree stands.  The scratch is one allocation,
// kept for the next build when it is small; the triangles go to the device as
// they are (144 bytes each, over NVLink-C2C) and their positions are picked out
// there, and the blob's three parts are copied straight into the caller's buffer
// when it fits.
#include <algorithm>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

#include "wf_bvh.h"
#include "wf_device.cuh"

namespace wf {

namespace {

constexpr uint32_t kMaxBins = 64;
constexpr uint32_t kChunk = 1024;      // positions a block of the large-node phase takes at a time: 32 words of side bits
constexpr uint32_t kChunkThreads = 256;
static_assert(kChunk == 1024 && kChunkThreads == 256, "a warp holds four of a chunk's 32 words");
#ifndef WF_BVH_SMALL
#define WF_BVH_SMALL 128
#endif
constexpr uint32_t kSmall = WF_BVH_SMALL;   // subtrees at most this large are built by one warp
static_assert(kSmall >= 32 && kSmall <= 65536, "16-bit local positions");
constexpr uint32_t kNone = 0xFFFFFFFFu;
constexpr uint32_t kBinWords = 7;      // count, min xyz, max xyz (order-preserving keys)
constexpr uint32_t kBoxWords = 18;     // node min/max, centroid min/max keys, first-zero positions

thread_local std::string g_err;

// Order-preserving float <-> uint32 keys for atomicMin / atomicMax.
__device__ __forceinline__ uint32_t fenc(float f) {
    uint32_t b = __float_as_uint(f);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float fdec(uint32_t k) { return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k); }
// glm::min / glm::max (func_common.inl:17-35)
__device__ __forceinline__ float gmin(float x, float y) { return (y < x) ? y : x; }
__device__ __forceinline__ float gmax(float x, float y) { return (x < y) ? y : x; }
__device__ __forceinline__ float half_area(const float* mn, const float* mx) {
    float ex = mx[0] - mn[0], ey = mx[1] - mn[1], ez = mx[2] - mn[2];
    return ex * ey + ey * ez + ez * ex;
}
__device__ __forceinline__ float comp(float4 v, uint32_t a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }

struct Ctx {
    uint32_t n, bins, single, max_leaf;
    const float* pos;        // 9 floats per triangle (original order)
    float4* cen;             // centroid
    float4* tmn;             // triangle min corner
    float4* tmx;             // triangle max corner
    uint32_t* idx[2];        // index permutation: a node at depth d has its range in idx[d & 1]; the leaves'
                             // ranges end in idx[0]
    uint32_t* F;             // per-position scratch: front right-goers by rank
    uint32_t* G;             // per-position scratch: back left-goers by rank
    float4* ta;              // temporary nodes {min xyz, first}
    float4* tb;              //                 {max xyz, count}
    uint32_t* tleft;         // left child (kNone for leaves); right child = left + 1
    uint32_t* tparent;
    uint32_t* tdepth;
    uint32_t* tcount;        // [0] nodes allocated, [1] internal nodes, [2] small roots, [3] error
    uint32_t* small_list;
};

// Split plan of one node, shared by the large and the small phase.
struct Plan {
    uint32_t axis, pos, nl, p, partition, children;
    float lo, scale;
};

// c = the triangle's centroid component on P.axis.
__device__ __forceinline__ bool goes_left_c(const Ctx& C, const Plan& P, float c) {
    if (P.pos == 0) return false;
    int32_t bin = (int32_t)((c - P.lo) * P.scale);
    if ((int32_t)C.bins - 1 < bin) bin = (int32_t)C.bins - 1;
    return (uint32_t)bin < P.pos;
}
__device__ __forceinline__ bool goes_left(const Ctx& C, const Plan& P, uint32_t t) {
    return goes_left_c(C, P, comp(C.cen[t], P.axis));
}

// find_best_split_plane's sweep (bvh_builder.cpp:196-249) by one warp over bins
// laid out [axis][bin][count, min xyz key, max xyz key]: every lane returns the
// same (cheapest, axis, pos) and nl = the triangles in bins [0, pos).  Lane l
// holds bins [q*l, q*l + q) (q = 1 for up to 32 bins, else 2); shuffle scans
// give each plane its left prefix and right suffix.  Prefix and suffix boxes
// are min/max folds and counts are integer sums, so every plane's box, area
// and cost are the same floats the sequential sweep computes (a bound that
// folds -0.0 with +0.0 may keep the other zero, which changes no area); the
// first minimum in (axis, plane) order wins, as with the strict "<".
__device__ float warp_sweep(const uint32_t* bins, uint32_t B, const float* cmn, const float* cmx, uint32_t lane,
                            uint32_t& axis, uint32_t& pos, uint32_t& nl) {
    float cheapest = FLT_MAX;
    axis = 0;
    pos = 0;
    nl = 0;
    const uint32_t q = (B + 31) >> 5;
    for (uint32_t a = 0; a < 3; ++a) {
        if (cmn[a] == cmx[a]) continue;
        const uint32_t* ab = bins + a * B * kBinWords;
        uint32_t cnt[2];
        float bmn[2][3], bmx[2][3];
        for (uint32_t k = 0; k < 2; ++k) {
            const uint32_t j = lane * q + k;
            const bool have = k < q && j < B;
            const uint32_t* e = ab + j * kBinWords;
            cnt[k] = have ? e[0] : 0u;
            for (int c = 0; c < 3; ++c) {
                bmn[k][c] = have ? fdec(e[1 + c]) : FLT_MAX;
                bmx[k][c] = have ? fdec(e[4 + c]) : -FLT_MAX;
            }
        }
        // lane totals, then inclusive scans up (prefix) and down (suffix)
        uint32_t pc = cnt[0] + cnt[1], sc = pc;
        float pmn[3], pmx[3], smn[3], smx[3];
        for (int c = 0; c < 3; ++c) {
            pmn[c] = smn[c] = gmin(bmn[0][c], bmn[1][c]);
            pmx[c] = smx[c] = gmax(bmx[0][c], bmx[1][c]);
        }
        for (uint32_t off = 1; off < 32; off <<= 1) {
            const uint32_t oc = __shfl_up_sync(0xffffffffu, pc, off), uc = __shfl_down_sync(0xffffffffu, sc, off);
            float omn[3], omx[3], umn[3], umx[3];
            for (int c = 0; c < 3; ++c) {
                omn[c] = __shfl_up_sync(0xffffffffu, pmn[c], off);
                omx[c] = __shfl_up_sync(0xffffffffu, pmx[c], off);
                umn[c] = __shfl_down_sync(0xffffffffu, smn[c], off);
                umx[c] = __shfl_down_sync(0xffffffffu, smx[c], off);
            }
            if (lane >= off) {
                pc += oc;
                for (int c = 0; c < 3; ++c) { pmn[c] = gmin(pmn[c], omn[c]); pmx[c] = gmax(pmx[c], omx[c]); }
            }
            if (lane + off < 32) {
                sc += uc;
                for (int c = 0; c < 3; ++c) { smn[c] = gmin(smn[c], umn[c]); smx[c] = gmax(smx[c], umx[c]); }
            }
        }
        // exclusive: lanes below (prefix) and above (suffix)
        uint32_t ec = __shfl_up_sync(0xffffffffu, pc, 1), xc = __shfl_down_sync(0xffffffffu, sc, 1);
        float emn[3], emx[3], xmn[3], xmx[3];
        for (int c = 0; c < 3; ++c) {
            emn[c] = __shfl_up_sync(0xffffffffu, pmn[c], 1);
            emx[c] = __shfl_up_sync(0xffffffffu, pmx[c], 1);
            xmn[c] = __shfl_down_sync(0xffffffffu, smn[c], 1);
            xmx[c] = __shfl_down_sync(0xffffffffu, smx[c], 1);
        }
        if (lane == 0) {
            ec = 0;
            for (int c = 0; c < 3; ++c) { emn[c] = FLT_MAX; emx[c] = -FLT_MAX; }
        }
        if (lane == 31) {
            xc = 0;
            for (int c = 0; c < 3; ++c) { xmn[c] = FLT_MAX; xmx[c] = -FLT_MAX; }
        }
        // planes j (between bin j and j + 1) held by this lane, first minimum
        float bc = INFINITY;
        uint32_t bi = 0xFFFFFFFFu, bl = 0;
        for (uint32_t k = 0; k < 2; ++k) {
            const uint32_t j = lane * q + k;
            if (k >= q || j + 1 >= B) continue;
            uint32_t lc = ec + cnt[0], rc = xc;
            float lmn[3], lmx[3], rmn[3], rmx[3];
            for (int c = 0; c < 3; ++c) {
                lmn[c] = gmin(emn[c], bmn[0][c]);
                lmx[c] = gmax(emx[c], bmx[0][c]);
                rmn[c] = xmn[c];
                rmx[c] = xmx[c];
            }
            if (k == 1) {
                lc += cnt[1];
                for (int c = 0; c < 3; ++c) { lmn[c] = gmin(lmn[c], bmn[1][c]); lmx[c] = gmax(lmx[c], bmx[1][c]); }
            } else if (q == 2) {
                rc += cnt[1];
                for (int c = 0; c < 3; ++c) { rmn[c] = gmin(rmn[c], bmn[1][c]); rmx[c] = gmax(rmx[c], bmx[1][c]); }
            }
            const float cost = (float)lc * half_area(lmn, lmx) + (float)rc * half_area(rmn, rmx);
            if (cost < FLT_MAX && cost < bc) { bc = cost; bi = j; bl = lc; }
        }
        for (uint32_t off = 16; off > 0; off >>= 1) {
            const float oc = __shfl_xor_sync(0xffffffffu, bc, off);
            const uint32_t oi = __shfl_xor_sync(0xffffffffu, bi, off), ol = __shfl_xor_sync(0xffffffffu, bl, off);
            if (oc < bc || (oc == bc && oi < bi)) { bc = oc; bi = oi; bl = ol; }
        }
        if (bc < cheapest) { axis = a; pos = bi + 1; cheapest = bc; nl = bl; }
    }
    return cheapest;
}

// The plan of a node from its cheapest plane (p placed only where every
// triangle goes one way).
__device__ __forceinline__ Plan plan_from(const Ctx& C, float cost, uint32_t axis, uint32_t pos, uint32_t nl,
                                          uint32_t count, const float* nmn, const float* nmx, const float* cmn,
                                          const float* cmx) {
    Plan P{};
    bool leaf;
    if (C.single) {
        leaf = count == 1;
    } else {
        bool force = C.max_leaf > 0 && count > C.max_leaf;
        float parent = (float)count * half_area(nmn, nmx);
        leaf = !force && cost >= parent;
    }
    P.axis = axis;
    P.pos = pos;
    P.partition = leaf ? 0u : 1u;
    if (leaf) return P;
    const float lo = axis == 0 ? cmn[0] : axis == 1 ? cmn[1] : cmn[2], hi = axis == 0 ? cmx[0] : axis == 1 ? cmx[1] : cmx[2];
    P.lo = lo;
    P.scale = pos > 0 ? (float)C.bins / (hi - lo) : 0.0f;
    P.nl = pos > 0 ? nl : 0u;
    P.p = count;
    P.children = (P.nl > 0 && P.nl < count) ? 1u : 0u;
    return P;
}

// Destination of local position i (closed form of the two-pointer loop).
__device__ __forceinline__ uint32_t partition_dst(const Ctx& C, const Plan& P, uint32_t first, uint32_t count,
                                                  uint32_t i, bool left, uint32_t lpre) {
    if (i < P.p) {
        if (left) return i;
        uint32_t m = i - lpre + 1;
        return (m == 1 ? count : C.G[first + m - 2]) - 1;
    }
    if (!left) return i - 1;
    uint32_t m = P.nl - lpre;
    return C.F[first + m - 1];
}

__device__ __forceinline__ void partition_rank(const Ctx& C, const Plan& P, uint32_t first, uint32_t i, bool left,
                                               uint32_t lpre) {
    if (i < P.p && !left) {
        C.F[first + (i - lpre)] = i;               // m = i - lpre + 1
    } else if (i >= P.p && left) {
        C.G[first + (P.nl - lpre) - 1] = i;        // m = nL - lpre
    }
}

// ---------------------------------------------------------------- bounds
__device__ __forceinline__ void box_init(float* v) {
    for (int k = 0; k < 3; ++k) { v[k] = FLT_MAX; v[3 + k] = -FLT_MAX; v[6 + k] = FLT_MAX; v[9 + k] = -FLT_MAX; }
}
__device__ __forceinline__ void box_add(float* v, const Ctx& C, uint32_t t) {
    float4 mn = C.tmn[t], mx = C.tmx[t], c = C.cen[t];
    v[0] = gmin(v[0], mn.x); v[1] = gmin(v[1], mn.y); v[2] = gmin(v[2], mn.z);
    v[3] = gmax(v[3], mx.x); v[4] = gmax(v[4], mx.y); v[5] = gmax(v[5], mx.z);
    v[6] = gmin(v[6], c.x); v[7] = gmin(v[7], c.y); v[8] = gmin(v[8], c.z);
    v[9] = gmax(v[9], c.x); v[10] = gmax(v[10], c.y); v[11] = gmax(v[11], c.z);
}
// Signed zeros.  A bound equal to zero is +0.0 or -0.0 in the reference
// depending on which zero its glm fold met first (calc_node_min_max walks the
// node's triangles in index-list order and keeps the running value on ties).
// Alongside the value reductions the builder records, per box component, the
// first index-list position whose triangle bound is zero; a zero result takes
// that triangle's bits.
__device__ __forceinline__ float tri_comp(const Ctx& C, uint32_t t, int k) {
    const float4 v = k < 3 ? C.tmn[t] : C.tmx[t];
    return comp(v, (uint32_t)(k % 3));
}
__device__ __forceinline__ void zero_init(uint32_t* zp) {
    for (int k = 0; k < 6; ++k) zp[k] = kNone;
}
__device__ __forceinline__ void zero_add(uint32_t* zp, const Ctx& C, uint32_t t, uint32_t position) {
    const float4 mn = C.tmn[t], mx = C.tmx[t];
    const float v[6] = {mn.x, mn.y, mn.z, mx.x, mx.y, mx.z};
    for (int k = 0; k < 6; ++k)
        if (v[k] == 0.0f) zp[k] = min(zp[k], position);   // positions come in any order
}
__device__ __forceinline__ void zero_fix(const Ctx& C, const uint32_t* idx, float* v, const uint32_t* zp) {
    for (int k = 0; k < 6; ++k)
        if (v[k] == 0.0f && zp[k] != kNone) v[k] = tri_comp(C, idx[zp[k]], k);
}
// Warp-wide bounds from per-lane folds: v = node min / max, centroid min / max.
__device__ __forceinline__ void box_warp_redux(float* v) {
#pragma unroll
    for (int k = 0; k < 12; ++k)
        v[k] = fdec((k % 6) < 3 ? __reduce_min_sync(0xffffffffu, fenc(v[k])) : __reduce_max_sync(0xffffffffu, fenc(v[k])));
}
// A warp's folds into a box's keys (shared or global memory).  Only a warp whose
// own bound is zero can hold the first zero of a zero bound.
__device__ __forceinline__ void box_warp_atomic(uint32_t* keys, float* v, const uint32_t* zp, uint32_t lane) {
    box_warp_redux(v);
#pragma unroll
    for (int k = 0; k < 12; ++k) {
        if (lane == (uint32_t)k) {
            if ((k % 6) < 3) atomicMin(&keys[k], fenc(v[k]));
            else atomicMax(&keys[k], fenc(v[k]));
        }
    }
#pragma unroll
    for (int k = 0; k < 6; ++k) {
        if (v[k] == 0.0f) {
            const uint32_t z = __reduce_min_sync(0xffffffffu, zp[k]);
            if (lane == 0 && z != kNone) atomicMin(&keys[12 + k], z);
        }
    }
}
__device__ __forceinline__ void box_merge(uint32_t* to, uint32_t key, uint32_t k) {
    if (k >= 12 || (k % 6) < 3) atomicMin(&to[k], key);
    else atomicMax(&to[k], key);
}

__device__ __forceinline__ uint32_t key_init(uint32_t k) {
    return k >= 12 ? kNone : (((k % 6) < 3) ? fenc(FLT_MAX) : fenc(-FLT_MAX));
}

__device__ __forceinline__ void bins_reset(uint32_t* sb, uint32_t words, uint32_t tid, uint32_t nthreads) {
    for (uint32_t w = tid; w < words; w += nthreads) {
        uint32_t k = w % kBinWords;
        sb[w] = k == 0 ? 0u : (k < 4 ? fenc(FLT_MAX) : fenc(-FLT_MAX));
    }
}

// ---------------------------------------------------------------- large-node phase
// Nodes of more than kSmall triangles, level by level, in one cooperative
// launch: each step of a level (bins, plans, sides, ranks, move) is a phase of
// the grid, with a grid-wide barrier after it.  Bound by the barriers and the
// latency of a step where a level has few chunks, by the partition's scattered
// reads (centroid, box) where it has many.  A launch per step (12 per level),
// with the level's node count read back by the host, took about 100 us per
// level however few triangles it had; us per wf_bvh_build, so / in one launch,
// with the renumbering below: 80 triangles 296 / 190, 1,280: 672 / 356, 20,480:
// 1,634 / 851, 100,820: 2,684 / 1,560, 499,280: 7,423 / 6,180 (1.00 ms of it
// k_large, 0.98 k_small, most of the rest the host's; 4,450 to 6,000 by the state
// of the caller's output pages since the positions are picked out on the GPU).
//
// A slot is a node of the level, a chunk kChunk consecutive positions of one
// slot; a block takes chunks in turn.  Slots and chunks of the next level are
// numbered as their parents are planned (their order changes nothing).
struct Large {
    uint32_t* slot_tmp[2];      // by level parity: node id per slot
    uint32_t* slot_box[2];      // kBoxWords keys per slot
    uint32_t* slot_done[2];     // 1: nothing left but to end in idx[0]
    uint32_t* slot_chunk[2];    // first chunk per slot
    uint32_t* chunk_slot[2];
    Plan* plan;                 // per slot
    uint32_t* child_slot;       // per slot x 2: next-level slot or kNone
    uint32_t* bins;             // slot x 3 x B x 7
    uint32_t* chunk_l;          // left-goers per chunk
    uint32_t* side;             // 32 words per chunk: bit = the position's triangle goes left
    uint32_t* cnt;              // [0..1] slots, [2..3] chunks by parity, [4] arrivals at the barrier
};

// Everything a build starts from (one block): the root as node 0 and, when it
// is large, as the first level's slot.
__global__ void k_init(Ctx C, Large G) {
    const uint32_t t = threadIdx.x, nch = (C.n + kChunk - 1) / kChunk;
    const bool large = C.n > kSmall;
    if (t == 0) {
        C.ta[0] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(0u));
        C.tb[0] = make_float4(0.0f, 0.0f, 0.0f, __uint_as_float(C.n));
        C.tleft[0] = kNone;
        C.tparent[0] = 0u;
        C.tdepth[0] = 0u;
        C.tcount[0] = 1u; C.tcount[1] = 0u; C.tcount[2] = large ? 0u : 1u; C.tcount[3] = 0u;
        C.small_list[0] = 0u;
        G.slot_tmp[0][0] = 0u; G.slot_done[0][0] = 0u; G.slot_chunk[0][0] = 0u;
        G.cnt[0] = large ? 1u : 0u; G.cnt[1] = 0u; G.cnt[2] = large ? nch : 0u; G.cnt[3] = 0u; G.cnt[4] = 0u;
    }
    if (t < kBoxWords) G.slot_box[0][t] = key_init(t);
    if (!large) return;
    for (uint32_t k = t; k < nch; k += blockDim.x) G.chunk_slot[0][k] = 0u;
    bins_reset(G.bins, 3 * C.bins * kBinWords, t, blockDim.x);
}

// Positions {v0, v1, v2} of m triangle_t (three 48-byte vertices each).
__global__ void k_gather(const float4* __restrict__ tris, uint32_t m, float* __restrict__ pos) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t q = blockIdx.x * blockDim.x + threadIdx.x; q < 3 * m; q += stride) {
        const float4 p = tris[3ull * q];
        pos[3ull * q] = p.x; pos[3ull * q + 1] = p.y; pos[3ull * q + 2] = p.z;
    }
}

// Centroid and box per triangle, and the root's bounds.
__global__ void __launch_bounds__(256) k_prep(Ctx C, uint32_t* root_box) {
    __shared__ uint32_t s_box[kBoxWords];
    if (threadIdx.x < kBoxWords) s_box[threadIdx.x] = key_init(threadIdx.x);
    __syncthreads();
    float v[12];
    uint32_t zp[6];
    box_init(v);
    zero_init(zp);
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < C.n; t += stride) {
        const float* p = C.pos + 9ull * t;
        float c[3], mn[3], mx[3];
        for (int a = 0; a < 3; ++a) {
            float p0 = p[a], p1 = p[3 + a], p2 = p[6 + a];
            c[a] = ((p0 + p1) + p2) * 0.3333f;
            mn[a] = gmin(gmin(p0, p1), p2);
            mx[a] = gmax(gmax(p0, p1), p2);
            v[a] = fminf(v[a], mn[a]);
            v[3 + a] = fmaxf(v[3 + a], mx[a]);
            v[6 + a] = fminf(v[6 + a], c[a]);
            v[9 + a] = fmaxf(v[9 + a], c[a]);
            if (mn[a] == 0.0f && zp[a] == kNone) zp[a] = t;
            if (mx[a] == 0.0f && zp[3 + a] == kNone) zp[3 + a] = t;
        }
        C.cen[t] = make_float4(c[0], c[1], c[2], 0.0f);
        C.tmn[t] = make_float4(mn[0], mn[1], mn[2], 0.0f);
        C.tmx[t] = make_float4(mx[0], mx[1], mx[2], 0.0f);
        C.idx[0][t] = t;
    }
    if (!root_box) return;
    box_warp_atomic(s_box, v, zp, threadIdx.x & 31u);
    __syncthreads();
    if (threadIdx.x < kBoxWords) box_merge(root_box, s_box[threadIdx.x], threadIdx.x);
}

// All blocks of the (cooperative) grid; false once it waited too long, which a
// correct run never does: the build then ends with an error.
__device__ bool grid_barrier(uint32_t* arrivals, uint32_t* error, uint32_t& round) {
    __shared__ uint32_t s_ok;
    __syncthreads();
    ++round;
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(arrivals, 1u);
        const uint32_t target = round * gridDim.x;
        uint32_t ok = 1u, spins = 0;
        while ((int32_t)(*(volatile uint32_t*)arrivals - target) < 0) {
            if (++spins > (1u << 22) || *(volatile uint32_t*)error) {
                atomicOr(error, 2u);
                ok = 0u;
                break;
            }
            __nanosleep(32);
        }
        __threadfence();
        s_ok = ok;
    }
    __syncthreads();
    return s_ok != 0u;
}

// A chunk: its slot and positions [i0, i1) of the slot's [first, first + count).
struct Chunk {
    uint32_t slot, first, count, i0, i1;
};
__device__ __forceinline__ Chunk chunk_of(const Ctx& C, const Large& G, uint32_t cur, uint32_t b) {
    Chunk k;
    k.slot = G.chunk_slot[cur][b];
    const uint32_t t = G.slot_tmp[cur][k.slot];
    k.first = __float_as_uint(C.ta[t].w);
    k.count = __float_as_uint(C.tb[t].w);
    k.i0 = (b - G.slot_chunk[cur][k.slot]) * kChunk;
    k.i1 = min(k.count, k.i0 + kChunk);
    return k;
}

__device__ __forceinline__ void bin_element(const Ctx& C, uint32_t* sb, uint32_t t, const bool* deg, const float* lo,
                                            const float* scale) {
    const float4 c = C.cen[t], mn = C.tmn[t], mx = C.tmx[t];
    for (uint32_t a = 0; a < 3; ++a) {
        if (deg[a]) continue;
        int32_t bin = (int32_t)((comp(c, a) - lo[a]) * scale[a]);
        if ((int32_t)C.bins - 1 < bin) bin = (int32_t)C.bins - 1;
        uint32_t* e = sb + (a * C.bins + (uint32_t)bin) * kBinWords;
        atomicAdd(&e[0], 1u);
        atomicMin(&e[1], fenc(mn.x)); atomicMin(&e[2], fenc(mn.y)); atomicMin(&e[3], fenc(mn.z));
        atomicMax(&e[4], fenc(mx.x)); atomicMax(&e[5], fenc(mx.y)); atomicMax(&e[6], fenc(mx.z));
    }
}

// A chunk's bins, summed in shared memory and merged into its slot's.
__device__ __forceinline__ void bin_chunk(const Ctx& C, const Large& G, uint32_t cur, const uint32_t* idx, uint32_t b,
                                          uint32_t* sb) {
    const Chunk k = chunk_of(C, G, cur, b);
    if (G.slot_done[cur][k.slot]) return;
    const uint32_t* key = G.slot_box[cur] + kBoxWords * k.slot;
    bool deg[3];
    float lo[3], scale[3];
    for (int a = 0; a < 3; ++a) {
        lo[a] = fdec(key[6 + a]);
        float hi = fdec(key[9 + a]);
        deg[a] = lo[a] == hi;
        scale[a] = deg[a] ? 0.0f : (float)C.bins / (hi - lo[a]);
    }
    const uint32_t words = 3 * C.bins * kBinWords;
    bins_reset(sb, words, threadIdx.x, blockDim.x);
    __syncthreads();
    for (uint32_t i = k.i0 + threadIdx.x; i < k.i1; i += blockDim.x) bin_element(C, sb, idx[k.first + i], deg, lo, scale);
    __syncthreads();
    uint32_t* gb = G.bins + (size_t)k.slot * words;
    for (uint32_t w = threadIdx.x; w < words; w += blockDim.x) {
        const uint32_t q = w % kBinWords, e = w - q;
        if (sb[e] == 0u) continue;   // an empty bin (or a degenerate axis)
        if (q == 0) atomicAdd(&gb[w], sb[w]);
        else if (q < 4) atomicMin(&gb[w], sb[w]);
        else atomicMax(&gb[w], sb[w]);
    }
    __syncthreads();
}

// One warp: a slot's plan, its children and, where they are large, their slots
// and chunks at the next level.
__device__ __forceinline__ void plan_slot(const Ctx& C, const Large& G, uint32_t cur, const uint32_t* idx, uint32_t s,
                                          uint32_t lane) {
    const uint32_t nxt = cur ^ 1u, X = G.slot_tmp[cur][s];
    const uint32_t first = __float_as_uint(C.ta[X].w), count = __float_as_uint(C.tb[X].w);
    Plan P{};
    uint32_t cs[2] = {kNone, kNone};
    // slot j of the next level: node Y with c triangles
    auto add_slot = [&](uint32_t Y, uint32_t c, uint32_t done) -> uint32_t {
        const uint32_t nch = (c + kChunk - 1) / kChunk;
        uint32_t j = 0, base = 0;
        if (lane == 0) {
            j = atomicAdd(&G.cnt[nxt], 1u);
            base = atomicAdd(&G.cnt[2 + nxt], nch);
            G.slot_tmp[nxt][j] = Y;
            G.slot_done[nxt][j] = done;
            G.slot_chunk[nxt][j] = base;
        }
        j = __shfl_sync(0xffffffffu, j, 0);
        base = __shfl_sync(0xffffffffu, base, 0);
        if (lane < kBoxWords) G.slot_box[nxt][kBoxWords * j + lane] = key_init(lane);
        for (uint32_t q = lane; q < nch; q += 32) G.chunk_slot[nxt][base + q] = j;
        return j;
    };
    if (!G.slot_done[cur][s]) {
        const uint32_t* key = G.slot_box[cur] + kBoxWords * s;
        float box[6], cmn[3], cmx[3];
        for (int a = 0; a < 3; ++a) {
            box[a] = fdec(key[a]); box[3 + a] = fdec(key[3 + a]);
            cmn[a] = fdec(key[6 + a]); cmx[a] = fdec(key[9 + a]);
        }
        zero_fix(C, idx, box, key + 12);
        uint32_t axis, pos, nl;
        const float cost = warp_sweep(G.bins + (size_t)s * 3 * C.bins * kBinWords, C.bins, cmn, cmx, lane, axis, pos, nl);
        P = plan_from(C, cost, axis, pos, nl, count, box, box + 3, cmn, cmx);
        // the element at position nl decides where the front part ends
        if (P.partition && P.nl < count) P.p = P.nl + (goes_left(C, P, idx[first + P.nl]) ? 0u : 1u);
        if (lane == 0) {
            C.ta[X] = make_float4(box[0], box[1], box[2], __uint_as_float(first));
            C.tb[X] = make_float4(box[3], box[4], box[5], __uint_as_float(count));
        }
        if (P.children) {
            uint32_t L = 0;
            if (lane == 0) {
                L = atomicAdd(&C.tcount[0], 2u);
                const uint32_t d = C.tdepth[X] + 1;
                for (uint32_t q = 0; q < 2; ++q) {
                    C.ta[L + q] = make_float4(0, 0, 0, __uint_as_float(q ? first + P.nl : first));
                    C.tb[L + q] = make_float4(0, 0, 0, __uint_as_float(q ? count - P.nl : P.nl));
                    C.tleft[L + q] = kNone;
                    C.tparent[L + q] = X;
                    C.tdepth[L + q] = d;
                }
                C.tleft[X] = L;
            }
            L = __shfl_sync(0xffffffffu, L, 0);
            for (uint32_t q = 0; q < 2; ++q) {
                const uint32_t c = q ? count - P.nl : P.nl;
                if (c > kSmall) cs[q] = add_slot(L + q, c, 0u);
                else if (lane == 0) C.small_list[atomicAdd(&C.tcount[2], 1u)] = L + q;
            }
        } else if (P.partition && cur == 0u) {
            // a rotated leaf lands in idx[1]: the next level moves it back
            add_slot(X, count, 1u);
        }
    }
    if (lane == 0) {
        G.plan[s] = P;
        G.child_slot[2 * s] = cs[0];
        G.child_slot[2 * s + 1] = cs[1];
    }
}

// A chunk's side bits and its left-goers.
__device__ __forceinline__ void side_chunk(const Ctx& C, const Large& G, uint32_t cur, const uint32_t* idx, uint32_t b,
                                           uint32_t* s_w) {
    const Chunk k = chunk_of(C, G, cur, b);
    const Plan P = G.plan[k.slot];
    if (!P.partition) return;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t sum = 0;
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
        const uint32_t w = 4 * warp + r, i = k.i0 + 32 * w + lane;
        const unsigned m = __ballot_sync(0xffffffffu, i < k.i1 && goes_left(C, P, idx[k.first + i]));
        if (lane == 0) G.side[32 * (size_t)b + w] = m;
        sum += __popc(m);
    }
    if (lane == 0) s_w[warp] = sum;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t all = 0;
        for (uint32_t w = 0; w < kChunkThreads / 32; ++w) all += s_w[w];
        G.chunk_l[b] = all;
    }
    __syncthreads();
}

// Ranks (MOVE = false) or destinations (true) of a chunk's positions; moving,
// the bounds of the large children too.  A slot that is not partitioned and
// lies in idx[1] is copied to idx[0].
template <bool MOVE>
__device__ __forceinline__ void part_chunk(const Ctx& C, const Large& G, uint32_t cur, uint32_t b, uint32_t (*s_box)[kBoxWords]) {
    const Chunk k = chunk_of(C, G, cur, b);
    const Plan P = G.plan[k.slot];
    const uint32_t* from = cur ? C.idx[1] : C.idx[0];
    uint32_t* to = cur ? C.idx[0] : C.idx[1];
    if (!P.partition) {
        if (MOVE && cur)
            for (uint32_t i = k.i0 + threadIdx.x; i < k.i1; i += blockDim.x) to[k.first + i] = from[k.first + i];
        return;
    }
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    // left-goers before the chunk, then before each of its 32 words
    uint32_t pre = 0;
    for (uint32_t q = G.slot_chunk[cur][k.slot] + lane; q < b; q += 32) pre += G.chunk_l[q];
    pre = __reduce_add_sync(0xffffffffu, pre);
    const uint32_t word = G.side[32 * (size_t)b + lane];
    uint32_t incl = __popc(word);
    for (uint32_t off = 1; off < 32; off <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, incl, off);
        if (lane >= off) incl += o;
    }
    const uint32_t before = pre + incl - __popc(word);
    uint32_t j0 = kNone, j1 = kNone;
    if (MOVE) { j0 = G.child_slot[2 * k.slot]; j1 = G.child_slot[2 * k.slot + 1]; }
    const bool bounds = j0 != kNone || j1 != kNone;
    if (MOVE && bounds) {
        if (threadIdx.x < 2 * kBoxWords) s_box[threadIdx.x / kBoxWords][threadIdx.x % kBoxWords] = key_init(threadIdx.x % kBoxWords);
        __syncthreads();
    }
    float v0[12], v1[12];
    uint32_t z0[6], z1[6];
    box_init(v0);
    box_init(v1);
    zero_init(z0);
    zero_init(z1);
#pragma unroll
    for (uint32_t r = 0; r < 4; ++r) {
        const uint32_t w = 4 * warp + r, i = k.i0 + 32 * w + lane;
        const unsigned m = __shfl_sync(0xffffffffu, word, w);
        const uint32_t lpre = __shfl_sync(0xffffffffu, before, w) + __popc(m & ((1u << lane) - 1u));
        if (i >= k.i1) continue;
        const bool left = (m >> lane) & 1u;
        if (!MOVE) {
            partition_rank(C, P, k.first, i, left, lpre);
            continue;
        }
        const uint32_t t = from[k.first + i], dst = partition_dst(C, P, k.first, k.count, i, left, lpre);
        to[k.first + dst] = t;
        if (dst < P.nl) {
            if (j0 != kNone) { box_add(v0, C, t); zero_add(z0, C, t, k.first + dst); }
        } else if (j1 != kNone) {
            box_add(v1, C, t);
            zero_add(z1, C, t, k.first + dst);
        }
    }
    if (MOVE && bounds) {
        __syncwarp();
        if (j0 != kNone) box_warp_atomic(s_box[0], v0, z0, lane);
        if (j1 != kNone) box_warp_atomic(s_box[1], v1, z1, lane);
        __syncthreads();
        if (threadIdx.x < 2 * kBoxWords) {
            const uint32_t side = threadIdx.x / kBoxWords, q = threadIdx.x % kBoxWords, j = side ? j1 : j0;
            if (j != kNone && s_box[side][q] != key_init(q)) box_merge(G.slot_box[cur ^ 1u] + kBoxWords * j, s_box[side][q], q);
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(kChunkThreads) k_large(Ctx C, Large G) {
    __shared__ uint32_t s_bins[3 * kMaxBins * kBinWords];
    __shared__ uint32_t s_w[kChunkThreads / 32];
    __shared__ uint32_t s_box[2][kBoxWords];
    const uint32_t lane = threadIdx.x & 31u, words = 3 * C.bins * kBinWords;
    uint32_t cur = 0, round = 0;
    for (;;) {
        const uint32_t nslots = G.cnt[cur], nchunks = G.cnt[2 + cur], nxt = cur ^ 1u;
        if (nslots == 0u) return;
        const uint32_t* idx = cur ? C.idx[1] : C.idx[0];
        for (uint32_t b = blockIdx.x; b < nchunks; b += gridDim.x) bin_chunk(C, G, cur, idx, b, s_bins);
        if (blockIdx.x == 0 && threadIdx.x == 0) { G.cnt[nxt] = 0u; G.cnt[2 + nxt] = 0u; }
        if (!grid_barrier(&G.cnt[4], &C.tcount[3], round)) return;
        for (uint32_t s = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; s < nslots; s += (gridDim.x * blockDim.x) >> 5)
            plan_slot(C, G, cur, idx, s, lane);
        if (!grid_barrier(&G.cnt[4], &C.tcount[3], round)) return;
        const uint32_t nnext = G.cnt[nxt];
        for (uint32_t b = blockIdx.x; b < nchunks; b += gridDim.x) side_chunk(C, G, cur, idx, b, s_w);
        for (uint32_t s = blockIdx.x; s < nnext; s += gridDim.x)
            bins_reset(G.bins + (size_t)s * words, words, threadIdx.x, blockDim.x);
        if (!grid_barrier(&G.cnt[4], &C.tcount[3], round)) return;
        for (uint32_t b = blockIdx.x; b < nchunks; b += gridDim.x) part_chunk<false>(C, G, cur, b, s_box);
        if (!grid_barrier(&G.cnt[4], &C.tcount[3], round)) return;
        for (uint32_t b = blockIdx.x; b < nchunks; b += gridDim.x) part_chunk<true>(C, G, cur, b, s_box);
        if (!grid_barrier(&G.cnt[4], &C.tcount[3], round)) return;
        cur = nxt;
    }
}

// ---------------------------------------------------------------- small-subtree phase
// One CTA of kSmallWarps warps builds a whole subtree of at most kSmall
// triangles with the subtree held in shared memory: each triangle's centroid,
// min and max corner (component k of local triangle j at d[k * kSmall + j]),
// its index, and a 16-bit permutation of local triangles that the partitions
// reorder.  The subtree grows level by level: a warp per node, the children
// listed for the next level, one barrier between levels.  Only the node records
// and the final index list go to global memory.  Node ids come from one
// reservation of 2 * (count - 1) per subtree (a subtree of count triangles
// splits at most count - 1 times); ids a subtree does not use keep tdepth =
// kNone and are skipped by the renumbering.
//
// What bounds it: instructions per node (and, in small meshes with few
// subtrees, the latency of a node times the subtree's depth).  Most nodes hold
// few triangles, so nodes of at most kDirect triangles skip the bins: a lane
// per (axis, triangle) sums the two sides of the plane after its triangle's bin
// over the node's triangles.  Only those planes can be the first minimum: the
// planes behind them with no triangle in between have the same sides and a
// higher number, and a plane with an empty side costs NaN.
#ifndef WF_BVH_SMALL_WARPS
#define WF_BVH_SMALL_WARPS 4
#endif
constexpr uint32_t kSmallWarps = WF_BVH_SMALL_WARPS;
constexpr uint32_t kDirect = 10;   // 3 axes x 10 triangles: one lane each

struct SmallSmem {
    float* d;
    uint32_t* oidx;
    uint16_t *perm, *ptmp, *F, *G;
    uint32_t* task[2];   // nodes of a level: first | count << 8 | (id's offset in the reservation + 1) << 16
    uint32_t* bins;      // per warp
};
static_assert(kSmall <= 128, "task words hold 8-bit counts and first positions");

__host__ __device__ constexpr size_t small_smem_bytes(uint32_t bins) {
    return (9ull + 1ull + 2ull) * 4ull * kSmall + 4ull * 2ull * kSmall + 4ull * 3ull * bins * kBinWords * kSmallWarps;
}

// The cheapest plane of a node of c <= kDirect triangles (see above): what
// warp_sweep returns over the node's bins.
__device__ __forceinline__ float direct_sweep(const SmallSmem& S, uint32_t B, uint32_t f, uint32_t c, const float* cmn,
                                              const float* cmx, uint32_t lane, uint32_t& axis, uint32_t& pos,
                                              uint32_t& nl) {
    const unsigned FULL = 0xffffffffu;
    const uint32_t a = lane / kDirect, i = lane - a * kDirect;
    const float lo = a == 0 ? cmn[0] : a == 1 ? cmn[1] : cmn[2], hi = a == 0 ? cmx[0] : a == 1 ? cmx[1] : cmx[2];
    const bool valid = a < 3 && i < c && lo != hi;
    uint32_t bin = 0;
    if (valid) {
        int32_t b = (int32_t)((S.d[a * kSmall + S.perm[f + i]] - lo) * ((float)B / (hi - lo)));
        if ((int32_t)B - 1 < b) b = (int32_t)B - 1;
        bin = (uint32_t)b;
    }
    float l[6], r[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) l[k] = r[k] = k < 3 ? FLT_MAX : -FLT_MAX;
    uint32_t lc = 0;
    for (uint32_t k = 0; k < c; ++k) {
        const uint32_t j = S.perm[f + k];
        const uint32_t kb = __shfl_sync(FULL, bin, a < 3 ? a * kDirect + k : 0u);
        const bool left = kb <= bin;
        lc += left ? 1u : 0u;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            const float e = S.d[(3 + q) * kSmall + j];
            const float none = q < 3 ? FLT_MAX : -FLT_MAX;
            l[q] = q < 3 ? fminf(l[q], left ? e : none) : fmaxf(l[q], left ? e : none);
            r[q] = q < 3 ? fminf(r[q], left ? none : e) : fmaxf(r[q], left ? none : e);
        }
    }
    const float cost = (float)lc * half_area(l, l + 3) + (float)(c - lc) * half_area(r, r + 3);
    const uint32_t key = valid && lc < c && cost < FLT_MAX ? fenc(cost + 0.0f) : kNone;
    const uint32_t best = __reduce_min_sync(FULL, key);
    axis = pos = nl = 0;
    if (best == kNone) return FLT_MAX;
    const uint32_t code = (a << 8) | bin;
    const uint32_t first = __reduce_min_sync(FULL, key == best ? code : kNone);
    const int src = __ffs(__ballot_sync(FULL, key == best && code == first)) - 1;
    axis = first >> 8;
    pos = (first & 0xFFu) + 1u;
    nl = __shfl_sync(FULL, lc, src);
    return fdec(best);
}

// One warp, one node (positions [f, f + c) of the subtree): its record, its
// split, and the partition of its positions.  Returns nl, the left child's
// triangles (0: no children).
__device__ __forceinline__ uint32_t small_node(const Ctx& C, const SmallSmem& S, uint32_t* bins, uint32_t X,
                                               uint32_t gfirst, uint32_t f, uint32_t c, uint32_t dep, uint32_t lane) {
    // node bounds, centroid bounds and first zero positions
    float v[12];
    uint32_t zp[6];
    box_init(v);
    zero_init(zp);
    for (uint32_t i = lane; i < c; i += 32) {
        const uint32_t j = S.perm[f + i];
        float e[9];
#pragma unroll
        for (int k = 0; k < 9; ++k) e[k] = S.d[k * kSmall + j];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            v[a] = fminf(v[a], e[3 + a]);
            v[3 + a] = fmaxf(v[3 + a], e[6 + a]);
            v[6 + a] = fminf(v[6 + a], e[a]);
            v[9 + a] = fmaxf(v[9 + a], e[a]);
        }
#pragma unroll
        for (int k = 0; k < 6; ++k)
            if (e[3 + k] == 0.0f && zp[k] == kNone) zp[k] = i;
    }
    box_warp_redux(v);
#pragma unroll
    for (int k = 0; k < 6; ++k)
        if (v[k] == 0.0f) {
            const uint32_t z = __reduce_min_sync(0xffffffffu, zp[k]);
            if (z != kNone) v[k] = S.d[(3 + k) * kSmall + S.perm[f + z]];
        }
    if (lane == 0) {
        C.ta[X] = make_float4(v[0], v[1], v[2], __uint_as_float(gfirst + f));
        C.tb[X] = make_float4(v[3], v[4], v[5], __uint_as_float(c));
        C.tleft[X] = kNone;
        C.tdepth[X] = dep;
    }
    uint32_t axis, pos, nl;
    float cost;
    if (c <= kDirect) {
        cost = direct_sweep(S, C.bins, f, c, v + 6, v + 9, lane, axis, pos, nl);
    } else {
        bool deg[3];
        float lo[3], scale[3];
        for (int a = 0; a < 3; ++a) {
            lo[a] = v[6 + a];
            deg[a] = v[6 + a] == v[9 + a];
            scale[a] = deg[a] ? 0.0f : (float)C.bins / (v[9 + a] - v[6 + a]);
        }
        bins_reset(bins, 3 * C.bins * kBinWords, lane, 32);
        __syncwarp();
        for (uint32_t i = lane; i < c; i += 32) {
            const uint32_t j = S.perm[f + i];
            for (uint32_t a = 0; a < 3; ++a) {
                if (deg[a]) continue;
                int32_t bin = (int32_t)((S.d[a * kSmall + j] - lo[a]) * scale[a]);
                if ((int32_t)C.bins - 1 < bin) bin = (int32_t)C.bins - 1;
                uint32_t* e = bins + (a * C.bins + (uint32_t)bin) * kBinWords;
                atomicAdd(&e[0], 1u);
                atomicMin(&e[1], fenc(S.d[3 * kSmall + j]));
                atomicMin(&e[2], fenc(S.d[4 * kSmall + j]));
                atomicMin(&e[3], fenc(S.d[5 * kSmall + j]));
                atomicMax(&e[4], fenc(S.d[6 * kSmall + j]));
                atomicMax(&e[5], fenc(S.d[7 * kSmall + j]));
                atomicMax(&e[6], fenc(S.d[8 * kSmall + j]));
            }
        }
        __syncwarp();
        cost = warp_sweep(bins, C.bins, v + 6, v + 9, lane, axis, pos, nl);
    }
    Plan P = plan_from(C, cost, axis, pos, nl, c, v, v + 3, v + 6, v + 9);
    if (!P.partition) return 0;
    // the closed form of the two-pointer partition (see the file head),
    // positions relative to the node's first position f
    if (P.nl < c) P.p = P.nl + (goes_left_c(C, P, S.d[P.axis * kSmall + S.perm[f + P.nl]]) ? 0u : 1u);
    if (c <= 32) {
        const bool valid = lane < c;
        const uint32_t j = valid ? S.perm[f + lane] : 0u;
        const bool left = valid && goes_left_c(C, P, S.d[P.axis * kSmall + j]);
        const unsigned m = __ballot_sync(0xffffffffu, left);
        const uint32_t lpre = __popc(m & ((1u << lane) - 1u));
        if (valid) {
            if (lane < P.p && !left) S.F[f + (lane - lpre)] = (uint16_t)lane;
            else if (lane >= P.p && left) S.G[f + (P.nl - lpre) - 1] = (uint16_t)lane;
        }
        __syncwarp();
        if (valid) {
            uint32_t dst;
            if (lane < P.p) {
                const uint32_t mm = lane - lpre + 1;
                dst = left ? lane : (mm == 1 ? c : (uint32_t)S.G[f + mm - 2]) - 1;
            } else {
                dst = !left ? lane - 1 : (uint32_t)S.F[f + (P.nl - lpre) - 1];
            }
            S.perm[f + dst] = (uint16_t)j;
        }
        __syncwarp();
    } else {
        for (int pass = 0; pass < 2; ++pass) {
            uint32_t run = 0;
            for (uint32_t base = 0; base < c; base += 32) {
                const uint32_t i = base + lane;
                const bool valid = i < c;
                const uint32_t j = valid ? S.perm[f + i] : 0u;
                const bool left = valid && goes_left_c(C, P, S.d[P.axis * kSmall + j]);
                const unsigned m = __ballot_sync(0xffffffffu, left);
                const uint32_t lpre = run + __popc(m & ((1u << lane) - 1u));
                if (valid) {
                    if (pass == 0) {
                        if (i < P.p && !left) S.F[f + (i - lpre)] = (uint16_t)i;
                        else if (i >= P.p && left) S.G[f + (P.nl - lpre) - 1] = (uint16_t)i;
                    } else {
                        uint32_t dst;
                        if (i < P.p) {
                            const uint32_t mm = i - lpre + 1;
                            dst = left ? i : (mm == 1 ? c : (uint32_t)S.G[f + mm - 2]) - 1;
                        } else {
                            dst = !left ? i - 1 : (uint32_t)S.F[f + (P.nl - lpre) - 1];
                        }
                        S.ptmp[f + dst] = (uint16_t)j;
                    }
                }
                run += __popc(m);
            }
            __syncwarp();
        }
        for (uint32_t i = lane; i < c; i += 32) S.perm[f + i] = S.ptmp[f + i];
        __syncwarp();
    }
    return P.children ? P.nl : 0u;
}

__global__ void __launch_bounds__(32 * kSmallWarps) k_small(Ctx C, uint32_t tcap) {
    extern __shared__ __align__(16) uint8_t smem_raw[];
    __shared__ uint32_t s_count[2], s_base, s_splits;
    SmallSmem S;
    S.d = reinterpret_cast<float*>(smem_raw);
    S.oidx = reinterpret_cast<uint32_t*>(S.d + 9 * kSmall);
    S.task[0] = S.oidx + kSmall;
    S.task[1] = S.task[0] + kSmall;
    S.perm = reinterpret_cast<uint16_t*>(S.task[1] + kSmall);
    S.ptmp = S.perm + kSmall;
    S.F = S.ptmp + kSmall;
    S.G = S.F + kSmall;
    S.bins = reinterpret_cast<uint32_t*>(S.G + kSmall);
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    uint32_t* bins = S.bins + warp * 3 * C.bins * kBinWords;
    const uint32_t nsmall = C.tcount[2];
    for (uint32_t w = blockIdx.x; w < nsmall; w += gridDim.x) {
        const uint32_t R = C.small_list[w];
        const uint32_t gfirst = __float_as_uint(C.ta[R].w), count = __float_as_uint(C.tb[R].w);
        uint32_t dep = C.tdepth[R];
        const uint32_t* from = (dep & 1u) ? C.idx[1] : C.idx[0];
        for (uint32_t i = t; i < count; i += 32 * kSmallWarps) {
            const uint32_t id = from[gfirst + i];
            const float4 c = C.cen[id], mn = C.tmn[id], mx = C.tmx[id];
            S.d[0 * kSmall + i] = c.x;  S.d[1 * kSmall + i] = c.y;  S.d[2 * kSmall + i] = c.z;
            S.d[3 * kSmall + i] = mn.x; S.d[4 * kSmall + i] = mn.y; S.d[5 * kSmall + i] = mn.z;
            S.d[6 * kSmall + i] = mx.x; S.d[7 * kSmall + i] = mx.y; S.d[8 * kSmall + i] = mx.z;
            S.oidx[i] = id;
            S.perm[i] = (uint16_t)i;
        }
        if (t == 0) {
            s_base = atomicAdd(&C.tcount[0], 2u * (count - 1));
            s_count[0] = 1u;
            s_count[1] = 0u;
            s_splits = 0u;
            S.task[0][0] = 0u | (count << 8);
        }
        __syncthreads();
        const uint32_t L0 = s_base;
        if ((uint64_t)L0 + 2ull * (count - 1) > tcap) {   // cannot happen for tcap = 2n + 2n / kSmall + 4
            if (t == 0) atomicOr(&C.tcount[3], 1u);
            __syncthreads();
            continue;
        }
        uint32_t cur = 0;
        for (uint32_t nodes = 1; nodes > 0;) {
            for (uint32_t q = warp; q < nodes; q += kSmallWarps) {
                const uint32_t task = S.task[cur][q];
                const uint32_t f = task & 0xFFu, c = (task >> 8) & 0xFFu, k = task >> 16;
                const uint32_t X = k == 0u ? R : L0 + k - 1u;
                const uint32_t nl = small_node(C, S, bins, X, gfirst, f, c, dep, lane);
                if (nl && lane == 0) {
                    const uint32_t kl = 2u * atomicAdd(&s_splits, 1u);
                    C.tleft[X] = L0 + kl;
                    C.tparent[L0 + kl] = C.tparent[L0 + kl + 1u] = X;
                    const uint32_t at = atomicAdd(&s_count[cur ^ 1], 2u);
                    S.task[cur ^ 1][at] = f | (nl << 8) | ((kl + 1u) << 16);
                    S.task[cur ^ 1][at + 1] = (f + nl) | ((c - nl) << 8) | ((kl + 2u) << 16);
                }
                __syncwarp();
            }
            __syncthreads();
            nodes = s_count[cur ^ 1];
            if (t == 0) s_count[cur] = 0u;   // read by no one now, filled after the next barrier
            __syncthreads();
            cur ^= 1u;
            if (nodes) ++dep;
        }
        for (uint32_t i = t; i < count; i += 32 * kSmallWarps) C.idx[0][gfirst + i] = S.oidx[S.perm[i]];
        __syncthreads();
    }
}

// ---------------------------------------------------------------- renumbering and output
// Two launches instead of two per depth that each read every node (139 + 4 us at
// 20,480 triangles, 264 + 15 at 499,280).
//
// Internal nodes of every subtree, from the leaves up: the second child to
// arrive at a node sums both and goes on.  On the way each child's word for the
// way down is set: {parent, what the child's pre-order rank among the internal
// nodes is above its parent's}.
__global__ void k_count(Ctx C, uint32_t* arrived, uint32_t* ic, uint2* up) {
    const uint32_t stride = gridDim.x * blockDim.x, T = C.tcount[0];
    for (uint32_t X = blockIdx.x * blockDim.x + threadIdx.x; X < T; X += stride) {
        if (C.tdepth[X] == kNone || C.tleft[X] != kNone) continue;   // unused id, or not a leaf
        uint32_t cur = X, mine = 0;
        for (;;) {
            ic[cur] = mine;
            if (cur == 0u) {
                C.tcount[1] = mine;
                break;
            }
            const uint32_t p = C.tparent[cur];
            __threadfence();
            if (atomicAdd(&arrived[p], 1u) == 0u) break;
            __threadfence();
            const uint32_t L = C.tleft[p];
            const uint32_t a = __ldcg(&ic[L]), b = __ldcg(&ic[L + 1]);
            up[L] = make_uint2(p, 1u);
            up[L + 1] = make_uint2(p, 1u + a);
            mine = 1u + a + b;
            cur = p;
        }
    }
}

// The nodes at their places: a node's rank is the sum of the words up to the
// root; left children have odd ids (pairs are handed out from id 1).
__global__ void k_emit(Ctx C, const uint2* up, float4* out) {
    const uint32_t stride = gridDim.x * blockDim.x, T = C.tcount[0];
    for (uint32_t X = blockIdx.x * blockDim.x + threadIdx.x; X < T; X += stride) {
        if (C.tdepth[X] == kNone) continue;   // id reserved by a small subtree but not used
        const float4 a = C.ta[X], b = C.tb[X];
        const bool internal = C.tleft[X] != kNone;
        uint32_t rank = 0, above = 0;
        for (uint32_t cur = X; cur != 0u;) {
            const uint2 u = up[cur];
            if (cur == X) above = u.y;
            rank += u.y;
            cur = u.x;
        }
        const uint32_t f = X == 0u ? 0u : 2u + 2u * (rank - above) + ((X & 1u) ? 0u : 1u);
        out[2ull * f] = make_float4(a.x, a.y, a.z, internal ? __uint_as_float(2 + 2 * rank) : a.w);
        out[2ull * f + 1] = make_float4(b.x, b.y, b.z, internal ? __uint_as_float(0u) : b.w);
        if (X == 0u) out[2] = out[3] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);   // node 1 is unused
    }
}

__global__ void k_leaf_tris(Ctx C, float4* out) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < C.n; i += stride) {
        const uint32_t t = C.idx[0][i];
        const float* p = C.pos + 9ull * t;
        out[3ull * i] = make_float4(p[0], p[1], p[2], __uint_as_float(t));
        out[3ull * i + 1] = make_float4(p[3] - p[0], p[4] - p[1], p[5] - p[2], 0.0f);
        out[3ull * i + 2] = make_float4(p[6] - p[0], p[7] - p[1], p[8] - p[2], 0.0f);
    }
}

// ---------------------------------------------------------------- host side
// One device allocation for all of a build's scratch, carved into 256-byte
// aligned parts (one cudaMalloc / cudaFree per build instead of one per array).
struct Arena {
    size_t bytes = 0;
    template <typename T>
    size_t part(size_t count) {
        const size_t off = bytes;
        bytes += (std::max<size_t>(count, 1) * sizeof(T) + 255) & ~size_t(255);
        return off;
    }
};

// A build's scratch: back to the kept blocks once the stream is done with it,
// else (an error on the way) freed, which waits.
struct DeviceBlock {
    void* p = nullptr;
    bool done = false;
    ~DeviceBlock() {
        if (done) scratch_give(p);
        else dfree(p);
    }
};

// k_large's grid: a block per 128 triangles up to 2 per SM (a block per 256 or
// 512: 356 -> 364 / 385 us at 1,280 triangles; 1 per SM: 2,045 -> 2,199 us at
// 200,000, 4: the same).
constexpr uint32_t kLargeBlocksPerSm = 2, kLargePerBlock = 128;
unsigned blocks_for(uint64_t n, unsigned threads, unsigned cap = 152u * 16u) {
    uint64_t b = (n + threads - 1) / threads;
    return (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(b, cap));
}

#define BVH_CUDA(call)                                                               \
    do {                                                                             \
        cudaError_t e_ = (call);                                                     \
        if (e_ != cudaSuccess) {                                                     \
            g_err = std::string(#call) + ": " + cudaGetErrorString(e_);              \
            return e_ == cudaErrorMemoryAllocation ? WF_ERR_OOM : WF_ERR_CUDA;       \
        }                                                                            \
    } while (0)

}  // namespace

const char* bvh_last_error() { return g_err.c_str(); }

int gpu_bvh_build(const triangle_t* tris, uint32_t n, const wf_bvh_options& o, cudaStream_t st, BvhBuildOut* out) {
    if (n == 0 || !tris || !out) { g_err = "gpu_bvh_build: empty mesh"; return WF_ERR_INVALID; }
    if (o.interval_count < 2 || o.interval_count > kMaxBins) {
        g_err = "gpu_bvh_build: interval_count must be 2..64";
        return WF_ERR_INVALID;
    }
    if (n > (1u << 30)) { g_err = "gpu_bvh_build: too many triangles"; return WF_ERR_CAPACITY; }
    const uint32_t B = o.interval_count;
    // 2n + 2 ids hold any binary tree over n triangles; the small phase reserves
    // 2 * (count - 1) per subtree, which can leave up to 2 * (large leaves) more
    const uint64_t tcap = 2ull * n + 2ull * (n / kSmall) + 4;
    const uint32_t maxslots = n / kSmall + 2;
    const uint32_t maxchunks = n / kChunk + maxslots + 1;
    const uint64_t max_nodes = 2ull * n;   // 2 + 2 * (internal nodes <= n - 1)

    Arena A;
    const size_t o_pos = A.part<float>(9ull * n), o_cen = A.part<float4>(3ull * n), o_idx = A.part<uint32_t>(n),
                 o_idx_tmp = A.part<uint32_t>(n), o_FG = A.part<uint32_t>(std::max<uint64_t>(2ull * n, tcap)),
                 o_ta = A.part<float4>(tcap), o_tb = A.part<float4>(tcap), o_tleft = A.part<uint32_t>(tcap),
                 o_tparent = A.part<uint32_t>(tcap), o_tdepth = A.part<uint32_t>(tcap),
                 o_tcount = A.part<uint32_t>(4), o_small = A.part<uint32_t>(n), o_ic = A.part<uint32_t>(tcap);
    size_t o_par[2][5];
    for (auto& q : o_par) {
        q[0] = A.part<uint32_t>(maxslots); q[1] = A.part<uint32_t>((size_t)kBoxWords * maxslots);
        q[2] = A.part<uint32_t>(maxslots); q[3] = A.part<uint32_t>(maxslots); q[4] = A.part<uint32_t>(maxchunks);
    }
    const size_t o_bins = A.part<uint32_t>((size_t)maxslots * 3 * B * kBinWords),
                 o_chl = A.part<uint32_t>(maxchunks), o_side = A.part<uint32_t>(32ull * maxchunks),
                 o_plan = A.part<Plan>(maxslots), o_child = A.part<uint32_t>(2ull * maxslots),
                 o_cnt = A.part<uint32_t>(5);
    const size_t o_nodes = out->keep_device ? 0 : A.part<float4>(2 * max_nodes);
    DeviceBlock scratch;
    {
        const cudaError_t e = scratch_take(&scratch.p, A.bytes);
        if (e != cudaSuccess) {
            cudaGetLastError();
            g_err = std::string("gpu_bvh_build: cudaMalloc: ") + cudaGetErrorString(e);
            return WF_ERR_OOM;
        }
    }
    uint8_t* base = static_cast<uint8_t*>(scratch.p);
    auto at = [base](size_t off) { return static_cast<void*>(base + off); };

    Ctx C{};
    C.n = n; C.bins = B; C.single = o.subdivide_single_prim ? 1u : 0u; C.max_leaf = o.max_leaf_prims;
    float* d_pos = static_cast<float*>(at(o_pos));
    C.pos = d_pos;
    C.cen = static_cast<float4*>(at(o_cen)); C.tmn = C.cen + n; C.tmx = C.tmn + n;
    C.idx[0] = static_cast<uint32_t*>(at(o_idx)); C.idx[1] = static_cast<uint32_t*>(at(o_idx_tmp));
    C.F = static_cast<uint32_t*>(at(o_FG)); C.G = C.F + n;
    C.ta = static_cast<float4*>(at(o_ta)); C.tb = static_cast<float4*>(at(o_tb));
    C.tleft = static_cast<uint32_t*>(at(o_tleft)); C.tparent = static_cast<uint32_t*>(at(o_tparent));
    C.tdepth = static_cast<uint32_t*>(at(o_tdepth));
    C.tcount = static_cast<uint32_t*>(at(o_tcount));
    C.small_list = static_cast<uint32_t*>(at(o_small));
    Large G{};
    for (int q = 0; q < 2; ++q) {
        G.slot_tmp[q] = static_cast<uint32_t*>(at(o_par[q][0]));
        G.slot_box[q] = static_cast<uint32_t*>(at(o_par[q][1]));
        G.slot_done[q] = static_cast<uint32_t*>(at(o_par[q][2]));
        G.slot_chunk[q] = static_cast<uint32_t*>(at(o_par[q][3]));
        G.chunk_slot[q] = static_cast<uint32_t*>(at(o_par[q][4]));
    }
    G.bins = static_cast<uint32_t*>(at(o_bins)); G.chunk_l = static_cast<uint32_t*>(at(o_chl));
    G.side = static_cast<uint32_t*>(at(o_side)); G.plan = static_cast<Plan*>(at(o_plan));
    G.child_slot = static_cast<uint32_t*>(at(o_child)); G.cnt = static_cast<uint32_t*>(at(o_cnt));
    // free once the tree stands: the partition's ranks take the arrivals, the
    // triangles' boxes the words up the tree (2 tcap words in 12 n)
    uint32_t* arrived = C.F;
    uint2* up = reinterpret_cast<uint2*>(C.cen);
    uint32_t* ic = static_cast<uint32_t*>(at(o_ic));

    // the triangles in turns through the words of the node table, not used yet
    const uint64_t turn = std::min<uint64_t>(n, 32ull * tcap / sizeof(triangle_t));
    for (uint64_t t0 = 0; t0 < n; t0 += turn) {
        const uint32_t m = (uint32_t)std::min<uint64_t>(turn, n - t0);
        BVH_CUDA(cudaMemcpyAsync(C.ta, tris + t0, m * sizeof(triangle_t), cudaMemcpyHostToDevice, st));
        k_gather<<<blocks_for(m, 256), 256, 0, st>>>(C.ta, m, d_pos + 9 * t0);
    }
    // ids that a small subtree reserves but does not use keep depth kNone
    BVH_CUDA(cudaMemsetAsync(C.tdepth, 0xFF, 4ull * tcap, st));
    k_init<<<1, 256, 0, st>>>(C, G);
    k_prep<<<blocks_for(n, 256, 152u * 4u), 256, 0, st>>>(C, n > kSmall ? G.slot_box[0] : nullptr);
    if (n > kSmall) {
        // a cooperative launch: its blocks wait for one another
        int per_sm = 0;
        BVH_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_large, kChunkThreads, 0));
        const unsigned most = (unsigned)sm_count() * (unsigned)std::max(1, std::min(per_sm, (int)kLargeBlocksPerSm));
        const unsigned grid = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>(most, n / kLargePerBlock));
        void* args[] = {&C, &G};
        BVH_CUDA(cudaLaunchCooperativeKernel(reinterpret_cast<const void*>(k_large), dim3(grid), dim3(kChunkThreads), args, 0, st));
    }
    // under the 48 KiB that need no leave: asking for a call's own size would
    // set another thread's maximum
    static_assert(small_smem_bytes(kMaxBins) <= 46u * 1024u, "");
    const size_t smem = small_smem_bytes(B);
    k_small<<<blocks_for(n, 48, 1u << 16), 32 * kSmallWarps, smem, st>>>(C, (uint32_t)tcap);
    BVH_CUDA(cudaMemsetAsync(arrived, 0, 4ull * tcap, st));
    k_count<<<blocks_for(tcap, 256), 256, 0, st>>>(C, arrived, ic, up);
    BVH_CUDA(cudaGetLastError());
    uint32_t counts[4];
    BVH_CUDA(cudaMemcpyAsync(counts, C.tcount, 16, cudaMemcpyDeviceToHost, st));
    BVH_CUDA(cudaStreamSynchronize(st));
    if (counts[3] != 0) {
        g_err = (counts[3] & 2u) ? "gpu_bvh_build: a grid barrier gave up"
                                 : "gpu_bvh_build: small-subtree node ids exceeded the reserved range";
        return (counts[3] & 2u) ? WF_ERR_TIMEOUT : WF_ERR_CAPACITY;
    }
    const uint32_t nc = 2 + 2 * counts[1];
    float4* d_nodes = nullptr;
    float4* d_tris = nullptr;
    if (out->keep_device) {
        BVH_CUDA(dmalloc(reinterpret_cast<void**>(&d_nodes), 32ull * nc));
        if (dmalloc(reinterpret_cast<void**>(&d_tris), 48ull * n) != cudaSuccess) {
            dfree(d_nodes);
            cudaGetLastError();
            g_err = "gpu_bvh_build: cudaMalloc failed";
            return WF_ERR_OOM;
        }
    } else {
        d_nodes = static_cast<float4*>(at(o_nodes));
    }
    auto drop = [&]() {
        if (out->keep_device) {
            dfree(d_nodes);
            dfree(d_tris);
        }
    };
    cudaError_t e = cudaSuccess;
    k_emit<<<blocks_for(counts[0], 256), 256, 0, st>>>(C, up, d_nodes);
    if (d_tris) k_leaf_tris<<<blocks_for(n, 256), 256, 0, st>>>(C, d_tris);
    if (e == cudaSuccess) e = cudaGetLastError();
    // blob: [header | nodes | bvh_triangle_t (original order) | index list], written
    // straight into the caller's buffer when it is large enough
    const uint64_t nodes_bytes = 32ull * nc, tri_bytes = 36ull * n, idx_bytes = 4ull * n;
    const uint64_t size = 12 + nodes_bytes + tri_bytes + idx_bytes;
    uint8_t* blob;
    if (out->dst && out->dst_capacity >= size) {
        blob = out->dst;
        out->in_dst = true;
    } else {
        out->blob.resize(size);
        blob = out->blob.data();
        out->in_dst = false;
    }
    out->blob_size = size;
    if (e == cudaSuccess) e = cudaMemcpyAsync(blob + 12, d_nodes, nodes_bytes, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(blob + 12 + nodes_bytes, d_pos, tri_bytes, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(blob + 12 + nodes_bytes + tri_bytes, C.idx[0], idx_bytes, cudaMemcpyDeviceToHost, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
        drop();
        g_err = std::string("gpu_bvh_build: ") + cudaGetErrorString(e);
        return WF_ERR_CUDA;
    }
    scratch.done = true;
    bvh_header_t h;
    h.nodes_offset = 12;
    h.triangles_offset = (uint32_t)(12 + nodes_bytes);
    h.indices_offset = (uint32_t)(12 + nodes_bytes + tri_bytes);
    std::memcpy(blob, &h, 12);
    bvh_node_t root;
    std::memcpy(&root, blob + 12, 32);
    std::memcpy(out->root_min, root.aabb_min, 12);
    std::memcpy(out->root_max, root.aabb_max, 12);
    out->node_count = nc;
    out->d_nodes = out->keep_device ? d_nodes : nullptr;
    out->d_tris = d_tris;
    return WF_OK;
}

}  // namespace wf
