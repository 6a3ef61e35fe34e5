// wf_traverse.cuh — software TLAS -> BLAS traversal (closest hit / any hit).
//
// Per ray it follows trace_ray_tlas / trace_ray_bvh_instance /
// trace_ray_bvh_local (accelstruct.hlsl:58-218) step for step: TLAS root box
// test, near-child-first descent with ties to the left, far child pushed only
// when it was hit, leaf triangles tested in index-list order with strict
// "t < ray.t" acceptance (the first triangle found wins an exact tie),
// instance rays transformed by world_to_local without renormalising.  The
// reference pushes whole node copies; this pushes the 8 bytes a popped node
// needs ({left_first, prim_count} or {left_right, instance_idx}), which visits
// the same nodes in the same order.  Each level keeps its own 64-entry stack,
// as the reference; an overflow abandons the ray (reported as a miss) and
// raises ERRF_STACK where the reference would write past its array.
//
// GPU organisation: a persistent grid; every warp runs one warp-uniform loop.
// An iteration takes each of its lanes through the steps that apply to it, in
// the order instance entry, up to kInnerSteps interior visits (the same code
// for TLAS and BLAS nodes: two child boxes, one slab test each; a miss pops the
// level's stack), one triangle of a leaf, return from an exhausted level.  So
// lanes meet again at every kind of step instead of drifting apart in nested
// per-lane loops, and none waits for another's whole leaf or subtree.
// A warp's first rays are its own by its number; lanes whose ray finished take
// new rays in groups through one atomic per warp (kRefill idle lanes, or all
// of them) from a per-launch counter.
//
// What bounds it: issue slots (50-60 % busy, most of it integer, compare and
// min / max work around the box tests) and the latency of the dependent node
// loads at 13-15 active lanes of 32.  So the loop carries as little as it can:
// TLAS nodes are read as child pairs in the BLAS's form, which makes an interior
// step one code path with one pointer for both levels and a leaf test one
// compare, and one ballot per iteration serves hand-out and termination
// (separate TLAS and BLAS addressing and three ballots before: 1080p instanced
// frame 12.37 -> 11.73 ms, 720p frame 1.18 -> 1.11, 1M any-hit rays 419 -> 391
// us, 4.2M incoherent closest-hit rays 6.28 -> 6.13 ms); then, on the same
// four, packed box tests, the choice of child by booleans and one overflow test:
// 11.31 ms, 1.07, 370 us, 5.99 ms; several steps per iteration (one kind of
// step per lane and iteration before) with the world ray's reciprocal kept
// through an instance: 9.91 ms, 1.02, 316 us, 5.49 ms, and a whole-wave 256x256
// frame 222 -> 172 us; then nodes and instance rows in 32-byte loads, half the
// requests: 9.53 ms, 1.02, 298 us, 4.46 ms, and with new rays at 12 idle lanes
// again 9.29, 1.02, 290, 4.44 (quantized and exact 4-wide: 6.02 ->
// 6.01, 7.04 -> 6.07).  Each pair on one GPU; the 1M any-hit rays take 232 to
// 290 us from GPU to GPU, so their small steps show little by themselves.  One
// ray alone over a 4-wide layout takes 37 us where a step per iteration took 34
// (eight rays: 69 and 82).
#pragma once
#include <type_traits>
#include "wf_device.cuh"
#include "wf_grid.h"

namespace wf {

struct Hit {
    uint32_t inst, prim;
    float t, u, v;
};

struct LocalCounters {
    uint32_t tlas_nodes, instances, blas_nodes, tris;
};

constexpr uint32_t kNoRay = 0xFFFFFFFFu;
// Threads per block of the persistent traversal kernels.
#ifndef WF_TRACE_BLOCK
#define WF_TRACE_BLOCK 128
#endif
constexpr int kTraceBlock = WF_TRACE_BLOCK;
// Traversal stack: one LIFO for both levels (the TLAS entries below, the
// current instance's BLAS entries above them), 64 entries per level as the
// reference.  Its top WF_TRACE_RING entries live in a shared-memory ring (slot
// index % ring, one column per thread), the older ones in local memory; a
// push into a full ring moves the ring's oldest entry to local memory, a pop
// from an empty ring reads local memory.
#ifndef WF_TRACE_RING
#define WF_TRACE_RING 8
#endif
// A warp takes new rays once this many of its lanes are idle (or all are).  8 /
// 10 / 12 / 14 / 16: 1080p instanced frame 9.34 / 9.30 / 9.29 / 9.34 / 9.52 ms, 1M
// any-hit rays 290 / 289 / 290 / 293 / 298 us, a batch of scenes 8.69 / 8.60 /
// 8.54 / 8.53 / 8.46 ms.
#ifndef WF_TRACE_REFILL
#define WF_TRACE_REFILL 12
#endif
constexpr int kRefill = WF_TRACE_REFILL;
// Interior visits per loop iteration (binary layout), unrolled.  Each costs the
// warp the step's instructions as long as one lane takes it, and saves the
// lanes that do the rest of an iteration: 1 / 2 / 3 / 4 / 5 / 6 / 8 gave the
// 1080p instanced frame 10.86 / 10.22 / 10.09 / 9.88 / 9.98 / 10.07 / 10.57 ms
// and 4.2M incoherent rays 5.94 / 5.80 / 5.75 / 5.58 / 5.60 / 5.63 / 5.75.
// Ending the row when few lanes are left in it costs a ballot per visit: 10.10 ms.
// A 4-wide node's step is itself four boxes and a sort: one (two and four
// visits: quantized 6.04 -> 6.51 / 9.52 ms, exact 7.03 -> 6.95 / 7.50).
constexpr int kInnerSteps = 4;

// Ray sources / sinks.  load(i, o, d, tmax, no_cull); root(i, S) = the TLAS
// root node of the ray's scene, kInvalid for an empty scene; store(i, hit, ok)
// where ok is false when a traversal stack overflowed.  A source that mixes
// closest-hit and any-hit rays in one launch also has any(i) (true for an
// any-hit ray); the others take the kernel's ANY for every ray.
template <class IO, class = void>
struct MixedIO : std::false_type {};
template <class IO>
struct MixedIO<IO, std::void_t<decltype(std::declval<const IO&>().any(0u))>> : std::true_type {};

// A source whose entries are whole paths (kChain): load() may refuse an entry
// and also says whether the ray is an any-hit one; when a ray ends, next()
// takes its hit (t < 0: the stack overflowed, h a miss) and returns the path's
// next ray, or false at the path's end.
template <class IO, class = void>
struct ChainIO : std::false_type {};
template <class IO>
struct ChainIO<IO, std::void_t<decltype(IO::kChain)>> : std::true_type {};
// Lanes whose ray ended wait for the warp's last running lane, then the warp
// runs next() for all of them: shading's own latency is long enough that
// running it for 2 / 4 / 8 / 16 ended lanes at a time measured 370 / 305 / 255 /
// 247 us per 256x256 box frame against 235.

// The paths that n rays of a source stand for, as the ray counts count them.
template <class IO, class = void>
struct SharedIO : std::false_type {};
template <class IO>
struct SharedIO<IO, std::void_t<decltype(std::declval<const IO&>().paths_of(0u))>> : std::true_type {};
template <class IO>
__device__ __forceinline__ uint32_t paths_of(const IO& io, uint32_t n) {
    if constexpr (SharedIO<IO>::value) return io.paths_of(n);
    else return n;
}

struct AosIO {
    const float4* rays;   // RayDesc2
    uint32_t* hits;       // hit_result_t
    bool no_cull;
    __device__ __forceinline__ void load(uint32_t i, V3& o, V3& d, float& tmax, bool& nc) const {
        const float4 a = ldg4(rays + 2ull * i), b = ldg4(rays + 2ull * i + 1);
        o = xyz(a); d = xyz(b); tmax = b.w; nc = no_cull;
    }
    __device__ __forceinline__ uint32_t root(uint32_t, const SceneRefs& S) const { return S.inst_count ? 0u : kInvalid; }
    __device__ __forceinline__ void store(uint32_t i, const Hit& h, bool) const {
        uint32_t* o = hits + 5ull * i;
        o[0] = h.inst; o[1] = h.prim; o[2] = __float_as_uint(h.t); o[3] = __float_as_uint(h.u);
        o[4] = __float_as_uint(h.v);
    }
};

// The same rays traced in the order of a permutation (the k-th ray handed
// out is ray perm[k]); each hit still lands at its ray's own index.
struct PermutedAosIO {
    AosIO io;
    const uint32_t* perm;
    const uint32_t* varied;   // 0: the permutation was not built (identity)
    __device__ __forceinline__ uint32_t ray(uint32_t k) const { return *varied ? perm[k] : k; }
    __device__ __forceinline__ void load(uint32_t k, V3& o, V3& d, float& tmax, bool& nc) const {
        io.load(ray(k), o, d, tmax, nc);
    }
    __device__ __forceinline__ uint32_t root(uint32_t, const SceneRefs& S) const { return S.inst_count ? 0u : kInvalid; }
    __device__ __forceinline__ void store(uint32_t k, const Hit& h, bool ok) const { io.store(ray(k), h, ok); }
};

// LAY: the BLAS layout (0 = binary child pairs; 1 = quantized and 2 = exact
// 4-wide nodes, csrc/wf_qbvh.cu).  Over the 4-wide nodes closest-hit rays use
// the order-independent tie rule (smallest t, then smallest (instance,
// primitive); boxes entered at exactly t still visited), so their hits equal
// the binary traversal's whatever order the wider nodes visit leaves in.
// Any-hit rays keep "t < tmax": only whether they hit matters.
template <bool ANY, bool COUNT, int LAY, class IO>
__device__ __forceinline__ void trace_persistent(const SceneRefs& S, IO& io, uint32_t n, uint32_t* fetch,
                                                 LocalCounters& cnt, bool& overflow) {
    constexpr bool QB = LAY != 0;   // a 4-wide layout, with the tie rule
    constexpr bool CH = ChainIO<IO>::value;
    constexpr uint32_t kEnded = 2u;   // level of a lane without a running ray (w1 = 1: no step is its)
    const unsigned FULL = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t col = threadIdx.x;
    // State a step rarely touches lives in shared memory, one column per
    // thread, to keep the loop's registers (and so the resident warps) up:
    // the world ray and its 1/dir (w of the two and s_wiz; read back when the
    // ray leaves an instance) and the hit record (written on a hit, read when
    // the ray finishes).
    __shared__ float4 s_wo[kTraceBlock], s_wd[kTraceBlock];
    __shared__ uint32_t s_inst[kTraceBlock], s_prim[kTraceBlock];
    __shared__ float s_t[kTraceBlock], s_u[kTraceBlock], s_v[kTraceBlock], s_wiz[kTraceBlock];
    uint32_t ri = kNoRay;
    bool any_ray = ANY;   // this lane's ray stops at its first hit
    // current-space ray and 1/dir; ct = ray.t (the closest hit so far, shared
    // by world and object space because instance rays are not renormalised)
    V3 co = mk(0, 0, 0), cd = mk(0, 0, 0), ci = mk(0, 0, 0);
    float ct = 0.0f;
    bool no_cull = false, hit_here = false;
    // the current node's words, for both levels {first, 0} = an interior node whose
    // child pair lies at float4 2 first of nb (the TLAS pairs, or the instance's
    // BLAS nodes), {instance, 1} a TLAS leaf, {first triangle, count} a BLAS leaf
    uint32_t level = kEnded, w0 = 0, w1 = 1u, ii = 0;
    const float4* nb = nullptr;
    BlasRef B;
    B.nodes = nullptr; B.tris = nullptr;
    // stack: entries [0, sp); the TLAS level's are [0, tb) while inside an
    // instance (tb = 0 outside); [lo, sp) are in the ring, [0, lo) in local memory
    int sp = 0, lo = 0, tb = 0;
    uint2 deep[2 * kStack];
    __shared__ uint2 ring[WF_TRACE_RING][kTraceBlock];
    // false: the level's 64 entries are taken
    auto stack_push = [&](uint2 e) -> bool {
        if (sp - tb == kStack) return false;
        if (sp - lo == WF_TRACE_RING) {
            deep[lo] = ring[lo % WF_TRACE_RING][col];
            lo++;
        }
        ring[sp % WF_TRACE_RING][col] = e;
        sp++;
        return true;
    };
    auto stack_pop = [&]() -> uint2 {
        sp--;
        if (sp >= lo) return ring[sp % WF_TRACE_RING][col];
        lo = sp;
        return deep[sp];
    };
    auto hit_record = [&]() {
        Hit h;
        h.inst = s_inst[col]; h.prim = s_prim[col]; h.t = s_t[col]; h.u = s_u[col]; h.v = s_v[col];
        return h;
    };
    auto clear_hit = [&]() {
        s_inst[col] = kInvalid; s_prim[col] = kInvalid; s_t[col] = FLT_MAX; s_u[col] = 0.0f; s_v[col] = 0.0f;
    };

    // Hand-out.  A warp's first rays are its own by its number, with no atomic,
    // `width` of them: a launch of fewer rays than the grid has lanes spreads
    // them over all its warps.  Such a launch takes as long as its slowest ray,
    // and a warp iteration costs the sum of the kinds of step its lanes are at,
    // so fewer lanes per warp make it shorter: 64 host rays 141 -> 98 us per
    // call, a 613x377 frame whose deep queues are short 2.58 -> 2.39 ms, a
    // 720p frame 1.33 -> 1.18 ms; launches larger than the grid gain the first
    // round's atomics (1M any-hit rays 426 -> 419 us).  Later rays come from
    // the launch's counter, once every lane of the grid had one.
    const uint32_t nwarps = gridDim.x * (kTraceBlock / 32u);
    const uint32_t width = n / nwarps >= 32u ? 32u : (n + nwarps - 1u) / nwarps;
    // the ray in co, cd, ct: its world copy, an empty hit, the TLAS root's box
    auto enter_root = [&](uint32_t k) {
        ci = rcp(cd);
        s_wo[col] = make_float4(co.x, co.y, co.z, ci.x);
        s_wd[col] = make_float4(cd.x, cd.y, cd.z, ci.y);
        s_wiz[col] = ci.z;
        clear_hit();
        const uint32_t root = io.root(k, S);
        bool miss = root == kInvalid;
        if (!miss && !in_bounds(root, S.tnode_count, S.status)) miss = true;
        if (!miss) {
            float4 n0, n1;
            ldg8(S.tnodes + 2ull * root, n0, n1);
            if (COUNT) cnt.tlas_nodes++;
            miss = ((QB && !any_ray) ? slab_le(xyz(n0), xyz(n1), co, ci, ct)
                                     : slab(xyz(n0), xyz(n1), co, ci, ct)) == FLT_MAX;
            const bool leaf = __float_as_uint(n0.w) == 0u;   // a single instance
            level = 0; nb = S.tpairs;
            w0 = leaf ? __float_as_uint(n1.w) : 2u * root;
            w1 = leaf ? 1u : 0u;
            sp = 0; lo = 0; tb = 0;
        }
        return !miss;
    };
    auto start = [&](uint32_t k) {
        if (k < n) {
            if constexpr (CH) {
                if (io.load(k, co, cd, ct, no_cull, any_ray)) {
                    ri = k;
                    if (!enter_root(k)) { level = kEnded; w1 = 1u; }
                }
            } else {
                ri = k;
                io.load(k, co, cd, ct, no_cull);
                if constexpr (MixedIO<IO>::value) any_ray = io.any(k);
                if (!enter_root(k)) { io.store(k, hit_record(), true); ri = kNoRay; level = kEnded; w1 = 1u; }
            }
        }
    };
    if (lane < width) start((blockIdx.x * (kTraceBlock / 32u) + (threadIdx.x >> 5)) * width + lane);
    bool more = width == 32u;   // the counter may have rays left (uniform over the warp)
    for (;;) {
        if constexpr (CH) {
            // ---- the paths whose ray ended go on
            const bool ended = ri != kNoRay && level == kEnded;
            const unsigned run = __ballot_sync(FULL, ri != kNoRay && !ended);
            if (run == 0u && ended) {
                if (io.next(ri, hit_record(), xyz(s_wd[col]), co, cd, ct, no_cull, any_ray)) {
                    if (!enter_root(ri)) { level = kEnded; w1 = 1u; }
                } else {
                    ri = kNoRay;
                }
            }
        }
        // ---- refill idle lanes (one atomic per warp)
        const unsigned idle = __ballot_sync(FULL, ri == kNoRay);
        if (idle) {
            if (more && (idle == FULL || __popc(idle) >= kRefill)) {
                const int leader = __ffs(idle) - 1;
                uint32_t base = 0;
                if ((int)lane == leader) base = atomicAdd(fetch, (uint32_t)__popc(idle));
                base = __shfl_sync(FULL, base, leader) + gridDim.x * kTraceBlock;
                more = base < n && n - base > (uint32_t)__popc(idle);
                if (ri == kNoRay) start(base + (uint32_t)__popc(idle & ((1u << lane) - 1u)));
            } else if (idle == FULL) {
                break;
            }
        }

        // ---- the lane's steps
        bool finish = false, ok = true;
        bool pop = false;
        if (w1 != 0u && level == 0u) {
            // TLAS leaf: enter the instance (trace_ray_bvh_instance); at level
            // 0 the current ray is the world ray
            ii = w0;
            const float4* ip = S.tinst + 4ull * ii;
            if (!in_bounds(ii, S.inst_count, S.status)) {
                w1 = 0u;
                pop = true;
            } else {
                float4 c0, c1, c2, c3;
                ldg8(ip, c0, c1);
                ldg8(ip + 2, c2, c3);
                if (COUNT) cnt.instances++;
                const uint32_t mesh = __float_as_uint(c0.w);
                if (!in_bounds(mesh, S.mesh_count, S.status)) {
                    w1 = 0u;
                    pop = true;
                } else {
                    co = xform(co, 1.0f, c0, c1, c2, c3);
                    cd = xform(cd, 0.0f, c0, c1, c2, c3);
                    ci = rcp(cd);
                    B = S.blas[mesh];
                    if (QB) {
                        // node 0, or the one leaf of a single-leaf BLAS
                        w0 = 0u;
                        w1 = B.root_count;
                    } else {
                        float4 r0, r1;
                        ldg8(B.nodes, r0, r1);
                        if (COUNT) cnt.blas_nodes++;
                        w0 = __float_as_uint(r0.w);
                        w1 = __float_as_uint(r1.w);
                    }
                    nb = B.nodes;
                    level = 1; tb = sp; hit_here = false;
                }
            }
        }
#pragma unroll
        for (int r = 0; r < (QB ? 1 : kInnerSteps); ++r) {
            if (w1 == 0u && !pop && !finish) {
            if (QB && level == 1u) {
                // 4-wide BLAS node: up to four child boxes (quantized: origin + q *
                // 2^e per plane; exact: the planes as stored), visited nearest
                // first, the others pushed
                if (!in_bounds(w0, B.qnode_count, S.status)) {
                    pop = true;
                } else {
                    const bool tie = !any_ray;
                    float d[4];
                    uint2 e[4];
                    if constexpr (LAY == 1) {
                        const float4* qp = B.qnodes + 4ull * w0;
                        float4 q0, q1, q2, q3;
                        ldg8(qp, q0, q1);
                        ldg8(qp + 2, q2, q3);
                        if (COUNT) cnt.blas_nodes += 2;   // 64 bytes, as a binary child pair
                        const uint32_t meta = __float_as_uint(q0.w);
                        const float sx = __uint_as_float((meta & 0xFFu) << 23);
                        const float sy = __uint_as_float(((meta >> 8) & 0xFFu) << 23);
                        const float sz = __uint_as_float(((meta >> 16) & 0xFFu) << 23);
                        const uint32_t nch = meta >> 24;
                        const uint32_t lx = __float_as_uint(q1.x), ly = __float_as_uint(q1.y), lz = __float_as_uint(q1.z);
                        const uint32_t hx = __float_as_uint(q2.x), hy = __float_as_uint(q2.y), hz = __float_as_uint(q2.z);
                        const uint32_t cl = __float_as_uint(q1.w), chi = __float_as_uint(q2.w);
                        const uint32_t kid[4] = {__float_as_uint(q3.x), __float_as_uint(q3.y), __float_as_uint(q3.z),
                                                 __float_as_uint(q3.w)};
    #pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const uint32_t sh = 8u * (uint32_t)i;
                            const V3 bmn = mk(q0.x + (float)((lx >> sh) & 0xFFu) * sx, q0.y + (float)((ly >> sh) & 0xFFu) * sy,
                                              q0.z + (float)((lz >> sh) & 0xFFu) * sz);
                            const V3 bmx = mk(q0.x + (float)((hx >> sh) & 0xFFu) * sx, q0.y + (float)((hy >> sh) & 0xFFu) * sy,
                                              q0.z + (float)((hz >> sh) & 0xFFu) * sz);
                            const float di = tie ? slab_le(bmn, bmx, co, ci, ct) : slab(bmn, bmx, co, ci, ct);
                            d[i] = (uint32_t)i < nch ? di : FLT_MAX;
                            e[i] = make_uint2(kid[i], ((cl >> sh) & 0xFFu) | (((chi >> sh) & 0xFFu) << 8));
                        }
                    } else {
                        const float4* wp = B.qnodes + 8ull * w0;
                        float4 xl, xh, yl, yh, zl, zh, en, cn;
                        ldg8(wp, xl, xh);
                        ldg8(wp + 2, yl, yh);
                        ldg8(wp + 4, zl, zh);
                        ldg8(wp + 6, en, cn);
                        if (COUNT) cnt.blas_nodes += 4;   // 128 bytes, as two binary child pairs
                        const uint32_t nch = __float_as_uint(cn.x) >> 24;
                        auto lane4 = [](const float4& v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; };
    #pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const V3 bmn = mk(lane4(xl, i), lane4(yl, i), lane4(zl, i));
                            const V3 bmx = mk(lane4(xh, i), lane4(yh, i), lane4(zh, i));
                            const float di = tie ? slab_le(bmn, bmx, co, ci, ct) : slab(bmn, bmx, co, ci, ct);
                            d[i] = (uint32_t)i < nch ? di : FLT_MAX;
                            const uint32_t c = __float_as_uint(lane4(cn, i));
                            e[i] = make_uint2(__float_as_uint(lane4(en, i)), i == 0 ? (c & 0x00FFFFFFu) : c);
                        }
                    }
                    // order the four by entry distance (a five-comparator network)
                    auto cswap = [&](int a, int b) {
                        if (d[a] > d[b]) {
                            const float td = d[a]; d[a] = d[b]; d[b] = td;
                            const uint2 te = e[a]; e[a] = e[b]; e[b] = te;
                        }
                    };
                    cswap(0, 1); cswap(2, 3); cswap(0, 2); cswap(1, 3); cswap(1, 2);
                    if (d[0] == FLT_MAX) {
                        pop = true;
                    } else {
                        w0 = e[0].x; w1 = e[0].y;
    #pragma unroll
                        for (int i = 3; i >= 1; --i) {
                            if (d[i] != FLT_MAX && !finish) {
                                if (!stack_push(e[i])) {
                                    clear_hit();
                                    w1 = 0u;
                                    finish = true; ok = false; overflow = true;
                                }
                            }
                        }
                    }
                }
            } else {
                // interior node, TLAS or BLAS: the two children, nearer first
                const float4* pa = nb + 2ull * w0;
                if (level == 0u ? !in_bounds(w0 >> 1, S.tnode_count, S.status)
                                : !in_bounds(w0 + 1ull, B.node_count, S.status)) {
                    pop = true;
                } else {
                    float4 a0, a1, b0, b1;
                    ldg8(pa, a0, a1);
                    ldg8(pa + 2, b0, b1);
                    if (COUNT) { if (level == 0u) cnt.tlas_nodes += 2; else cnt.blas_nodes += 2; }
                    float dl, dr;
                    bool hl, hr;   // the children entered before the current hit
                    if (QB && !any_ray) {
                        dl = slab_le(xyz(a0), xyz(a1), co, ci, ct); hl = dl != FLT_MAX;
                        dr = slab_le(xyz(b0), xyz(b1), co, ci, ct); hr = dr != FLT_MAX;
                    } else {
                        hl = slab_hit(a0, a1, co, ci, ct, dl);
                        hr = slab_hit(b0, b1, co, ci, ct, dr);
                    }
                    // the nearer first, ties to the left
                    const bool right = hr && (!hl || dl > dr);
                    pop = !hl && !hr;
                    w0 = __float_as_uint(right ? b0.w : a0.w);
                    w1 = pop ? 0u : __float_as_uint(right ? b1.w : a1.w);
                    if (pop && sp > tb) {
                        const uint2 e = stack_pop();
                        w0 = e.x; w1 = e.y;
                        pop = false;
                    }
                    if (hl && hr) {
                        const uint2 far = make_uint2(__float_as_uint(right ? a0.w : b0.w), __float_as_uint(right ? a1.w : b1.w));
                        if (!stack_push(far)) {
                            clear_hit();
                            w1 = 0u;
                            finish = true; ok = false; overflow = true;
                        }
                    }
                }
            }
        }
        }
        if (w1 != 0u && level == 1u) {
            if (!in_bounds(w0, B.tri_count, S.status)) {
                w1 = 0u;
                pop = true;
            } else {
                // BLAS leaf: one triangle, in index-list order (w0 = the next one,
                // w1 = triangles left).  Two per iteration: 1080p 10.22 -> 10.31 ms
                const float4* tp = B.tris + 3ull * w0;
                const float4 a = ldg4(tp), b = ldg4(tp + 1), c = ldg4(tp + 2);
                if (COUNT) cnt.tris++;
                float bu, bv;
                bool accepted;
                if (QB && !any_ray) {
                    // the current hit: this instance once it has one here, else the outer one
                    const uint32_t bi = hit_here ? ii : s_inst[col];
                    const uint32_t pr = __float_as_uint(a.w);
                    const bool wins = ii < bi || (ii == bi && pr < s_prim[col]);
                    accepted = tri_hit_tie(xyz(a), xyz(b), xyz(c), co, cd, ct, bu, bv, no_cull, wins);
                } else {
                    accepted = tri_hit(xyz(a), xyz(b), xyz(c), co, cd, ct, bu, bv, no_cull);
                }
                if (accepted) {
                    s_prim[col] = __float_as_uint(a.w);
                    s_u[col] = bu; s_v[col] = bv;
                    hit_here = true;
                    if (any_ray) { s_inst[col] = ii; s_t[col] = ct; finish = true; }
                }
                w0++;
                w1--;
                pop = !finish && w1 == 0u;
            }
        }
        if (pop) {
            if (sp == tb && level == 1u) {
                // leave the instance: ray.t = ray_local.t (accelstruct.hlsl:146, 170-174)
                if (hit_here) { s_inst[col] = ii; s_t[col] = ct; }
                level = 0; nb = S.tpairs; tb = 0;
                const float4 so = s_wo[col], sd = s_wd[col];
                co = xyz(so); cd = xyz(sd); ci = mk(so.w, sd.w, s_wiz[col]);
            }
            if (sp > tb) {
                const uint2 e = stack_pop();
                w0 = e.x; w1 = e.y;
            } else {
                finish = true;
            }
        }
        if (finish) {
            level = kEnded; w1 = 1u;
            if constexpr (CH) {
                if (!ok) s_t[col] = -1.0f;
            } else {
                io.store(ri, hit_record(), ok);
                ri = kNoRay;
            }
        }
    }
}

// One ray traced by one thread in nested TLAS / BLAS loops (the structure of
// accelstruct.hlsl:58-218 as written), for the megakernel path.  It visits the
// same nodes and triangles in the same order as trace_persistent and returns
// the same hit; false when a stack overflowed (the hit is then a miss).
template <bool ANY>
__device__ __forceinline__ bool trace_single(const SceneRefs& S, uint32_t root, V3 wo, V3 wd, float tmax,
                                             bool no_cull, Hit& h) {
    h.inst = kInvalid; h.prim = kInvalid; h.t = FLT_MAX; h.u = 0.0f; h.v = 0.0f;
    if (root == kInvalid || !in_bounds(root, S.tnode_count, S.status)) return true;
    const V3 wi = rcp(wd);
    float wt = tmax;
    float4 n0 = ldg4(S.tnodes + 2ull * root), n1 = ldg4(S.tnodes + 2ull * root + 1);
    if (slab(xyz(n0), xyz(n1), wo, wi, wt) == FLT_MAX) return true;
    uint32_t t0 = __float_as_uint(n0.w), t1 = __float_as_uint(n1.w);
    uint2 tstack[kStack];
    int tsp = 0;
    for (;;) {
        if (t0 == 0u) {
            // trace_ray_bvh_instance: the ray in object space, t shared
            const uint32_t ii = t1;
            const float4* ip = S.tinst + 4ull * ii;
            const float4 c0 = in_bounds(ii, S.inst_count, S.status) ? ldg4(ip) : make_float4(0.f, 0.f, 0.f, 0.f);
            if (!in_bounds(ii, S.inst_count, nullptr) || !in_bounds(__float_as_uint(c0.w), S.mesh_count, S.status)) {
                if (tsp == 0) break;
                const uint2 e = tstack[--tsp];
                t0 = e.x; t1 = e.y;
                continue;
            }
            const float4 c1 = ldg4(ip + 1), c2 = ldg4(ip + 2), c3 = ldg4(ip + 3);
            const V3 co = xform(wo, 1.0f, c0, c1, c2, c3);
            const V3 cd = xform(wd, 0.0f, c0, c1, c2, c3);
            const V3 ci = rcp(cd);
            float ct = wt;
            const BlasRef B = S.blas[__float_as_uint(c0.w)];
            const float4 r0 = ldg4(B.nodes), r1 = ldg4(B.nodes + 1);
            uint32_t b0 = __float_as_uint(r0.w), b1 = __float_as_uint(r1.w);
            uint2 bstack[kStack];
            int bsp = 0;
            bool hit_here = false;
            for (;;) {
                bool pop = false;
                if (b1 > 0u && !in_bounds((uint64_t)b0 + b1 - 1u, B.tri_count, S.status)) {
                    pop = true;
                } else if (b1 > 0u) {
                    for (uint32_t i = b0; i < b0 + b1; ++i) {
                        const float4* tp = B.tris + 3ull * i;
                        const float4 a = ldg4(tp), b = ldg4(tp + 1), c = ldg4(tp + 2);
                        float bu, bv;
                        if (tri_hit(xyz(a), xyz(b), xyz(c), co, cd, ct, bu, bv, no_cull)) {
                            h.prim = __float_as_uint(a.w);
                            h.u = bu; h.v = bv;
                            hit_here = true;
                            if (ANY) { h.inst = ii; h.t = ct; return true; }
                        }
                    }
                    pop = true;
                } else if (!in_bounds(b0 + 1ull, B.node_count, S.status)) {
                    pop = true;
                } else {
                    const float4* pa = B.nodes + 2ull * b0;
                    const float4 a0 = ldg4(pa), a1 = ldg4(pa + 1), q0 = ldg4(pa + 2), q1 = ldg4(pa + 3);
                    float dl = slab(xyz(a0), xyz(a1), co, ci, ct);
                    float dr = slab(xyz(q0), xyz(q1), co, ci, ct);
                    uint2 L = make_uint2(__float_as_uint(a0.w), __float_as_uint(a1.w));
                    uint2 R = make_uint2(__float_as_uint(q0.w), __float_as_uint(q1.w));
                    if (dl > dr) { float td = dl; dl = dr; dr = td; uint2 tn = L; L = R; R = tn; }
                    if (dl == FLT_MAX) {
                        pop = true;
                    } else {
                        b0 = L.x; b1 = L.y;
                        if (dr != FLT_MAX) {
                            if (bsp == kStack) {
                                h.inst = kInvalid; h.prim = kInvalid; h.t = FLT_MAX; h.u = 0.0f; h.v = 0.0f;
                                return false;
                            }
                            bstack[bsp++] = R;
                        }
                    }
                }
                if (pop) {
                    if (bsp == 0) break;
                    const uint2 e = bstack[--bsp];
                    b0 = e.x; b1 = e.y;
                }
            }
            wt = ct;
            if (hit_here) { h.inst = ii; h.t = wt; }
            if (tsp == 0) break;
            const uint2 e = tstack[--tsp];
            t0 = e.x; t1 = e.y;
            continue;
        }
        if (!(in_bounds(t0 >> 16, S.tnode_count, S.status) && in_bounds(t0 & 0xFFFFu, S.tnode_count, S.status))) {
            if (tsp == 0) break;
            const uint2 e = tstack[--tsp];
            t0 = e.x; t1 = e.y;
            continue;
        }
        const float4* pa = S.tnodes + 2ull * (t0 >> 16);
        const float4* pb = S.tnodes + 2ull * (t0 & 0xFFFFu);
        const float4 a0 = ldg4(pa), a1 = ldg4(pa + 1), q0 = ldg4(pb), q1 = ldg4(pb + 1);
        float dl = slab(xyz(a0), xyz(a1), wo, wi, wt);
        float dr = slab(xyz(q0), xyz(q1), wo, wi, wt);
        uint2 L = make_uint2(__float_as_uint(a0.w), __float_as_uint(a1.w));
        uint2 R = make_uint2(__float_as_uint(q0.w), __float_as_uint(q1.w));
        if (dl > dr) { float td = dl; dl = dr; dr = td; uint2 tn = L; L = R; R = tn; }
        if (dl == FLT_MAX) {
            if (tsp == 0) break;
            const uint2 e = tstack[--tsp];
            t0 = e.x; t1 = e.y;
        } else {
            t0 = L.x; t1 = L.y;
            if (dr != FLT_MAX) {
                if (tsp == kStack) {
                    h.inst = kInvalid; h.prim = kInvalid; h.t = FLT_MAX; h.u = 0.0f; h.v = 0.0f;
                    return false;
                }
                tstack[tsp++] = R;
            }
        }
    }
    return true;
}

// Adds a thread's fetch counts to the global counters (one atomic per warp).
__device__ __forceinline__ void flush_counters(const LocalCounters& c, Counters* g) {
    unsigned long long a = c.tlas_nodes, b = c.instances, x = c.blas_nodes, y = c.tris;
    for (int off = 16; off > 0; off >>= 1) {
        a += __shfl_down_sync(0xffffffffu, a, off);
        b += __shfl_down_sync(0xffffffffu, b, off);
        x += __shfl_down_sync(0xffffffffu, x, off);
        y += __shfl_down_sync(0xffffffffu, y, off);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&g->tlas_node_loads, a);
        atomicAdd(&g->instance_loads, b);
        atomicAdd(&g->blas_node_loads, x);
        atomicAdd(&g->triangle_tests, y);
    }
}

// Minimum resident blocks per SM asked of the compiler for the traversal
// kernels (it caps their registers at 65536 / (128 * blocks)): 9 blocks = 56
// registers, 36 warps per SM, for a few bytes of spills in the closest-hit
// kernel (measured fastest against 7-8 blocks without spills and 10 blocks
// with 50+ bytes of spills).
#ifndef WF_TRACE_MIN_BLOCKS
#define WF_TRACE_MIN_BLOCKS 9
#endif
// The same for the 4-wide BLAS layouts, whose node step holds four child
// boxes and their sort keys at once: 8 blocks (64 registers) measured 1-3 %
// faster than 9 (56 registers, 40-72 bytes of spills) on both layouts.
#ifndef WF_TRACE_QB_MIN_BLOCKS
#define WF_TRACE_QB_MIN_BLOCKS 8
#endif
// The traversal kernel: a persistent grid over count rays (read from
// count_ptr on the device when it is non-null), rays handed out from *fetch.
// total (optional) accumulates the number of rays of each launch.
template <bool ANY, bool COUNT, int LAY, class IO>
__global__ void __launch_bounds__(kTraceBlock, LAY ? WF_TRACE_QB_MIN_BLOCKS : WF_TRACE_MIN_BLOCKS) k_trace(SceneRefs S, IO io, const uint32_t* count_ptr, uint32_t count,
                                                  uint32_t* fetch, uint32_t* status, Counters* counters,
                                                  unsigned long long* total) {
    const uint32_t n = count_ptr ? *count_ptr : count;
    if (total && blockIdx.x == 0 && threadIdx.x == 0) atomicAdd(total, (unsigned long long)paths_of(io, n));
    LocalCounters c = {0, 0, 0, 0};
    bool overflow = false;
    trace_persistent<ANY, COUNT, LAY>(S, io, n, fetch, c, overflow);
    if (overflow) atomicOr(status, ERRF_STACK);
    if (COUNT) flush_counters(c, counters);
}

}  // namespace wf
