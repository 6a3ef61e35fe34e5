// wf_finish.cu — a short wave, or the tail of one, in one launch: its paths run
// through all their (remaining) bounces without going back to the queues.
//
// A staged depth (extend, shade, connect launches) lasts at least as long as
// its slowest ray, about 90 us for extend and 50 for connect, however few rays
// are left, while most of the grid idles.  Here a lane keeps its path: its ray
// steps in the warp-uniform traversal loop of trace_persistent (the same nodes
// in the same order), and when it ends the path's next() shades the hit
// (shade_one) and hands back the shadow ray, then the next extension ray.  The
// launch lasts as long as the longest path's own rays, not as long as the sum
// over the depths of each depth's slowest ray.
//
// The path state is the wavefront's own (queue entry i, ps_T / ps_flags / ps_L
// by path, in L2): only the traversal's state and the depth live in registers,
// so the loop keeps its occupancy and next() alone pays for the loads.  A
// path's additions stay in the staged order (the event of depth d, its shadow
// ray, depth d + 1), so its radiance is the same bit for bit.
//
// What bounds it: the latency of a warp's dependent node fetches.  A 256x256
// box frame (65,536 paths, depth 4): 299 -> 235 us against the staged launches
// (wf_api.cu, kWholePaths); the tail of a 1080p instanced frame from 100,000
// paths: 17.31 ms per frame with one thread per path in nested loops, 16.55 here
// (16.69 staged).
#include "wf_shade.cuh"
#include "wf_traverse.cuh"

namespace wf {

namespace {

// Resident blocks of 128 asked of the compiler: 4 (128 registers, the shading's
// need) 255 us per 256x256 box frame, 6 (80 registers, 320 bytes of spills)
// 275, 8: 299, all with lanes waiting for 8 others.
#ifndef WF_FINISH_MIN_BLOCKS
#define WF_FINISH_MIN_BLOCKS 4
#endif

struct FinishIO {
    static constexpr bool kChain = true;
    const ShadeRefs& SH;
    const RenderBuffers& B;
    const WaveParams& W;
    uint32_t* s_ext;        // shared, kMaxDepth: extension rays started at depths after the first
    uint32_t* s_sh;         // shared, kMaxDepth: shadow rays started
    uint32_t depth0;        // the depth of the queue's entries
    // this lane's path
    uint32_t depth = 0;
    uint32_t kind = 0;      // its ray: kExtend, or a shadow ray of a path that continues / has ended
    enum : uint32_t { kExtend = 0, kShadow = 1, kShadowLast = 2 };

    // selects, not dynamic indices into the parameter
    __device__ __forceinline__ float4* qo() const { return (depth0 & 1u) ? B.q_o[1] : B.q_o[0]; }
    __device__ __forceinline__ float4* qd() const { return (depth0 & 1u) ? B.q_d[1] : B.q_d[0]; }
    __device__ __forceinline__ const uint32_t* qp() const { return (depth0 & 1u) ? B.q_path[1] : B.q_path[0]; }
    __device__ __forceinline__ float4* sc() const { return (depth0 & 1u) ? B.s_c[1] : B.s_c[0]; }

    __device__ __forceinline__ uint32_t path_of(uint32_t i) const {
        const uint32_t p = depth0 ? qp()[i] : i;
        return in_bounds(p, W.npaths, B.status) ? p : 0u;   // checked builds: flagged, path 0 stands in
    }
    __device__ __forceinline__ uint32_t root(uint32_t, const SceneRefs& S) const { return S.inst_count ? 0u : kInvalid; }

    __device__ __forceinline__ void queued_ray(uint32_t i, V3& o, V3& d, float& tmax, bool& nc, bool& any) {
        const float4 a = qo()[i], b = qd()[i];
        o = xyz(a); d = xyz(b); tmax = FLT_MAX;
        nc = (__float_as_uint(a.w) & kFlagInside) != 0u;
        any = false;
        kind = kExtend;
    }
    __device__ __forceinline__ bool load(uint32_t i, V3& o, V3& d, float& tmax, bool& nc, bool& any) {
        depth = depth0;
        if (depth0 == 0u) {
            const uint32_t pixel = W.pix0 + i / W.nsamples;
            primary_ray(W, pixel % W.width, pixel / W.width, o, d);
            tmax = FLT_MAX; nc = false; any = false;
            kind = kExtend;
            return true;
        }
        if (!in_bounds(i, B.capacity, B.status)) return false;
        queued_ray(i, o, d, tmax, nc, any);
        return true;
    }

    __device__ __forceinline__ bool next(uint32_t i, const Hit& h, V3 rd, V3& o, V3& d, float& tmax, bool& nc,
                                         bool& any) {
        const uint32_t path = path_of(i);
        if (kind != kExtend) {
            if (h.inst == kInvalid && h.t >= 0.0f) {
                const float4 k = sc()[i];
                float4 acc = B.ps_L[path];
                acc.x = acc.x + k.x;
                acc.y = acc.y + k.y;
                acc.z = acc.z + k.z;
                B.ps_L[path] = acc;
            }
            if (kind == kShadowLast) return false;
            depth++;
            atomicAdd(&s_ext[depth], 1u);
            queued_ray(i, o, d, tmax, nc, any);
            return true;
        }
        ShadeCtl K;
        K.frame_seed = W.frame_seed; K.max_bounces = W.max_bounces; K.nee = W.nee; K.rr_start = W.rr_start;
        K.cosine = W.cosine; K.env_strength = W.env_strength; K.env0 = W.env[0]; K.env1 = W.env[1]; K.env2 = W.env[2];
        K.lights = SH.lights; K.light_count = SH.light_count; K.light_total = SH.light_total;
        K.env_tex = W.env_tex; K.view_mode = 0u; K.far_plane = W.far_plane;
        ShadeIn in;
        in.rd = rd;
        in.tuvp = make_float4(h.t < 0.0f ? FLT_MAX : h.t, h.u, h.v, __uint_as_float(h.prim));
        in.inst = h.inst;
        if (depth) {
            const float4 T4 = B.ps_T[path];
            in.T = xyz(T4);
            in.last_pdf = T4.w;
            in.flags = B.ps_flags[path];
        } else {
            in.T = mk(1.0f, 1.0f, 1.0f);
            in.last_pdf = 0.0f;
            in.flags = kFlagSpecular;
        }
        in.pixel = W.pix0 + path / W.nsamples;
        in.sample = W.s0 + path % W.nsamples;
        in.depth = depth;
        const AdjointRefs none = {};
        ShadeOut out;
        shade_one(SH, K, in, none, 0u, 0u, out);
        if (out.has_add || depth == 0u) {
            float4 acc = depth ? B.ps_L[path] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            if (out.has_add) {
                acc.x = acc.x + out.add.x;
                acc.y = acc.y + out.add.y;
                acc.z = acc.z + out.add.z;
            }
            B.ps_L[path] = acc;
        }
        if (out.enqueue) {
            B.ps_T[path] = make_float4(out.T.x, out.T.y, out.T.z, out.pdf);
            B.ps_flags[path] = out.flags;
        }
        if (out.shadow) {
            if (out.enqueue) {
                qo()[i] = make_float4(out.org.x, out.org.y, out.org.z, __uint_as_float(out.flags & kFlagInside));
                qd()[i] = make_float4(out.dir.x, out.dir.y, out.dir.z, FLT_MAX);
            }
            sc()[i] = make_float4(out.contrib.x, out.contrib.y, out.contrib.z, 0.0f);
            atomicAdd(&s_sh[depth], 1u);
            o = out.spos; d = out.sdir; tmax = out.stmax; nc = false;
            any = true;
            kind = out.enqueue ? kShadow : kShadowLast;
            return true;
        }
        if (!out.enqueue) return false;
        depth++;
        atomicAdd(&s_ext[depth], 1u);
        o = out.org; d = out.dir; tmax = FLT_MAX;
        nc = (out.flags & kFlagInside) != 0u;
        return true;
    }
};

__global__ void __launch_bounds__(kTraceBlock, WF_FINISH_MIN_BLOCKS)
    k_finish(const __grid_constant__ SceneRefs S, const __grid_constant__ ShadeRefs SH,
             const __grid_constant__ RenderBuffers B, const __grid_constant__ WaveParams W, uint32_t depth0,
             uint32_t* fetch, unsigned long long* totals) {
    const uint32_t n = depth0 ? B.counts[depth0] : W.npaths;
    __shared__ uint32_t s_ext[kMaxDepth], s_sh[kMaxDepth];
    if (threadIdx.x < kMaxDepth) { s_ext[threadIdx.x] = 0u; s_sh[threadIdx.x] = 0u; }
    __syncthreads();
    FinishIO io{SH, B, W, s_ext, s_sh, depth0};
    LocalCounters c = {0, 0, 0, 0};
    bool overflow = false;
    trace_persistent<false, false, 0>(S, io, n, fetch, c, overflow);
    if (overflow) atomicOr(B.status, ERRF_STACK);
    __syncthreads();
    if (threadIdx.x < kMaxDepth) {
        const uint32_t e = s_ext[threadIdx.x], s = s_sh[threadIdx.x];
        if (e) { atomicAdd(&B.counts[threadIdx.x], e); atomicAdd(&totals[0], (unsigned long long)e); }
        if (s) { atomicAdd(&B.counts[kMaxDepth + threadIdx.x], s); atomicAdd(&totals[1], (unsigned long long)s); }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (depth0 == 0u) B.counts[0] = n;
        atomicAdd(&totals[0], (unsigned long long)n);
    }
}

}  // namespace

cudaError_t launch_finish(const SceneRefs& S, const ShadeRefs& SH, const RenderBuffers& B, const WaveParams& W,
                          uint32_t depth, unsigned long long* totals, cudaStream_t stream) {
    k_finish<<<persistent_grid<k_finish, kTraceBlock>(), kTraceBlock, 0, stream>>>(S, SH, B, W, depth,
                                                                    B.counts + 2 * kMaxDepth + depth, totals);
    return cudaGetLastError();
}

}  // namespace wf
