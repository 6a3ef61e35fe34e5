// wf_shade.cu — shade (shade.hlsl:42-174 plus the added metal / dielectric /
// next-event / Russian-roulette steps; at depth 0 it also stands in for
// clear_buffers.hlsl + generate.hlsl: the camera rays themselves are made in
// the depth-0 traversal launch) and post-process (post_process.hlsl:25-72).
//
// The per-path arithmetic is the CPU oracle's (oracle/orc_impl.h) operation
// for operation; both are compiled without fused multiply-add.
#include "wf_shade.cuh"

namespace wf {

namespace {

constexpr int kBlock = 256;

unsigned grid_for(uint32_t n) {
    unsigned blocks = (n + kBlock - 1) / kBlock;
    unsigned cap = (unsigned)sm_count() * 8u;
    if (blocks > cap) blocks = cap;
    return blocks ? blocks : 1u;
}

// Shade's block size and, for path tracing, the resident blocks per SM asked of
// the compiler (which caps its registers accordingly): 768 threads per SM (80
// registers, some spills) measured 7 % faster per frame's shade than 512 (126
// registers).  6 blocks of 128 rather than 3 of 256, whose barriers hold more
// warps up: 613x377 textured frame 1.770 -> 1.758 ms, 1080p instanced frame 9.87
// -> 9.85; 5 of 128: 1.786 and 9.98.
#ifndef WF_SHADE_BLOCK
#define WF_SHADE_BLOCK 128
#endif
#ifndef WF_SHADE_MIN_BLOCKS
#define WF_SHADE_MIN_BLOCKS 6
#endif
constexpr int kShadeBlock = WF_SHADE_BLOCK;

// Path tracing (kPlain), path tracing that also keeps the radiance sums'
// rounding errors and records the hits (kRecord, wf_adjoint's forward pass),
// and the debug views (kViews, at 2 resident blocks).
enum ShadeMode { kPlain, kRecord, kViews };
template <int MODE>
__global__ void __launch_bounds__(kShadeBlock, MODE == kViews ? 2 : WF_SHADE_MIN_BLOCKS)
    k_shade(ShadeRefs SH, RenderBuffers B, WaveParams W, uint32_t depth) {
    const AdjointRefs none = {};
    // depth 0 shades the camera paths of the wave in path order, their state
    // the one a path starts with (throughput 1, specular flag, no radiance),
    // so nothing is read but the hit; it also records the depth-0 count
    const uint32_t n = depth ? B.counts[depth] : W.npaths;
    if (depth == 0 && blockIdx.x == 0 && threadIdx.x == 0) B.counts[0] = W.npaths;
    const int cur = depth & 1, nxt = cur ^ 1;
    ShadeCtl K;
    K.frame_seed = W.frame_seed; K.max_bounces = W.max_bounces; K.nee = W.nee; K.rr_start = W.rr_start;
    K.cosine = W.cosine; K.env_strength = W.env_strength; K.env0 = W.env[0]; K.env1 = W.env[1]; K.env2 = W.env[2];
    K.lights = SH.lights; K.light_count = SH.light_count; K.light_total = SH.light_total;
    K.env_tex = W.env_tex; K.view_mode = MODE == kViews ? W.view_mode : 0u; K.far_plane = W.far_plane;
    // shadow queue of this depth's parity (selects, not a dynamic index into the parameter)
    float4* const s_o = cur ? B.s_o[1] : B.s_o[0];
    float4* const s_d = cur ? B.s_d[1] : B.s_d[0];
    float4* const s_c = cur ? B.s_c[1] : B.s_c[0];
    __shared__ BlockAppend<kShadeBlock> append;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += stride) {
        const uint32_t i = base + threadIdx.x;
        ShadeOut o;
        o.enqueue = false; o.shadow = false;
        o.dir = mk(0, 0, 0); o.sdir = mk(0, 0, 0);
        uint32_t path = 0;
        if (i < n) {
            ShadeIn in;
            if (depth == 0) {
                path = i;
                in.pixel = W.pix0 + path / W.nsamples;
                V3 ro;
                primary_ray(W, in.pixel % W.width, in.pixel / W.width, ro, in.rd);
                in.T = mk(1.0f, 1.0f, 1.0f);
                in.last_pdf = 0.0f;
                in.flags = kFlagSpecular;
            } else {
                path = B.q_path[cur][i];
                if (!in_bounds(path, W.npaths, B.status)) path = 0u;   // checked builds: flagged, path 0 stands in
                in.pixel = W.pix0 + path / W.nsamples;
                in.rd = xyz(B.q_d[cur][i]);
                const float4 T4 = B.ps_T[path];
                in.T = xyz(T4);
                in.last_pdf = T4.w;
                in.flags = B.ps_flags[path];
            }
            const uint32_t hit = depth ? i : i / W.camera_share;
            in.tuvp = B.h_tuvp[hit];
            in.inst = B.h_inst[hit];
            in.sample = W.s0 + path % W.nsamples;
            in.depth = depth;
            if (MODE == kRecord) {
                const size_t at = (size_t)depth * W.npaths + path;
                B.tape_tuvp[at] = in.tuvp;
                B.tape_inst[at] = in.inst;
            }
            shade_one(SH, K, in, none, 0u, 0u, o);
            if (o.has_add || depth == 0) {
                // the path's radiance starts at zero here
                float4 acc = depth ? B.ps_L[path] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (MODE == kRecord) {
                    float4 lc = depth ? B.ps_Lc[path] : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                    if (o.has_add) {
                        float e;
                        acc.x = two_sum(acc.x, o.add.x, e); lc.x = lc.x + e;
                        acc.y = two_sum(acc.y, o.add.y, e); lc.y = lc.y + e;
                        acc.z = two_sum(acc.z, o.add.z, e); lc.z = lc.z + e;
                    }
                    B.ps_Lc[path] = lc;
                } else if (o.has_add) {
                    acc.x = acc.x + o.add.x;
                    acc.y = acc.y + o.add.y;
                    acc.z = acc.z + o.add.z;
                }
                B.ps_L[path] = acc;
            }
        }
        uint2 slots;
        if (MODE == kPlain) {
            slots = append(&B.counts[depth + 1], o.enqueue, o.dir, &B.counts[kMaxDepth + depth], o.shadow, o.sdir);
        } else {
            // the adjoint's tape is written by path, and loses more to a queue out
            // of path order (33.0 -> 34.1 ms) than its rays gain
            slots.x = warp_append(&B.counts[depth + 1], o.enqueue);
            slots.y = warp_append(&B.counts[kMaxDepth + depth], o.shadow);
        }
        const uint32_t slot = slots.x, sslot = slots.y;
        if (o.enqueue && in_bounds(slot, B.capacity, B.status)) {
            B.q_o[nxt][slot] = make_float4(o.org.x, o.org.y, o.org.z, __uint_as_float(o.flags & kFlagInside));
            B.q_d[nxt][slot] = make_float4(o.dir.x, o.dir.y, o.dir.z, FLT_MAX);
            B.q_path[nxt][slot] = path;
            B.ps_T[path] = make_float4(o.T.x, o.T.y, o.T.z, o.pdf);
            B.ps_flags[path] = o.flags;
        }
        if (o.shadow && in_bounds(sslot, B.capacity, B.status)) {
            s_o[sslot] = make_float4(o.spos.x, o.spos.y, o.spos.z, o.stmax);
            s_d[sslot] = make_float4(o.sdir.x, o.sdir.y, o.sdir.z, __uint_as_float(path));
            s_c[sslot] = make_float4(o.contrib.x, o.contrib.y, o.contrib.z, __uint_as_float(o.light_inst));
        }
    }
}

// The adjoint's replay, one path per thread: every event of the path is shaded
// again from the hit that the forward pass recorded, so no ray is traced and no
// queue written; the path's state and its radiance so far (with its rounding
// errors) stay in registers, summed in the forward pass's order.  The gradients
// go out as shade_one's atomics, the emitters' into 32 replicas: a path sums its
// terms of one emitter, a shadow ray's and the emission it ends at, and a warp
// its paths'.  One number
// per emitter sums millions of terms whose signs cancel where the image
// gradient's do, so paths, warps and replicas add in double: over 12 image
// gradients of the adjoint below, 1e-8 to 1.1e-6 from the FP64 sum over the
// image, against 2e-7 to 2.4e-5 with float replicas and up to 5e-5 with one
// float per emitter.  (An atomic per shadow ray instead took 50.7 ms with
// next-event estimation, 43.1 so; without, where the kernel leaves that code out,
// 28.85 and 28.10.)
//
// Bound by the gathers of shade_one and the albedo atomics.  A 512x512 x 64
// sample adjoint of depth 6 took 70.6 ms with a replay that traced every ray
// again through the staged launches, 39.2 ms so on the traversal loop of that
// time and 28.0 ms now.  4 / 5 / 6 / 7 resident blocks: 28.04 / 28.03 / 28.08 /
// 27.87 ms, with next-event estimation 43.98 / 43.04 / 42.94 / 42.83.
constexpr int kReplayBlock = 128, kReplayMinBlocks = 5;
template <bool NEE>
__global__ void __launch_bounds__(kReplayBlock, kReplayMinBlocks)
    k_replay(ShadeRefs SH, RenderBuffers B, WaveParams W, AdjointRefs A) {
    const uint32_t path = blockIdx.x * kReplayBlock + threadIdx.x;
    ShadeCtl K;
    K.frame_seed = W.frame_seed; K.max_bounces = W.max_bounces; K.nee = NEE ? 1u : 0u; K.rr_start = W.rr_start;
    K.cosine = W.cosine; K.env_strength = W.env_strength; K.env0 = W.env[0]; K.env1 = W.env[1]; K.env2 = W.env[2];
    K.lights = SH.lights; K.light_count = SH.light_count; K.light_total = SH.light_total;
    K.env_tex = W.env_tex; K.view_mode = 0u; K.far_plane = W.far_plane;
    uint32_t em_key = kInvalid;
    double em_val = 0.0;
    if (path < W.npaths) {
        ShadeIn in;
        in.pixel = W.pix0 + path / W.nsamples;
        in.sample = W.s0 + path % W.nsamples;
        V3 ro;
        primary_ray(W, in.pixel % W.width, in.pixel / W.width, ro, in.rd);
        in.T = mk(1.0f, 1.0f, 1.0f);
        in.last_pdf = 0.0f;
        in.flags = kFlagSpecular;
        in.Lb = mk(0.0f, 0.0f, 0.0f);
        in.Lb_lo = in.Lb;
        auto gather = [&](V3 c) {
            float e;
            in.Lb.x = two_sum(in.Lb.x, c.x, e); in.Lb_lo.x = in.Lb_lo.x + e;
            in.Lb.y = two_sum(in.Lb.y, c.y, e); in.Lb_lo.y = in.Lb_lo.y + e;
            in.Lb.z = two_sum(in.Lb.z, c.z, e); in.Lb_lo.z = in.Lb_lo.z + e;
        };
        auto emitted = [&](uint32_t key, float v) {
            if (key != em_key) {
                if (em_key != kInvalid) atomicAdd(&A.g_em_rep[(size_t)(path & 31u) * A.instances + em_key], em_val);
                em_key = key;
                em_val = 0.0;
            }
            em_val += v;
        };
        for (uint32_t depth = 0; depth <= W.max_bounces; ++depth) {
            const size_t at = (size_t)depth * W.npaths + path;
            in.tuvp = B.tape_tuvp[at];
            in.inst = B.tape_inst[at];
            in.depth = depth;
            ShadeOut o;
            shade_one(SH, K, in, A, path, in.pixel, o);
            if (o.has_add) gather(o.add);
            if (o.em_key != kInvalid) emitted(o.em_key, o.em_val);   // the path ends at an emitter
            if (NEE && o.shadow && B.tape_clear[at]) {
                gather(o.contrib);
                // linear in the emitter's strength
                if (in_bounds(o.light_inst, A.instances, B.status)) {
                    const float strength = SH.sinst[(size_t)kInstRows * o.light_inst + 5].w;
                    if (strength != 0.0f) {
                        const float4 g = A.dimage[in.pixel];
                        const float v = (g.x * A.inv_spp) * o.contrib.x + (g.y * A.inv_spp) * o.contrib.y +
                                        (g.z * A.inv_spp) * o.contrib.z;
                        emitted(o.light_inst, v / strength);
                    }
                }
            }
            if (!o.enqueue) break;
            in.rd = o.dir;
            in.T = o.T;
            in.last_pdf = o.pdf;
            in.flags = o.flags;
        }
    }
    const uint32_t rep = (blockIdx.x * (kReplayBlock / 32) + (threadIdx.x >> 5)) & 31u;
    warp_add_by_key(A.g_em_rep + (size_t)rep * A.instances, em_key, em_val);
}

// post_process.hlsl:25-72 with accumulate on: average, NaN/Inf -> magenta,
// Reinhard, linear -> sRGB, RGBA8.
__device__ __forceinline__ float srgb(float c) {
    float x = fminf(fmaxf(c, 0.0f), 1.0f);
    return (x <= 0.0031308f) ? x * 12.92f : 1.055f * powf(x, 1.0f / 2.4f) - 0.055f;
}
__device__ __forceinline__ unsigned char unorm8(float c) {
    return (unsigned char)(fminf(fmaxf(c, 0.0f), 1.0f) * 255.0f + 0.5f);
}
__device__ __forceinline__ bool bad(float x) { return isnan(x) || isinf(x); }

__global__ void k_post(const float4* __restrict__ accum, uint32_t npix, uint32_t view_mode, uchar4* __restrict__ out) {
    const bool tonemap = view_mode == RENDER_VIEW_MODE_NONE;
    const bool to_srgb = tonemap || view_mode == RENDER_VIEW_MODE_MATERIAL_BASE_COLOR ||
                         view_mode == RENDER_VIEW_MODE_MATERIAL_EMISSIVE;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += stride) {
        float4 a = accum[i];
        float inv = a.w > 0.0f ? 1.0f / a.w : 0.0f;
        float r = a.x * inv, g = a.y * inv, b = a.z * inv;
        if (bad(r) || bad(g) || bad(b)) { r = 1.0f; g = 0.0f; b = 1.0f; }
        if (tonemap) { r = r / (1.0f + r); g = g / (1.0f + g); b = b / (1.0f + b); }
        if (to_srgb) { r = srgb(r); g = srgb(g); b = srgb(b); }
        out[i] = make_uchar4(unorm8(r), unorm8(g), unorm8(b), 255);
    }
}

__global__ void k_wave_resolve(RenderBuffers B, WaveParams W) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t p = blockIdx.x * blockDim.x + threadIdx.x; p < W.np; p += stride) {
        float4 acc = B.accum[W.pix0 + p];
        sum_samples(B.ps_L + (size_t)p * W.nsamples, W.nsamples, acc);
        B.accum[W.pix0 + p] = acc;
    }
}

__global__ void k_resolve(const float4* __restrict__ accum, uint32_t npix, float4* __restrict__ out) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < npix; i += stride) {
        float4 a = accum[i];
        out[i] = a.w > 0.0f ? make_float4(a.x / a.w, a.y / a.w, a.z / a.w, a.w) : make_float4(0, 0, 0, 0);
    }
}

__global__ void k_reduce_replicas(float4* g, uint32_t triangles, uint32_t replicas) {
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < triangles; t += stride) {
        float4 a = g[t];
        for (uint32_t r = 1; r < replicas; ++r) {
            const float4 b = g[(size_t)r * triangles + t];
            a.x += b.x; a.y += b.y; a.z += b.z;
        }
        g[t] = a;
    }
}

}  // namespace

cudaError_t launch_shade(const ShadeRefs& SH, const RenderBuffers& B, const WaveParams& W, uint32_t depth,
                         uint32_t max_rays, cudaStream_t stream) {
    unsigned blocks = (max_rays + kShadeBlock - 1) / kShadeBlock;
    const unsigned cap = (unsigned)sm_count() * 8u * (256u / kShadeBlock);
    if (blocks > cap) blocks = cap;
    if (blocks == 0) blocks = 1;
    if (B.ps_Lc) k_shade<kRecord><<<blocks, kShadeBlock, 0, stream>>>(SH, B, W, depth);
    else if (W.view_mode == 0u) k_shade<kPlain><<<blocks, kShadeBlock, 0, stream>>>(SH, B, W, depth);
    else k_shade<kViews><<<blocks, kShadeBlock, 0, stream>>>(SH, B, W, depth);
    return cudaGetLastError();
}

cudaError_t launch_replay(const ShadeRefs& SH, const RenderBuffers& B, const WaveParams& W, const AdjointRefs& A,
                          cudaStream_t stream) {
    const auto replay = W.nee ? k_replay<true> : k_replay<false>;
    replay<<<(W.npaths + kReplayBlock - 1) / kReplayBlock, kReplayBlock, 0, stream>>>(SH, B, W, A);
    return cudaGetLastError();
}

cudaError_t launch_reduce_replicas(float4* g, uint32_t triangles, uint32_t replicas, cudaStream_t stream) {
    k_reduce_replicas<<<grid_for(triangles), kBlock, 0, stream>>>(g, triangles, replicas);
    return cudaGetLastError();
}

namespace {
__global__ void k_depth_counts(const uint32_t* counts, unsigned long long* per_depth) {
    const uint32_t d = threadIdx.x;
    if (d < 2 * kMaxDepth) per_depth[d] += counts[d];
}
}  // namespace

cudaError_t launch_depth_counts(const uint32_t* counts, unsigned long long* per_depth, cudaStream_t stream) {
    k_depth_counts<<<1, 2 * kMaxDepth, 0, stream>>>(counts, per_depth);
    return cudaGetLastError();
}

cudaError_t launch_wave_resolve(const RenderBuffers& B, const WaveParams& W, cudaStream_t stream) {
    k_wave_resolve<<<grid_for(W.np), kBlock, 0, stream>>>(B, W);
    return cudaGetLastError();
}

cudaError_t launch_post(const float4* accum, uint32_t npix, uint32_t view_mode, uchar4* out, cudaStream_t stream) {
    k_post<<<grid_for(npix), kBlock, 0, stream>>>(accum, npix, view_mode, out);
    return cudaGetLastError();
}

cudaError_t launch_resolve(const float4* accum, uint32_t npix, float4* out, cudaStream_t stream) {
    k_resolve<<<grid_for(npix), kBlock, 0, stream>>>(accum, npix, out);
    return cudaGetLastError();
}

}  // namespace wf
