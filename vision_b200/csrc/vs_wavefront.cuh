// Device side of the wavefront path tracer: the per-slot path state and the
// bodies of the bounce kernels (traversal, shading), shared by
// the single-scene renderer (wavefront.cu) and the job server (server.cu).
// `Scenes` maps a slot's scene id to its DeviceScene (one scene for vs_render,
// a table of resident scenes for the server); the scene id of a slot lives in
// st.w, that of a shadow query in sh_c.w.
#pragma once

#include "vs_integrator.cuh"
#include "vs_wavefront.h"

namespace vs {
namespace wf {

__device__ __forceinline__ float comp(const float4 &v, int i) {
    return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
}

template <int N>
__device__ __forceinline__ float4 pack4(const float *a) {
    return make_float4(a[0], N > 1 ? a[1] : 0.0f, N > 2 ? a[2] : 0.0f, N > 3 ? a[3] : 0.0f);
}

template <int N>
__device__ __forceinline__ void store(const WfBuffers &b, uint32_t slot, const PathState<N> &ps, uint32_t scene) {
    b.o[slot] = make_float4(ps.ro.x, ps.ro.y, ps.ro.z, ps.scatter_pdf);
    b.d[slot] = make_float4(ps.rd.x, ps.rd.y, ps.rd.z, ps.eta_scale);
    b.tp[slot] = pack4<N>(ps.throughput.v);
    b.lam[slot] = pack4<N>(ps.wl.lambda);
    b.pdf[slot] = pack4<N>(ps.wl.pdf);
    b.L[slot] = make_float4(ps.L.x, ps.L.y, ps.L.z, ps.filter_w);
    b.st[slot] = make_uint4(static_cast<uint32_t>(ps.smp.state), static_cast<uint32_t>(ps.smp.state >> 32),
                            ps.bounce, scene);
}

// Loads slot `slot`; returns its scene id.
template <int N, class Scenes>
__device__ __forceinline__ uint32_t load(const Scenes &scenes, const WfBuffers &b, uint32_t slot, PathState<N> &ps) {
    const uint4 st = b.st[slot];
    const DeviceScene &s = scenes(st.w);
    const float4 o = b.o[slot], d = b.d[slot], tp = b.tp[slot], lam = b.lam[slot], pdf = b.pdf[slot],
                 L = b.L[slot];
    ps.ro = make3(o.x, o.y, o.z);
    ps.scatter_pdf = o.w;
    ps.rd = make3(d.x, d.y, d.z);
    ps.eta_scale = d.w;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        ps.throughput.v[i] = comp(tp, i);
        ps.wl.lambda[i] = comp(lam, i);
        ps.wl.pdf[i] = comp(pdf, i);
    }
    ps.L = make3(L.x, L.y, L.z);
    ps.filter_w = L.w;
    ps.smp.state = static_cast<uint64_t>(st.x) | (static_cast<uint64_t>(st.y) << 32);
    ps.smp.kind = s.ip.sampler;
    ps.smp.seed = s.ip.seed;
    ps.bounce = st.z;
    return st.w;
}

// Camera paths of a wave: slot i holds path base + i of `cam` (frame-major
// over frames frame_begin, ...), queued for the first bounce; clears every
// counter of the wave.  A scene of max_depth 0 writes each path's (zero)
// radiance directly.
template <int N>
__device__ __forceinline__ void generate(const DeviceScene &s, const Camera &cam, const WfBuffers &b,
                                         uint32_t frame_begin, uint64_t base, uint32_t n, float4 *radiance) {
    const uint32_t npix = cam.width * cam.height;
    if (blockIdx.x == 0 && threadIdx.x < kWfCounters) b.count[threadIdx.x] = threadIdx.x == 0 ? n : 0u;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const uint64_t p = base + i;
        const uint32_t frame = frame_begin + static_cast<uint32_t>(p / npix);
        const uint32_t pix = static_cast<uint32_t>(p % npix);
        PathState<N> ps;
        path_start<N>(s, cam, pix % cam.width, pix / cam.width, frame, ps);
        if (s.ip.max_depth == 0u) {
            radiance[p] = make_float4(0.0f, 0.0f, 0.0f, 1.0f);
            continue;
        }
        store<N>(b, i, ps, 0u);
        b.queue[0][i] = i;
    }
}

// The calling thread's lane in its warp (any block shape: a 16 x 8 block's
// warps hold two rows of threadIdx.x, so threadIdx.x % 32 is not the lane).
__device__ __forceinline__ int lane_id() {
    unsigned lane;
    asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
    return static_cast<int>(lane);
}

// Appends one entry per calling lane to a device queue: one atomicAdd per
// converged group of lanes, positions in lane order.
__device__ __forceinline__ uint32_t queue_push(uint32_t *counter) {
    const unsigned mask = __activemask();
    const int lane = lane_id();
    const int leader = __ffs(mask) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(counter, static_cast<uint32_t>(__popc(mask)));
    base = __shfl_sync(mask, base, leader);
    return base + static_cast<uint32_t>(__popc(mask & ((1u << lane) - 1u)));
}

// Appends the calling lane's slot to the queue of its shading class: one
// atomicAdd per class present among the converged lanes.
__device__ __forceinline__ uint32_t class_push(uint32_t *counts, uint32_t cls) {
    const unsigned active = __activemask();
    const unsigned group = __match_any_sync(active, cls);
    const int lane = lane_id();
    const int leader = __ffs(group) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(counts + cls, static_cast<uint32_t>(__popc(group)));
    base = __shfl_sync(active, base, leader);
    return base + static_cast<uint32_t>(__popc(group & ((1u << lane) - 1u)));
}

// Lanes of a warp that must be idle before the warp takes new rays.
#ifndef VS_REFILL_LANES
#define VS_REFILL_LANES 8
#endif

// Ray replacement for the traversal kernels: the idle lanes of a warp (at
// least VS_REFILL_LANES of them, or all) claim the next rays of a queue of `n`
// with one atomicAdd on `fetch`; returns the claimed index of the calling
// lane (>= n: none) and sets `drained` once the queue is exhausted.  Called by
// all 32 lanes.
__device__ __forceinline__ uint32_t refill(uint32_t *fetch, uint32_t n, bool active, bool &drained) {
    const unsigned idle = __ballot_sync(0xffffffffu, !active);
    const uint32_t k = static_cast<uint32_t>(__popc(idle));
    if (k < VS_REFILL_LANES && k != 32u) return n;
    const int lane = lane_id();
    const int leader = __ffs(idle) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(fetch, k);
    base = __shfl_sync(0xffffffffu, base, leader);
    if (base + k >= n) drained = true;
    if (active) return n;
    return base + static_cast<uint32_t>(__popc(idle & ((1u << lane) - 1u)));
}

// The traversal pass of bounce `round`: the closest hits of the path queue,
// sorted into the shading-class queues, then the shadow queries that the
// shading of the bounce before left (none at round 0; at the round after the
// last bounce the path queue is empty).  Each warp keeps 32 rays in flight and
// refills finished lanes from the queue.  A query adds its contribution when
// unoccluded and writes the radiance of a path that ended at its bounce.
//
// Neither needs the other's results, so one pass does both: a warp that finds
// the path queue empty goes on to the shadow rays while others still trace
// their last paths.
// Against two kernels per bounce: the large scene's 1024 x 1024 at 8 spp
// 29.6 -> 27.0 ms, the instanced scene's 640 x 360 at 4 spp 7.27 -> 5.96 ms, the
// box room's 256 x 256 at 16 spp 2.08 -> 2.01 ms.  Handing out both kinds from
// one queue, lane by lane, cost a third of the box room's throughput.
//
// Also clears the counters that the next passes fill (their previous users
// have finished, as kernels of one stream run in order): the other path queue,
// the shadow queue of this parity, and the class and fetch counters of the
// other one.  All start at zero (cleared by the wave's generate kernel).
template <int Levels, class Scenes>
__device__ __forceinline__ void trace(const Scenes &scenes, const WfBuffers &b, uint32_t round, uint64_t base,
                                      float4 *radiance) {
    const uint32_t cur = round & 1u;
    if (blockIdx.x == 0 && threadIdx.x < kWfClasses) {
        b.count[kWfClass + (cur ^ 1u) * kWfClasses + threadIdx.x] = 0u;
        if (threadIdx.x < 2) b.count[kWfFetch + 2u * (cur ^ 1u) + threadIdx.x] = 0u;
        if (threadIdx.x == 0) {
            b.count[cur ^ 1u] = 0u;
            b.count[kWfShadow + cur] = 0u;
        }
    }
    uint2 stack[kStackSize];
    {
        const uint32_t n = b.count[cur];
        const uint32_t *q = b.queue[cur];
        bool active = false, drained = n == 0u;
        uint32_t slot = 0;
        const DeviceScene *s = nullptr;
        RayPre r;
        TravState t;
        for (;;) {
            if (!drained) {
                const uint32_t i = refill(b.count + kWfFetch + 2u * cur, n, active, drained);
                if (i < n) {
                    slot = q[i];
                    const float4 o = b.o[slot], d = b.d[slot];
                    s = &scenes(b.st[slot].w);
                    r = precompute_ray(make3(o.x, o.y, o.z), make3(d.x, d.y, d.z), s->bound);
                    trav_init(t, r, 3.402823466e+38f);
                    active = true;
                }
            }
            if (!__any_sync(0xffffffffu, active)) break;
            if (active && closest_step<Levels>(*s, r, t, stack)) {
                const Hit h = trav_hit(*s, t);
                uint32_t cls = 0u;
                if (h.inst_id != kInvalid) {
                    const uint32_t type = s->materials[s->instances[h.inst_id].mat_id].type;
                    if (type != kMatBlackBody) cls = 1u + type;
                }
                b.hit[slot] = h;
                b.tq[static_cast<size_t>(cls) * b.capacity + class_push(b.count + kWfClass + cur * kWfClasses, cls)] =
                    slot;
                active = false;
            }
        }
    }
    {
        const uint32_t n = b.count[kWfShadow + (cur ^ 1u)];
        bool active = false, drained = n == 0u;
        uint32_t i = 0;
        const DeviceScene *s = nullptr;
        RayPre r;
        TravState t;
        for (;;) {
            if (!drained) {
                const uint32_t k = refill(b.count + kWfFetch + 2u * cur + 1u, n, active, drained);
                if (k < n) {
                    i = b.sh_perm ? b.sh_perm[k] : k;
                    const float4 o = b.sh_o[i], d = b.sh_d[i];
                    s = &scenes(__float_as_uint(b.sh_c[i].w));
                    r = precompute_ray(make3(o.x, o.y, o.z), make3(d.x, d.y, d.z), s->bound);
                    trav_init(t, r, o.w);
                    active = true;
                }
            }
            if (!__any_sync(0xffffffffu, active)) break;
            bool occluded = false;
            if (active && any_step<Levels>(*s, r, t, stack, occluded)) {
                const uint32_t tag = __float_as_uint(b.sh_d[i].w);
                const uint32_t slot = tag & 0x7fffffffu;
                float4 L = b.L[slot];
                if (!occluded) {
                    const float4 c = b.sh_c[i];
                    f3 l = make3(L.x, L.y, L.z);
                    l += make3(c.x, c.y, c.z);
                    L = make_float4(l.x, l.y, l.z, L.w);
                    b.L[slot] = L;
                }
                if (tag & 0x80000000u) {
                    const f3 Lw = make3(L.x, L.y, L.z) * L.w;
                    radiance[base + slot] = make_float4(Lw.x, Lw.y, Lw.z, 1.0f);
                }
                active = false;
            }
        }
    }
}

// The shading-class mask of path_shade for class C.
template <uint32_t C>
struct ClassMask {
    static constexpr uint32_t value = C == 0u ? 1u << kMatBlackBody : 1u << (C - 1u);
};

// One bounce (path_shade) of every path of shading class C after its closest
// hit: survivors go to path queue cur ^ 1, next-event estimates to the shadow
// queue; a path that ends without a pending shadow query writes its radiance
// to radiance[base + slot].
template <int N, uint32_t C, class Scenes>
__device__ __forceinline__ void shade(const Scenes &scenes, const WfBuffers &b, uint32_t cur, uint64_t base,
                                      float4 *radiance) {
    const uint32_t n = b.count[kWfClass + cur * kWfClasses + C];
    const uint32_t *q = b.tq + static_cast<size_t>(C) * b.capacity;
    for (uint32_t first = blockIdx.x * blockDim.x; first < n; first += gridDim.x * blockDim.x) {
        if constexpr (C == kWfClassPrincipled) __syncthreads();
        const uint32_t i = first + threadIdx.x;
        if (i >= n) continue;
        const uint32_t slot = q[i];
        PathState<N> ps;
        const uint32_t scene = load<N>(scenes, b, slot, ps);
        const DeviceScene &s = scenes(scene);
        const Hit h = b.hit[slot];
        ShadowQuery sq;
        bool more =
            path_shade<N, false, ClassMask<C>::value>(s, ps, C != 0u || h.inst_id != kInvalid, h, nullptr, sq);
        if (more) more = ++ps.bounce < s.ip.max_depth;
        if (more) {
            store<N>(b, slot, ps, scene);
            b.queue[cur ^ 1u][queue_push(&b.count[cur ^ 1u])] = slot;
        } else {
            b.L[slot] = make_float4(ps.L.x, ps.L.y, ps.L.z, ps.filter_w);
        }
        if (sq.valid) {
            const uint32_t k = queue_push(&b.count[kWfShadow + cur]);
            b.sh_o[k] = make_float4(sq.o.x, sq.o.y, sq.o.z, sq.tmax);
            b.sh_d[k] = make_float4(sq.d.x, sq.d.y, sq.d.z, __uint_as_float(slot | (more ? 0u : 0x80000000u)));
            b.sh_c[k] = make_float4(sq.c.x, sq.c.y, sq.c.z, __uint_as_float(scene));
        } else if (!more) {
            const f3 Lw = ps.L * ps.filter_w;
            radiance[base + slot] = make_float4(Lw.x, Lw.y, Lw.z, 1.0f);
        }
    }
}

}  // namespace wf
}  // namespace vs
