// queues.cuh -- ray queues shared by the path machines (wavefront.cu) and the
// shift machines (reuse_passes.cu): warp-aggregated append, and the closest /
// shadow traversal kernels over a queue of record indices.
//
// A record type R provides closest_ray / set_hit for closest-hit rays and
// shadow_ray / set_occluded for visibility rays; the kernels only move rays
// and results, so one traversal kernel serves every kind of machine.
#pragma once

#include <algorithm>

#include "passes.cuh"

namespace crisb {
namespace {

// lanes that may go without a ray into a traversal of a persistent kernel rather
// than have the others wait for one more step (0 / 4 / 8 / 16 / 24: 14.79, 14.64,
// 14.57, 14.70, 14.86 ms per 1080p frame with two to three rounds a flow)
constexpr int kMostIdle = 8;

// Warp-aggregated append of `val` to queue q (count cnt) for the lanes with
// `take` set.  Every lane of the warp must call this.
RT_D void q_append(uint32_t* q, uint32_t* cnt, bool take, uint32_t val) {
    const unsigned mask = __ballot_sync(0xffffffffu, take);
    if (!mask) return;
    const int lane = threadIdx.x & 31;
    const int leader = __ffs(mask) - 1;
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(cnt, static_cast<uint32_t>(__popc(mask)));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (take) q[base + __popc(mask & ((1u << lane) - 1u))] = val;
}

// path states (FlowPath::save): a shadow ray's result is a triangle if occluded
RT_D void closest_ray(const PathState& p, V3& o, V3& d) {
    const uint4 a = p.w[1], b = p.w[2];
    o = V3{__uint_as_float(a.x), __uint_as_float(a.y), __uint_as_float(a.z)};
    d = V3{__uint_as_float(b.x), __uint_as_float(b.y), __uint_as_float(b.z)};
}
RT_D void set_hit(PathState& p, float4 h) {
    p.hit = make_uint4(__float_as_uint(h.x), __float_as_uint(h.y), __float_as_uint(h.z), __float_as_uint(h.w));
}
RT_D void shadow_ray(const PathState& p, V3& o, V3& d, float& tmax) {
    closest_ray(p, o, d);
    tmax = __uint_as_float(p.w[5].x);
}
RT_D void set_occluded(PathState& p, uint32_t v) { p.hit.x = v ? 0u : CRISB_INVALID_PRIM; }

// shift machine records: one ray in flight in o / d
RT_D void closest_ray(const ShiftJob& j, V3& o, V3& d) {
    const float4 a = j.o, b = j.d;
    o = V3{a.x, a.y, a.z};
    d = V3{b.x, b.y, b.z};
}
RT_D void set_hit(ShiftJob& j, float4 h) { j.hit = h; }
RT_D void shadow_ray(const ShiftJob& j, V3& o, V3& d, float& tmax) {
    const float4 a = j.o, b = j.d;
    o = V3{a.x, a.y, a.z};
    d = V3{b.x, b.y, b.z};
    tmax = a.w;
}
RT_D void set_occluded(ShiftJob& j, uint32_t v) { j.hit.x = __uint_as_float(v); }

// Grid-stride loops over the queue, each lane walking its ray to the end.
// Warps lose most of their lanes to that (a warp runs 2.4x the node visits
// its rays need on the 1080p workload), but refilling finished lanes measured
// slower every time: with 4-wide nodes (per-warp batches, 31 ms against 20 ms
// of trace per frame: the per-step convergence removes the latency hiding
// between diverged inner-node and leaf lanes) and with compressed nodes
// (per-warp chunks of the queue, every idle lane refilled at once when at most
// 8-31 lanes are busy: 19.1-19.8 against 12.1 ms: lanes on different rays and
// depths no longer load the same nodes in the same instruction).
// One launch per round over both queues: entries [0, nc) of the closest-hit
// queue, then [nc, nc + ns) of the shadow queue, so the two queues' tails
// (the last, slowest rays) overlap instead of running back to back.
// Block sizes of the traversal kernel (crisb_set_trace_block, tuned by
// crisb_autotune): resident blocks per SM chosen so every size has the
// register budget of 8 x 128 threads (64 registers).  On the 1080p workload
// 7 / 8 / 9 / 10 blocks of 128 threads render a frame in 15.47 / 15.09 / 15.09 /
// 15.29 ms, the 256 x 256 Cornell box in 677 / 683 / 702 / 707 us.
template <int kB>
struct TraceShape {
    static constexpr int kMinBlocks = 8 * 128 / kB;
};

template <class R, int kB, int kFmt>
__global__ void __launch_bounds__(kB, TraceShape<kB>::kMinBlocks) k_q_trace(SceneView s, const uint32_t* qc,
                                                                          const uint32_t* ccnt, const uint32_t* qs,
                                                                          const uint32_t* scnt, R* rec) {
    const uint32_t nc = *ccnt, ns = *scnt;
    const uint32_t n = nc + ns;
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        V3 o, d;
        if (t < nc) {
            const uint32_t i = qc[t];
            closest_ray(rec[i], o, d);
            count_ray(s, 0);
            const TraceResult h = traverse_fmt<kFmt, false>(s, make_ray(o, d), 1e-3f, 1e16f);
            set_hit(rec[i], make_float4(__uint_as_float(h.prim), h.t, h.u, h.v));
        } else {
            const uint32_t i = qs[t - nc];
            float tmax;
            shadow_ray(rec[i], o, d, tmax);
            count_ray(s, 1);
            const bool occ = traverse_fmt<kFmt, true>(s, make_ray(o, d), 1e-3f, tmax).prim != CRISB_INVALID_PRIM;
            set_occluded(rec[i], occ ? 1u : 0u);
        }
    }
}

inline unsigned grid_for(uint32_t n) { return (n + kPassBlock - 1) / kPassBlock; }

// all blocks of `kernel` at `block` threads that are resident on the device at once
inline unsigned persistent_grid(const void* kernel, int block = kPassBlock) {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) == cudaSuccess &&
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, block, 0) == cudaSuccess && sms > 0 &&
        per_sm > 0)
        return static_cast<unsigned>(sms * per_sm);
    return 148u * 4u;
}

template <class R, int kB, int kFmt>
unsigned trace_grid_of() {
    static const unsigned g = persistent_grid(reinterpret_cast<const void*>(k_q_trace<R, kB, kFmt>), kB);
    return g;
}

template <class R, int kB, int kFmt>
void launch_trace_as(uint32_t m, uint32_t most, cudaStream_t st, const SceneView& s, const uint32_t* qc,
                     const uint32_t* ccnt, const uint32_t* qs, const uint32_t* scnt, R* rec) {
    const unsigned g = std::min(trace_grid_of<R, kB, kFmt>() * m, std::max(most, 1u) / kB + 1);
    k_q_trace<R, kB, kFmt><<<g, kB, 0, st>>>(s, qc, ccnt, qs, scnt, rec);
}

template <class R, int kFmt>
void launch_trace_fmt(uint32_t block, uint32_t m, uint32_t most, cudaStream_t st, const SceneView& s,
                      const uint32_t* qc, const uint32_t* ccnt, const uint32_t* qs, const uint32_t* scnt, R* rec) {
    if (block == 64) launch_trace_as<R, 64, kFmt>(m, most, st, s, qc, ccnt, qs, scnt, rec);
    else if (block == 256) launch_trace_as<R, 256, kFmt>(m, most, st, s, qc, ccnt, qs, scnt, rec);
    else launch_trace_as<R, 128, kFmt>(m, most, st, s, qc, ccnt, qs, scnt, rec);
}

// one traversal launch over a closest-hit and a shadow queue that hold at most
// `most` rays together: `block` threads (64, 128 or 256) and `mult` x the blocks
// resident at once, but no more than the rays fill (a 256 x 256 frame: 513
// instead of 9,472 blocks a launch, 343 -> 341 us); the kernel instance of the
// scene tree's node format
template <class R>
void launch_trace(uint32_t block, uint32_t mult, uint32_t most, cudaStream_t st, const SceneView& s,
                  const uint32_t* qc, const uint32_t* ccnt, const uint32_t* qs, const uint32_t* scnt, R* rec) {
    const uint32_t m = std::max(mult, 1u);
    if (s.qnodes) launch_trace_fmt<R, kFmtCompressed8>(block, m, most, st, s, qc, ccnt, qs, scnt, rec);
    else launch_trace_fmt<R, kFmtWide4>(block, m, most, st, s, qc, ccnt, qs, scnt, rec);
}

}  // namespace
}  // namespace crisb
