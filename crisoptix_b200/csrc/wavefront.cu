// wavefront.cu -- the path machine of wavefront.cuh run for one pass, in two ways
// that a flow combines (flow_rounds):
//   by rounds: a begin kernel starts every pixel's path and queues its first ray;
//     each round traces the queued rays in one traversal launch and takes the
//     results to the paths' next rays in a shading launch.  Traversal runs at its
//     own register budget (32 warps per SM) over rays in pixel order: the faster
//     way while a round has rays for the whole GPU several times over;
//   on persistent warps: each lane holds one path in registers, traces its ray,
//     steps, and takes another path when it has ended.  20 warps per SM, but no
//     launch waits for its slowest ray: a late round of a 960x540 frame held 5%
//     of the paths and still took 100 us.
// The rounds come first, then the persistent kernel finishes the paths left.
//
// Flows (which records a path writes):
//   prefix: TracePrefix into the canonical prefix record (prefix pass);
//   suffix: TraceSuffix into the canonical suffix record from the pixel's
//           reservoir prefix (suffix temporal pass);
//   gather: TracePrefix, then TraceSuffix when the prefix ends without NEE,
//           into fresh records (final gather, FinalGatherCanon).
#include <algorithm>

#include "queues.cuh"
#include "wavefront.cuh"

namespace crisb {

namespace {

// ---- by rounds -----------------------------------------------------------------------
// queue the ray of pixel i's path for round `round` (two queue pairs, used in turn)
RT_D void push_ray(const Bufs& b, int round, uint32_t phase, uint32_t i) {
    const int q = 2 * (round & 1);
    q_append(b.path_queue[q], &b.path_counts[2 * round], phase == kPhHit || phase == kPhRecon, i);
    q_append(b.path_queue[q + 1], &b.path_counts[2 * round + 1], phase == kPhShadow, i);
}

// starts every pixel's path and queues its first ray
template <int kFlow, bool kTex>
__global__ void __launch_bounds__(kPassBlock, 6) k_flow_begin(SceneView s, FrameParams fp, Bufs b) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    FlowPath<kFlow, kTex> path;
    path.phase = kPhDone;
    if (i < pixel_count(fp)) {
        path.begin(s, fp, b, i);
        if (kFlow == 1 && path.phase == kPhStart) path.vertex(s, fp, b, i, TraceResult{CRISB_INVALID_PRIM, 0.0f, 0.0f, 0.0f});
        if (path.phase != kPhDone) path.save(b.paths + i);
    }
    push_ray(b, 0, path.phase, i);
}

// takes the result of every ray of round `round` to its path's next ray, queued
// for the next round, or its end (5 resident blocks per SM; 6 / 7 / 8: 0.1-0.2 ms
// more per 1080p frame)
template <int kFlow, bool kTex>
__global__ void __launch_bounds__(kPassBlock, 5) k_flow_shade(SceneView s, FrameParams fp, Bufs b, int round) {
    const uint32_t nc = b.path_counts[2 * round], total = nc + b.path_counts[2 * round + 1];
    const uint32_t* qc = b.path_queue[2 * (round & 1)];
    const uint32_t* qs = b.path_queue[2 * (round & 1) + 1];
    for (uint32_t base = blockIdx.x * blockDim.x; base < total; base += gridDim.x * blockDim.x) {
        const uint32_t t = base + threadIdx.x;
        FlowPath<kFlow, kTex> path;
        path.phase = kPhDone;
        uint32_t i = 0;
        if (t < total) {
            i = t < nc ? qc[t] : qs[t - nc];
            PathState* st = b.paths + i;
            path.load(st);
            path.step(s, fp, b, i, FlowPath<kFlow, kTex>::result(st));
            if (path.phase != kPhDone) path.save(st);
        }
        push_ray(b, round + 1, path.phase, i);
    }
}

// ---- on persistent warps -------------------------------------------------------------
// Each lane holds a path, traces the ray it waits for (rays of every kind side by
// side in one traversal), steps, and takes another path when it has ended:
// every pixel's path from its start (round < 0), or the paths whose rays are
// queued for round `round`.
template <int kFlow, bool kTex, int kFmt>
__global__ void __launch_bounds__(kPassBlock, 5) k_flow(SceneView s, FrameParams fp, Bufs b, int round) {
    constexpr unsigned kFull = 0xffffffffu;
    const bool fresh = round < 0;
    const uint32_t nc = fresh ? pixel_count(fp) : b.path_counts[2 * round];
    const uint32_t* qc = b.path_queue[2 * (round & 1)];
    const uint32_t* qs = b.path_queue[2 * (round & 1) + 1];
    WorkPool pool(fresh ? nc : nc + b.path_counts[2 * round + 1], b.path_next);
    FlowPath<kFlow, kTex> path;
    path.phase = kPhDone;
    uint32_t pixel = 0;
    bool traced = false;  // the lane's ray has its result in h
    TraceResult h{CRISB_INVALID_PRIM, 0.0f, 0.0f, 0.0f};
    while (true) {
        // lanes with a result or at a suffix's first vertex step; lanes whose path
        // has ended take another, until all but a few have a ray or none is left
        while (true) {
            if (traced || (kFlow == 1 && path.phase == kPhStart)) {
                path.step(s, fp, b, pixel, h);
                traced = false;
            }
            if (pool.more()) {
                const bool want = path.phase == kPhDone;
                if (__any_sync(kFull, want)) {
                    const uint32_t i = pool.take(want);
                    if (i != 0xffffffffu) {
                        if (fresh) {
                            pixel = i;
                            path.begin(s, fp, b, i);
                        } else {
                            pixel = i < nc ? qc[i] : qs[i - nc];
                            path.load(b.paths + pixel);
                        }
                    }
                }
            }
            const unsigned lacking =
                __ballot_sync(kFull, path.phase == kPhStart || (path.phase == kPhDone && pool.more()));
            if (!lacking) break;
            if (__popc(lacking) <= kMostIdle && __any_sync(kFull, path.phase > kPhStart)) break;
        }
        if (!__any_sync(kFull, path.phase != kPhDone)) break;
        if (path.phase > kPhStart) {
            const bool shadow = path.phase == kPhShadow;
            count_ray_kind(s, shadow);
            h = traverse_ray<kFmt>(s, path.o, path.d, 1e-3f, shadow ? path.tmax : 1e16f, shadow);
            traced = true;
        }
    }
}

// the most rays a path of the flow traces
int most_rays(const crisb_params& p, int flow) {
    if (p.renderer_type == CRISB_RENDERER_RESTIR_PT) return p.max_path_len + 1;  // every vertex and a light
    // n vertices of the suffix, the first of them known: rays to the others, to the
    // light and to its reconnection vertex
    const int n = std::max(p.max_path_len - p.prefix_len, 0);
    return (flow != 1 ? p.prefix_len : 0) + (flow != 0 && n > 0 ? n + 1 : 0);
}
// whether paths may be left after `rounds` rounds (a suffix may be longer than
// the parameters say: temporal reuse keeps prefixes of other lengths)
bool needs_tail(const crisb_params& p, int flow, int rounds) { return flow == 1 || rounds < most_rays(p, flow); }

template <int kFlow, bool kTex, int kFmt>
void launch_flow_as(const SceneView& s, const FrameParams& fp, const Bufs& b, cudaStream_t st, Marker* m) {
    static const unsigned g_flow = persistent_grid(reinterpret_cast<const void*>(k_flow<kFlow, kTex, kFmt>));
    static const unsigned g_shade = persistent_grid(reinterpret_cast<const void*>(k_flow_shade<kFlow, kTex>));
    const unsigned most = grid_for(fp.width * fp.height);  // a path a pixel
    const int rounds = flow_rounds(fp, kFlow, kTex);
    if (rounds > 0) {
        k_flow_begin<kFlow, kTex><<<most, kPassBlock, 0, st>>>(s, fp, b);
        if (m) m->mark(kClsShade, st);
    }
    for (int r = 0; r < rounds; ++r) {
        const int q = 2 * (r & 1);
        launch_trace<PathState>(fp.trace_block, fp.trace_grid, fp.width * fp.height, st, s, b.path_queue[q],
                                b.path_counts + 2 * r, b.path_queue[q + 1], b.path_counts + 2 * r + 1, b.paths);
        if (m) m->mark(kClsTrace, st);
        k_flow_shade<kFlow, kTex><<<std::min(g_shade, most), kPassBlock, 0, st>>>(s, fp, b, r);
        if (m) m->mark(kClsShade, st);
    }
    if (rounds > 0 && !needs_tail(fp.p, kFlow, rounds)) return;
    k_flow<kFlow, kTex, kFmt><<<std::min(g_flow, most), kPassBlock, 0, st>>>(s, fp, b, rounds > 0 ? rounds : -1);
    if (m) m->mark(kClsTrace, st);
}

template <int kFlow>
void launch_flow(const SceneView& s, const FrameParams& fp, const Bufs& b, cudaStream_t st, Marker* m) {
    const auto launch = s.qnodes ? (s.mat_tex ? launch_flow_as<kFlow, true, kFmtAny>
                                              : launch_flow_as<kFlow, false, kFmtAny>)
                                 : (s.mat_tex ? launch_flow_as<kFlow, true, kFmtWide4>
                                              : launch_flow_as<kFlow, false, kFmtWide4>);
    launch(s, fp, b, st, m);
}

}  // namespace

// Rounds before the persistent kernel.  Frames whose pixels fit the resident lanes
// (94,720) once or a little more run on persistent warps alone: 256x192 conditional
// frames of the Cornell box 505 us against 542-581 with 1-4 rounds, 512x384 ones
// already 859 against 827.  Textured shading diverges more, so its paths stay in
// rounds sooner (400x300: 989 against 816 us).  RestirPt's one flow, whose late
// vertices are few, runs best persistent at every size measured to 1080p
// untextured (room 6.23 against 6.41 ms in rounds alone), and in five rounds
// textured (641x479: 765 us, 826 with one).  Above those sizes one round (two for
// the gather, whose prefix takes the first) was fastest to 800x600 and 960x540
// (4.95 ms, 5.03 with one more each), two and three at 1080p (14.31 ms, 14.47 and
// 14.55 with one fewer and one more); views that render beside one another fill
// each other's late rounds, so theirs go on longest (16 views 75.9 ms, 78.7 with
// the single view's rounds).  That line is drawn for batches that fill the GPU (8 views
// of 512x512 12.5 ms, 13.3 with 2 / 2 / 3 rounds and one of shifts, 14.0 with 1 / 1 / 2,
// 17.0 with none; two of 1080p 24.5, 25.0, 25.4, 31.5).  Around a million pixels it makes
// no difference (4 of 512x512 7.05, 7.05, 7.45, 8.89), and smaller batches would run
// faster with fewer: 2 of 256x256 2.82, 2.47, 2.40, 2.24, 16 of 64x64 2.24, 1.98, 1.89,
// 1.53.  (With rounds to the last ray these four took 15.4, 8.92, 3.80 and 5.74, the
// 1080p pair 29.8.)  By rounds to the last ray, the three flows of a
// 1080p frame took 0.5 ms more, those of a 960x540 frame 0.4.
int flow_rounds(const FrameParams& fp, int flow, bool textured) {
    const uint32_t pixels = fp.width * fp.height;
    const bool restir_pt = fp.p.renderer_type == CRISB_RENDERER_RESTIR_PT;
    int r;
    if (fp.concurrent) r = flow == 0 ? 2 : flow == 1 ? 4 : 5;
    else if (pixels <= (textured ? 49152u : 131072u)) r = 0;
    else if (restir_pt) r = textured ? 5 : 0;
    else if (pixels < (1u << 20)) r = flow == 2 ? 2 : 1;
    else r = flow == 2 ? 3 : 2;
    return std::min(r, most_rays(fp.p, flow));
}
uint32_t flow_launches(const FrameParams& fp, int flow, bool textured) {
    const int r = flow_rounds(fp, flow, textured);
    return r > 0 ? 1 + 2 * static_cast<uint32_t>(r) + (needs_tail(fp.p, flow, r) ? 1u : 0u) : 1;
}

void launch_wf_prefix(const SceneView& s, const FrameParams& fp, const Bufs& b, cudaStream_t st, Marker* m) {
    launch_flow<0>(s, fp, b, st, m);
}
void launch_wf_suffix(const SceneView& s, const FrameParams& fp, const Bufs& b, cudaStream_t st, Marker* m) {
    launch_flow<1>(s, fp, b, st, m);
}
void launch_wf_gather(const SceneView& s, const FrameParams& fp, const Bufs& b, cudaStream_t st, Marker* m) {
    launch_flow<2>(s, fp, b, st, m);
}

}  // namespace crisb
