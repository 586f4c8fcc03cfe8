// adjoint.cu -- path-replay adjoint of the unidirectional path tracer.
//
// The estimator differentiated is TraceCompletePath
// (include/graph/restir/path_gen.h:389-472; CompletePath here) with its
// sampling frozen: every random decision, BRDF-sampled direction and sampling
// pdf comes from a fixed copy of the materials (theta0, taken when the adjoint
// context is made), while the BRDF values, emissions and emitter colours come
// from the scene's current tables (theta).  At theta = theta0 it is the path
// tracer sample for sample; for any theta it is an unbiased estimator of the
// rendering integral at theta (importance sampling with a fixed proposal), and
// it is a smooth function of theta, so its gradient is what central
// differences of the same estimator measure.
//
// The estimator has one term per path: at the vertex j where NEE is chosen,
//   L = T_j * brdf_j(light) * Le / d^2 (+ emission_j when j is the first hit),
//   T_j = prod_{i<j} brdf_i(dir_i) / (pdf0_i (1 - neeProb)) / neeProb.
// The backward kernel replays each pixel's path from its seed (no tape) and
// carries d T / d(diffuse rgb, roughness) for every material met so far
// (forward mode), then turns dLoss/dL into gradients of the diffuse albedo,
// roughness and emission of each material and the colour of each emitter.
// Gradients gather in shared memory per block and reach global memory with one
// atomic per touched parameter per block.
#include <algorithm>
#include <stdexcept>
#include <string>
#include <vector>

#include "adjoint_common.cuh"
#include "queues.cuh"

namespace crisb {
namespace {

struct AdjView {
    SceneView eval;           // current materials / emitters (theta)
    const crisb_material* sample_mats;  // theta0
    uint32_t num_mats, num_emitters;
};

// One path of the frozen-sampling estimator cut at its rays (as CompletePath):
// a lane holds the ray in flight, step() takes its result to the next ray or the
// end.  With kGrad the path also adds its gradient for the pixel adjoint `dl`
// to the sink when it ends in a visible light.
template <bool kGrad>
struct FrozenPath {
    V3 o, d;      // the ray in flight
    float tmax;   // 1e16 for an extension ray, the light distance for a shadow ray
    bool shadow;
    V3 tp, radiance;
    uint32_t depth;
    Rng rng;
    Isect it;     // kGrad: the vertex the shadow ray starts from ...
    V3 color;     // ... and the light's colour and emitter
    uint32_t em;
    int nt;

    RT_D void begin(V3 origin, V3 dir, const Rng& r) {
        o = origin;
        d = dir;
        tmax = 1e16f;
        shadow = false;
        tp = splat(1.0f);
        radiance = splat(0.0f);
        depth = 0;
        rng = r;
        nt = 0;
    }

    // the light connection's value and, with a sink, its gradient
    RT_D V3 connect(const AdjView& a, const Isect& v, V3 light_dir, float dist, V3 col, uint32_t ei, V3 dl,
                    const Touched* tl, GradSink* sink) const {
        const uint32_t mi = material_of(a.eval, v.prim);
        const crisb_material mat = a.eval.mats[mi];
        const BrdfGrad bg = brdf_grad(mat, v.nrm, -v.dir, light_dir);
        const float dist_factor = 1.0f / (dist * dist);
        V3 r = tp * bg.brdf * col * dist_factor;
        // brdf_eval reports the emission only past its facing checks
        const bool emit = depth == 1 && dot(v.nrm, -v.dir) > 0.0f && dot(v.nrm, light_dir) >= 0.0f;
        if (emit) r = r + mat_vals(mat).emission;
        if (!kGrad || !sink) return r;
        const V3 lw = col * dist_factor;  // light weight
        for (int t = 0; t < nt; ++t) {
            const V3 c_diff = dl * tl[t].d_diff * bg.brdf * lw;
            sink->add_mat(tl[t].mat, 0, c_diff.x);
            sink->add_mat(tl[t].mat, 1, c_diff.y);
            sink->add_mat(tl[t].mat, 2, c_diff.z);
            const V3 c_r = dl * tl[t].d_rough * bg.brdf * lw;
            sink->add_mat(tl[t].mat, 3, (c_r.x + c_r.y) + c_r.z);
        }
        const V3 c_diff = dl * tp * bg.d_diff * lw;
        sink->add_mat(mi, 0, c_diff.x);
        sink->add_mat(mi, 1, c_diff.y);
        sink->add_mat(mi, 2, c_diff.z);
        const V3 c_r = dl * tp * bg.d_rough * lw;
        sink->add_mat(mi, 3, (c_r.x + c_r.y) + c_r.z);
        const V3 c_e = dl * tp * bg.brdf * dist_factor;
        sink->add_em(ei, 0, c_e.x);
        sink->add_em(ei, 1, c_e.y);
        sink->add_em(ei, 2, c_e.z);
        if (emit) {
            sink->add_mat(mi, 4, dl.x);
            sink->add_mat(mi, 5, dl.y);
            sink->add_mat(mi, 6, dl.z);
        }
        return r;
    }

    // the path's next ray is in o, d, tmax, shadow; false: ended with `radiance`
    RT_D bool step(const AdjView& a, const FrameParams& fp, const TraceResult& h, V3 dl, Touched* tl, GradSink* sink) {
        if (shadow) {
            if (h.prim != CRISB_INVALID_PRIM) radiance = splat(0.0f);
            else if (kGrad) connect(a, it, d, tmax, color, em, dl, tl, sink);
            return false;
        }
        Isect v;
        hit_isect(a.eval, h, d, v);
        if (!v.valid) return false;
        ++depth;
        const float nee = fp.p.nee_prob;
        if (rng.next_float() < nee) {
            tp = tp / nee;
            if (kGrad)
                for (int t = 0; t < nt; ++t) {
                    tl[t].d_diff = tl[t].d_diff / nee;
                    tl[t].d_rough = tl[t].d_rough / nee;
                }
            const EmitterSample es = sample_emitter(a.eval, rng);
            const V3 light_dir = normalize(es.pos - v.pos);
            const float dist = length(es.pos - v.pos);
            if (kGrad) {
                it = v;
                color = es.color;
                em = es.index;
            } else {
                // the value does not depend on the shadow ray: evaluated before it
                radiance = connect(a, v, light_dir, dist, es.color, es.index, dl, nullptr, nullptr);
                if ((__float_as_uint(radiance.x) | __float_as_uint(radiance.y) | __float_as_uint(radiance.z)) == 0u)
                    return false;  // +0 whether or not the light is visible
            }
            o = v.pos;
            d = light_dir;
            tmax = dist;
            shadow = true;
            return true;
        }
        SceneView ss = a.eval;  // sampling view: theta0 materials
        ss.mats = a.sample_mats;
        const uint32_t mi = material_of(a.eval, v.prim);
        const BrdfSample bs = brdf_sample<false>(ss, v, rng);  // direction and pdf at theta0
        if (bs.pdf <= 0.0f) return false;
        const BrdfGrad bg = brdf_grad(a.eval.mats[mi], v.nrm, -v.dir, bs.dir);
        const float inv = 1.0f / (bs.pdf * (1.0f - nee));
        const V3 w = bg.brdf * inv;
        if (kGrad) {
            for (int t = 0; t < nt; ++t) {
                tl[t].d_diff = tl[t].d_diff * w;
                tl[t].d_rough = tl[t].d_rough * w;
            }
            int slot = -1;
            for (int t = 0; t < nt; ++t)
                if (tl[t].mat == mi) slot = t;
            if (slot < 0 && nt < kMaxTouched) {
                slot = nt++;
                tl[slot].mat = mi;
                tl[slot].d_diff = tl[slot].d_rough = splat(0.0f);
            }
            if (slot >= 0) {
                tl[slot].d_diff = tl[slot].d_diff + tp * bg.d_diff * inv;
                tl[slot].d_rough = tl[slot].d_rough + tp * bg.d_rough * inv;
            }
        }
        o = v.pos;
        d = bs.dir;
        tp = tp * w;
        return depth < static_cast<uint32_t>(fp.p.max_path_len);
    }
};

// The pixels' paths of a pool: a lane takes the next pixel when its path ends and
// traces one ray of either kind a turn.  kGrad: `d_img` is the image's adjoint,
// whose zero and non-finite pixels trace nothing; else `out` is the image.
template <bool kGrad, int kFmt, class Pool>
RT_D void frozen_pixels(const AdjView& a, const FrameParams& fp, Pool pool, const float* d_img, float* out,
                        GradSink* sink) {
    FrozenPath<kGrad> path;
    Touched tl[kGrad ? kMaxTouched : 1];
    V3 dl = splat(0.0f);
    uint32_t pixel = 0xffffffffu;
    while (true) {
        const unsigned idle = __ballot_sync(0xffffffffu, pixel == 0xffffffffu);
        if (idle) {
            const bool more = pool.more();
            if (idle == 0xffffffffu && !more) break;
            if (more) {
                const uint32_t i = pool.take(pixel == 0xffffffffu);
                bool start = i != 0xffffffffu;
                if (kGrad && start) {
                    dl = V3{d_img[3 * i], d_img[3 * i + 1], d_img[3 * i + 2]};
                    start = !nonfinite(dl) && (dl.x != 0.0f || dl.y != 0.0f || dl.z != 0.0f);
                }
                if (start) {
                    pixel = i;
                    Rng rng = rng_seeded(tea64(i, fp.random));
                    const V3 dir = camera_dir(fp, i % fp.width, i / fp.width, rng);
                    path.begin(ld3(fp.cam.pos), dir, rng);
                }
            }
        }
        if (pixel != 0xffffffffu) {
            const TraceResult h = traverse_ray<kFmt>(a.eval, path.o, path.d, 1e-3f, path.tmax, path.shadow);
            if (!path.step(a, fp, h, dl, tl, sink)) {
                if (!kGrad) {
                    V3 L = path.radiance;
                    if (nonfinite(L)) L = splat(0.0f);
                    out[3 * pixel] = L.x;
                    out[3 * pixel + 1] = L.y;
                    out[3 * pixel + 2] = L.z;
                }
                pixel = 0xffffffffu;
            }
        }
    }
}

// 6 resident blocks per SM (80 registers; 4 and 5 blocks: 2-4% slower)
template <int kFmt>
__global__ void __launch_bounds__(kPassBlock, 6) k_frozen_forward(AdjView a, FrameParams fp, float* out) {
    frozen_pixels<false, kFmt>(a, fp, PixelPool(fp.width * fp.height), nullptr, out, nullptr);
}

// Backward: a block per group of 128 pixels, whose lanes take the group's pixels in
// turn and whose gradients gather in one shared-memory block of all parameters (12 KB
// for the large scene) that reaches global memory once.  The group, not the block,
// sets how the gradients' float sums are split: larger ones, as persistent warps
// would have, change them by 2e-5 through what a global sum of 1e9 takes from each
// addition.  Forward and backward of 8 views of 512 x 512: 11.3 ms with 64 threads a
// group (10 blocks per SM, 96 registers), 12.3 with 128, 11.9 with 96, 11.7 with 32;
// 15.9 with a thread a pixel, each warp running until its longest path ended.
// Images whose groups are all resident at once with a thread a pixel take that
// instead: two pixels a lane then only make the chain longer (one view, backward,
// 64 x 64 283 against 431 us, 256 x 256 413 / 509, 320 x 320, just above the line,
// 586 / 604, 384 x 384 779 / 719).
constexpr uint32_t kGroup = 128;
constexpr int kGroupThreads = 64;

template <int kFmt>
__global__ void __launch_bounds__(kGroup, 5) k_frozen_backward(AdjView a, FrameParams fp, const float* d_img,
                                                               float* g_mat, float* g_em, int use_shared) {
    extern __shared__ float sh[];
    __shared__ uint32_t taken;
    const uint32_t n_sh = a.num_mats * kMatGrad + a.num_emitters * kEmGrad;
    if (threadIdx.x == 0) taken = 0;
    if (use_shared)
        for (uint32_t k = threadIdx.x; k < n_sh; k += blockDim.x) sh[k] = 0.0f;
    __syncthreads();
    GradSink sink{use_shared ? sh : nullptr, g_mat, g_em, a.num_mats};
    const uint32_t first = blockIdx.x * kGroup;
    frozen_pixels<true, kFmt>(a, fp, GroupPool{first, min(kGroup, fp.width * fp.height - first), &taken}, d_img, nullptr, &sink);
    if (use_shared) {
        __syncthreads();
        for (uint32_t k = threadIdx.x; k < n_sh; k += blockDim.x) {
            const float v = sh[k];
            if (v == 0.0f) continue;
            if (k < a.num_mats * kMatGrad) atomicAdd(&g_mat[k], v);
            else atomicAdd(&g_em[k - a.num_mats * kMatGrad], v);
        }
    }
}

template <int kFmt>
void forward(const SceneView& eval, const crisb_material* sample_mats, uint32_t num_mats, const FrameParams& fp,
             float* out, cudaStream_t st) {
    const AdjView a{eval, sample_mats, num_mats, eval.num_emitters};
    const uint32_t P = fp.width * fp.height;
    static const unsigned resident = persistent_grid(reinterpret_cast<const void*>(k_frozen_forward<kFmt>));
    k_frozen_forward<kFmt><<<std::min((P + kPassBlock - 1) / kPassBlock, resident), kPassBlock, 0, st>>>(a, fp, out);
}

template <int kFmt>
void backward(const SceneView& eval, const crisb_material* sample_mats, uint32_t num_mats, const FrameParams& fp,
              const float* d_img, float* g_mat, float* g_em, cudaStream_t st) {
    const AdjView a{eval, sample_mats, num_mats, eval.num_emitters};
    const uint32_t P = fp.width * fp.height;
    const size_t sh_bytes = (static_cast<size_t>(num_mats) * kMatGrad + eval.num_emitters * kEmGrad) * sizeof(float);
    const int use_shared = sh_bytes <= kSharedGradBytes ? 1 : 0;
    const size_t shb = use_shared ? sh_bytes : 0;
    allow_shared_grads(reinterpret_cast<const void*>(k_frozen_backward<kFmt>), shb);
    static const unsigned resident = persistent_grid(reinterpret_cast<const void*>(k_frozen_backward<kFmt>));
    const unsigned groups = (P + kGroup - 1) / kGroup;
    const unsigned threads = groups <= resident ? kGroup : kGroupThreads;
    k_frozen_backward<kFmt><<<groups, threads, shb, st>>>(a, fp, d_img, g_mat, g_em, use_shared);
}

}  // namespace

// host side, called from api.cu
void adjoint_forward(const SceneView& eval, const crisb_material* sample_mats, uint32_t num_mats,
                     const FrameParams& fp, float* out, cudaStream_t st) {
    const auto run = eval.qnodes ? forward<kFmtAny> : forward<kFmtWide4>;
    run(eval, sample_mats, num_mats, fp, out, st);
}

void adjoint_backward(const SceneView& eval, const crisb_material* sample_mats, uint32_t num_mats,
                      const FrameParams& fp, const float* d_img, float* g_mat, float* g_em, cudaStream_t st) {
    const auto run = eval.qnodes ? backward<kFmtAny> : backward<kFmtWide4>;
    run(eval, sample_mats, num_mats, fp, d_img, g_mat, g_em, st);
}

}  // namespace crisb
