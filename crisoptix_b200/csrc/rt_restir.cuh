// rt_restir.cuh -- path generation, hybrid shift mappings, pairwise MIS and
// reservoir streaming of Conditional ReSTIR PT.
//
// Device restatement of include/graph/restir/path_gen.h, prefix_reuse.h,
// suffix_reuse.h and Reservoir.h.  Records are modified in place with the
// reference's field-by-field semantics (fields a function does not write keep
// their previous value).
#pragma once

#include "rt_scene.cuh"

namespace crisb {

// Frame-constant parameters (LaunchParams + RestirParams knobs)
struct FrameParams {
    crisb_params p;
    crisb_camera_data cam;
    uint32_t width, height;
    uint32_t random;
    uint32_t frame_idx;  // for the accumulation blend factor
    int front, back;     // 0/1 buffer selection
    uint32_t k;          // gatherM - 1
    uint32_t trace_grid; // traversal launches: blocks per resident block (host side only)
    uint32_t trace_block; // traversal launches: threads per block, 64 / 128 / 256 (host side only)
    uint32_t concurrent = 0;  // other views' frames run beside this one (host side only)
    const float2* motion = nullptr;  // CRISB_MOTION_VECTORS: per-pixel motion vectors
    crisb_camera_data prev_cam{};    // CRISB_MOTION_REPROJECT: the previous frame's camera
    uint32_t has_prev_cam = 0;
};

// ---- temporal reprojection (prevPixelCoord) ---------------------------------------
// G-buffer prev_xy: x | y << 16, or kPrevNone when the pixel has no previous
// pixel (IsPixelValid false); resolutions stay below 65535 so no valid pixel
// packs to it.
constexpr uint32_t kPrevNone = 0xffffffffu;

RT_HD uint32_t pack_prev(uint32_t px, uint32_t py, uint32_t w, uint32_t h) {
    return (px < w && py < h) ? (px | (py << 16)) : kPrevNone;
}

// glm::uvec2(vec2) as it compiles on the GPU (cvt.rzi.u32.f32): truncation
// toward zero, saturating at 0 and 2^32 - 1, NaN to 0
RT_HD uint32_t f2u_sat(float v) {
    if (!(v > 0.0f)) return 0u;
    if (v >= 4294967296.0f) return 0xffffffffu;
    return static_cast<uint32_t>(v);
}

// prevPixelCoord = uvec2(vec2(pixelCoord) + vec2(0.5) + motionVector)
// (prefix_gen_temp_reuse.cu:136, the commented-out form)
RT_HD uint32_t prev_from_motion(uint32_t x, uint32_t y, float mx, float my, uint32_t w, uint32_t h) {
    const float fx = (static_cast<float>(x) + 0.5f) + mx;
    const float fy = (static_cast<float>(y) + 0.5f) + my;
    return pack_prev(f2u_sat(fx), f2u_sat(fy), w, h);
}

// The pixel of camera `c` whose footprint holds world point p: the inverse of
// camera_dir (d = U ux + V uy + W with U, V, W orthogonal), ux = 2 x / width -
// 1 over the pixel's footprint [x, x + 1).  None behind the camera or off
// screen.
RT_HD uint32_t reproject(const crisb_camera_data& c, V3 p, uint32_t w, uint32_t h) {
    const V3 U = ld3(c.u), V = ld3(c.v), W = ld3(c.w);
    const V3 d = p - ld3(c.pos);
    const float t = dot(d, W) / dot(W, W);
    if (!(t > 0.0f)) return kPrevNone;
    const float ux = dot(d, U) / (t * dot(U, U));
    const float uy = dot(d, V) / (t * dot(V, V));
    const float xc = (ux + 1.0f) * 0.5f * static_cast<float>(w);
    const float yc = (uy + 1.0f) * 0.5f * static_cast<float>(h);
    if (!(xc >= 0.0f && xc < static_cast<float>(w) && yc >= 0.0f && yc < static_cast<float>(h))) return kPrevNone;
    return pack_prev(static_cast<uint32_t>(xc), static_cast<uint32_t>(yc), w, h);
}

RT_HD uint32_t prev_index(uint32_t prev_xy, uint32_t w) { return (prev_xy & 0xffffu) + (prev_xy >> 16) * w; }

// ---- reservoir (include/graph/restir/Reservoir.h:28-50) ------------------------
template <typename T>
RT_D bool res_update(Res<T>& r, const T& s, float w, Rng& rng, float in_conf) {
    if (isnan(w) || isinf(w)) w = 0.0f;
    r.w_sum += w;
    r.conf += in_conf;
    r.conf = gmin(r.conf, CRISB_CONFIDENCE_MAX);
    if (rng.next_float() < w / r.w_sum) {
        r.s = s;
        return true;
    }
    return false;
}
// res_update without the sample: the same weight and confidence arithmetic and
// the same random draw; true when the candidate replaces the current sample
RT_D bool res_choose(float& w_sum, float& conf, float w, Rng& rng, float in_conf) {
    if (isnan(w) || isinf(w)) w = 0.0f;
    w_sum += w;
    conf += in_conf;
    conf = gmin(conf, CRISB_CONFIDENCE_MAX);
    return rng.next_float() < w / w_sum;
}

template <typename T>
RT_D void res_finalize(Res<T>& r) {
    const float phat = luminance(r.s.f);
    if (phat == 0.0f) r.w_sum = 0.0f;
    else r.w_sum /= phat;
}

// ---- pairwise MIS (include/graph/restir/path_gen.h:15-48) ----------------------
RT_D float mis_canonical(V3 b_at_b, V3 b_at_n, float jac, float K, float cM, float nM) {
    float w = 1.f;
    if (luminance(b_at_b) > 0.f) {
        const float at_basis = luminance(b_at_b) * cM;
        w = at_basis / (at_basis + luminance(b_at_n) * jac * nM * K);
    }
    return w;
}
RT_D float mis_neighbor(V3 n_at_b, V3 n_at_n, float jac, float K, float cM, float nM) {
    float w = 0.f;
    if (luminance(n_at_n) > 0.f) {
        w = luminance(n_at_n) * nM / (luminance(n_at_n) * nM + luminance(n_at_b) * jac * cM / K);
    }
    return w;
}

// SelectSpatialNeighbor (path_gen.h:50-57) with a configurable window radius
RT_D void select_spatial_neighbor(uint32_t px, uint32_t py, uint32_t radius, Rng& rng, uint32_t& nx, uint32_t& ny) {
    const uint32_t ws = 2 * radius + 1;
    const uint32_t x = (px + radius) - (rng.next_u32() % ws);
    const uint32_t y = (py + radius) - (rng.next_u32() % ws);
    if (x == px && y == py) {
        nx = px + 1;
        ny = py + 1;
        return;
    }
    nx = x;
    ny = y;
}

// CalcReconnectionJacobian (path_gen.h:59-72)
RT_D float recon_jacobian(V3 old_xi, V3 new_xi, V3 target, V3 target_n) {
    const float term1 =
        fabsf(dot(normalize(new_xi - target), target_n) / dot(normalize(old_xi - target), target_n));
    const float term2 = dot(target - old_xi, target - old_xi);
    const float term3 = dot(target - new_xi, target - new_xi);
    const float result = term1 * term2 / term3;
    if (isinf(result) || isnan(result)) return 0.0f;
    return gmax(0.0f, result);
}

// ---- path generation -----------------------------------------------------------------
// TraceCompletePath (path_gen.h:389-472) cut at its rays: a lane holds the ray
// its path waits for, and step() takes the ray's result to the next ray or the
// end.  The radiance of a light connection does not depend on the shadow ray, so
// it is evaluated before the ray and the ray only selects between it and zero
// (a radiance that is bitwise +0 needs no ray).
struct CompletePath {
    V3 o, d;        // the ray in flight
    float tmax;     // 1e16 for an extension ray, the light distance for a shadow ray
    bool shadow;
    V3 tp, radiance;
    uint32_t depth;
    Rng rng;

    RT_D void begin(V3 origin, V3 dir, const Rng& r) {
        o = origin;
        d = dir;
        tmax = 1e16f;
        shadow = false;
        tp = splat(1.0f);
        radiance = splat(0.0f);
        depth = 0;
        rng = r;
    }
    // the path's next ray is in o, d, tmax, shadow; false: ended with `radiance`
    template <bool kTex>
    RT_D bool step(const SceneView& s, const FrameParams& fp, const TraceResult& h) {
        if (shadow) {
            if (h.prim != CRISB_INVALID_PRIM) radiance = splat(0.0f);
            return false;
        }
        Isect it;
        hit_isect(s, h, d, it);
        if (!it.valid) return false;
        ++depth;
        const float nee = fp.p.nee_prob;
        if (rng.next_float() < nee) {
            tp = tp / nee;
            const EmitterSample es = sample_emitter(s, rng);
            const V3 light_dir = normalize(es.pos - it.pos);
            const float dist = length(es.pos - it.pos);
            const BrdfEval be = brdf_eval<kTex>(s, it, light_dir);
            const float dist_factor = 1.0f / (dist * dist);
            radiance = tp * be.brdf * es.color * dist_factor;
            if (depth == 1) radiance = radiance + be.emission;
            if ((__float_as_uint(radiance.x) | __float_as_uint(radiance.y) | __float_as_uint(radiance.z)) == 0u)
                return false;
            o = it.pos;
            d = light_dir;
            tmax = dist;
            shadow = true;
            return true;
        }
        const BrdfSample bs = brdf_sample<kTex>(s, it, rng);
        if (bs.pdf <= 0.0f) return false;
        tp = tp * (bs.brdf / bs.pdf);
        tp = tp / (1.0f - nee);
        o = it.pos;
        d = bs.dir;
        return depth < static_cast<uint32_t>(fp.p.max_path_len);
    }
};

// TracePrefixForFinalGather (path_gen.h:474-531)
RT_D bool trace_prefix_for_gather(const SceneView& s, V3& tp, float& p, Isect& last, V3 origin, V3 dir,
                                  uint32_t max_len, Rng& rng) {
    V3 cur_pos = origin, cur_dir = dir;
    tp = splat(1.0f);
    p = 1.0f;
    last.valid = false;
    for (uint32_t ti = 0; ti < max_len; ++ti) {
        trace_closest(s, cur_pos, cur_dir, 1e-3f, 1e16f, last);
        if (!last.valid) return false;
        const BrdfSample bs = brdf_sample(s, last, rng);
        if (bs.pdf <= 0.0f) return false;
        cur_pos = last.pos;
        cur_dir = bs.dir;
        tp = tp * bs.brdf;
        p *= bs.pdf;
    }
    return true;
}

// SpawnCameraRay's direction (include/graph/Camera.h:14-22) at viewport
// coordinates (ux, uy)
RT_D V3 spawn_camera_dir(V3 U, V3 V, V3 W, float ux, float uy) { return normalize(U * ux + V * uy + W); }

// jittered camera ray of the pixel (prefix_gen_temp_reuse.cu:124-126); the x
// jitter is drawn before the y jitter.
RT_D V3 camera_dir(const FrameParams& fp, uint32_t x, uint32_t y, Rng& rng) {
    const float jx = rng.next_float();
    const float jy = rng.next_float();
    float ux = (static_cast<float>(x) + jx) / static_cast<float>(fp.width);
    float uy = (static_cast<float>(y) + jy) / static_cast<float>(fp.height);
    ux = 2.0f * ux - 1.0f;
    uy = 2.0f * uy - 1.0f;
    return spawn_camera_dir(ld3(fp.cam.u), ld3(fp.cam.v), ld3(fp.cam.w), ux, uy);
}

}  // namespace crisb
