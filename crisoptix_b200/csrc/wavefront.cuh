// wavefront.cuh -- TracePrefix and TraceSuffix as one resumable machine.
//
// The per-pixel loops of include/graph/restir/path_gen.h:74-387 are cut at
// every ray they trace: a step takes the result of the path's ray through the
// loop body of one vertex up to the path's next closest-hit ray (extension,
// reconnection vertex) or shadow ray (NEE), and the path's end.  The arithmetic
// of each step is the loop body of the reference function, in the same order,
// so a path ends with the same record bits as the per-pixel loop.
//
// Prefix and suffix vertices run through the same code (one light sample, one
// BRDF evaluation, one BRDF sample), so lanes in either loop shade together; the
// NEE BRDF, which does not depend on visibility, is evaluated with its vertex and
// not after the shadow ray.  On persistent warps, with a copy of that code per
// loop and per ray kind (five BRDF bodies in one kernel), a 1080p frame took 22.4
// instead of 15.6 ms.
#pragma once

#include "passes.cuh"
#include "records.cuh"

namespace crisb {
namespace {

RT_D float4 f4(V3 v, float w) { return make_float4(v.x, v.y, v.z, w); }

enum WfPhase : uint32_t {
    kPhDone = 0,
    kPhStart = 1,   // a suffix at its first vertex, which no ray leads to
    kPhHit = 2,     // extension ray
    kPhShadow = 3,  // NEE shadow ray
    kPhRecon = 4,   // reconnection-vertex ray of a suffix
};

// Vertex fields of the record in hand that the path has written
enum : uint32_t { kSetPrimary = 1u, kSetRecon = 2u, kSetLast = 4u };

// A lane's path.  Flows: 0 TracePrefix into the canonical prefix record, 1
// TraceSuffix into the canonical suffix record from the pixel's reservoir prefix,
// 2 the gather's fresh prefix and then its suffix.  The running values stay in
// registers; vertex fields and reconOutDir go to the record when a step sets
// them, the running values when the path ends.  Canonical records keep the fields
// that no step sets from the frames before; the gather's records are fresh, so
// their unset fields are written.
template <int kFlow, bool kTex>
struct FlowPath {
    uint32_t phase;
    uint32_t ctr;   // bits 0-7 loop index, bit 8 post-reconnection, bit 9 suffix, 10-12 set fields, 16-23
                    // max length, 24-31 prefix length
    V3 o, d;        // the ray in flight (Start: o is unused)
    float tmax;     // shadow ray: the light distance
    uint32_t flags; // record flags, throughput, post-reconnection throughput, pdf
    V3 f, prf;
    float p, path_len;
    Rng rng;
    // the vertex and light of a shadow ray (and of the reconnection ray after it)
    uint32_t prim;
    float bu, bv;
    V3 in_dir, brdf, col;
    bool dark;      // the BRDF towards the light has no density

    RT_D uint32_t idx() const { return ctr & 0xffu; }
    RT_D bool post() const { return (ctr >> 8) & 1u; }
    RT_D bool suffix() const { return kFlow == 1 || (kFlow == 2 && ((ctr >> 9) & 1u)); }
    RT_D uint32_t set() const { return (ctr >> 10) & 7u; }
    RT_D uint32_t max_len() const { return (ctr >> 16) & 0xffu; }
    RT_D uint32_t pre_len() const { return ctr >> 24; }
    RT_D void mark(uint32_t fields) { ctr |= fields << 10; }

    RT_D static crisb_prefix_rec& prefix_rec(const Bufs& b, uint32_t i) {
        return kFlow == 0 ? b.canon_prefix[i] : b.gather_cp[i];
    }
    RT_D static crisb_suffix_rec& suffix_rec(const Bufs& b, uint32_t i) {
        return kFlow == 1 ? b.canon_suffix[i].sample : b.gather_cs[i].sample;
    }
    RT_D static Hit no_hit() { return Hit{CRISB_INVALID_PRIM, 0.0f, 0.0f, splat(0.0f)}; }

    // ---- starts -------------------------------------------------------------------
    // pixel i's path; leaves phase Done where none runs
    RT_D void begin(const SceneView& s, const FrameParams& fp, const Bufs& b, uint32_t i) {
        if (kFlow == 1) {
            const uint32_t pflags = pres_flags(b.pres[fp.front], i);
            if (!fl_valid(pflags) || fl_nee(pflags)) {
                Res<Suffix> cur = ld_sres(b.sres_cur, i);
                invalidate(cur);
                st_sres(b.sres_next, i, cur);  // the temporal pass writes sres_next
                b.nval_next[i] = 0;
                b.pass_status[i] = kWfIdle;
                return;
            }
            rng = Rng{b.gbuf[i].rng};
            b.pass_status[i] = kWfPath;
            const Hit last = pres_last(b.pres[fp.front], i);
            if (begin_suffix(fp, b, i, fl_len(pflags), last, last.valid() && last.prim < s.num_tris)) {
                prim = last.prim;
                bu = last.bu;
                bv = last.bv;
                in_dir = last.dir;
                phase = kPhStart;
            } else {
                end_suffix(b, i);
            }
            return;
        }
        if (kFlow == 2) {
            if (b.canon_prefix[i].primary.prim == CRISB_INVALID_PRIM) {
                b.pass_status[i] = kWfIdle;
                if (b.gather_ext) b.gather_ext[3 * static_cast<size_t>(i)] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                return;
            }
            rng = Rng{b.gbuf[i].rng};
            b.pass_status[i] = kWfPath;
        } else {
            rng = rng_seeded(tea64(i, fp.random));
        }
        o = ld3(fp.cam.pos);
        d = camera_dir(fp, i % fp.width, i / fp.width, rng);
        // gatherN > 1: the extra prefixes start along the same ray
        if (kFlow == 2 && b.gather_ext)
            b.gather_ext[3 * static_cast<size_t>(i)] = make_float4(d.x, d.y, d.z, 1.0f);
        const int len = fp.p.renderer_type == CRISB_RENDERER_RESTIR_PT ? fp.p.max_path_len : fp.p.prefix_len;
        ctr = (static_cast<uint32_t>(len) & 0xffu) << 16;
        flags = fl_set_valid(0u, true);
        f = prf = splat(1.0f);
        p = 1.0f;
        path_len = 0.0f;
        prefix_rec(b, i).rng = rng.state;
        phase = kPhHit;
    }

    // the suffix of a valid prefix of `len` vertices that did not end in NEE,
    // from its last vertex; false: it has no vertex
    RT_D bool begin_suffix(const FrameParams& fp, const Bufs& b, uint32_t i, uint32_t len, const Hit& last,
                           bool last_valid) {
        crisb_suffix_rec& r = suffix_rec(b, i);
        r.rng = rng.state;
        st_hit(r.last_prefix, last);
        flags = 0u;
        f = prf = splat(1.0f);
        p = 1.0f;
        const uint32_t n = static_cast<uint32_t>(fp.p.max_path_len) - len;
        ctr = (1u << 9) | ((n & 0xffu) << 16) | (len << 24);
        return last_valid && n != 0;
    }

    // ---- ends ---------------------------------------------------------------------
    RT_D void end_prefix(const Bufs& b, uint32_t i) {
        crisb_prefix_rec& r = prefix_rec(b, i);
        r.flags = flags;
        st3(r.f, f);
        st3(r.post_recon_f, prf);
        r.p = p;
        r.path_len = path_len;
        if (kFlow == 2) {
            const uint32_t have = set();
            if (!(have & kSetPrimary)) st_hit(r.primary, no_hit());
            if (!(have & kSetLast)) st_hit(r.last, no_hit());
            if (!(have & kSetRecon)) {
                st_hit(r.recon, no_hit());
                st3(r.recon_out_dir, splat(0.0f));
            }
        }
        phase = kPhDone;
        b.gbuf[i].rng = rng.state;  // for the pass's next kernels
    }
    RT_D void end_suffix(const Bufs& b, uint32_t i) {
        crisb_suffix_rec& r = suffix_rec(b, i);
        r.flags = flags;
        st3(r.f, f);
        st3(r.post_recon_f, prf);
        r.p = p;
        if (kFlow == 2 && !(set() & kSetRecon)) {
            st_hit(r.recon, no_hit());
            st3(r.recon_out_dir, splat(0.0f));
        }
        phase = kPhDone;
        b.gbuf[i].rng = rng.state;
    }
    RT_D void end(const Bufs& b, uint32_t i) {
        if (suffix()) end_suffix(b, i);
        else end_prefix(b, i);
    }
    // an end that leaves a prefix invalid (a suffix is only valid once finished)
    RT_D void fail(const Bufs& b, uint32_t i) {
        if (!suffix()) flags = fl_set_valid(flags, false);
        end(b, i);
    }

    RT_D void set_recon(const Bufs& b, uint32_t i, const Hit& h, V3 out_dir) {
        if (suffix()) {
            st_hit(suffix_rec(b, i).recon, h);
            st3(suffix_rec(b, i).recon_out_dir, out_dir);
        } else {
            st_hit(prefix_rec(b, i).recon, h);
            st3(prefix_rec(b, i).recon_out_dir, out_dir);
        }
        mark(kSetRecon);
    }

    // ---- steps --------------------------------------------------------------------
    RT_D void finish_nee_suffix(const Bufs& b, uint32_t i, float light_len) {
        const float dist_factor = 1.0f / (light_len * light_len);
        f = f * (brdf * col * dist_factor);
        prf = prf * (col * dist_factor);
        if (fl_recon(flags) < fl_len(flags)) prf = prf * brdf;
        flags = fl_set_valid(flags, true);
        end_suffix(b, i);
    }

    // path_gen.h:167-222 and 300-345 after the shadow ray
    RT_D void shadow_done(const SceneView& s, const Bufs& b, uint32_t i, bool occluded) {
        if (occluded) {
            fail(b, i);
            return;
        }
        if (suffix()) {
            flags = fl_set_len(flags, fl_len(flags) + 1);
            if (post()) {
                finish_nee_suffix(b, i, tmax);
                return;
            }
            phase = kPhRecon;  // from the vertex along the light direction: o, d as they are
            return;
        }
        const Hit v{prim, bu, bv, in_dir};
        if (!post()) {
            // the reference re-traces the same ray here; the result is `v`
            flags = fl_set_recon(flags, fl_len(flags));
            set_recon(b, i, v, in_dir);
        }
        if (dark) {
            fail(b, i);
            return;
        }
        const float dist_factor = 1.0f / (tmax * tmax);
        f = f * (brdf * col * dist_factor);
        prf = prf * (brdf * col * dist_factor);
        if (fl_len(flags) == 1) {
            const crisb_material& m = s.mats[material_of(s, prim)];
            f = f + V3{m.emission[0], m.emission[1], m.emission[2]} * dist_factor;
        }
        flags = fl_set_nee(flags, true);
        flags = fl_set_valid(flags, true);
        st_hit(prefix_rec(b, i).last, v);
        mark(kSetLast);
        end_prefix(b, i);
    }

    RT_D void recon_done(const Bufs& b, uint32_t i, const TraceResult& h) {
        if (h.prim == CRISB_INVALID_PRIM) {
            end_suffix(b, i);
            return;
        }
        flags = fl_set_recon(flags, fl_len(flags));
        flags = fl_set_recon_vert(flags, fl_len(flags) - 1);  // the NEE vertex
        set_recon(b, i, Hit{h.prim, h.u, h.v, d}, splat(0.0f));
        finish_nee_suffix(b, i, tmax);
    }

    // the vertex at the end of an extension ray, or a suffix's first vertex
    RT_D void vertex(const SceneView& s, const FrameParams& fp, const Bufs& b, uint32_t i, const TraceResult& h) {
        Isect it;
        it.valid = true;
        if (kFlow == 1 && phase == kPhStart) {
            it.prim = prim;
            it.bu = bu;
            it.bv = bv;
            it.dir = in_dir;
        } else {
            if (h.prim == CRISB_INVALID_PRIM) {
                fail(b, i);
                return;
            }
            it.prim = h.prim;
            it.bu = h.u;
            it.bv = h.v;
            it.dir = d;
        }
        const ShadeTri t = load_shade(s, it.prim);
        it.pos = interp(it.bu, it.bv, t.p0, t.p1, t.p2);
        const V3 nrm = interp(it.bu, it.bv, t.n0, t.n1, t.n2);
        // an interaction from a trace has its normal normalised, one unpacked
        // from a record (a suffix's first vertex) does not
        it.nrm = kFlow == 1 && phase == kPhStart ? nrm : normalize(nrm);
        V3 from = kFlow == 1 && phase == kPhStart ? it.pos : o;
        if (kFlow != 1 && !suffix()) {
            path_len += distance(o, it.pos);
            flags = fl_set_len(flags, fl_len(flags) + 1);
            if (fl_len(flags) == 1) {
                st_hit(prefix_rec(b, i).primary, it.pack());
                mark(kSetPrimary);
            }
            if (fp.p.renderer_type == CRISB_RENDERER_CONDITIONAL_RESTIR && idx() == max_len() - 1) {
                if (!post()) {
                    flags = fl_set_recon(flags, fl_len(flags));
                    set_recon(b, i, it.pack(), splat(0.0f));
                }
                flags = fl_set_valid(flags, true);
                st_hit(prefix_rec(b, i).last, it.pack());
                mark(kSetLast);
                const uint32_t len = fl_len(flags);
                end_prefix(b, i);
                if (kFlow == 0) return;
                // FinalGatherCanon: the canonical suffix continues the canonical prefix
                if (!begin_suffix(fp, b, i, len, it.pack(), true)) {
                    end_suffix(b, i);
                    return;
                }
                it.nrm = nrm;
                from = it.pos;
            }
        }
        const bool suf = suffix();
        const float nee = fp.p.nee_prob;
        const bool force_nee = (suf || fp.p.renderer_type == CRISB_RENDERER_RESTIR_PT) && idx() == max_len() - 1;
        if (rng.next_float() < nee || force_nee) {
            if (!suf || !force_nee) p *= nee;
            const EmitterSample es = sample_emitter(s, rng);
            const V3 light_vec = es.pos - it.pos;
            const float light_len = length(light_vec);
            const V3 light_dir = normalize(light_vec);
            if (suf && nonfinite(light_dir)) {
                end_suffix(b, i);
                return;
            }
            const BrdfEval be = brdf_eval<kTex>(s, it, light_dir);
            dark = be.pdf <= 0.0f;
            if (suf && dark) {  // ends the same way whether or not the light is visible
                end_suffix(b, i);
                return;
            }
            prim = it.prim;
            bu = it.bu;
            bv = it.bv;
            in_dir = it.dir;
            brdf = be.brdf;
            col = es.color;
            o = it.pos;
            d = light_dir;
            tmax = light_len;
            phase = kPhShadow;
            return;
        }
        const BrdfSample bs = brdf_sample<kTex>(s, it, rng);
        if (bs.pdf <= 0.0f) {
            fail(b, i);
            return;
        }
        const float recon_dist = distance(from, it.pos);
        const bool can_recon = recon_dist > fp.p.recon_min_distance && bs.roughness > fp.p.recon_min_roughness &&
                               (suf ? pre_len() >= 1 : fl_len(flags) >= 2);
        const bool was_post = post();
        if (!was_post && can_recon) {
            flags = fl_set_recon(flags, suf ? pre_len() : fl_len(flags));
            if (suf) flags = fl_set_recon_vert(flags, fl_len(flags));  // the loop index
            set_recon(b, i, it.pack(), bs.dir);
            ctr |= 1u << 8;
        }
        f = f * bs.brdf;
        p *= bs.pdf * (1.0f - nee);
        // a prefix's post-reconnection throughput starts at the reconnection
        // vertex, a suffix's after it
        if (suf ? was_post : post()) prf = prf * bs.brdf;
        if (suf) flags = fl_set_len(flags, fl_len(flags) + 1);
        if (idx() + 1 < max_len()) {
            o = it.pos;
            d = bs.dir;
            ctr += 1u;
            phase = kPhHit;
            return;
        }
        if (!suf) {
            st_hit(prefix_rec(b, i).last, it.pack());
            mark(kSetLast);
        }
        end(b, i);
    }

    // ---- between launches ---------------------------------------------------------
    RT_D static TraceResult result(const PathState* st) {
        const uint4 h = st->hit;
        return TraceResult{h.x, uf(h.y), uf(h.z), uf(h.w)};
    }
    RT_D void save(PathState* st) const {
        st->w[0] = make_uint4(phase | (dark ? 16u : 0u), ctr, flags, __float_as_uint(p));
        st->w[1] = make_uint4(fu(o.x), fu(o.y), fu(o.z), fu(path_len));
        st->w[2] = make_uint4(fu(d.x), fu(d.y), fu(d.z), fu(f.x));
        st->w[3] = make_uint4(fu(f.y), fu(f.z), fu(prf.x), fu(prf.y));
        st->w[4] = make_uint4(fu(prf.z), 0u, static_cast<uint32_t>(rng.state), static_cast<uint32_t>(rng.state >> 32));
        if (phase == kPhHit) return;
        st->w[5] = make_uint4(fu(tmax), prim, fu(bu), fu(bv));
        st->w[6] = make_uint4(fu(in_dir.x), fu(in_dir.y), fu(in_dir.z), fu(brdf.x));
        st->w[7] = make_uint4(fu(brdf.y), fu(brdf.z), fu(col.x), fu(col.y));
        st->w[8] = make_uint4(fu(col.z), 0u, 0u, 0u);
    }
    RT_D void load(const PathState* st) {
        const uint4 a = st->w[0], q = st->w[1], c = st->w[2], e = st->w[3], g = st->w[4];
        phase = a.x & 15u;
        dark = (a.x & 16u) != 0u;
        ctr = a.y;
        flags = a.z;
        p = uf(a.w);
        o = V3{uf(q.x), uf(q.y), uf(q.z)};
        path_len = uf(q.w);
        d = V3{uf(c.x), uf(c.y), uf(c.z)};
        f = V3{uf(c.w), uf(e.x), uf(e.y)};
        prf = V3{uf(e.z), uf(e.w), uf(g.x)};
        rng.state = static_cast<uint64_t>(g.z) | (static_cast<uint64_t>(g.w) << 32);
        if (phase == kPhHit) return;
        const uint4 k = st->w[5], l = st->w[6], m = st->w[7], n = st->w[8];
        tmax = uf(k.x);
        prim = k.y;
        bu = uf(k.z);
        bv = uf(k.w);
        in_dir = V3{uf(l.x), uf(l.y), uf(l.z)};
        brdf = V3{uf(l.w), uf(m.x), uf(m.y)};
        col = V3{uf(m.z), uf(m.w), uf(n.x)};
    }
    RT_D static uint32_t fu(float v) { return __float_as_uint(v); }
    RT_D static float uf(uint32_t v) { return __uint_as_float(v); }

    RT_D void step(const SceneView& s, const FrameParams& fp, const Bufs& b, uint32_t i, const TraceResult& h) {
        if (phase == kPhShadow) shadow_done(s, b, i, h.prim != CRISB_INVALID_PRIM);
        else if (kFlow != 0 && phase == kPhRecon) recon_done(b, i, h);
        else vertex(s, fp, b, i, h);
    }
};

}  // namespace
}  // namespace crisb
