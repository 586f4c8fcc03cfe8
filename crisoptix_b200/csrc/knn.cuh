// knn.cuh -- the prefix-endpoint neighbour search (device side).
//
// Replaces the OptiX custom-primitive acceleration structure over per-pixel
// AABBs and its intersection program (src/PrefixAccelStruct.cpp:14-221,
// shader/prefix_search_hit.cu:9-73).  An entry is an endpoint position with a
// radius; a query point q collects every entry j with |p_j - q| <= r_j and
// keeps the k nearest, ordered by (distance, entry index) -- a deterministic
// definition of the reference's "first k hits in traversal order".  The
// entries sit in an LBVH (lbvh.cuh) whose boxes are conservative: an entry
// that passes the distance test always has q inside its box.
#pragma once

#include "lbvh.cuh"

namespace crisb {

struct KnnView {
    const BvhNode* nodes;
    const float4* leaf;       // leaf order: x, y, z, radius
    const uint32_t* index;    // leaf order -> entry index
    const uint32_t* n;        // number of entries in the structure
};

struct NeighborList {
    float dist[CRISB_MAX_GATHER_M];
    uint32_t pix[CRISB_MAX_GATHER_M];
    uint32_t count;
};

// float <-> order-preserving unsigned, for atomic min / max of floats
RT_D unsigned int float_to_ordered(float f) {
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
RT_D float ordered_to_float(unsigned int u) {
    return __uint_as_float((u & 0x80000000u) ? (u & 0x7FFFFFFFu) : ~u);
}

// conservative box of an entry: a candidate passes dist <= radius only if the
// query lies inside this box
RT_D lbvh::Box entry_box(float4 e) {
    const float h = e.w * 1.0001f + 4e-7f * (fabsf(e.x) + fabsf(e.y) + fabsf(e.z) + 1.0f);
    lbvh::Box bx;
    bx.lo[0] = e.x - h;
    bx.lo[1] = e.y - h;
    bx.lo[2] = e.z - h;
    bx.hi[0] = e.x + h;
    bx.hi[1] = e.y + h;
    bx.hi[2] = e.z + h;
    return bx;
}

// An entry is rejected on its squared distance where d > radius is certain: the
// rounded root d of d2 is at most r only if d2 <= r^2 (1 + 2^-23).
constexpr float kRejectScale = 1.0000005f;

RT_D bool knn_before(float d, uint32_t p, float d2, uint32_t p2) { return d < d2 || (d == d2 && p < p2); }

// A 64-byte node as two 32-byte loads.  A query is a chain of dependent node loads,
// each lane's its own: with these, the reject above the square root and both leaf
// children in one loop, 262,144 queries of 8 neighbours take 183 us instead of 213.
RT_D BvhNode ld_node(const BvhNode* p) {
    BvhNode n;
    float d0, d1, d2, d3;
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(n.a.x), "=f"(n.a.y), "=f"(n.a.z), "=f"(n.a.w), "=f"(n.b.x), "=f"(n.b.y), "=f"(n.b.z), "=f"(n.b.w)
        : "l"(p));
    asm("ld.global.nc.v8.f32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
        : "=f"(n.c.x), "=f"(n.c.y), "=f"(n.c.z), "=f"(n.c.w), "=f"(d0), "=f"(d1), "=f"(d2), "=f"(d3)
        : "l"(reinterpret_cast<const char*>(p) + 32));
    n.d = make_int4(__float_as_int(d0), __float_as_int(d1), __float_as_int(d2), __float_as_int(d3));
    return n;
}

RT_D void knn_error(int* err, int code) {
    if (err) atomicOr(err, code);
}

// The k (<= CRISB_MAX_GATHER_M) nearest entries whose radius covers q.  A
// query that visits more than max_visits nodes stops with the neighbours found
// so far and sets kDevErrKnn in *err.
RT_D void knn_query(const KnnView& v, int* err, V3 q, uint32_t k, NeighborList& nl,
                    uint32_t max_visits = kKnnMaxVisits) {
    nl.count = 0;
    bool alive = *v.n != 0 && k != 0 && !nonfinite(q);
    int stack[kTraversalStack];
    int sp = 0;
    int cur = 0;
    uint32_t visits = 0;
    while (alive) {
        if (++visits > max_visits) {
            knn_error(err, kDevErrKnn);
            return;
        }
        const BvhNode nd = ld_node(v.nodes + cur);
        const bool in_l = q.x >= nd.a.x && q.y >= nd.a.y && q.z >= nd.a.z && q.x <= nd.a.w && q.y <= nd.b.x &&
                          q.z <= nd.b.y;
        const bool in_r = q.x >= nd.b.z && q.y >= nd.b.w && q.z >= nd.c.x && q.x <= nd.c.y && q.y <= nd.c.z &&
                          q.z <= nd.c.w;
        // the entries of the leaf children the query lies in: siblings' ranges of
        // the leaf order touch, so both together are one range too
        const bool leaf_l = in_l && nd.d.x < 0, leaf_r = in_r && nd.d.y < 0;
        int i = -1 - (leaf_l ? nd.d.x : nd.d.y);
        const int end = i + (leaf_l ? nd.d.z : 0) + (leaf_r ? nd.d.w : 0);
        for (; i < end; ++i) {
            const float4 e = __ldg(&v.leaf[i]);
            const V3 w = q - V3{e.x, e.y, e.z};
            const float d2 = dot(w, w);
            if (d2 > e.w * e.w * kRejectScale && e.w > 1e-18f) continue;
            const float d = sqrtf(d2);
            if (d > e.w) continue;
            const uint32_t j = __ldg(&v.index[i]);
            if (nl.count == k) {
                if (!knn_before(d, j, nl.dist[k - 1], nl.pix[k - 1])) continue;
                --nl.count;
            }
            uint32_t pos = nl.count;
            while (pos > 0 && knn_before(d, j, nl.dist[pos - 1], nl.pix[pos - 1])) {
                nl.dist[pos] = nl.dist[pos - 1];
                nl.pix[pos] = nl.pix[pos - 1];
                --pos;
            }
            nl.dist[pos] = d;
            nl.pix[pos] = j;
            ++nl.count;
        }
        const bool go_l = in_l && !leaf_l, go_r = in_r && !leaf_r;
        if (go_l || go_r) {
            cur = go_l ? nd.d.x : nd.d.y;
            if (go_l && go_r) {
                if (sp >= kTraversalStack) {
                    knn_error(err, kDevErrStack);
                    return;
                }
                stack[sp++] = nd.d.y;
            }
        } else if (sp > 0) {
            cur = stack[--sp];
        } else {
            alive = false;
        }
    }
}

}  // namespace crisb
