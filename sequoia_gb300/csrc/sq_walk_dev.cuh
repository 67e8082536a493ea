// sq_walk_dev.cuh -- the order-free traversals of the reference, a warp's
// rays or packets from one pool of node ranges.
//
// trace() / traverse() (src/tracer.cpp:47-65, 195-230) and trace_packet<k>
// (src/tracer.cpp:88-123, 232-281) test every child of every node that a ray
// (any ray of a packet) hits, in no order that matters and with no early
// exit: the result is a count and a hit flag.  So a ray's node ranges need
// not be walked by the ray's own lane.  The warp keeps one pool of (node
// range, owner) entries in shared memory, and each step every lane takes an
// entry of any owner, tests up to two nodes against the owner's K rays (a
// node counts once a packet, so the first ray that hits ends its test) and
// puts the hit nodes' child ranges back.  Triangles of hit leaves go to a
// second pool and are tested 32 at a time.
//
// trace_bundle<k> (src/tracer.cpp:126-156, 292-362) adds owners that are
// bundles: tested by their direction bounds, walked while the middle
// direction hits, and where only the bounds hit, all packets of the bundle go
// on alone from that node.  Such a node is one entry of a third kind (node,
// packets [first, first + n)), halved each time it is taken until it is one
// packet's, so no entry taken puts more than two back.
//
// What bounds it: with a ray per lane the kernel waited for its longest rays
// (a ray through the middle of the 2M-triangle soup tests thousands of boxes,
// its neighbours in the warp tens): 14 of 32 lanes busy and 30% of the warps
// resident on average.  Bundles waited for one walk after another: the bundle
// the same on all 32 lanes, its packets 8 lanes each.
#pragma once

#include "sq_trace_dev.cuh"

namespace sq {

constexpr uint32_t kPoolCap = 768;      // node ranges in a warp's pool (more cost resident warps)
constexpr uint32_t kTriCap = 128;       // 31 waiting + 64 of one step fit
constexpr uint32_t kCountBits = 27;     // an entry: node, owner << 27 | node count
constexpr uint32_t kCountMask = (1u << kCountBits) - 1u;

// intersect_bundle_aabb (src/tracer.h:37-80)
__device__ __forceinline__ void bundle_box(const NodeRec& nd, const float* pos, const float* imin, const float* imax,
                                           const float* imid, bool& any_hit, bool& mid_hit)
{
    float tmin_mid[3], tmin_any[3], tmax_mid[3], tmax_any[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float lo = nd.mn[k] - pos[k], hi = nd.mx[k] - pos[k];
        const float t1a = lo * imin[k], t1b = lo * imax[k], t2a = hi * imin[k], t2b = hi * imax[k];
        const float t1 = lo * imid[k], t2 = hi * imid[k];
        const float t1min = ref_min(t1a, t1b), t1max = simd_max(t1a, t1b);
        const float t2min = ref_min(t2a, t2b), t2max = simd_max(t2a, t2b);
        tmin_mid[k] = ref_min(t1, t2);
        tmin_any[k] = ref_min(t1min, t2min);
        tmax_mid[k] = simd_max(t1, t2);
        tmax_any[k] = simd_max(t1max, t2max);
    }
    const float front_mid = ref_max(ref_max(tmin_mid[0], tmin_mid[1]), tmin_mid[2]);
    const float front_any = ref_max(ref_max(tmin_any[0], tmin_any[1]), tmin_any[2]);
    const float back_mid = ref_min(ref_min(tmax_mid[0], tmax_mid[1]), tmax_mid[2]);
    const float back_any = ref_min(ref_min(tmax_any[0], tmax_any[1]), tmax_any[2]);
    mid_hit = back_mid >= front_mid;
    any_hit = back_any >= front_any;
}

// K rays per owner, PW owners per warp, and NB bundles of PW / NB owners each
// (0: the owners start by themselves).  Owner numbers: 0 to PW - 1 the owners,
// then the bundles, then the bundles' entries of the third kind; at most 32.
template <int K, int PW, bool TRI, int NB = 0>
struct WalkPool {
    static_assert(PW + 2 * NB <= 32, "an owner number has 5 bits");
    // places kept for the one-at-a-time walk (walk_pool): the deepest walk of
    // one ray or packet that is asked for has 128 pending ranges, one of a
    // bundle 128 more, and a range, a fan and the places checked for come on
    // top
    static constexpr uint32_t kOpen = kPoolCap - (NB ? 272u : 136u);
    uint2 node[kPoolCap];
    uint2 tri[TRI ? kTriCap : 1];
    float inv[3][K][PW];                      // reciprocal directions
    float o[3][TRI ? PW : 1], d[3][TRI ? PW : 1], tmax[TRI ? PW : 1];
    float bun[9][NB ? NB : 1];                // bundles: reciprocals of the least, largest and middle direction
    uint32_t cnt[PW + NB];                    // box tests of each owner and bundle
    uint32_t hit;                             // bit per owner: a triangle was hit
};

struct WalkStats {
    uint32_t tri_tests;  // this lane's
    bool overflow, bad;  // pool full; an index outside the node or triangle array
};

// Walks nodes [root, root + group) for every owner in `owners` (a mask, the
// same in all lanes; with bundles, of bundles); pool.inv (and o, d, tmax with TRI) hold the owners'
// rays.  Without TRI all rays start at `org` and end at 10000.  hit_tri(tri, o, d)
// tests one triangle.  Afterwards pool.cnt and pool.hit have the results.
//
// The pool grows by at most two ranges per entry taken, so as it fills fewer
// entries are taken a step, down to one at a time where only the reserve is
// left: the rest of the range goes above the children that were found, and a
// bundle's packets above both, so this is the reference's own order (all of a
// group, then the last hit child's; src/tracer.cpp:47-65, 126-156) and needs
// the places of the reference's own stack.  (Halving long ranges here too left
// half a group behind at every level of a chain of groups of 17 nodes.)
template <int K, int PW, bool TRI, int NB, class HitTri>
__device__ __forceinline__ void walk_pool(WalkPool<K, PW, TRI, NB>& pool, uint32_t owners, const Node* __restrict__ nodes,
                                          uint32_t nn, uint32_t nt, uint32_t root, uint32_t group, const float* org,
                                          WalkStats& st, HitTri hit_tri)
{
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    if (lane < (uint32_t)(PW + NB)) pool.cnt[lane] = 0;
    if (lane == 0) pool.hit = 0;
    // a range of 2^26 nodes or more (no node has one, a caller's root group
    // may) is walked in pieces
    for (uint32_t g0 = 0; g0 < group;) {
        const uint32_t piece = min(group - g0, 1u << 26);
        if ((owners >> lane) & 1u)
            pool.node[__popc(owners & lt)] = make_uint2(root + g0, piece | (lane << kCountBits));
        g0 += piece;
        uint32_t size = __popc(owners), tris = 0;
        __syncwarp();
        for (;;) {
            if (TRI && (tris >= 32u || (size == 0u && tris))) {
                const uint32_t take = min(32u, tris);
                uint2 e = make_uint2(0u, 0u);
                if (lane < take) e = pool.tri[tris - 1u - lane];
                tris -= take;
                const uint32_t w = e.y >> kCountBits, c = e.y & kCountMask;
                if (lane < take) {
                    const float o[3] = {pool.o[0][w], pool.o[1][w], pool.o[2][w]};
                    const float d[3] = {pool.d[0][w], pool.d[1][w], pool.d[2][w]};
                    bool hit = false;
                    for (uint32_t k = 0; k < c; ++k) hit |= hit_tri(e.x + k, o, d);
                    st.tri_tests += c;
                    if (hit) atomicOr(&pool.hit, 1u << w);
                }
                __syncwarp();
                continue;
            }
            if (size == 0) break;
            constexpr uint32_t kOpen = WalkPool<K, PW, TRI, NB>::kOpen;
            const uint32_t room = size < kOpen ? (kOpen - size) / 2u : 0u;
            const bool one = room == 0u;
            const uint32_t take = one ? 1u : min(min(32u, size), room);
            if (size + 2u > kPoolCap) {
                st.overflow = true;
                break;
            }
            uint2 e = make_uint2(0u, 0u);
            if (lane < take) e = pool.node[size - 1u - lane];
            size -= take;
            uint32_t w = e.y >> kCountBits, c = e.y & kCountMask;
            uint32_t fan = 0, fan_first = 0;  // packets that go on alone from node e.x
            if (NB && w >= (uint32_t)(PW + NB)) {
                fan = c & 0xFFu;
                fan_first = c >> 8;
                c = 1;
                if (fan == 1u) {
                    w = fan_first;
                    fan = 0;
                }
            }
            if ((uint64_t)e.x + c > nn) {
                st.bad = true;
                c = 0;
            }
            // up to two nodes now, the rest of the range back to the pool; a
            // long range is halved instead
            const bool halve = (c > 16u && !one) || (NB && fan);
            const uint32_t two = NB && one ? 1u : 2u;
            const uint32_t k = halve ? 0u : min(c, two);
            uint2 put[3];
            bool has[3] = {halve, halve, !halve && c > two}, leaf[2] = {false, false};
            put[0] = make_uint2(e.x, (c >> 1) | (w << kCountBits));
            put[1] = make_uint2(e.x + (c >> 1), (c - (c >> 1)) | (w << kCountBits));
            put[2] = make_uint2(e.x + two, (c - two) | (w << kCountBits));
            if (NB && fan) {
                const uint32_t h = fan >> 1;
                put[0] = make_uint2(e.x, h | (fan_first << 8) | (w << kCountBits));
                put[1] = make_uint2(e.x, (fan - h) | ((fan_first + h) << 8) | (w << kCountBits));
            }
            if (NB && k && w >= (uint32_t)PW) {
                const uint32_t g = w - (uint32_t)PW;
                const NodeRec n0 = load_node(nodes, e.x), n1 = load_node(nodes, e.x + (k > 1u ? 1u : 0u));
                float imin[3], imax[3], imid[3];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    imin[a] = pool.bun[a][g];
                    imax[a] = pool.bun[3 + a][g];
                    imid[a] = pool.bun[6 + a][g];
                }
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (q && k < 2u) break;
                    const NodeRec& nd = q ? n1 : n0;
                    bool any_hit, mid_hit;
                    bundle_box(nd, org, imin, imax, imid, any_hit, mid_hit);
                    const uint32_t cc = node_count(nd.cf);
                    if (mid_hit) {
                        has[q] = !node_is_leaf(nd.cf) && cc;
                        put[q] = make_uint2(nd.child, cc | (w << kCountBits));
                    } else if (any_hit) {
                        constexpr uint32_t PK = (uint32_t)(NB ? PW / NB : 1);
                        has[q] = true;
                        put[q] = make_uint2(e.x + (uint32_t)q, PK | ((g * PK) << 8) | ((w + (uint32_t)NB) << kCountBits));
                        if (one && has[2]) {  // on top of the rest of the range
                            const uint2 rest = put[2];
                            put[2] = put[0];
                            put[0] = rest;
                        }
                    }
                }
                atomicAdd(&pool.cnt[w], k);
            } else if (k) {
                float o[3], tmax;
#pragma unroll
                for (int a = 0; a < 3; ++a) o[a] = TRI ? pool.o[a][w] : org[a];
                tmax = TRI ? pool.tmax[w] : 10000.0f;
                const NodeRec n0 = load_node(nodes, e.x), n1 = load_node(nodes, e.x + (k > 1u ? 1u : 0u));
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    if (q && k < 2u) break;
                    const NodeRec& nd = q ? n1 : n0;
                    bool hit = false;
                    for (int m = 0; m < K && !hit; ++m) {
                        const float inv[3] = {pool.inv[0][m][w], pool.inv[1][m][w], pool.inv[2][m][w]};
                        hit = box_ref(nd, o, inv, tmax);
                    }
                    const uint32_t cc = node_count(nd.cf);
                    if (hit && cc) {
                        put[q] = make_uint2(nd.child, cc | (w << kCountBits));
                        if (!node_is_leaf(nd.cf)) has[q] = true;
                        else if (TRI) {
                            if ((uint64_t)nd.child + cc > nt) st.bad = true;
                            else leaf[q] = true;
                        }
                    }
                }
                atomicAdd(&pool.cnt[w], k);
            }
            __syncwarp();  // every lane has its entry before any is overwritten
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const uint32_t b = __ballot_sync(FULL, has[q]);
                if (has[q]) pool.node[size + __popc(b & lt)] = put[q];
                size += __popc(b);
            }
            if (TRI) {
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    const uint32_t b = __ballot_sync(FULL, leaf[q]);
                    if (leaf[q]) pool.tri[tris + __popc(b & lt)] = put[q];
                    tris += __popc(b);
                }
            }
            __syncwarp();
        }
        __syncwarp();
    }
}

}  // namespace sq
