// sq_bvh8.cu -- 8-wide BVH with 8-bit quantised child boxes (the precision
// form), built by collapsing a binary range-tree BVH (node layout in
// sq_bvh8_dev.cuh; its traversal is in sq_bvh8_trace.cu).
//
// Child box on axis a: [origin_a + qlo * 2^e_a, origin_a + qhi * 2^e_a], each
// bound computed exactly as the traversal computes it (one rounded add of an
// exact product) and moved outward until it contains the binary node's FP32
// box, so a quantised box is never smaller than the FP32 box it replaces.
// This is the compressed wide BVH idea of Ylitie, Karras and Laine
// ("Efficient Incoherent Ray Traversal on GPUs Through Compressed Wide
// BVHs", HPG 2017), laid out our own way.
//
// Collapse: each 8-wide node starts from a binary inner record's two children
// and repeatedly opens the inner child of largest surface area until it has 8
// children or no inner child is left.  Leaf-cluster records (and single leaf
// records) become leaf children; their triangles are copied into a 48-byte
// triangle array in leaf order, with the original triangle index in the
// fourth float of the first vertex.  A cluster that does not fit its parent
// becomes a node of its own, one triangle per slot.
//
// Schedule: the nodes that open records depend on their parents, level by
// level (k_collapse_coop).  The cluster nodes -- five in six of all nodes --
// depend on nothing but their place, so a parent only leaves a placeholder
// (record, first triangle slot) in the cluster's node, and k_collapse_clusters
// writes them all in one pass afterwards.
#include "sq_bvh8_dev.cuh"

#include <algorithm>
#include <type_traits>
#include <utility>

namespace {

using namespace sq;

__device__ __forceinline__ float node_sa(const Node& r)
{
    const float lx = r.mxx - r.mnx, ly = r.mxy - r.mny, lz = r.mxz - r.mnz;
    return lx * ly + lx * lz + ly * lz;
}


// Exponent of the quantisation step so that origin + 255 * 2^e >= hi.
__device__ int quant_exp(float lo, float hi)
{
    const float ext = hi - lo;
    int e = -126;
    if (ext > 0.0f) {
        int ex;
        frexpf(ext, &ex);  // ext in [2^(ex-1), 2^ex)
        e = ex - 8;        // 255 * 2^e >= 2^(ex-1) * 255/128 ... adjusted below
        if (e < -126) e = -126;
        while (e > -126 && fmaf(255.0f, pow2f(e - 1), lo) >= hi) --e;
        while (fmaf(255.0f, pow2f(e), lo) < hi && e < 127) ++e;
    }
    return e;
}

// (v - origin) / 2^e is computed as (v - origin) * 2^-e: both are the
// correctly rounded value of the same real number (2^-e is exact for every
// exponent quant_exp returns), and the multiply is far cheaper.
__device__ __forceinline__ uint8_t quant_lo(float v, float origin, int e)
{
    const float s = pow2f(e);
    float q = floorf((v - origin) * ldexpf(1.0f, -e));
    int qi = q < 0.0f ? 0 : (q > 255.0f ? 255 : (int)q);
    while (qi > 0 && fmaf((float)qi, s, origin) > v) --qi;
    return (uint8_t)qi;
}

__device__ __forceinline__ uint8_t quant_hi(float v, float origin, int e)
{
    const float s = pow2f(e);
    float q = ceilf((v - origin) * ldexpf(1.0f, -e));
    int qi = q < 0.0f ? 0 : (q > 255.0f ? 255 : (int)q);
    while (qi < 255 && fmaf((float)qi, s, origin) < v) ++qi;
    return (uint8_t)qi;
}


// One warp's staging area: a node per group of eight lanes.
struct GroupSmem {
    Node8 node[4];
    uint32_t off[4][8], cnt[4][8], child[4][8];
};

// A cluster node that k_collapse_clusters is still to write: the cluster's
// record and its first triangle slot stand in the node's second 16 bytes,
// marked by a `valid` word no node has (slot 0's rank is 0).
constexpr uint32_t kPlaceholder = 0xFFFFFFFFu;

__device__ __forceinline__ uint4* placeholder_of(Node8* node) { return reinterpret_cast<uint4*>(node) + 1; }

// Quantise and write a node, eight lanes per node (all 32 lanes call this):
// lane k holds slot k's child box (ok: the slot is used), `self` the node's
// own box.  Each lane quantises its slot's six planes; the exponents take one
// lane per axis.
__device__ __forceinline__ void write_node8(bool active, int k, int g, const Node& self, const Node& child, bool ok,
                                            uint32_t imask, uint32_t valid, uint32_t child_base, uint32_t tri_base,
                                            GroupSmem& sm, Node8* __restrict__ dst)
{
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    Node8& sn = sm.node[g];
    const float lo[3] = {self.mnx, self.mny, self.mnz}, hi[3] = {self.mxx, self.mxy, self.mxz};
    const int ea = active ? quant_exp(k == 0 ? lo[0] : (k == 1 ? lo[1] : lo[2]), k == 0 ? hi[0] : (k == 1 ? hi[1] : hi[2]))
                          : 0;
    int e[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) e[a] = __shfl_sync(FULL, ea, a, 8);
    if (active) {
        uint32_t ql[3] = {255u, 255u, 255u}, qh[3] = {0u, 0u, 0u};
        if (ok) {
            const float cl[3] = {child.mnx, child.mny, child.mnz}, ch[3] = {child.mxx, child.mxy, child.mxz};
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                ql[a] = quant_lo(cl[a], lo[a], e[a]);
                qh[a] = quant_hi(ch[a], lo[a], e[a]);
            }
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) { sn.qlo[a][k] = (uint8_t)ql[a]; sn.qhi[a][k] = (uint8_t)qh[a]; }
    }
    __syncwarp();
    if (active && k == 0) {
        uint32_t counts = 0, ranks = 0;  // a rank at an empty or leaf slot is not read
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            counts |= sm.cnt[g][q] << (4 * q);
            ranks |= (uint32_t)__popc(imask & ((1u << q) - 1u)) << (8 + 3 * q);
        }
        sn.ox = self.mnx; sn.oy = self.mny; sn.oz = self.mnz;
        sn.exps_imask = (uint32_t)(e[0] + 127) | ((uint32_t)(e[1] + 127) << 8) | ((uint32_t)(e[2] + 127) << 16) |
                        (imask << 24);
        sn.child_base = child_base;
        sn.tri_base = (tri_base & kTriBaseMask) | ((uint32_t)__popc(valid) << 27);
        sn.counts = counts;
        sn.valid = valid | ranks;
    }
    __syncwarp();
    // the node: five 16-byte words
    if (active && k < 5) reinterpret_cast<float4*>(dst)[k] = reinterpret_cast<const float4*>(&sn)[k];
}

__device__ __forceinline__ void write_tri8(float4* __restrict__ d, const float* __restrict__ tris, uint32_t id)
{
    float tv[9];
    load_tri(tris, id, tv);
    d[0] = make_float4(tv[0], tv[1], tv[2], __uint_as_float(id));
    d[1] = make_float4(tv[3], tv[4], tv[5], 0.0f);
    d[2] = make_float4(tv[6], tv[7], tv[8], 0.0f);
}

// Build 8-wide nodes from binary records, eight lanes per node and four
// nodes per warp.  Lane k of a group holds candidate child slot k (its binary
// record in registers), so the records a step opens are loaded in parallel
// and the six dequantised planes of each slot are computed by the slot's own
// lane.  The decisions are those of a sequential scan over the slots: open
// the first child of largest surface area that still fits, until none does.
// All 32 lanes must call this; a group whose `active` is false only takes
// part in the warp-wide shuffles.  Inner children become nodes
// [child_base, child_base + n) and leaf triangles take the triangle slots
// [tri_base, ...), those of the cluster children after the node's own.
// The warp's four groups allocate together: lane 0 calls
// alloc(nodes, tris, tasks, node_base, tri_base, task_base) once with the
// warp's totals (same-address atomics serialise in L2), and each group takes
// its share in group order.  publish(task, node, record) is called by the
// lane of each child that opens records itself, with task = task_base + the
// child's rank among those; cluster children get a placeholder.  published()
// is called by the whole warp once that is done: what follows (the node's
// planes and the triangle copies) is of no matter to the next level.  sm: this
// warp's staging area.
// A node that cannot be made (a record of more than eight children, a leaf of
// more than 15 triangles, no room for its children) is refused: the error word
// is set and the node is written without children, so that neither the cluster
// pass nor a trace before the error is seen meets a node that nothing wrote.
template <class Alloc, class Publish, class Published>
__device__ void collapse_node_group(const Node* __restrict__ rec, uint32_t leaf0, const float* __restrict__ tris,
                                    bool active, uint32_t rec_i, uint32_t node_i, Node8* __restrict__ nodes8,
                                    float4* __restrict__ tris8, uint32_t capacity, uint32_t* err, GroupSmem& sm,
                                    Alloc alloc, Publish publish, Published published)
{
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    const int lane = (int)(threadIdx.x & 31u);
    const int k = lane & 7;   // slot of this lane
    const int g = lane >> 3;  // group (node) of this lane
    const int gs = lane & ~7; // first lane of the group
    auto gballot = [&](bool pr) -> uint32_t { return (__ballot_sync(FULL, pr) >> gs) & 0xFFu; };
    const bool owns = active;
    Node self;
    uint32_t c0 = 0, cn = 0;
    if (active) {
        self = rec[rec_i];
        c0 = self.child;
        cn = node_count(self.count_flags);
        if (cn > 8) {
            if (k == 0) raise_error(err, SQ_DEVERR_NODE_COUNT);
            active = false;
        }
    }
    // slot state of this lane
    Node e_node;
    e_node.child = 0;
    e_node.count_flags = 0;
    uint32_t e_rec = 0, e_kind = 0, e_cnt = 0;
    float e_sa = 0.0f;
    auto load_entry = [&](uint32_t i) {
        e_node = rec[i];
        e_rec = i;
        e_sa = node_sa(e_node);
        e_cnt = node_count(e_node.count_flags);
        if (node_is_leaf(e_node.count_flags)) e_kind = 2;
        else e_kind = (e_node.child < leaf0 && e_cnt > 0) ? 0u : 1u;
        // the records an opening of this entry would load, towards L2 now:
        // the collapse is a chain of dependent record loads
        if (e_kind != 2 && e_cnt > 0) asm volatile("prefetch.global.L2 [%0];" ::"l"(rec + e_node.child));
    };
    if (active && k < (int)cn) load_entry(c0 + (uint32_t)k);
    // the start set is a binary record's two children or a cluster's leaves;
    // open the child of largest area (a binary record into its two children,
    // a leaf cluster into its single-triangle leaves) while it fits in 8 slots
    int nc = active ? (int)cn : 0;
    bool opening = active;
    for (;;) {
        const bool can = opening && k < nc &&
                         (e_kind == 0 ? (nc + 1 <= 8) : (e_kind == 1 && nc + (int)e_cnt - 1 <= 8));
        const uint32_t canm = gballot(can);
        opening = opening && canm != 0;
        if (!__any_sync(FULL, opening)) break;
        int best = -1;
        float bsa = 0.0f;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const float sq = __shfl_sync(FULL, e_sa, q, 8);
            if (((canm >> q) & 1u) && (best < 0 || sq > bsa)) { best = q; bsa = sq; }
        }
        const int bs = best < 0 ? 0 : best;
        const uint32_t bkind = __shfl_sync(FULL, e_kind, bs, 8), bcnt = __shfl_sync(FULL, e_cnt, bs, 8);
        const uint32_t bchild = __shfl_sync(FULL, e_node.child, bs, 8);
        const uint32_t m = bkind == 0 ? 2u : bcnt;
        const bool drop = opening && m == 0;
        if (__any_sync(FULL, drop)) {
            // drop the empty cluster: the group's last slot moves into its place
            const int src = nc > 0 ? nc - 1 : 0;
            Node t;
            t.mnx = __shfl_sync(FULL, e_node.mnx, src, 8); t.mny = __shfl_sync(FULL, e_node.mny, src, 8);
            t.mnz = __shfl_sync(FULL, e_node.mnz, src, 8);
            t.count_flags = __shfl_sync(FULL, e_node.count_flags, src, 8);
            t.mxx = __shfl_sync(FULL, e_node.mxx, src, 8); t.mxy = __shfl_sync(FULL, e_node.mxy, src, 8);
            t.mxz = __shfl_sync(FULL, e_node.mxz, src, 8); t.child = __shfl_sync(FULL, e_node.child, src, 8);
            const uint32_t trec = __shfl_sync(FULL, e_rec, src, 8), tkind = __shfl_sync(FULL, e_kind, src, 8);
            const uint32_t tcnt = __shfl_sync(FULL, e_cnt, src, 8);
            const float tsa = __shfl_sync(FULL, e_sa, src, 8);
            if (drop) {
                if (k == best) { e_node = t; e_rec = trec; e_kind = tkind; e_cnt = tcnt; e_sa = tsa; }
                --nc;
            }
        }
        if (opening && m != 0) {
            if (k == best) load_entry(bchild);
            else if (k >= nc && k < nc + (int)m - 1) load_entry(bchild + 1u + (uint32_t)(k - nc));
            nc += (int)m - 1;
        }
    }
    // a cluster of 2..8 triangles that did not fit becomes a wide child node
    // of its own (its triangles one per slot), so every triangle keeps its own
    // box; larger clusters stay leaf children of up to 15 triangles
    const bool own_node = k < nc && e_kind == 1 && e_cnt >= 2 && e_cnt <= 8;
    if (own_node) e_kind = 0;
    // children with an empty box (empty grid cells and subtrees of them) take
    // no slot
    const bool ok = k < nc && e_node.mnx <= e_node.mxx && e_node.mny <= e_node.mxy && e_node.mnz <= e_node.mxz;
    const bool inner = ok && e_kind == 0;
    const bool leafc = ok && e_kind != 0;
    if (gballot(leafc && e_cnt > 15u)) {
        if (active && k == 0) raise_error(err, SQ_DEVERR_NODE_COUNT);
        active = false;
    }
    // triangle slots: the leaf children's in the low half, the cluster
    // children's in the high half (at most 64 and 120)
    const uint32_t cntk = leafc ? e_cnt : 0u;
    const uint32_t both = cntk | (inner && own_node ? e_cnt << 16 : 0u);
    uint32_t imask = gballot(inner);
    uint32_t valid = gballot(ok);
    const uint32_t tmask = gballot(inner && !own_node);
    const uint32_t leafrec = gballot(k < nc && node_is_leaf(e_node.count_flags));
    uint32_t incl = both;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const uint32_t y = __shfl_up_sync(FULL, incl, o, 8);
        if (k >= o) incl += y;
    }
    const uint32_t all = __shfl_sync(FULL, incl, 7, 8);
    const uint32_t n_tris = all & 0xFFFFu;
    const uint32_t tri_off = (incl - both) & 0xFFFFu;
    // the warp's totals and this group's offsets (groups in lane order):
    // tasks and nodes (at most 32 each) in one word
    const uint32_t n_nt = active ? __popc(imask) | (__popc(tmask) << 16) : 0u;
    const uint32_t n_place = active ? n_tris + (all >> 16) : 0u;
    uint32_t pre_nt = 0, pre_t = 0, sum_nt = 0, sum_t = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const uint32_t a = __shfl_sync(FULL, n_nt, 8 * q), b = __shfl_sync(FULL, n_place, 8 * q);
        if (q < g) { pre_nt += a; pre_t += b; }
        sum_nt += a;
        sum_t += b;
    }
    uint32_t node_base = 0, tri_base = 0, task_base = 0;
    if (lane == 0 && (sum_nt | sum_t)) alloc(sum_nt & 0xFFFFu, sum_t, sum_nt >> 16, node_base, tri_base, task_base);
    const uint32_t child_base = __shfl_sync(FULL, node_base, 0) + (pre_nt & 0xFFFFu);
    tri_base = __shfl_sync(FULL, tri_base, 0) + pre_t;
    task_base = __shfl_sync(FULL, task_base, 0) + (pre_nt >> 16);
    if (active && inner) {
        const uint32_t node = child_base + __popc(imask & ((1u << k) - 1u));
        if (!own_node) publish(task_base + __popc(tmask & ((1u << k) - 1u)), node, e_rec);
        else if (node < capacity)
            *placeholder_of(nodes8 + node) = make_uint4(e_rec, tri_base + n_tris + ((incl - both) >> 16), 0u, kPlaceholder);
    }
    published();
    if (imask && child_base + __popc(imask) > capacity) active = false;
    if (!active) imask = valid = 0;
    sm.off[g][k] = tri_off;
    sm.cnt[g][k] = active ? cntk : 0u;
    sm.child[g][k] = e_node.child;
    write_node8(owns, k, g, self, e_node, ok && active, imask, valid, child_base, tri_base, sm, nodes8 + node_i);
    if (active) {
        // leaf triangles, spread over the group: triangle t of the node
        // belongs to the leaf slot whose [off, off + cnt) holds it
        for (uint32_t t = (uint32_t)k; t < n_tris; t += 8u) {
            int q = 0;
#pragma unroll
            for (int r = 1; r < 8; ++r)
                if (sm.cnt[g][r] && sm.off[g][r] <= t) q = r;
            const uint32_t j = t - sm.off[g][q], qc = sm.child[g][q];
            // a leaf record is its own triangle; a cluster's are its leaves
            write_tri8(tris8 + 3ull * (tri_base + t), tris, ((leafrec >> q) & 1u) ? qc + j : rec[qc + j].child);
        }
    }
    __syncwarp();  // the staging area is reused by the warp's next nodes
}

// The cluster nodes, four per warp: lane k of a group has the cluster's
// triangle k, its box from its leaf record.  One pass over the node array
// (80 B a node read or written, the leaf records and the triangles gathered):
// bound by those gathers.  A placeholder is taken only where its record and
// its triangle slots are inside the arrays (ntris triangles, leaf records from
// leaf0 on): where the collapse ran out of room, the last counted nodes were
// written by nothing.  A collapse that gave up (a barrier wait that ran out,
// too many levels) left no count: its trees become empty roots, so that a
// trace before the error is seen, as in a batch, reads nothing else.
__global__ void __launch_bounds__(256) k_collapse_clusters(const Node* __restrict__ rec, uint32_t leaf0,
                                                           const float* __restrict__ tris, uint32_t ntris,
                                                           const uint32_t* __restrict__ count, uint32_t nroots,
                                                           uint32_t* __restrict__ meta, Node8* __restrict__ nodes8,
                                                           float4* __restrict__ tris8)
{
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    __shared__ GroupSmem s_group[8];
    GroupSmem& sm = s_group[threadIdx.x >> 5];
    const int lane = (int)(threadIdx.x & 31u), k = lane & 7, g = lane >> 3, gs = lane & ~7;
    const uint32_t n = *count;
    if (n == 0) {
        for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < 5u * nroots; i += gridDim.x * blockDim.x)
            reinterpret_cast<uint4*>(nodes8)[i] = make_uint4(0u, 0u, 0u, 0u);
        if (meta && blockIdx.x == 0 && threadIdx.x < 2) meta[threadIdx.x] = 1u;
        return;
    }
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t base = 4u * ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); base < n; base += 4u * warps) {
        const uint32_t i = base + (uint32_t)g;
        uint4 ph = make_uint4(0u, 0u, 0u, 0u);
        if (i < n) ph = *placeholder_of(nodes8 + i);
        const bool active = i < n && ph.w == kPlaceholder;
        if (!__any_sync(FULL, active)) continue;
        Node self, child;
        bool ok = false;
        uint32_t id = 0;
        if (active && ph.x < leaf0) {
            self = rec[ph.x];
            const uint32_t c = node_count(self.count_flags);
            if (k < (int)c && c <= 8u && self.child >= leaf0 && (uint64_t)self.child + c <= (uint64_t)leaf0 + ntris &&
                (uint64_t)ph.y + c <= ntris) {
                child = rec[self.child + (uint32_t)k];
                id = child.child;
                ok = id < ntris && child.mnx <= child.mxx && child.mny <= child.mxy && child.mnz <= child.mxz;
            }
        }
        const uint32_t valid = (__ballot_sync(FULL, ok) >> gs) & 0xFFu;
        sm.cnt[g][k] = ok ? 1u : 0u;
        write_node8(active, k, g, self, child, ok, 0u, valid, 0u, ph.y, sm, nodes8 + i);
        if (ok) write_tri8(tris8 + 3ull * (ph.y + __popc(valid & ((1u << k) - 1u))), tris, id);
        __syncwarp();  // the staging area is reused by the warp's next nodes
    }
}

// Nodes and triangle slots of one warp from the counter pair at ctr (nodes
// after the roots in word 0, triangles in word 1: one 64-bit atomic).  On
// overflow of the node capacity the error word is set and the nodes land at
// `capacity`, where nothing is written.
__device__ __forceinline__ void alloc_nodes_tris(uint32_t* ctr, uint32_t kn, uint32_t kt, uint32_t nroots,
                                                 uint32_t capacity, uint32_t* err, uint32_t& nb, uint32_t& tb)
{
    const unsigned long long v =
        atomicAdd(reinterpret_cast<unsigned long long*>(ctr), ((unsigned long long)kt << 32) | kn);
    nb = (uint32_t)v + nroots;
    tb = (uint32_t)(v >> 32);
    if ((unsigned long long)nb + kn > capacity) {
        raise_error(err, SQ_DEVERR_SAH_QUEUE);
        nb = capacity;
    }
}

// Workspace words: the counters, then two task lists (record and node of
// each task), `capacity` words a list half.
struct CollapseWs {
    uint32_t* head;  // see the indices below
    uint32_t *rec[2], *node[2];
};
constexpr uint32_t kMaxLevels = 64;
// Words that atomics go to and words that are stored stand on lines of their
// own: with the level's cluster mark stored beside the counters the collapse
// of the 2M soup took 858 us instead of 215.
constexpr uint32_t kWsNodes = 0;               // a 64-bit pair: nodes beyond the roots, triangle slots
constexpr uint32_t kWsBarrier = 32;            // arrivals at the level barriers
constexpr uint32_t kWsCount = 64;              // final node count, then the number of levels
constexpr uint32_t kWsClusters = 66;           // levels that the deepest cluster node makes
constexpr uint32_t kWsBefore = 67;             // nodes before the level
constexpr uint32_t kWsOpen = 96;               // a 64-bit word: tasks of the level opened last, its number above
constexpr uint32_t kWsLevel = 128;             // tasks of level l at kWsLevel + l
constexpr uint32_t kWsHead = kWsLevel + kMaxLevels + 32;

__host__ __device__ inline CollapseWs collapse_ws(uint32_t* ws, uint32_t capacity)
{
    CollapseWs w;
    w.head = ws;
    uint32_t* p = ws + kWsHead;
    for (int i = 0; i < 2; ++i) {
        w.rec[i] = p;
        w.node[i] = p + capacity;
        p += 2ull * capacity;
    }
    return w;
}

// The work of one task group of level `level`: allocation from the head's
// counters, open-record children to the next level's list.  Wide node r
// (r < nroots) is the tree of record root + r; the other nodes follow.
// next_count: the next level's task counter.
template <class Published>
__device__ __forceinline__ void collapse_task(const Node* __restrict__ rec, uint32_t leaf0,
                                              const float* __restrict__ tris, bool active, uint32_t rec_i,
                                              uint32_t node_i, uint32_t level, uint32_t* next_count, uint32_t nroots,
                                              const CollapseWs& w,
                                              Node8* __restrict__ nodes8, float4* __restrict__ tris8, uint32_t capacity,
                                              uint32_t* err, GroupSmem& sm, Published published)
{
    uint32_t* head = w.head;
    uint32_t *next_rec = w.rec[(level + 1) & 1], *next_node = w.node[(level + 1) & 1];
    auto alloc = [&](uint32_t kn, uint32_t kt, uint32_t kj, uint32_t& nb, uint32_t& tb, uint32_t& jb) {
        if (kj) jb = atomicAdd(next_count, kj);
        alloc_nodes_tris(head + kWsNodes, kn, kt, nroots, capacity, err, nb, tb);
    };
    // (a node past the capacity is listed too: its task is counted, and the
    // next level passes it over)
    auto publish = [&](uint32_t j, uint32_t node, uint32_t record) {
        if (j >= capacity) return;
        next_rec[j] = record;
        next_node[j] = node;
    };
    collapse_node_group(rec, leaf0, tris, active, rec_i, node_i, nodes8, tris8, capacity, err, sm, alloc, publish,
                        published);
}

// One level per launch (where a cooperative launch is not possible): group i
// (four per warp) takes task i of the level's list and so on in strides of the
// grid.  The task counts of four levels take turns, so the depth has no limit
// here.
constexpr int kCollapseBlock = 128;

__device__ __forceinline__ uint32_t* level_slot(uint32_t* head, uint32_t level) { return head + kWsLevel + (level & 3u); }

__global__ void __launch_bounds__(kCollapseBlock) k_collapse_level(
    const Node* __restrict__ rec, uint32_t leaf0, const float* __restrict__ tris, uint32_t root, uint32_t nroots,
    uint32_t level, CollapseWs w, uint32_t capacity, Node8* __restrict__ nodes8, float4* __restrict__ tris8, uint32_t* err)
{
    __shared__ GroupSmem s_group[kCollapseBlock / 32];
    const uint32_t ntasks = level ? min(*level_slot(w.head, level), capacity) : nroots;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t base = 4u * ((blockIdx.x * blockDim.x + threadIdx.x) >> 5); base < ntasks; base += 4u * warps) {
        const uint32_t i = base + ((threadIdx.x & 31u) >> 3);
        const bool listed = i < ntasks;
        const uint32_t rec_i = !listed ? 0u : (level ? w.rec[level & 1][i] : root + i);
        const uint32_t node_i = !listed ? 0u : (level ? w.node[level & 1][i] : i);
        const bool active = listed && node_i < capacity;
        collapse_task(rec, leaf0, tris, active, rec_i, node_i, level, level_slot(w.head, level + 1u), nroots, w, nodes8,
                      tris8, capacity, err, s_group[threadIdx.x >> 5], [] {});
    }
}

// After level `level`, before anything of the next one: a level that made
// more nodes than tasks made cluster nodes, one level below its own.  Returns
// the next level's tasks.  (Relaxed loads, so they are in flight together: the
// caller has ordered them after the level's atomics.)
__device__ __forceinline__ uint32_t collapse_level_end(uint32_t* head, uint32_t level, const uint32_t* next_count)
{
    const uint32_t nodes = ld_relaxed_u32(head + kWsNodes), tasks = ld_relaxed_u32(next_count);
    const uint32_t before = ld_relaxed_u32(head + kWsBefore);
    if (nodes - before > tasks) st_relaxed_u32(head + kWsClusters, level + 2u);
    st_relaxed_u32(head + kWsBefore, nodes);
    return tasks;
}

// The final counts: nodes, and levels (levels of tasks, or one more where the
// deepest nodes are clusters).
__device__ __forceinline__ void collapse_done(uint32_t* head, uint32_t levels, uint32_t nroots, uint32_t capacity,
                                              uint32_t* meta)
{
    const uint32_t nodes = ld_acquire_u32(head + kWsNodes) + nroots, deep = ld_acquire_u32(head + kWsClusters);
    head[kWsCount] = nodes < capacity ? nodes : capacity;
    head[kWsCount + 1] = deep > levels ? deep : levels;
    if (meta) {
        meta[0] = head[kWsCount];
        meta[1] = head[kWsCount + 1];
    }
}

__global__ void k_collapse_level_end(CollapseWs w, uint32_t level)
{
    collapse_level_end(w.head, level, level_slot(w.head, level + 1u));
    *level_slot(w.head, level) = 0;
}

// (tasks left after the last level that was launched: no count, so the trees
// are empty)
__global__ void k_collapse_done(CollapseWs w, uint32_t levels, uint32_t nroots, uint32_t capacity, uint32_t* err)
{
    if (*level_slot(w.head, levels)) raise_error(err, SQ_DEVERR_SAH_QUEUE);
    else collapse_done(w.head, levels, nroots, capacity, nullptr);
}

// All levels in one cooperative launch (every block is resident): a
// grid-stride loop over a level's tasks, a grid barrier, the next level.  No
// host round trip per level, and a CUDA graph can hold it.  The barrier's
// wait is bounded (barrier_wait): a block that gives up raises
// SQ_DEVERR_SAH_QUEUE and returns (the other blocks then give up at their next
// barrier too).  Task lists are read through L2 (__ldcg): the same lists are
// rewritten every other level, so an SM's L1 may hold stale lines of them.
// The failure-detection tests pass one phantom block (barrier_extra = 1) that
// never arrives: every block then gives up at the first barrier.
//
// The bound is half a second of polling, which no level of 2^27 triangles comes
// near (8 million take less than a millisecond in all); polls alone are not
// counted, since how long one takes depends on what else the GPU does (2^24 of
// them, at a sleep and an L2 round trip each, are ten seconds or more).  A poll
// adds at most 0.1 ms, so the time that the kernel is not on the GPU at all
// does not count.
struct BarrierLimit {
    uint32_t polls, ns;  // polls before the time starts, and the time
};
constexpr BarrierLimit kBarrierLimit = {1u << 10, 500000000u};
constexpr uint32_t kBarrierPollNs = 100000u;

// Grid barrier of a level in two halves.  barrier_arrive: every warp calls it
// once, when its writes before the barrier are done; the block's last warp
// arrives for the block, and the grid's last block (arrivals are counted from
// the first level on: `target` of them) runs on_last(), with every write of
// before the barrier visible to it, and opens the next level.  barrier_wait:
// the block waits (thread 0 polls), and every thread gets the next level's
// tasks, which are in the polled word; false when the wait gave up.  s_warps:
// a shared counter, zero before the first use.  Each access that depends on
// one before it is an L2 round trip, most of a thin level's time: the count
// reset and the tasks read after the wait took two to three more (2M soup 12 us
// over 12 levels, 1,280 triangles 3 us over four).
template <class OnLast>
__device__ __forceinline__ void barrier_arrive(uint32_t* arrivals, uint32_t target, uint32_t* s_warps, OnLast on_last)
{
    __syncwarp();
    if ((threadIdx.x & 31u) != 0) return;
    __threadfence();
    if (atomicAdd(s_warps, 1u) + 1u != (blockDim.x >> 5)) return;
    __threadfence();
    *s_warps = 0;  // every warp of the block has counted; the next use is after barrier_wait's block barrier
    if (atomicAdd(arrivals, 1u) + 1u == target) {
        __threadfence();
        on_last();
    }
}

__device__ __forceinline__ void open_level(uint32_t* head, uint32_t level, uint32_t tasks)
{
    asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(head + kWsOpen),
                 "l"(((unsigned long long)level << 32) | tasks)
                 : "memory");
}

// Low word of the GPU's nanosecond clock (differences of up to four seconds).
__device__ __forceinline__ uint32_t global_ns()
{
    uint32_t t;
    asm volatile("mov.u32 %0, %%globaltimer_lo;" : "=r"(t));
    return t;
}

__device__ __forceinline__ bool barrier_wait(const uint32_t* head, uint32_t level, BarrierLimit limit, uint32_t* err,
                                             uint32_t& tasks)
{
    __shared__ uint32_t s_ok, s_tasks;
    if (threadIdx.x == 0) {
        uint32_t ok = 1, polls = 0, waited = 0, last = 0;
        unsigned long long v;
        for (;;) {
            asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(head + kWsOpen) : "memory");
            if ((uint32_t)(v >> 32) == level) break;
            if (++polls > limit.polls) {
                const uint32_t now = global_ns();
                if (polls > limit.polls + 1u) waited += min(now - last, kBarrierPollNs);
                last = now;
                if (waited >= limit.ns) {
                    raise_error(err, SQ_DEVERR_SAH_QUEUE);
                    ok = 0;
                    break;
                }
            }
            __nanosleep(32);
        }
        s_ok = ok;
        s_tasks = (uint32_t)v;
    }
    __syncthreads();
    const bool ok = s_ok != 0;
    tasks = s_tasks;
    __syncthreads();  // read by every thread before the next wait writes them
    return ok;
}

// A warp arrives at a level's barrier as soon as its last task's children are
// published and writes that task's node and triangles while it waits: a thin
// level (the top and the bottom of the tree, most levels) is a chain of
// dependent loads, and what the next level does not need is off it.
__global__ void __launch_bounds__(256) k_collapse_coop(const Node* __restrict__ rec, uint32_t leaf0,
                                                       const float* __restrict__ tris, uint32_t root, uint32_t nroots,
                                                       CollapseWs w, uint32_t capacity, Node8* __restrict__ nodes8,
                                                       float4* __restrict__ tris8, uint32_t* meta, uint32_t* err,
                                                       uint32_t barrier_extra, BarrierLimit limit)
{
    __shared__ GroupSmem s_group[8];
    __shared__ uint32_t s_warps;
    if (threadIdx.x == 0) s_warps = 0;
    __syncthreads();
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t wid = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    uint32_t ntasks = nroots;
    // (an overflow of the node capacity has raised the error word; the lists
    // hold no more than `capacity` tasks)
    for (uint32_t level = 0; ntasks; ++level, ntasks = min(ntasks, capacity)) {
        if (level + 1 >= kMaxLevels) {
            if (blockIdx.x == 0 && threadIdx.x == 0) raise_error(err, SQ_DEVERR_SAH_QUEUE);
            return;
        }
        uint32_t* next_count = w.head + kWsLevel + level + 1u;
        auto arrive = [&] {
            barrier_arrive(w.head + kWsBarrier, (gridDim.x + barrier_extra) * (level + 1u), &s_warps,
                           [&] { open_level(w.head, level + 1u, collapse_level_end(w.head, level, next_count)); });
        };
        if (4u * wid >= ntasks) arrive();
        for (uint32_t base = 4u * wid; base < ntasks; base += 4u * warps) {
            const uint32_t i = base + ((threadIdx.x & 31u) >> 3);
            const bool listed = i < ntasks;
            const uint32_t rec_i = !listed ? 0u : (level ? __ldcg(w.rec[level & 1] + i) : root + i);
            const uint32_t node_i = !listed ? 0u : (level ? __ldcg(w.node[level & 1] + i) : i);
            const bool active = listed && node_i < capacity;
            const bool last = ntasks - base <= 4u * warps;
            collapse_task(rec, leaf0, tris, active, rec_i, node_i, level, next_count, nroots, w, nodes8, tris8, capacity,
                          err, s_group[threadIdx.x >> 5], [&] { if (last) arrive(); });
        }
        if (!barrier_wait(w.head, level + 1u, limit, err, ntasks)) return;
        if (!ntasks && blockIdx.x == 0 && threadIdx.x == 0) collapse_done(w.head, level + 1, nroots, capacity, meta);
    }
}

}  // namespace

namespace sqk {

// A wide node has at least two children except the root and nodes next to
// empty grid cells (at most 64 of those), so n + 130 nodes beside the roots
// always suffice.
uint32_t bvh8_capacity(uint32_t n) { return n + 130u; }
size_t bvh8_node_bytes(uint32_t n, uint32_t nroots) { return sizeof(Node8) * ((size_t)bvh8_capacity(n) + nroots); }
size_t bvh8_ws_words(uint32_t n, uint32_t nroots) { return 4ull * (bvh8_capacity(n) + nroots) + kWsHead; }
size_t bvh8_tri_bytes(uint32_t n) { return sizeof(float4) * 3ull * ((size_t)n + 1); }

// Blocks per SM of the cooperative collapse: every block must be resident
// (0: no cooperative launch on this device).
static int coop_blocks()
{
    static PerDevice<int> cache;
    return cache.get([] {
        int coop = 0, occ = 0;
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, current_device());
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_collapse_coop, 256, 0);
        return (coop && occ > 0) ? occ : 0;
    });
}

static cudaError_t launch_clusters(const Node* rec, uint32_t leaf0, const float* tris, uint32_t n, const CollapseWs& w,
                                   uint32_t nroots, uint32_t* meta, void* nodes8, void* tris8, cudaStream_t s)
{
    static PerDevice<int> cache;
    const int grid = cache.get([] { return blocks_per_sm(k_collapse_clusters, 256) * sm_count(); });
    k_collapse_clusters<<<grid, 256, 0, s>>>(rec, leaf0, tris, n, w.head + kWsCount, nroots, meta,
                                             static_cast<Node8*>(nodes8), static_cast<float4*>(tris8));
    return cudaGetLastError();
}

// The collapse as one kernel launch per level of tasks (the host reads each
// level's task count), where a cooperative launch does not fit (by_level: the
// tests ask for it).  The node count is host_ctl[0] and the number of levels
// host_ctl[3].
static int build_bvh8_levels(const Node* rec, uint32_t root, uint32_t leaf0, const float* tris, uint32_t n,
                             void* nodes8, void* tris8, const CollapseWs& w, uint32_t* host_ctl, uint32_t* err,
                             cudaStream_t s)
{
    const uint32_t capacity = bvh8_capacity(n) + 1u;
    cudaError_t e;
    uint32_t ntasks = 1, level = 0;
    for (; ntasks; ++level) {
        k_collapse_level<<<(ntasks + 15) / 16, kCollapseBlock, 0, s>>>(rec, leaf0, tris, root, 1u, level, w, capacity,
                                                               static_cast<Node8*>(nodes8), static_cast<float4*>(tris8),
                                                               err);
        k_collapse_level_end<<<1, 1, 0, s>>>(w, level);
        if ((e = cudaMemcpyAsync(host_ctl, w.head + kWsLevel + ((level + 1u) & 3u), 4, cudaMemcpyDeviceToHost, s)) !=
            cudaSuccess)
            return (int)e;
        if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return (int)e;
        ntasks = std::min(host_ctl[0], capacity);
    }
    k_collapse_done<<<1, 1, 0, s>>>(w, level, 1u, capacity, err);
    if ((e = launch_clusters(rec, leaf0, tris, n, w, 1u, nullptr, nodes8, tris8, s)) != cudaSuccess) return (int)e;
    uint32_t m[2];
    if ((e = cudaMemcpyAsync(m, w.head + kWsCount, sizeof m, cudaMemcpyDeviceToHost, s)) != cudaSuccess) return (int)e;
    if ((e = cudaStreamSynchronize(s)) != cudaSuccess) return (int)e;
    host_ctl[0] = m[0];
    host_ctl[3] = m[1];
    host_ctl[4] = 2 * level + 2;  // launches
    return (int)cudaGetLastError();
}

// The cooperative collapse and the cluster pass of the trees of records
// root .. root + nroots - 1 over n triangles: nothing waits on the host, so a
// CUDA graph can hold it.  meta (device, 2 words, may be null): node and level
// counts.
static cudaError_t enqueue_collapse(const Node* rec, uint32_t root, uint32_t nroots, uint32_t leaf0, const float* tris,
                                    uint32_t n, void* nodes8, void* tris8, uint32_t* ws, uint32_t* meta, uint32_t* err,
                                    int per_sm, const BarrierStall* stall, cudaStream_t s)
{
    uint32_t capacity = bvh8_capacity(n) + nroots;
    CollapseWs w = collapse_ws(ws, capacity);
    const uint32_t extra = stall ? 1u : 0u;
    const BarrierLimit limit = stall && stall->spin_limit ? BarrierLimit{stall->spin_limit, 0u} : kBarrierLimit;
    void* args[] = {(void*)&rec, (void*)&leaf0, (void*)&tris, (void*)&root, (void*)&nroots, (void*)&w, (void*)&capacity,
                    (void*)&nodes8, (void*)&tris8, (void*)&meta, (void*)&err, (void*)&extra, (void*)&limit};
    const cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_collapse_coop, dim3(per_sm * sm_count()), dim3(256),
                                                      args, 0, s);
    if (e != cudaSuccess) return e;
    return launch_clusters(rec, leaf0, tris, n, w, nroots, meta, nodes8, tris8, s);
}

int build_bvh8_queue(const Node* rec, uint32_t root0, uint32_t nroots, uint32_t leaf0, const float* tris, uint32_t n,
                     void* nodes8, void* tris8, uint32_t* ws, uint32_t* err, cudaStream_t s, bool by_level)
{
    const int per_sm = by_level ? 0 : coop_blocks();
    cudaError_t e;
    if ((e = cudaMemsetAsync(ws, 0, sizeof(uint32_t) * kWsHead, s)) != cudaSuccess) return (int)e;
    if (per_sm == 0) {
        // a fixed number of levels, as many as the cooperative kernel takes:
        // a level without tasks returns at once
        static PerDevice<int> cache;
        const int grid = cache.get([] { return blocks_per_sm(k_collapse_level, kCollapseBlock) * sm_count(); });
        const uint32_t capacity = bvh8_capacity(n) + nroots;
        const CollapseWs w = collapse_ws(ws, capacity);
        for (uint32_t level = 0; level + 1 < kMaxLevels; ++level) {
            k_collapse_level<<<grid, kCollapseBlock, 0, s>>>(rec, leaf0, tris, root0, nroots, level, w, capacity,
                                                             static_cast<Node8*>(nodes8), static_cast<float4*>(tris8),
                                                             err);
            k_collapse_level_end<<<1, 1, 0, s>>>(w, level);
        }
        k_collapse_done<<<1, 1, 0, s>>>(w, kMaxLevels - 1, nroots, capacity, err);
        return (int)launch_clusters(rec, leaf0, tris, n, w, nroots, nullptr, nodes8, tris8, s);
    }
    return (int)enqueue_collapse(rec, root0, nroots, leaf0, tris, n, nodes8, tris8, ws, nullptr, err, per_sm, nullptr, s);
}

int build_bvh8(const Node* rec, uint32_t root, uint32_t leaf0, const float* tris, uint32_t n, void* nodes8, void* tris8,
               uint32_t* ws, uint32_t* host_ctl, uint32_t* err, cudaStream_t s, uint32_t* meta,
               const BarrierStall* stall, bool by_level)
{
    host_ctl[5] = 0;
    cudaError_t e;
    if ((e = cudaMemsetAsync(ws, 0, sizeof(uint32_t) * kWsHead, s)) != cudaSuccess) return (int)e;
    const int per_sm = by_level ? 0 : coop_blocks();
    if (per_sm == 0)
        return build_bvh8_levels(rec, root, leaf0, tris, n, nodes8, tris8, collapse_ws(ws, bvh8_capacity(n) + 1u),
                                 host_ctl, err, s);
    if ((e = enqueue_collapse(rec, root, 1u, leaf0, tris, n, nodes8, tris8, ws, meta, err, per_sm, stall, s)) !=
        cudaSuccess)
        return (int)e;
    host_ctl[4] = 2;  // the cooperative kernel and the cluster pass
    host_ctl[5] = 1;  // node count and levels stay in meta until asked for
    return 0;
}

}  // namespace sqk
