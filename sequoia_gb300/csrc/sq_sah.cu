// sq_sah.cu -- binned SAH and grid BVH builders on the GPU.
//
// Same logical tree as the reference's binned SAH build (recurse /
// recurse_omp / build_hierarchy, src/builder.cpp:1053-1156, 1365-1477,
// 1576-1618) and grid build (src/builder.cpp:1665-1753, 2133-2194), with the
// bin count and leaf size as parameters:
//   leaf        count <= leaf_size, or centroid box area <= 0
//   axis        choose_axis (src/builder.cpp:334-345)
//   bins        bin = int(k1 * (c[axis] - cmin)), k1 = bins*(1-2^-23)/extent
//               (src/builder.cpp:372-398)
//   plane       left-to-right unions, right-to-left sweep, score
//               sa(L)*nL + sa(R)*nR, strict <, ties to the higher plane
//               (src/builder.cpp:488-523)
//   partition   bin <= plane goes left.  The reference swaps in place
//               (src/builder.cpp:599-628); this builder partitions stably.
//               Both yield the same two sets, so the same tree.
//   children    their primitive and centroid boxes come from the bins.
// Records are written in the range-tree layout (oracle/sq_oracle.c), so the
// result is record-for-record the oracle's.
//
// Schedule:
//   large nodes (> kMid triangles): level by level, two kernels a level.
//     k_large_split  one warp per node picks the plane from the node's bins,
//                    places the children and scans the left counts of the
//                    node's chunks;
//     k_large_move   one block per chunk (256 or 2048 triangles, by mesh
//                    size) moves the chunk's triangles to their side, stably,
//                    and bins each one for the child that it goes to, so the
//                    next level's split finds its bins ready.
//     A triangle's box is read once a level: the bin it falls in is kept as a
//     byte beside its id, and the next partition needs only that byte.
//   middle nodes (> kSmall, at most kMid triangles): one block per subtree, in
//     shared memory, down to the small nodes.
//   small nodes: one warp per subtree, smaller child first (stack depth
//     O(log n)), binning and partitioning with warp intrinsics only.
#include "sq_common.cuh"
#include "sq_lbvh_dev.cuh"

#include <type_traits>
#include <utility>

namespace {

using namespace sq;

// Triangles per chunk of a large level: 2048 from 1M triangles up, 256 below
// (a small mesh then still spreads a level over many blocks; each thread
// handles one triangle of a chunk instead of eight dependent ones).
constexpr uint32_t kChunk = 2048;
constexpr uint32_t kChunkSmall = 256;
constexpr uint32_t kChunkSmallBelow = 1u << 20;
constexpr uint32_t kSmall = 128;
constexpr uint32_t kMid = 1024;
constexpr int kMaxBins = 32;
constexpr int kBinWords = 13;  // -pmin xyz, pmax xyz, -cmin xyz, cmax xyz (ordered ints), count
constexpr int kStackDepth = 24;
// Large-phase levels of the batched build (device-side counts, no host
// round trip): larger tasks left then are finished by k_small_big.
constexpr uint32_t kBatchLargeLevels = 20;
// Large-phase levels a single build queues between two host reads of the
// task count, after a first group sized to the mesh (build_sah).
constexpr uint32_t kSahLevelsPerCheck = 4;
constexpr uint32_t kNone = 0xFFFFFFFFu;

struct __align__(16) Task {
    uint32_t begin, count, slot, flags;  // flags: bit0 = ids live in buffer B, bit1 = root-like record
    float pmn[3], pmx[3], cmn[3], cmx[3];
};
static_assert(sizeof(Task) == 64, "Task is 64 bytes");

struct LeafRange {
    uint32_t begin, count, slot, flags;
    float pmn[3], pmx[3];
    uint32_t pad[2];
};
static_assert(sizeof(LeafRange) == 48, "LeafRange is 48 bytes");

// What k_large_move needs to move one task's chunks: the task's own range
// and plane (a bin at or below it goes left; -1: the task became a leaf and
// its triangles stay), and for each side that is a large task the bins and
// chunks it collects into and how it bins.
struct __align__(16) Part {
    uint32_t begin, count, nl, chunk0;
    int plane;
    uint32_t flags;  // bit 0: ids in buffer B; bit 1: several chunks
    int axis[2];     // binning axis of the large children
    uint32_t task[2], child_chunk0[2];  // kNone: the side is not a large task
    float k1[2], cmin[2];
};
static_assert(sizeof(Part) == 64, "Part is 64 bytes");

// Task counts.  level[l % 3] holds the tasks (low word) and chunks (high
// word) of level l: k_large_split of level l reads it and adds its large
// children to level[(l + 1) % 3]; k_large_move of level l, which runs while
// neither is needed, clears level[(l + 2) % 3].  The kernels read the counts
// on the device, so a level needs no host round trip.
struct Ctl {
    unsigned long long level[3];
    uint32_t n_mid, n_small, n_leaf;
    uint32_t mid_pop, small_pop;  // tasks taken by k_mid's blocks and k_small's warps
    uint32_t odd;                 // a triangle with a NaN bound is among them (encode_boxes)
};
static_assert(sizeof(Ctl) == 48, "Ctl is 48 bytes");

__device__ __forceinline__ float box_sa(const float* mn, const float* mx)
{
    const float lx = mx[0] - mn[0], ly = mx[1] - mn[1], lz = mx[2] - mn[2];
    const float xy = lx * ly, xz = lx * lz, yz = ly * lz;
    float s = xy + xz;
    s = s + yz;
    return s * 2.0f;
}

__device__ __forceinline__ int choose_axis(const float* mn, const float* mx)
{
    const float lx = mx[0] - mn[0], ly = mx[1] - mn[1], lz = mx[2] - mn[2];
    int r = 0;
    r += 2 * (lz > lx && lz > ly);
    r += 1 * (ly > lx && ly >= lz);
    return r;
}

__device__ __forceinline__ float bin_k1(int nb, float ext)
{
    const float eps = 1.1920929e-7f;
    const float one_minus = 1.0f - eps;
    const float num = (float)nb * one_minus;
    return num / ext;
}

__device__ __forceinline__ int bin_of(float k1, float c, float cmin, int nb)
{
    const float d = c - cmin;
    const float x = k1 * d;
    int b = (x == x) ? (int)x : 0;  // cvt.rzi saturates; NaN -> 0
    b = b < 0 ? 0 : b;
    return b > nb - 1 ? nb - 1 : b;
}

__device__ __forceinline__ void load_box(const float4* __restrict__ tb, uint32_t id, float* mn, float* mx)
{
    const float4 a = __ldg(tb + 2ull * id), b = __ldg(tb + 2ull * id + 1);
    mn[0] = a.x; mn[1] = a.y; mn[2] = a.z;
    mx[0] = b.x; mx[1] = b.y; mx[2] = b.z;
}

__device__ __forceinline__ float sel(const float* v, int k) { return k == 0 ? v[0] : (k == 1 ? v[1] : v[2]); }

// The twelve words of a triangle in a bin: order-preserving integers of
// (-pmin, pmax, -cmin, cmax), so that a bin is their maxima.  A NaN bound is
// passed over, as in the reference's comparisons (src/vec3.h:179-180): it gives
// 0, below every number.  (float_to_ordered of a NaN is whatever the compiler
// makes of its sign operations.)  ODD: look for one.  The setup kernels leave
// in Ctl::odd whether the build has any, and the binning kernels are compiled
// both ways: a look for each triangle, or at the flag, took 3% of k_small and
// 8% of k_large_move.
template <bool ODD>
__device__ __forceinline__ void encode_boxes(const float* mn, const float* mx, const float* c, uint32_t* e)
{
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        e[a] = float_to_ordered(-mn[a]);
        e[3 + a] = float_to_ordered(mx[a]);
        e[6 + a] = float_to_ordered(-c[a]);
        e[9 + a] = float_to_ordered(c[a]);
    }
    if (ODD) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            if (isnan(mn[a])) e[a] = 0u;
            if (isnan(mx[a])) e[3 + a] = 0u;
            if (isnan(c[a])) e[6 + a] = e[9 + a] = 0u;
        }
    }
}

// A triangle with a NaN bound has a NaN centroid.  (Infinities of both signs
// only cost the look.)
__device__ __forceinline__ bool odd_box(const float* c)
{
    const float sum = (c[0] + c[1]) + c[2];
    return sum != sum;
}

// ---------------------------------------------------------------------------
// setup: triangle boxes, identity ids, root boxes

__global__ void __launch_bounds__(256) k_sah_setup(const float* __restrict__ tris, uint32_t n, float4* __restrict__ tb,
                                                   uint32_t* __restrict__ ids, uint32_t* __restrict__ root_ord,
                                                   Ctl* __restrict__ ctl)
{
    float v[12];
    bool odd = false;
#pragma unroll
    for (int k = 0; k < 12; ++k) v[k] = -FLT_MAX;  // max of (-pmin, pmax, -cmin, cmax)
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float t[9];
        load_tri(tris, i, t);
        const Box b = tri_box(t);
        tb[2ull * i] = make_float4(b.mn[0], b.mn[1], b.mn[2], 0.0f);
        tb[2ull * i + 1] = make_float4(b.mx[0], b.mx[1], b.mx[2], 0.0f);
        ids[i] = i;
        float c[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            c[k] = (b.mn[k] + b.mx[k]) * 0.5f;
            v[k] = fmaxf(v[k], -b.mn[k]);
            v[3 + k] = fmaxf(v[3 + k], b.mx[k]);
            v[6 + k] = fmaxf(v[6 + k], -c[k]);
            v[9 + k] = fmaxf(v[9 + k], c[k]);
        }
        odd = odd || odd_box(c);
    }
    if (odd) ctl->odd = 1u;
#pragma unroll
    for (int k = 0; k < 12; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v[k] = fmaxf(v[k], __shfl_xor_sync(0xFFFFFFFFu, v[k], o));
    }
    __shared__ float s[8][12];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
        for (int k = 0; k < 12; ++k) s[warp][k] = v[k];
    __syncthreads();
    if (threadIdx.x < 12) {
        float m = s[0][threadIdx.x];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmaxf(m, s[w][threadIdx.x]);
        atomicMax(root_ord + threadIdx.x, float_to_ordered(m));
    }
}

// A bound from its word (0: no triangle had one, with NaN bounds only).
template <bool ODD = true>
__device__ __forceinline__ float dec_neg(uint32_t u) { return !ODD || u ? -ordered_to_float(u) : FLT_MAX; }
template <bool ODD = true>
__device__ __forceinline__ float dec_pos(uint32_t u) { return !ODD || u ? ordered_to_float(u) : -FLT_MAX; }

// Where the large tasks of one level are listed: the tasks, each task's
// first chunk, the task of each chunk, and the bins and per-chunk bin counts
// that k_large_move fills.
struct LevelLists {
    Task* tasks;
    uint32_t *chunk0, *chunk_task, *bins, *counts;
};

// 32-bit words of a chunk's bin counts (16 bits a bin: a chunk holds at most
// 2048 triangles)
__host__ __device__ __forceinline__ uint32_t count_words(int nb) { return ((uint32_t)nb + 1u) >> 1; }

// Where the other tasks go.
struct DoneLists {
    Task *mid, *small;
    LeafRange* leaves;
    Ctl* ctl;
};

__device__ __forceinline__ bool is_leaf_task(const Task& t, uint32_t leaf_size)
{
    return t.count <= leaf_size || !(box_sa(t.cmn, t.cmx) > 0.0f);
}

__device__ __forceinline__ void list_leaf(const Task& t, const DoneLists& done)
{
    LeafRange lr;
    lr.begin = t.begin; lr.count = t.count; lr.slot = t.slot; lr.flags = t.flags;
    for (int a = 0; a < 3; ++a) { lr.pmn[a] = t.pmn[a]; lr.pmx[a] = t.pmx[a]; }
    lr.pad[0] = lr.pad[1] = 0;
    done.leaves[atomicAdd(&done.ctl->n_leaf, 1u)] = lr;
}

// Place a task (all lanes of a warp call it with the same task): leaf
// (recorded in the leaf list), large (listed for the level counted by *cnt),
// middle or small.  side: which child of `part` it is, for the large case.  zero:
// the bins are collected with atomics and must start from zero (else one
// block stores them whole).
template <uint32_t CHUNK>
__device__ void place_task(const Task& t, uint32_t leaf_size, int nb, const LevelLists& next, unsigned long long* cnt,
                           bool zero, const DoneLists& done, Part& part, int side)
{
    const uint32_t lane = threadIdx.x & 31u;
    part.task[side] = kNone;
    if (is_leaf_task(t, leaf_size)) {
        if (lane == 0) list_leaf(t, done);
        return;
    }
    if (t.count <= kMid) {
        if (lane == 0) {
            if (t.count <= kSmall) done.small[atomicAdd(&done.ctl->n_small, 1u)] = t;
            else done.mid[atomicAdd(&done.ctl->n_mid, 1u)] = t;
        }
        return;
    }
    const uint32_t chunks = (t.count + CHUNK - 1) / CHUNK;
    unsigned long long at = 0;
    if (lane == 0) at = atomicAdd(cnt, ((unsigned long long)chunks << 32) | 1ull);
    at = __shfl_sync(0xFFFFFFFFu, at, 0);
    const uint32_t k = (uint32_t)at, c0 = (uint32_t)(at >> 32);
    if (lane == 0) {
        next.tasks[k] = t;
        next.chunk0[k] = c0;
    }
    for (uint32_t c = lane; c < chunks; c += 32) next.chunk_task[c0 + c] = k;
    if (zero) {
        uint32_t* b = next.bins + (size_t)k * kMaxBins * kBinWords;
        for (int j = lane; j < nb * kBinWords; j += 32) b[j] = 0;
        if (chunks > 1) {
            const uint32_t cw = count_words(nb);
            uint32_t* cc = next.counts + (size_t)c0 * cw;
            for (uint32_t j = lane; j < chunks * cw; j += 32) cc[j] = 0;
        }
    }
    part.task[side] = k;
    part.child_chunk0[side] = c0;
    part.axis[side] = choose_axis(t.cmn, t.cmx);
    part.cmin[side] = sel(t.cmn, part.axis[side]);
    part.k1[side] = bin_k1(nb, sel(t.cmx, part.axis[side]) - part.cmin[side]);
}

// A root task: placed, and where it is large its Part makes k_large_move
// bin it in place (everything on side 0).
template <uint32_t CHUNK>
__device__ void place_root(const Task& t, uint32_t leaf_size, int nb, const LevelLists& l0, Part* __restrict__ parts,
                           const DoneLists& done)
{
    Part p;
    place_task<CHUNK>(t, leaf_size, nb, l0, &done.ctl->level[0], true, done, p, 0);
    if (p.task[0] == kNone) return;
    p.begin = t.begin;
    p.count = p.nl = t.count;
    p.chunk0 = p.child_chunk0[0];
    p.plane = kMaxBins;
    p.flags = (t.flags & 1u) | 2u;
    p.axis[1] = 0;
    p.task[1] = kNone;
    p.child_chunk0[1] = 0;
    p.k1[1] = p.cmin[1] = 0.0f;
    if ((threadIdx.x & 31u) == 0) parts[p.task[0]] = p;
}

template <uint32_t CHUNK>
__global__ void k_root_task(const uint32_t* __restrict__ root_ord, uint32_t n, uint32_t leaf_size, int nb,
                            LevelLists l0, Part* parts, DoneLists done, float* scene_out)
{
    Task t;  // one warp
    t.begin = 0; t.count = n; t.slot = 0; t.flags = 2u;
    for (int k = 0; k < 3; ++k) {
        t.pmn[k] = dec_neg(root_ord[k]);
        t.pmx[k] = dec_pos(root_ord[3 + k]);
        t.cmn[k] = dec_neg(root_ord[6 + k]);
        t.cmx[k] = dec_pos(root_ord[9 + k]);
        if (threadIdx.x == 0) {
            scene_out[k] = t.pmn[k];
            scene_out[3 + k] = t.pmx[k];
        }
    }
    place_root<CHUNK>(t, leaf_size, nb, l0, parts, done);
}

// ---------------------------------------------------------------------------
// grid: cells, Morton order, cell tasks

// Morton slot of grid cell (x, y, z) in a 4x4x4 grid: bits x0 y0 z0 x1 y1 z1
// (the inverse of compact_1_by_2, src/builder.cpp:27-35, 1726-1728).
__device__ __forceinline__ uint32_t cell_slot(uint32_t x, uint32_t y, uint32_t z)
{
    return (x & 1u) | ((y & 1u) << 1) | ((z & 1u) << 2) | ((x & 2u) << 2) | ((y & 2u) << 3) | ((z & 2u) << 4);
}

__global__ void __launch_bounds__(256) k_grid_bin(const float4* __restrict__ tb, uint32_t n,
                                                  const uint32_t* __restrict__ root_ord, uint32_t* __restrict__ keys,
                                                  uint32_t* __restrict__ cell_ord, uint32_t* __restrict__ hist)
{
    __shared__ uint32_t s_cell[64 * kBinWords];
    for (int j = threadIdx.x; j < 64 * kBinWords; j += blockDim.x) s_cell[j] = 0;
    __syncthreads();
    float cmn[3], k1[3];
    for (int a = 0; a < 3; ++a) {
        cmn[a] = dec_neg(root_ord[6 + a]);
        const float cmx = dec_pos(root_ord[9 + a]);
        k1[a] = bin_k1(4, cmx - cmn[a]);
    }
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        float mn[3], mx[3], c[3];
        load_box(tb, i, mn, mx);
        uint32_t g[3];
        for (int a = 0; a < 3; ++a) {
            c[a] = (mn[a] + mx[a]) * 0.5f;
            g[a] = (uint32_t)bin_of(k1[a], c[a], cmn[a], 4);
        }
        const uint32_t m = cell_slot(g[0], g[1], g[2]);
        keys[i] = m;
        uint32_t* cb = s_cell + m * kBinWords;
        uint32_t e[12];
        encode_boxes<true>(mn, mx, c, e);
#pragma unroll
        for (int k = 0; k < 12; ++k) atomicMax(cb + k, e[k]);
        atomicAdd(cb + 12, 1u);
    }
    __syncthreads();
    for (int j = threadIdx.x; j < 64 * kBinWords; j += blockDim.x) {
        const uint32_t v = s_cell[j];
        if ((j % kBinWords) == 12) {
            if (v) { atomicAdd(cell_ord + j, v); atomicAdd(hist + j / kBinWords, v); }
        } else if (v) {
            atomicMax(cell_ord + j, v);
        }
    }
}

// One warp per cell, in Morton order; cell m covers [begin_m, begin_m +
// count_m), begin_m summed by the warp from the earlier cells' counts.
template <uint32_t CHUNK>
__global__ void k_grid_tasks(const uint32_t* __restrict__ cell_ord, const uint32_t* __restrict__ root_ord, uint32_t n,
                             uint32_t leaf_size, uint32_t scene_box_cells, int nb, LevelLists l0, Part* parts,
                             DoneLists done, float* scene_out)
{
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (m >= 64) return;
    if (m == 0 && lane == 0)
        for (int k = 0; k < 3; ++k) { scene_out[k] = dec_neg(root_ord[k]); scene_out[3 + k] = dec_pos(root_ord[3 + k]); }
    uint32_t before = lane < m ? cell_ord[lane * kBinWords + 12] : 0u;
    if (lane + 32u < m) before += cell_ord[(lane + 32u) * kBinWords + 12];
    const uint32_t* cb = cell_ord + m * kBinWords;
    Task t;
    t.begin = __reduce_add_sync(0xFFFFFFFFu, before);
    t.count = cb[12];
    t.slot = 63u + m;
    t.flags = 2u;
    for (int k = 0; k < 3; ++k) {
        if (t.count) {
            t.pmn[k] = dec_neg(cb[k]); t.pmx[k] = dec_pos(cb[3 + k]);
            t.cmn[k] = dec_neg(cb[6 + k]); t.cmx[k] = dec_pos(cb[9 + k]);
        } else {
            t.pmn[k] = FLT_MAX; t.pmx[k] = -FLT_MAX; t.cmn[k] = FLT_MAX; t.cmx[k] = -FLT_MAX;
        }
    }
    if (scene_box_cells) {
        // the plain grid builder gives every cell node the scene box (src/builder.cpp:2173-2174)
        for (int k = 0; k < 3; ++k) { t.pmn[k] = dec_neg(root_ord[k]); t.pmx[k] = dec_pos(root_ord[3 + k]); }
    }
    place_root<CHUNK>(t, leaf_size, nb, l0, parts, done);
}

// heap of 63 inner nodes above the 64 cell nodes (src/builder.cpp:2181-2188),
// a level at a time, one lane per node
__global__ void k_grid_heap(Node* __restrict__ nodes)
{
    for (uint32_t width = 32; width; width >>= 1) {
        if (threadIdx.x < width) {
            const uint32_t i = width - 1u + threadIdx.x;
            const Node a = nodes[2 * i + 1], b = nodes[2 * i + 2];
            Box u;
            u.mn[0] = ref_min(a.mnx, b.mnx); u.mn[1] = ref_min(a.mny, b.mny); u.mn[2] = ref_min(a.mnz, b.mnz);
            u.mx[0] = ref_max(a.mxx, b.mxx); u.mx[1] = ref_max(a.mxy, b.mxy); u.mx[2] = ref_max(a.mxz, b.mxz);
            store_node(nodes + i, u, 2u * i + 1u, 2u, 0);
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------------------
// warp-level binning and plane choice

// Merge one element per lane (bin = nb for inactive lanes) into warp bins.
__device__ __forceinline__ void warp_bin_add(uint32_t* __restrict__ wb, int bin, int nb, const float* mn, const float* mx,
                                             const float* c)
{
    const int lane = threadIdx.x & 31;
    uint32_t e[12];
    encode_boxes<true>(mn, mx, c, e);
    const int b0 = __shfl_sync(0xFFFFFFFFu, bin, 0);
    if (__all_sync(0xFFFFFFFFu, bin == b0)) {
        // the whole warp in one bin: full-warp reductions and one writer
        if (b0 < nb) {
#pragma unroll
            for (int k = 0; k < 12; ++k) e[k] = __reduce_max_sync(0xFFFFFFFFu, e[k]);
            if (lane == 0) {
                uint32_t* b = wb + b0 * kBinWords;
#pragma unroll
                for (int k = 0; k < 12; ++k) b[k] = max(b[k], e[k]);
                b[12] += 32u;
            }
        }
    } else if (bin < nb) {
        // lanes spread over bins: shared-memory atomics per lane (reductions
        // with per-bin masks would run once per distinct bin)
        uint32_t* b = wb + bin * kBinWords;
#pragma unroll
        for (int k = 0; k < 12; ++k) atomicMax(b + k, e[k]);
        atomicAdd(b + 12, 1u);
    }
    __syncwarp();
}

struct PlaneResult {
    int plane;  // -1 if none
    uint32_t nl;
    float lp[6], rp[6], lc[6], rc[6];  // min xyz, max xyz
};

__device__ __forceinline__ float redux_min(float v)
{
    float r;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float redux_max(float v)
{
    float r;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// choose_plane (src/builder.cpp:488-523) for 32 / NBP nodes at once: lane =
// (node g, bin b), `cnt` and the boxes p of the lane's bin (FLT_MAX boxes
// where it is empty or b >= nb), c its centroid box.  Every lane of a group
// returns its node's plane (-1: none), left count, and both sides' boxes.
// The primitive boxes are scanned from both ends; the centroid boxes are
// needed at the chosen plane alone and are reduced once it is known.
template <int NBP>
__device__ __forceinline__ void choose_planes(int nb, uint32_t cnt, const float* p, const float* c, int& plane,
                                              uint32_t& nl, float* lp, float* rp, float* lc, float* rc)
{
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    const int lane = threadIdx.x & 31, b = lane & (NBP - 1), g0 = lane - b;
    float l[6], s[6];
    uint32_t lcnt = cnt, scnt = cnt;
#pragma unroll
    for (int k = 0; k < 6; ++k) l[k] = s[k] = p[k];
    // below 32 bins an empty bin follows the last one: its FLT_MAX box is
    // part of every right side's union
    const bool cap = nb < kMaxBins && b == NBP - 1;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        if (cap) { s[k] = fminf(s[k], FLT_MAX); s[3 + k] = fmaxf(s[3 + k], -FLT_MAX); }
    }
#pragma unroll
    for (int o = 1; o < NBP; o <<= 1) {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const float y = __shfl_up_sync(FULL, l[k], o, NBP), z = __shfl_down_sync(FULL, s[k], o, NBP);
            if (b >= o) l[k] = k < 3 ? fminf(l[k], y) : fmaxf(l[k], y);
            if (b + o < NBP) s[k] = k < 3 ? fminf(s[k], z) : fmaxf(s[k], z);
        }
        const uint32_t yc = __shfl_up_sync(FULL, lcnt, o, NBP), zc = __shfl_down_sync(FULL, scnt, o, NBP);
        if (b >= o) lcnt += yc;
        if (b + o < NBP) scnt += zc;
    }
    // right side of plane b = suffix(b + 1)
    float r[6];
#pragma unroll
    for (int k = 0; k < 6; ++k) r[k] = __shfl_down_sync(FULL, s[k], 1, NBP);
    const uint32_t rcnt = __shfl_down_sync(FULL, scnt, 1, NBP);
    bool valid = false;
    float score = 0.0f;
    if (b <= nb - 2) {
        const float sl = box_sa(l, l + 3) * (float)lcnt;
        const float sr = box_sa(r, r + 3) * (float)rcnt;
        score = sl + sr;
        valid = score < FLT_MAX;
    }
    // smallest score, ties to the highest plane
    int best = valid ? b : -1;
#pragma unroll
    for (int o = NBP / 2; o > 0; o >>= 1) {
        const int ob = __shfl_xor_sync(FULL, best, o);
        const float os = __shfl_xor_sync(FULL, score, o);
        if (ob >= 0 && (best < 0 || os < score || (os == score && ob > best))) { best = ob; score = os; }
    }
    plane = best;
    const int at = g0 + (best < 0 ? 0 : best);
    nl = __shfl_sync(FULL, lcnt, at);
#pragma unroll
    for (int k = 0; k < 6; ++k) { lp[k] = __shfl_sync(FULL, l[k], at); rp[k] = __shfl_sync(FULL, r[k], at); }
    // centroid boxes of bins [0, best] and (best, ...]
    const bool in_left = b <= best;
    if (NBP > 8) {
        // whole-warp reductions, once per node
#pragma unroll
        for (int q = 0; q < 32 / NBP; ++q) {
            const bool mine = NBP == 32 || g0 == q * NBP;
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float x0 = redux_min(mine && in_left ? c[k] : INFINITY);
                const float x1 = redux_max(mine && in_left ? c[3 + k] : -INFINITY);
                const float x2 = redux_min(mine && !in_left ? c[k] : INFINITY);
                const float x3 = redux_max(mine && !in_left ? c[3 + k] : -INFINITY);
                if (mine) { lc[k] = x0; lc[3 + k] = x1; rc[k] = x2; rc[3 + k] = x3; }
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < 6; ++k) {
            const float none = k < 3 ? INFINITY : -INFINITY;
            lc[k] = in_left ? c[k] : none;
            rc[k] = in_left ? none : c[k];
        }
#pragma unroll
        for (int o = NBP / 2; o > 0; o >>= 1) {
#pragma unroll
            for (int k = 0; k < 6; ++k) {
                const float y = __shfl_xor_sync(FULL, lc[k], o), z = __shfl_xor_sync(FULL, rc[k], o);
                lc[k] = k < 3 ? fminf(lc[k], y) : fmaxf(lc[k], y);
                rc[k] = k < 3 ? fminf(rc[k], z) : fmaxf(rc[k], z);
            }
        }
    }
    if (nb < kMaxBins) {
#pragma unroll
        for (int k = 0; k < 3; ++k) { rc[k] = fminf(rc[k], FLT_MAX); rc[3 + k] = fmaxf(rc[3 + k], -FLT_MAX); }
    }
}

// A bin's boxes from its encoded words (FLT_MAX boxes when it is empty).
template <bool ODD>
__device__ __forceinline__ uint32_t load_bin(const uint32_t* bin, bool in_range, float* p, float* c)
{
    const uint32_t cnt = in_range ? bin[12] : 0u;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        p[a] = c[a] = FLT_MAX;
        p[3 + a] = c[3 + a] = -FLT_MAX;
        if (cnt) {
            p[a] = dec_neg<ODD>(bin[a]); p[3 + a] = dec_pos<ODD>(bin[3 + a]);
            c[a] = dec_neg<ODD>(bin[6 + a]); c[3 + a] = dec_pos<ODD>(bin[9 + a]);
        }
    }
    return cnt;
}

// The plane of one node whose nb bins are given, one bin per lane; every lane
// returns the result.
__device__ __forceinline__ PlaneResult warp_choose_plane(const uint32_t* __restrict__ bins, int nb)
{
    const int lane = threadIdx.x & 31;
    PlaneResult r;
    float p[6], c[6];
    const uint32_t cnt = load_bin<true>(bins + lane * kBinWords, lane < nb, p, c);
    choose_planes<32>(nb, cnt, p, c, r.plane, r.nl, r.lp, r.rp, r.lc, r.rc);
    return r;
}

__device__ __forceinline__ Task child_task(uint32_t begin, uint32_t count, uint32_t slot, uint32_t buf, const float* p,
                                           const float* c)
{
    Task t;
    t.begin = begin; t.count = count; t.slot = slot; t.flags = buf;
    for (int k = 0; k < 3; ++k) { t.pmn[k] = p[k]; t.pmx[k] = p[3 + k]; t.cmn[k] = c[k]; t.cmx[k] = c[3 + k]; }
    return t;
}

// ---------------------------------------------------------------------------
// large phase
//
// Every kernel reads the level's task and chunk counts on the device and
// loops over its work (tasks per warp, chunks per block), so a fixed grid
// serves any level, with or without the host knowing the counts.

// Sum of the counts of bins [0, plane] of one chunk's count row.
__device__ __forceinline__ uint32_t left_count(const uint32_t* __restrict__ row, int plane)
{
    const int full = (plane + 1) >> 1;
    uint32_t n = 0;
    for (int w = 0; w < full; ++w) {
        const uint32_t v = row[w];
        n += (v & 0xFFFFu) + (v >> 16);
    }
    if ((plane + 1) & 1) n += row[full] & 0xFFFFu;
    return n;
}

// One warp per task: the plane, the node record, the two children, and the
// number of left triangles before each of the task's chunks.
template <uint32_t CHUNK>
__global__ void __launch_bounds__(128) k_large_split(LevelLists cur, LevelLists next, const Ctl* __restrict__ ctl_in,
                                                     uint32_t cur_i, uint32_t next_i, int nb, uint32_t base,
                                                     uint32_t leaf_size, Node* __restrict__ nodes,
                                                     Part* __restrict__ parts, uint32_t* __restrict__ chunk_left,
                                                     DoneLists done)
{
    chain_wait();  // a chained launch (enqueue_levels)
    chain_release();
    const uint32_t nt = (uint32_t)ctl_in->level[cur_i];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t warps = (gridDim.x * blockDim.x) >> 5;
    const uint32_t cw = count_words(nb);
    for (uint32_t t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < nt; t += warps) {
        const Task tk = cur.tasks[t];
        const uint32_t chunk0 = cur.chunk0[t];
        const uint32_t chunks = (tk.count + CHUNK - 1) / CHUNK;
        const PlaneResult r = warp_choose_plane(cur.bins + (size_t)t * kMaxBins * kBinWords, nb);
        Part p;
        p.begin = tk.begin;
        p.count = tk.count;
        p.nl = r.nl;
        p.chunk0 = chunk0;
        p.plane = r.plane;
        p.flags = (tk.flags & 1u) | (chunks > 1 ? 2u : 0u);
        p.task[0] = p.task[1] = kNone;
        p.axis[0] = p.axis[1] = 0;
        p.child_chunk0[0] = p.child_chunk0[1] = 0;
        p.k1[0] = p.k1[1] = p.cmin[0] = p.cmin[1] = 0.0f;
        if (r.plane < 0 || r.nl == 0 || r.nl == tk.count) {
            // no plane scored below FLT_MAX: the node becomes a leaf
            p.plane = -1;
            if (lane == 0) {
                list_leaf(tk, done);
                parts[t] = p;
            }
            continue;
        }
        const uint32_t q = tk.begin + r.nl;
        if (lane == 0) {
            Box pb;
            for (int a = 0; a < 3; ++a) { pb.mn[a] = tk.pmn[a]; pb.mx[a] = tk.pmx[a]; }
            store_node(nodes + tk.slot, pb, base + 2u * q, 2u, 0);
        }
        const uint32_t buf = (tk.flags & 1u) ^ 1u;
        const bool zero = chunks > 1;
        place_task<CHUNK>(child_task(tk.begin, r.nl, base + 2u * q, buf, r.lp, r.lc), leaf_size, nb, next,
                          &done.ctl->level[next_i], zero, done, p, 0);
        place_task<CHUNK>(child_task(q, tk.count - r.nl, base + 2u * q + 1u, buf, r.rp, r.rc), leaf_size, nb, next,
                          &done.ctl->level[next_i], zero, done, p, 1);
        if (lane == 0) parts[t] = p;
        // exclusive scan of the chunks' left counts, 128 chunks a round
        uint32_t carry = 0;
        if (chunks > 1)
            for (uint32_t c0 = 0; c0 < chunks; c0 += 128) {
                const uint32_t c = c0 + 4u * lane;
                uint32_t v[4], sum = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    v[k] = c + k < chunks ? left_count(cur.counts + (size_t)(chunk0 + c + k) * cw, r.plane) : 0u;
                    sum += v[k];
                }
                uint32_t x = sum;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xFFFFFFFFu, x, o);
                    if (lane >= (uint32_t)o) x += y;
                }
                uint32_t run = carry + x - sum;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    if (c + k < chunks) chunk_left[chunk0 + c + k] = run;
                    run += v[k];
                }
                carry += __shfl_sync(0xFFFFFFFFu, x, 31);
            }
    }
}

// One block per chunk: the chunk's triangles move to their side of the
// task's plane, in order, and each is binned for the large child it joins:
// its bin is stored as a byte beside its id, its boxes go into the child's
// bins, and where the task has several chunks the bin counts of the child's
// chunks are counted too (a side's run of one chunk lands in at most two).
// ROOT: the level's tasks are binned in place, nothing moves.
//
// The block's warps share kSlots / NBP copies of a side's bins (NBP: the bin count
// rounded up to 8, 16 or 32), a lane's copy by its number: shared-memory
// atomics on order-preserving integers, 13 a triangle, which were what bounded
// the kernel (half of all shared-memory cycles) while lanes of one bin waited
// for one another; full-warp reductions when 32 triangles share one side and
// bin.
constexpr int kSlots = 32;

struct MoveSmem {
    uint32_t bins[2 * kSlots * kBinWords];
    uint32_t cnt[2][2][kSlots];
    uint32_t w[8];
};

template <uint32_t CHUNK, int NBP, bool ROOT, bool ODD>
__device__ __forceinline__ void move_chunks(MoveSmem& sm, uint32_t chunks, const Part* __restrict__ parts,
                                            const LevelLists& cur, const LevelLists& next, uint32_t* __restrict__ ids_a,
                                            uint32_t* __restrict__ ids_b, uint8_t* __restrict__ bin_a,
                                            uint8_t* __restrict__ bin_b, const uint32_t* __restrict__ chunk_left,
                                            const float4* __restrict__ tb, int nb)
{
    uint32_t* s_bins = sm.bins;
    uint32_t (&s_cnt)[2][2][kSlots] = sm.cnt;
    uint32_t* s_w = sm.w;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t lt = (1u << lane) - 1u;
    const uint32_t copy = (lane * NBP) & (kSlots - 1);  // first bin of the lane's copy
    const uint32_t cw = count_words(nb);
    for (uint32_t c = blockIdx.x; c < chunks; c += gridDim.x) {
        const Part P = parts[cur.chunk_task[c]];
        if (P.plane < 0) continue;  // block-uniform
        const uint32_t off = (c - P.chunk0) * CHUNK;
        const uint32_t len = min(CHUNK, P.count - off);
        const bool from_b = P.flags & 1u;
        const uint32_t* in = (from_b ? ids_b : ids_a) + P.begin + off;
        const uint8_t* bin_in = (from_b ? bin_b : bin_a) + P.begin + off;
        uint32_t* out = ROOT ? nullptr : (from_b ? ids_a : ids_b) + P.begin;
        uint8_t* bin_out = (from_b != ROOT ? bin_a : bin_b) + P.begin;
        const bool large0 = P.task[0] != kNone, large1 = P.task[1] != kNone;
        for (int j = threadIdx.x; j < 2 * kSlots * kBinWords; j += 256) s_bins[j] = 0;
        for (int j = threadIdx.x; j < 4 * kSlots; j += 256) (&s_cnt[0][0][0])[j] = 0;
        // the warp's rows of 32 triangles
        const uint32_t rows = (len + 31u) >> 5, per = (rows + 7u) >> 3;
        const uint32_t r0 = warp * per, r1 = min(rows, r0 + per);
        uint32_t left_before = 0, lrun = 0;
        if (!ROOT) {
            uint32_t nl = 0;
            for (uint32_t r = r0; r < r1; ++r) {
                const uint32_t j = r * 32u + lane;
                nl += __popc(__ballot_sync(0xFFFFFFFFu, j < len && (int)bin_in[j] <= P.plane));
            }
            if (lane == 0) s_w[warp] = nl;
            left_before = (P.flags & 2u) ? chunk_left[c] : 0u;
        }
        __syncthreads();
        if (!ROOT)
            for (uint32_t w = 0; w < warp; ++w) lrun += s_w[w];
        lrun += left_before;  // left triangles of the task before this warp's row
        const uint32_t first[2] = {ROOT ? c - P.chunk0 : left_before / CHUNK,
                                   (off - left_before) / CHUNK};  // first chunk of each side's run
        for (uint32_t r = r0; r < r1; ++r) {
            const uint32_t j = r * 32u + lane;
            const bool valid = j < len;
            bool left = true;
            uint32_t id = 0, pos = off + j;  // pos: place in the task's range
            if (valid) id = in[j];
            if (!ROOT) {
                left = valid && (int)bin_in[j] <= P.plane;
                const uint32_t lb = __ballot_sync(0xFFFFFFFFu, left);
                const uint32_t lrank = lrun + __popc(lb & lt);
                lrun += __popc(lb);
                // a right triangle's rank is its index less the left ones before it
                pos = left ? lrank : off + j - lrank;
            }
            const uint32_t side = left ? 0u : 1u;
            const bool binned = valid && (left ? large0 : large1);
            const uint32_t to = pos + (left ? 0u : P.nl);
            if (!ROOT && valid) out[to] = id;
            uint32_t key = kNone;
            uint32_t e[12];
            if (binned) {
                float mn[3], mx[3], cc[3];
                load_box(tb, id, mn, mx);
#pragma unroll
                for (int a = 0; a < 3; ++a) cc[a] = (mn[a] + mx[a]) * 0.5f;
                const int b = bin_of(left ? P.k1[0] : P.k1[1], sel(cc, left ? P.axis[0] : P.axis[1]),
                                     left ? P.cmin[0] : P.cmin[1], nb);
                bin_out[to] = (uint8_t)b;
                key = side * kSlots + (uint32_t)b;
                encode_boxes<ODD>(mn, mx, cc, e);
                atomicAdd(&s_cnt[side][pos / CHUNK - (left ? first[0] : first[1])][copy + (uint32_t)b], 1u);
            }
            const uint32_t key0 = __shfl_sync(0xFFFFFFFFu, key, 0);
            if (__all_sync(0xFFFFFFFFu, key == key0)) {
                if (key0 != kNone) {
#pragma unroll
                    for (int k = 0; k < 12; ++k) e[k] = __reduce_max_sync(0xFFFFFFFFu, e[k]);
                    if (lane == 0) {
#pragma unroll
                        for (int k = 0; k < 12; ++k) atomicMax(&s_bins[key * kBinWords + k], e[k]);
                    }
                }
            } else if (binned) {
#pragma unroll
                for (int k = 0; k < 12; ++k) atomicMax(&s_bins[(key + copy) * kBinWords + k], e[k]);
            }
        }
        __syncthreads();
        const bool several = P.flags & 2u;
#pragma unroll
        for (int side = 0; side < 2; ++side) {
            if (P.task[side] == kNone) continue;  // block-uniform
            uint32_t* g = next.bins + (size_t)P.task[side] * kMaxBins * kBinWords;
            const uint32_t* sb = s_bins + side * kSlots * kBinWords;
            for (int j = threadIdx.x; j < nb * kBinWords; j += 256) {
                const int b = j / kBinWords;
                const bool is_count = j - b * kBinWords == 12;
                uint32_t v = 0;
#pragma unroll
                for (int q = 0; q < kSlots; q += NBP)
                    v = is_count ? v + s_cnt[side][0][b + q] + s_cnt[side][1][b + q] : max(v, sb[j + q * kBinWords]);
                if (!several) g[j] = v;
                else if (v) {
                    if (is_count) atomicAdd(g + j, v); else atomicMax(g + j, v);
                }
            }
            if (several && (side ? P.count - P.nl : P.nl) > CHUNK) {
                // the counts of the run's one or two chunks, two bins a word
                for (uint32_t j = threadIdx.x; j < 2u * cw; j += 256) {
                    const uint32_t slot = j >= cw ? 1u : 0u, w = j - slot * cw;
                    uint32_t v = 0;
#pragma unroll
                    for (int q = 0; q < kSlots; q += NBP)
                        v += s_cnt[side][slot][2 * w + q] +
                             (2 * w + 1 < (uint32_t)nb ? s_cnt[side][slot][2 * w + 1 + q] << 16 : 0u);
                    if (v) atomicAdd(next.counts + (size_t)(P.child_chunk0[side] + first[side] + slot) * cw + w, v);
                }
            }
        }
        __syncthreads();  // the shared bins are cleared for the next chunk
    }
}

template <uint32_t CHUNK, int NBP, bool ROOT>
__global__ void __launch_bounds__(256) k_large_move(const Part* __restrict__ parts, LevelLists cur, LevelLists next,
                                                    uint32_t cur_i, uint32_t* __restrict__ ids_a,
                                                    uint32_t* __restrict__ ids_b, uint8_t* __restrict__ bin_a,
                                                    uint8_t* __restrict__ bin_b, const uint32_t* __restrict__ chunk_left,
                                                    const float4* __restrict__ tb, int nb, Ctl* ctl)
{
    chain_wait();  // a chained launch (enqueue_levels)
    chain_release();
    __shared__ MoveSmem sm;
    if (!ROOT && blockIdx.x == 0 && threadIdx.x == 0) ctl->level[(cur_i + 2u) % 3u] = 0;
    const uint32_t chunks = (uint32_t)(ctl->level[cur_i] >> 32);
    if (ctl->odd) move_chunks<CHUNK, NBP, ROOT, true>(sm, chunks, parts, cur, next, ids_a, ids_b, bin_a, bin_b, chunk_left, tb, nb);
    else move_chunks<CHUNK, NBP, ROOT, false>(sm, chunks, parts, cur, next, ids_a, ids_b, bin_a, bin_b, chunk_left, tb, nb);
}

// ---------------------------------------------------------------------------
// leaves

// Leaf-region records for [b, b+c) and the range's own record at its slot.
__device__ void warp_emit_leaf(const uint32_t* __restrict__ ids, uint32_t b, uint32_t c, uint32_t slot, uint32_t flags,
                               const float* pmn, const float* pmx, const float4* __restrict__ tb, Node* __restrict__ nodes,
                               uint32_t leaf0, uint32_t* err)
{
    const int lane = threadIdx.x & 31;
    for (uint32_t j = lane; j < c; j += 32) {
        const uint32_t id = ids[b + j];
        Box bb;
        load_box(tb, id, bb.mn, bb.mx);
        store_node(nodes + leaf0 + b + j, bb, id, 1u, kLeafFlag);
        if (c == 1 && !(flags & 2u)) store_node(nodes + slot, bb, id, 1u, kLeafFlag);
    }
    if (lane == 0 && (c != 1 || (flags & 2u))) {
        // a record counts to 65535: a larger range is refused, its record empty
        // (the collapse and the traversals read it before the error is seen)
        const bool fits = c <= 65535u;
        if (!fits) raise_error(err, SQ_DEVERR_NODE_COUNT);
        Box pb;
        for (int a = 0; a < 3; ++a) { pb.mn[a] = pmn[a]; pb.mx[a] = pmx[a]; }
        store_node(nodes + slot, pb, leaf0 + b, fits ? c : 0u, 0);
    }
}

__global__ void k_emit_leaves(const LeafRange* __restrict__ leaves, const Ctl* __restrict__ ctl,
                              const uint32_t* __restrict__ ids_a, const uint32_t* __restrict__ ids_b,
                              const float4* __restrict__ tb, Node* __restrict__ nodes, uint32_t leaf0, uint32_t* err)
{
    const uint32_t nl = ctl->n_leaf;
    for (uint32_t w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < nl; w += (gridDim.x * blockDim.x) >> 5) {
        const LeafRange lr = leaves[w];
        const uint32_t* ids = (lr.flags & 1u) ? ids_b : ids_a;
        warp_emit_leaf(ids, lr.begin, lr.count, lr.slot, lr.flags, lr.pmn, lr.pmx, tb, nodes, leaf0, err);
    }
}

// ---------------------------------------------------------------------------
// middle phase: one block per subtree of kSmall + 1 to kMid triangles
//
// The subtree is staged in shared memory and split level by level, a warp per
// node for the planes (at most seven nodes of more than kSmall triangles exist
// at a time), the block's threads over the triangles for binning and the
// stable partition, until every node is small or a leaf; then the ids go back
// to their buffer in the final order.  A level here is four block barriers;
// as a level of the large phase it was two launches of 3 to 15 us, and the
// lower third of the large levels were these.
constexpr int kMidNodes = 8;
static_assert(kMid / (kSmall + 1) < kMidNodes, "a warp per middle node");

struct MidNode {
    Task t;  // begin relative to the subtree
    float k1, cmin;
    int axis, plane;  // plane -1: stays (a leaf)
    uint32_t nl, lstart, pad[2];
};

struct MidStage {
    float4 box[kMid][2];  // min xyz, id; max xyz
    uint32_t bins[kMidNodes][kMaxBins * kBinWords];
    MidNode node[2][kMidNodes];
    uint32_t n_node[2];
    uint32_t lbits[kMid / 32], lpre[kMid / 32];  // left flags by position, and left triangles before each word
    uint16_t loc[2][kMid];                       // the triangle at each position
    uint8_t bin[kMid];
    uint32_t task;
};

template <int NBP>
__global__ void __launch_bounds__(256) k_mid(uint32_t* __restrict__ ids_a, uint32_t* __restrict__ ids_b,
                                             const float4* __restrict__ tb, int nb, uint32_t leaf_size, uint32_t base,
                                             Node* __restrict__ nodes, DoneLists done)
{
    extern __shared__ __align__(16) unsigned char s_mid[];
    MidStage& sg = *reinterpret_cast<MidStage*>(s_mid);
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t copy = (lane * NBP) & (kMaxBins - 1);  // first bin of the lane's copy
    const uint32_t total = done.ctl->n_mid;
    const bool odd = done.ctl->odd != 0u;
    auto add_node = [&](int p, const Task& t) {
        MidNode& m = sg.node[p][atomicAdd(&sg.n_node[p], 1u)];
        m.t = t;
        m.axis = choose_axis(t.cmn, t.cmx);
        m.cmin = sel(t.cmn, m.axis);
        m.k1 = bin_k1(nb, sel(t.cmx, m.axis) - m.cmin);
    };
    for (;;) {
        if (tid == 0) {
            sg.task = atomicAdd(&done.ctl->mid_pop, 1u);
            sg.n_node[0] = sg.n_node[1] = 0;
        }
        __syncthreads();
        if (sg.task >= total) return;
        const Task root = done.mid[sg.task];
        const uint32_t rb = root.begin, count = root.count, parity = root.flags & 1u;
        uint32_t* ids = (parity ? ids_b : ids_a) + rb;
        for (uint32_t j = tid; j < count; j += 256) {
            const uint32_t id = ids[j];
            float4 lo = __ldg(tb + 2ull * id);
            lo.w = __uint_as_float(id);
            sg.box[j][0] = lo;
            sg.box[j][1] = __ldg(tb + 2ull * id + 1);
            sg.loc[0][j] = (uint16_t)j;
        }
        if (tid == 0) {
            Task t = root;
            t.begin = 0;
            add_node(0, t);
        }
        int cur = 0;
        for (;; cur ^= 1) {
            __syncthreads();
            const uint32_t active = sg.n_node[cur];
            if (active == 0) break;
            MidNode* node = sg.node[cur];
            for (uint32_t j = tid; j < active * (kMaxBins * kBinWords); j += 256) (&sg.bins[0][0])[j] = 0;
            __syncthreads();
            // the node of a position (kMidNodes: none, its triangles are done)
            auto node_at = [&](uint32_t pos) {
                uint32_t a = kMidNodes;
                for (uint32_t q = 0; q < active; ++q)
                    if (pos - node[q].t.begin < node[q].t.count) a = q;
                return a;
            };
            auto bin_all = [&](auto form) {
                for (uint32_t pos = tid; pos < count; pos += 256) {
                    const uint32_t a = node_at(pos);
                    if (a == kMidNodes) continue;
                    const uint32_t li = sg.loc[cur][pos];
                    const float4 lo = sg.box[li][0], hi = sg.box[li][1];
                    const float mn[3] = {lo.x, lo.y, lo.z}, mx[3] = {hi.x, hi.y, hi.z};
                    float cc[3];
#pragma unroll
                    for (int k = 0; k < 3; ++k) cc[k] = (mn[k] + mx[k]) * 0.5f;
                    const uint32_t b = (uint32_t)bin_of(node[a].k1, sel(cc, node[a].axis), node[a].cmin, nb);
                    sg.bin[pos] = (uint8_t)b;
                    uint32_t* w = sg.bins[a] + (copy + b) * kBinWords;
                    uint32_t e[12];
                    encode_boxes<decltype(form)::value>(mn, mx, cc, e);
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
#pragma unroll
                        for (int k = a; k < 12; k += 3) atomicMax(w + k, e[k]);
                    }
                    atomicAdd(w + 12, 1u);
                }
            };
            if (odd) bin_all(std::true_type{});
            else bin_all(std::false_type{});
            __syncthreads();
            if (warp < active) {
                MidNode& m = node[warp];
                uint32_t w[kBinWords];
#pragma unroll
                for (int k = 0; k < kBinWords; ++k) w[k] = 0;
                if (lane < (uint32_t)NBP) {
#pragma unroll
                    for (int q = 0; q < kMaxBins; q += NBP) {
                        const uint32_t* bw = sg.bins[warp] + (lane + q) * kBinWords;
#pragma unroll
                        for (int k = 0; k < 12; ++k) w[k] = max(w[k], bw[k]);
                        w[12] += bw[12];
                    }
                }
                float p[6], c[6];
                const uint32_t cnt = load_bin<true>(w, (int)lane < nb, p, c);
                PlaneResult r;
                choose_planes<32>(nb, cnt, p, c, r.plane, r.nl, r.lp, r.rp, r.lc, r.rc);
                if (lane == 0) {
                    const Task t = m.t;
                    const bool split = r.plane >= 0 && r.nl != 0 && r.nl != t.count;
                    m.plane = split ? r.plane : -1;
                    m.nl = r.nl;
                    if (!split) {
                        // no plane scored below FLT_MAX: the node becomes a leaf
                        Task g = t;
                        g.begin += rb;
                        list_leaf(g, done);
                    } else {
                        const uint32_t q = rb + t.begin + r.nl;
                        Box pb;
                        for (int k = 0; k < 3; ++k) { pb.mn[k] = t.pmn[k]; pb.mx[k] = t.pmx[k]; }
                        store_node(nodes + t.slot, pb, base + 2u * q, 2u, 0);
#pragma unroll
                        for (int side = 0; side < 2; ++side) {
                            Task ch = side ? child_task(t.begin + r.nl, t.count - r.nl, base + 2u * q + 1u, parity, r.rp, r.rc)
                                           : child_task(t.begin, r.nl, base + 2u * q, parity, r.lp, r.lc);
                            const bool leaf = is_leaf_task(ch, leaf_size);
                            if (!leaf && ch.count > kSmall) {
                                add_node(cur ^ 1, ch);
                                continue;
                            }
                            ch.begin += rb;
                            if (leaf) list_leaf(ch, done);
                            else done.small[atomicAdd(&done.ctl->n_small, 1u)] = ch;
                        }
                    }
                }
            }
            __syncthreads();
            // partition, stably: left flags by position, their prefix, the moves
            for (uint32_t w0 = warp * 32u; w0 < count; w0 += 256) {
                const uint32_t pos = w0 + lane;
                const uint32_t a = pos < count ? node_at(pos) : (uint32_t)kMidNodes;
                const uint32_t b = __ballot_sync(FULL, a != kMidNodes && (int)sg.bin[pos] <= node[a].plane);
                if (lane == 0) sg.lbits[w0 >> 5] = b;
            }
            __syncthreads();
            if (warp == 0) {
                const uint32_t words = (count + 31u) >> 5;
                const uint32_t v = lane < words ? (uint32_t)__popc(sg.lbits[lane]) : 0u;
                uint32_t x = v;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(FULL, x, o);
                    if (lane >= (uint32_t)o) x += y;
                }
                if (lane < words) sg.lpre[lane] = x - v;
                __syncwarp();
                if (lane < active) {
                    const uint32_t s0 = node[lane].t.begin;
                    node[lane].lstart = sg.lpre[s0 >> 5] + __popc(sg.lbits[s0 >> 5] & ((1u << (s0 & 31u)) - 1u));
                }
                if (lane == 0) sg.n_node[cur] = 0;
            }
            __syncthreads();
            for (uint32_t pos = tid; pos < count; pos += 256) {
                const uint32_t a = node_at(pos), li = sg.loc[cur][pos];
                uint32_t to = pos;
                if (a != kMidNodes && node[a].plane >= 0) {
                    const uint32_t word = sg.lbits[pos >> 5], bit = 1u << (pos & 31u);
                    const uint32_t lr = sg.lpre[pos >> 5] + __popc(word & (bit - 1u)) - node[a].lstart;
                    const uint32_t b0 = node[a].t.begin;
                    to = b0 + ((word & bit) ? lr : node[a].nl + (pos - b0) - lr);
                }
                sg.loc[cur ^ 1][to] = (uint16_t)li;
            }
        }
        for (uint32_t j = tid; j < count; j += 256) ids[j] = __float_as_uint(sg.box[sg.loc[cur][j]][0].w);
        __syncthreads();  // the stage is used again for the block's next task
    }
}

// ---------------------------------------------------------------------------
// small phase: one warp per subtree
//
// A subtree of at most kStage triangles (every small task of a single build:
// a task turns small at kSmall or fewer) is staged once in the warp's shared
// memory -- each triangle's box and id -- and built from there: only local
// indices move, and leaves read their boxes from the stage.
//
// The warp's nodes wait on a stack and are split G = 32 / NBP at a time (NBP:
// the bin count rounded up to 8, 16 or 32), lane = (node, bin) while the
// planes are swept and lane = triangle while the nodes' triangles are binned
// and partitioned, four rounds of 32 at most for all of them together.  A
// node holds 5 to 30 triangles mostly, so one node at a time left most lanes
// idle in the binning and 24 of 32 in a sweep of 8 bins; the sweep, a chain
// of shuffles, was what bounded a node.  The order of the stack does not
// matter: a node's records go to slots that its range gives.
//
// The large tasks left after a batch's fixed levels are split by k_small_big,
// one node at a time, in the global buffers.
constexpr uint32_t kStage = 128;
static_assert(kSmall <= kStage && kMid / 32 <= 32, "every small task is staged; one warp scans a middle task's words");

struct SmallNode {
    float p[6], c[6];  // primitive and centroid boxes (min xyz, max xyz)
    uint32_t slot;
    uint16_t begin, count;  // positions in the subtree
};
static_assert(sizeof(SmallNode) == 56, "SmallNode is 56 bytes");

struct SmallStage {
    float4 box[kStage][2];                   // min xyz, id; max xyz
    uint32_t bins[kMaxBins * kBinWords];
    SmallNode stack[kStage / 2];             // waiting nodes are disjoint and hold two triangles or more
    uint8_t loc[kStage];                     // the triangle at each position
};

// One small task from the stage.
template <int NBP, bool ODD>
__device__ void staged_subtree(const Task& root, SmallStage& sg, const uint32_t* __restrict__ ids,
                               const float4* __restrict__ tb, int nb, uint32_t leaf_size, uint32_t base,
                               Node* __restrict__ nodes, uint32_t leaf0)
{
    constexpr uint32_t FULL = 0xFFFFFFFFu;
    constexpr int G = 32 / NBP;
    constexpr int kRounds = kStage / 32;
    const uint32_t lane = threadIdx.x & 31u, lt = (1u << lane) - 1u;
    const uint32_t b = lane & (NBP - 1), g = lane / NBP;
    const uint32_t rb = root.begin;
    for (uint32_t j = lane; j < root.count; j += 32) {
        const uint32_t id = ids[rb + j];
        float4 lo = __ldg(tb + 2ull * id);
        lo.w = __uint_as_float(id);
        sg.box[j][0] = lo;
        sg.box[j][1] = __ldg(tb + 2ull * id + 1);
        sg.loc[j] = (uint8_t)j;
    }
    if (lane == 0) {
        SmallNode& s = sg.stack[0];
        for (int k = 0; k < 3; ++k) {
            s.p[k] = root.pmn[k]; s.p[3 + k] = root.pmx[k];
            s.c[k] = root.cmn[k]; s.c[3 + k] = root.cmx[k];
        }
        s.slot = root.slot; s.begin = 0; s.count = (uint16_t)root.count;
    }
    __syncwarp();
    uint32_t sp = 1;
    while (sp) {
        // the top m nodes of the stack, one per lane group (every one is
        // splittable: more than leaf_size triangles, centroid area > 0)
        const uint32_t m = min((uint32_t)G, sp);
        const bool act = g < m;
        const SmallNode& nd = sg.stack[sp - m + (act ? g : 0u)];
        const uint32_t begin = nd.begin, count = act ? nd.count : 0u, slot = nd.slot;
        float np[6];
#pragma unroll
        for (int k = 0; k < 6; ++k) np[k] = nd.p[k];
        const int axis = choose_axis(nd.c, nd.c + 3);
        const float cmin = sel(nd.c, axis);
        const float k1 = bin_k1(nb, sel(nd.c + 3, axis) - cmin);
        // the group's triangles are [start, start + count) of the warp's total
        uint32_t starts[G], total = 0, start = 0;
#pragma unroll
        for (int q = 0; q < G; ++q) {
            starts[q] = total;
            if (g == (uint32_t)q) start = total;
            total += __shfl_sync(FULL, count, q * NBP);
        }
        for (uint32_t j = lane; j < (uint32_t)(kMaxBins * kBinWords / 4); j += 32)
            reinterpret_cast<uint4*>(sg.bins)[j] = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
        // bin: lane = triangle
        uint32_t el[kRounds];  // the triangle's place in the stage, its bin and its node's group
#pragma unroll
        for (int it = 0; it < kRounds; ++it) {
            el[it] = 0;
            if (32u * it < total) {  // warp-uniform
                const uint32_t e = 32u * it + lane;
                uint32_t ge = 0;
#pragma unroll
                for (int q = 1; q < G; ++q) ge += ((uint32_t)q < m && e >= starts[q]) ? 1u : 0u;
                const int src = (int)ge * NBP;
                const uint32_t at = __shfl_sync(FULL, (begin - start) & 0xFFFFu, src);
                const int ax = __shfl_sync(FULL, axis, src);
                const float cm = __shfl_sync(FULL, cmin, src), kk = __shfl_sync(FULL, k1, src);
                if (e < total) {
                    const uint32_t li = sg.loc[(at + e) & 0xFFFFu];
                    const float4 lo = sg.box[li][0], hi = sg.box[li][1];
                    const float mn[3] = {lo.x, lo.y, lo.z}, mx[3] = {hi.x, hi.y, hi.z};
                    float cc[3];
#pragma unroll
                    for (int a = 0; a < 3; ++a) cc[a] = (mn[a] + mx[a]) * 0.5f;
                    const uint32_t bin = (uint32_t)bin_of(kk, sel(cc, ax), cm, nb);
                    el[it] = li | (bin << 8) | (ge << 16);
                    uint32_t* w = sg.bins + (ge * NBP + bin) * kBinWords;
                    uint32_t e[12];
                    encode_boxes<ODD>(mn, mx, cc, e);
#pragma unroll
                    for (int a = 0; a < 3; ++a) {
#pragma unroll
                        for (int k = a; k < 12; k += 3) atomicMax(w + k, e[k]);
                    }
                    atomicAdd(w + 12, 1u);
                }
            }
        }
        __syncwarp();
        // sweep: lane = (node, bin)
        int plane;
        uint32_t nl;
        float lp[6], rp[6], lc[6], rc[6];
        {
            float p[6], c[6];
            const uint32_t cnt = load_bin<ODD>(sg.bins + lane * kBinWords, act && (int)b < nb, p, c);
            choose_planes<NBP>(nb, cnt, p, c, plane, nl, lp, rp, lc, rc);
        }
        // the node's records and its children: lane 0 of a group has the
        // node, lanes 1 and 2 the left and the right child
        const bool has = act && plane >= 0 && nl != 0 && nl != count;
        const uint32_t nr = count - nl, q = rb + begin + nl;
        const bool leaf_l = has && (nl <= leaf_size || !(box_sa(lc, lc + 3) > 0.0f));
        const bool leaf_r = has && (nr <= leaf_size || !(box_sa(rc, rc + 3) > 0.0f));
        const bool right = b == 2;
        const bool push = has && (b == 1 || right) && !(right ? leaf_r : leaf_l);
        const uint32_t pushes = __ballot_sync(FULL, push);
        sp -= m;
        if (act && b <= 2) {
            const uint32_t cn = b == 0 ? count : (right ? nr : nl);
            Box pb;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                pb.mn[a] = b == 0 ? np[a] : (right ? rp[a] : lp[a]);
                pb.mx[a] = b == 0 ? np[3 + a] : (right ? rp[3 + a] : lp[3 + a]);
            }
            const uint32_t cslot = b == 0 ? slot : base + 2u * q + (right ? 1u : 0u);
            if (push) {
                SmallNode& s = sg.stack[sp + __popc(pushes & lt)];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    s.p[a] = pb.mn[a]; s.p[3 + a] = pb.mx[a];
                    s.c[a] = right ? rc[a] : lc[a]; s.c[3 + a] = right ? rc[3 + a] : lc[3 + a];
                }
                s.slot = cslot;
                s.begin = (uint16_t)(begin + (right ? nl : 0u));
                s.count = (uint16_t)cn;
            } else if (b == 0 && has) {
                store_node(nodes + slot, pb, base + 2u * q, 2u, 0);
            } else if (b == 0 || (has && cn != 1)) {
                // a leaf's range: this node's when no plane scored below
                // FLT_MAX, else the child's (a leaf child of one triangle has
                // that triangle's record at its slot)
                store_node(nodes + cslot, pb, leaf0 + rb + begin + (right ? nl : 0u), cn, 0);
            }
        }
        sp += __popc(pushes);
        // partition, stably: lane = triangle again
        uint32_t lb[kRounds], before[kRounds];
        const uint32_t say = (has ? 1u : 0u) | (leaf_l ? 2u : 0u) | (leaf_r ? 4u : 0u) | ((uint32_t)(plane & 31) << 3) |
                             (nl << 8) | (begin << 16) | (start << 24);
        uint32_t sum = 0;
#pragma unroll
        for (int it = 0; it < kRounds; ++it) {
            lb[it] = 0;
            before[it] = sum;
            if (32u * it < total) {
                const uint32_t x = __shfl_sync(FULL, say, (int)(el[it] >> 16) * NBP);
                lb[it] = __ballot_sync(FULL, 32u * it + lane < total && (x & 1u) && ((el[it] >> 8) & 0xFFu) <= ((x >> 3) & 31u));
                sum += __popc(lb[it]);
            }
        }
        // left triangles before this group's first
        uint32_t lstart = 0;
#pragma unroll
        for (int it = 0; it < kRounds; ++it)
            if (start >= 32u * it && start < 32u * it + 32u) lstart = before[it] + __popc(lb[it] & ((1u << (start & 31u)) - 1u));
        const uint32_t say2 = lstart | (count << 8);
#pragma unroll
        for (int it = 0; it < kRounds; ++it) {
            if (32u * it >= total) break;
            const uint32_t e = 32u * it + lane;
            const int src = (int)(el[it] >> 16) * NBP;
            const uint32_t x = __shfl_sync(FULL, say, src), y = __shfl_sync(FULL, say2, src);
            if (e < total) {
                const bool split = x & 1u, left = (lb[it] >> lane) & 1u;
                const uint32_t xnl = (x >> 8) & 0xFFu, xbegin = (x >> 16) & 0xFFu, rel = e - (x >> 24);
                const uint32_t lr = before[it] + __popc(lb[it] & lt) - (y & 0xFFu);
                const uint32_t pos = xbegin + (split ? (left ? lr : xnl + rel - lr) : rel);
                const uint32_t li = el[it] & 0xFFu;
                sg.loc[pos] = (uint8_t)li;
                if (!split || (x & (left ? 2u : 4u))) {
                    const float4 lo = sg.box[li][0], hi = sg.box[li][1];
                    Box bb;
                    bb.mn[0] = lo.x; bb.mn[1] = lo.y; bb.mn[2] = lo.z;
                    bb.mx[0] = hi.x; bb.mx[1] = hi.y; bb.mx[2] = hi.z;
                    const uint32_t id = __float_as_uint(lo.w);
                    store_node(nodes + leaf0 + rb + pos, bb, id, 1u, kLeafFlag);
                    if (split && (left ? xnl : (y >> 8) - xnl) == 1u)
                        store_node(nodes + base + 2u * (rb + xbegin + xnl) + (left ? 0u : 1u), bb, id, 1u, kLeafFlag);
                }
            }
        }
        __syncwarp();
    }
}

// One warp per small task of at most kStage triangles (the tasks
// left after the last level of a batch, larger ones, are k_small_big's).
template <int NBP>
__global__ void __launch_bounds__(128) k_small(const Task* __restrict__ small, Ctl* ctl,
                                               const uint32_t* __restrict__ ids_a, const uint32_t* __restrict__ ids_b,
                                               const float4* __restrict__ tb, int nb, uint32_t leaf_size, uint32_t base,
                                               Node* __restrict__ nodes, uint32_t leaf0)
{
    __shared__ __align__(16) SmallStage s_stage[4];
    chain_wait();  // a chained launch (launch_subtrees)
    chain_release();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t total = ctl->n_small;
    const bool odd = ctl->odd != 0u;
    for (;;) {
        uint32_t ti = 0;
        if (lane == 0) ti = atomicAdd(&ctl->small_pop, 1u);
        ti = __shfl_sync(0xFFFFFFFFu, ti, 0);
        if (ti >= total) return;
        const Task t = small[ti];
        const uint32_t* ids = (t.flags & 1u) ? ids_b : ids_a;
        if (odd) staged_subtree<NBP, true>(t, s_stage[warp], ids, tb, nb, leaf_size, base, nodes, leaf0);
        else staged_subtree<NBP, false>(t, s_stage[warp], ids, tb, nb, leaf_size, base, nodes, leaf0);
    }
}

// A task of more than kStage triangles: one warp, one node at a time,
// smaller child first (stack depth O(log n)), in the global buffers.
__device__ void big_subtree(Task cur, Task* st, uint32_t* wb, uint32_t* __restrict__ ids_a, uint32_t* __restrict__ ids_b,
                            const float4* __restrict__ tb, int nb, uint32_t leaf_size, uint32_t base,
                            Node* __restrict__ nodes, uint32_t leaf0, uint32_t* err)
{
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    auto emit_leaf = [&](const Task& t) {
        warp_emit_leaf((t.flags & 1u) ? ids_b : ids_a, t.begin, t.count, t.slot, t.flags, t.pmn, t.pmx, tb, nodes, leaf0,
                       err);
    };
    int sp = 0;
    for (;;) {
        // cur is splittable (count > leaf_size, centroid area > 0)
        const uint32_t pin = cur.flags & 1u, pout = pin ^ 1u;
        const uint32_t* in = pin ? ids_b : ids_a;
        uint32_t* out = pin ? ids_a : ids_b;
        const int axis = choose_axis(cur.cmn, cur.cmx);
        const float cmin = sel(cur.cmn, axis);
        const float k1 = bin_k1(nb, sel(cur.cmx, axis) - cmin);
        for (int j = lane; j < kMaxBins * kBinWords; j += 32) wb[j] = 0;
        __syncwarp();
        for (uint32_t j0 = 0; j0 < cur.count; j0 += 32) {
            const uint32_t j = j0 + lane;
            float mn[3], mx[3], cc[3];
            int bin = nb;
            if (j < cur.count) {
                load_box(tb, in[cur.begin + j], mn, mx);
                for (int a = 0; a < 3; ++a) cc[a] = (mn[a] + mx[a]) * 0.5f;
                bin = bin_of(k1, sel(cc, axis), cmin, nb);
            } else {
                for (int a = 0; a < 3; ++a) { mn[a] = mx[a] = cc[a] = 0.0f; }
            }
            warp_bin_add(wb, bin, nb, mn, mx, cc);
        }
        const PlaneResult r = warp_choose_plane(wb, nb);
        __syncwarp();
        bool have_next = false;
        if (r.plane < 0 || r.nl == 0 || r.nl == cur.count) {
            // no plane scored below FLT_MAX: leaf
            emit_leaf(cur);
        } else {
            const uint32_t q = cur.begin + r.nl;
            if (lane == 0) {
                Box pb;
                for (int a = 0; a < 3; ++a) { pb.mn[a] = cur.pmn[a]; pb.mx[a] = cur.pmx[a]; }
                store_node(nodes + cur.slot, pb, base + 2u * q, 2u, 0);
            }
            // stable partition into the other order
            uint32_t lc = 0, rc = 0;
            for (uint32_t j0 = 0; j0 < cur.count; j0 += 32) {
                const uint32_t j = j0 + lane;
                const bool valid = j < cur.count;
                uint32_t id = 0;
                bool left = false;
                if (valid) {
                    float mn[3], mx[3];
                    id = in[cur.begin + j];
                    load_box(tb, id, mn, mx);
                    const float cc = (sel(mn, axis) + sel(mx, axis)) * 0.5f;
                    left = bin_of(k1, cc, cmin, nb) <= r.plane;
                }
                const uint32_t lb = __ballot_sync(0xFFFFFFFFu, valid && left);
                const uint32_t rb = __ballot_sync(0xFFFFFFFFu, valid && !left);
                if (valid) {
                    if (left) out[cur.begin + lc + __popc(lb & lt)] = id;
                    else out[q + rc + __popc(rb & lt)] = id;
                }
                lc += __popc(lb);
                rc += __popc(rb);
            }
            __syncwarp();
            Task ch[2] = {child_task(cur.begin, r.nl, base + 2u * q, pout, r.lp, r.lc),
                          child_task(q, cur.count - r.nl, base + 2u * q + 1u, pout, r.rp, r.rc)};
            bool split_ch[2];
            for (int k = 0; k < 2; ++k) {
                split_ch[k] = !(ch[k].count <= leaf_size || !(box_sa(ch[k].cmn, ch[k].cmx) > 0.0f));
                if (!split_ch[k]) emit_leaf(ch[k]);
            }
            if (split_ch[0] && split_ch[1]) {
                const int small_k = ch[0].count <= ch[1].count ? 0 : 1;
                if (sp >= kStackDepth) {
                    raise_error(err, SQ_DEVERR_SAH_QUEUE);
                    return;
                }
                if (lane == 0) st[sp] = ch[1 - small_k];
                sp++;
                __syncwarp();
                cur = ch[small_k];
                have_next = true;
            } else if (split_ch[0] || split_ch[1]) {
                cur = split_ch[0] ? ch[0] : ch[1];
                have_next = true;
            }
        }
        if (!have_next) {
            if (sp == 0) break;
            --sp;
            __syncwarp();
            cur = st[sp];
            __syncwarp();
        }
    }
}

__global__ void __launch_bounds__(128) k_small_big(const Task* __restrict__ tasks,
                                                   const unsigned long long* __restrict__ level,
                                                   uint32_t* __restrict__ ids_a,
                                                   uint32_t* __restrict__ ids_b, const float4* __restrict__ tb, int nb,
                                                   uint32_t leaf_size, uint32_t base, Node* __restrict__ nodes,
                                                   uint32_t leaf0, uint32_t* err)
{
    __shared__ uint32_t s_bins[4][kMaxBins * kBinWords];
    __shared__ Task s_stack[4][kStackDepth];
    const uint32_t warp = threadIdx.x >> 5;
    const uint32_t total = (uint32_t)*level;
    for (uint32_t ti = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; ti < total; ti += (gridDim.x * blockDim.x) >> 5) {
        const Task cur = tasks[ti];
        big_subtree(cur, s_stack[warp], s_bins[warp], ids_a, ids_b, tb, nb, leaf_size, base, nodes, leaf0, err);
    }
}

int sms() { return sm_count(); }

// Workspace carving shared by the single and the batched build.
struct SahWs {
    float4* tb;
    uint32_t *ids_a, *ids_b;
    uint8_t *bin_a, *bin_b;
    LevelLists lists[2];
    Task *mid, *small;
    LeafRange* leaves;
    Part* parts;
    uint32_t *chunk_left, *cells, *hist, *root_ord;
    Ctl* ctl;
    DoneLists done() const { return DoneLists{mid, small, leaves, ctl}; }
};

// Most large tasks a level can have, and most chunks.
size_t sah_tasks(uint32_t n) { return n / kMid + 2; }
size_t sah_chunks(uint32_t n) { return (size_t)n / (n < kChunkSmallBelow ? kChunkSmall : kChunk) + sah_tasks(n) + 1; }

// Lays the workspace out at p (null: only the size is wanted) and returns its size.
size_t sah_layout(char* p, uint32_t n, uint32_t meshes, SahWs& w)
{
    const size_t tasks = sah_tasks(n), chunks = sah_chunks(n);
    size_t used = 0;
    auto take = [&](auto*& ptr, size_t count) {
        using T = std::remove_reference_t<decltype(*ptr)>;
        ptr = reinterpret_cast<T*>(p + used);
        used += (sizeof(T) * count + 255) / 256 * 256;
    };
    take(w.tb, 2ull * n);  // triangle boxes
    take(w.ids_a, n);
    take(w.ids_b, n);
    take(w.bin_a, n);
    take(w.bin_b, n);
    for (LevelLists& l : w.lists) {
        take(l.tasks, tasks);
        take(l.chunk0, tasks);
        take(l.chunk_task, chunks);
        take(l.bins, (size_t)kMaxBins * kBinWords * tasks);
        take(l.counts, (size_t)(kMaxBins / 2) * chunks);
    }
    take(w.mid, (size_t)n / kSmall + 2);
    take(w.small, (size_t)n / 2 + 2);
    take(w.leaves, (size_t)n + 66 + meshes);  // + 64 empty grid cells, + empty meshes
    take(w.parts, tasks);
    take(w.chunk_left, chunks);
    take(w.cells, 64 * kBinWords);
    take(w.hist, 64);
    take(w.root_ord, 16ull * (meshes ? meshes : 1));  // 12 words per mesh
    take(w.ctl, 1);
    return used;
}

size_t sah_ws_bytes(uint32_t n, uint32_t meshes)
{
    SahWs w;
    return sah_layout(nullptr, n, meshes, w);
}

SahWs carve(void* ws, uint32_t n, uint32_t meshes)
{
    SahWs w;
    sah_layout(static_cast<char*>(ws), n, meshes, w);
    return w;
}

// Calls f(std::integral_constant<uint32_t, CHUNK>) with the chunk size of a
// build over n triangles.
template <class F>
void with_chunk(uint32_t n, F f)
{
    if (n < kChunkSmallBelow) f(std::integral_constant<uint32_t, kChunkSmall>());
    else f(std::integral_constant<uint32_t, kChunk>());
}

// One k_large_move launch over the chunks of level `level` (in w.lists[cur]).
template <uint32_t CHUNK, bool ROOT>
void enqueue_move(const SahWs& w, uint32_t cur, uint32_t next, uint32_t cur_i, int nb, cudaStream_t s)
{
    auto kernel = nb <= 8 ? k_large_move<CHUNK, 8, ROOT> : nb <= 16 ? k_large_move<CHUNK, 16, ROOT>
                                                                    : k_large_move<CHUNK, 32, ROOT>;
    launch_chained(kernel, dim3(sms() * 8), dim3(256), 0, s, (const Part*)w.parts, w.lists[cur], w.lists[next], cur_i,
                   w.ids_a, w.ids_b, w.bin_a, w.bin_b, (const uint32_t*)w.chunk_left, (const float4*)w.tb, nb, w.ctl);
}

// The bins of the root tasks in w.lists[0].
template <uint32_t CHUNK>
void enqueue_root_bins(const SahWs& w, int nb, cudaStream_t s)
{
    enqueue_move<CHUNK, true>(w, 0, 0, 0, nb, s);
}

// Levels [level, level + count) of the large phase: two chained launches a
// level, each may launch while the one before it runs and waits for it on
// the device (chain_wait).  Levels past the tree's depth find no tasks.
template <uint32_t CHUNK>
void enqueue_levels(const SahWs& w, uint32_t level, uint32_t count, int nb, uint32_t base, uint32_t leaf_size,
                    Node* nodes, cudaStream_t s)
{
    const uint32_t grid = (uint32_t)sms() * 8u;
    for (uint32_t l = level; l < level + count; ++l) {
        launch_chained(k_large_split<CHUNK>, dim3(grid), dim3(128), 0, s, w.lists[l & 1], w.lists[(l + 1) & 1],
                       (const Ctl*)w.ctl, l % 3u, (l + 1) % 3u, nb, base, leaf_size, nodes, w.parts, w.chunk_left,
                       w.done());
        enqueue_move<CHUNK, false>(w, l & 1, (l + 1) & 1, l % 3u, nb, s);
    }
}

template <int NBP>
void launch_subtrees_n(const SahWs& w, int nb, uint32_t leaf_size, uint32_t base, Node* nodes, uint32_t leaf0,
                       cudaStream_t s)
{
    // above 48 KB of dynamic shared memory is a per-device opt-in
    static PerDevice<int> cache;
    const int per_sm = cache.get([] {
        cudaFuncSetAttribute(k_mid<NBP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(MidStage));
        return blocks_per_sm(k_mid<NBP>, 256, sizeof(MidStage));
    });
    k_mid<NBP><<<per_sm * sms(), 256, sizeof(MidStage), s>>>(w.ids_a, w.ids_b, w.tb, nb, leaf_size, base, nodes, w.done());
    launch_chained(k_small<NBP>, dim3(sms() * 8), dim3(128), 0, s, (const Task*)w.small, w.ctl, (const uint32_t*)w.ids_a,
                   (const uint32_t*)w.ids_b, (const float4*)w.tb, nb, leaf_size, base, nodes, leaf0);
}

void launch_subtrees(const SahWs& w, int nb, uint32_t leaf_size, uint32_t base, Node* nodes, uint32_t leaf0,
                     cudaStream_t s)
{
    if (nb <= 8) launch_subtrees_n<8>(w, nb, leaf_size, base, nodes, leaf0, s);
    else if (nb <= 16) launch_subtrees_n<16>(w, nb, leaf_size, base, nodes, leaf0, s);
    else launch_subtrees_n<32>(w, nb, leaf_size, base, nodes, leaf0, s);
}

// ---------------------------------------------------------------------------
// batch: many meshes in one build

// Boxes, ids and every mesh's root boxes (order-preserving words, 12 per
// mesh at a stride of 16).
__global__ void __launch_bounds__(256) k_sah_setup_seg(const float* __restrict__ tris, uint32_t n,
                                                       const uint32_t* __restrict__ off, uint32_t M,
                                                       float4* __restrict__ tb, uint32_t* __restrict__ ids,
                                                       uint32_t* __restrict__ root_ord, Ctl* __restrict__ ctl)
{
    seg_maxima<12>(n, off, M, root_ord, 16u, [&](uint32_t i, uint32_t* e) {
        float t[9];
        load_tri(tris, i, t);
        const Box b = tri_box(t);
        tb[2ull * i] = make_float4(b.mn[0], b.mn[1], b.mn[2], 0.0f);
        tb[2ull * i + 1] = make_float4(b.mx[0], b.mx[1], b.mx[2], 0.0f);
        ids[i] = i;
        float c[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) c[k] = (b.mn[k] + b.mx[k]) * 0.5f;
        if (odd_box(c)) ctl->odd = 1u;
        encode_boxes<true>(b.mn, b.mx, c, e);
    });
}

// One root task per mesh (one warp each): triangles [off[m], off[m + 1]),
// record root0 + m.
template <uint32_t CHUNK>
__global__ void k_root_tasks_seg(const uint32_t* __restrict__ root_ord, const uint32_t* __restrict__ off, uint32_t M,
                                 uint32_t leaf_size, uint32_t root0, int nb, LevelLists l0, Part* parts,
                                 DoneLists done)
{
    const uint32_t m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (m >= M) return;
    Task t;
    t.begin = off[m];
    t.count = off[m + 1] - off[m];
    t.slot = root0 + m;
    t.flags = 2u;
    const uint32_t* ro = root_ord + 16ull * m;
    for (int k = 0; k < 3; ++k) {
        if (t.count) {
            t.pmn[k] = dec_neg(ro[k]);
            t.pmx[k] = dec_pos(ro[3 + k]);
            t.cmn[k] = dec_neg(ro[6 + k]);
            t.cmx[k] = dec_pos(ro[9 + k]);
        } else {
            t.pmn[k] = t.cmn[k] = FLT_MAX;
            t.pmx[k] = t.cmx[k] = -FLT_MAX;
        }
    }
    place_root<CHUNK>(t, leaf_size, nb, l0, parts, done);
}

}  // namespace

namespace sqk {

size_t sah_workspace_bytes(uint32_t n) { return sah_ws_bytes(n, 0); }
size_t sah_batch_workspace_bytes(uint32_t n, uint32_t meshes) { return sah_ws_bytes(n, meshes); }

// Builds a SAH (grid = 0) or grid (grid = 1) BVH.  ws: workspace of
// sah_workspace_bytes(n) bytes; keys/vals/alt: 4n-word sort buffers (grid
// only); sort_ws: zeroed onesweep state for one 6-bit pass (grid only).
// host_ctl: pinned 32-byte buffer.  Returns 0 or a cudaError_t.
int build_sah(const float* tris, uint32_t n, uint32_t nb, uint32_t leaf_size, int grid, uint32_t scene_box_cells,
              sq::Node* nodes, float* scene_out, void* ws, uint32_t* sort_keys, uint32_t* sort_vals,
              uint32_t* sort_alt_keys, uint32_t* sort_alt_vals, uint32_t* sort_lookback, uint32_t* sort_counters,
              uint32_t* err, uint32_t* host_ctl, cudaStream_t s)
{
    const SahWs w = carve(ws, n, 0);
    const uint32_t base = grid ? 128u : 0u;
    const uint32_t leaf0 = base + 2u * n + 2u;
    cudaError_t e;
#define SQ_TRY(x) do { if ((e = (x)) != cudaSuccess) return (int)e; } while (0)
    if (grid) SQ_TRY(cudaMemsetAsync(w.cells, 0, sizeof(uint32_t) * 64 * kBinWords, s));
    if (grid) SQ_TRY(cudaMemsetAsync(w.hist, 0, sizeof(uint32_t) * 64, s));
    SQ_TRY(cudaMemsetAsync(w.root_ord, 0, sizeof(uint32_t) * 16, s));
    SQ_TRY(cudaMemsetAsync(w.ctl, 0, sizeof(Ctl), s));
    const uint32_t g = min((n + 255) / 256, (uint32_t)sms() * 8u);
    k_sah_setup<<<g, 256, 0, s>>>(tris, n, w.tb, w.ids_a, w.root_ord, w.ctl);
    if (grid) {
        // bin into 64 cells keyed by Morton slot, then stable sort by slot
        k_grid_bin<<<g, 256, 0, s>>>(w.tb, n, w.root_ord, sort_keys, w.cells, w.hist);
        SQ_TRY(cudaMemcpyAsync(sort_vals, w.ids_a, sizeof(uint32_t) * (size_t)n, cudaMemcpyDeviceToDevice, s));
        const int which = sort_passes(sort_keys, sort_vals, sort_alt_keys, sort_alt_vals, n, w.hist, sort_lookback,
                                      sort_counters, 6, 1, err, s);
        SQ_TRY(cudaMemcpyAsync(w.ids_a, which ? sort_alt_vals : sort_vals, sizeof(uint32_t) * (size_t)n,
                               cudaMemcpyDeviceToDevice, s));
    }
    with_chunk(n, [&](auto chunk) {
        constexpr uint32_t CHUNK = decltype(chunk)::value;
        if (grid)
            k_grid_tasks<CHUNK><<<16, 128, 0, s>>>(w.cells, w.root_ord, n, leaf_size, scene_box_cells, (int)nb,
                                                   w.lists[0], w.parts, w.done(), scene_out);
        else
            k_root_task<CHUNK><<<1, 32, 0, s>>>(w.root_ord, n, leaf_size, (int)nb, w.lists[0], w.parts, w.done(),
                                                scene_out);
        if (n > kMid) enqueue_root_bins<CHUNK>(w, (int)nb, s);
    });
    // large phase: levels are queued in groups and the host reads the next
    // level's task count (and waits) only between groups; levels past the
    // tree's depth find no tasks and cost two empty launches.  The first
    // group is a balanced tree's depth and two levels more, which is all of
    // most meshes' large phase; a mesh of at most kMid triangles has none.
    uint32_t group = 2;
    while (((uint64_t)kMid << (group - 2)) < n) ++group;
    if (n > kMid)
        for (uint32_t level = 0;; group = kSahLevelsPerCheck) {
            with_chunk(n, [&](auto chunk) {
                enqueue_levels<decltype(chunk)::value>(w, level, group, (int)nb, base, leaf_size, nodes, s);
            });
            level += group;
            SQ_TRY(cudaMemcpyAsync(host_ctl, &w.ctl->level[level % 3u], sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
            SQ_TRY(cudaStreamSynchronize(s));
            if (host_ctl[0] == 0) break;
        }
    // small phase and leaves
    const uint32_t sg = (uint32_t)sms() * 8u;
    launch_subtrees(w, (int)nb, leaf_size, base, nodes, leaf0, s);
    k_emit_leaves<<<sg, 256, 0, s>>>(w.leaves, w.ctl, w.ids_a, w.ids_b, w.tb, nodes, leaf0, err);
    if (grid) k_grid_heap<<<1, 32, 0, s>>>(nodes);
    return (int)cudaGetLastError();
#undef SQ_TRY
}

// Binned SAH trees of M meshes at once, with no host synchronisation (a
// fixed number of large-phase levels with device-side task counts, so the
// sequence can be captured in a CUDA graph).  Mesh m holds triangles
// [off[m], off[m + 1]) of the concatenated `tris` (off on the device, M + 1
// words); its root is record root0 + m, inner records at 2q and 2q + 1 for a
// split at q, leaf records at 2n + 2 + position -- the layout of a single
// build, shifted by the mesh's offset.  Large tasks left after the last
// fixed level go to the small phase (same splits, one warp per subtree).
int build_sah_batch(const float* tris, uint32_t n, const uint32_t* off, uint32_t M, uint32_t nb, uint32_t leaf_size,
                    uint32_t root0, sq::Node* nodes, void* ws, uint32_t* err, cudaStream_t s)
{
    const SahWs w = carve(ws, n, M);
    const uint32_t leaf0 = 2u * n + 2u;
    cudaError_t e;
#define SQ_TRY(x) do { if ((e = (x)) != cudaSuccess) return (int)e; } while (0)
    SQ_TRY(cudaMemsetAsync(w.root_ord, 0, sizeof(uint32_t) * 16ull * M, s));
    SQ_TRY(cudaMemsetAsync(w.ctl, 0, sizeof(Ctl), s));
    const uint32_t sm = (uint32_t)sms();
    if (n > 0) {
        const uint32_t g = min((n + 255) / 256, sm * 8u);
        k_sah_setup_seg<<<g, 256, 0, s>>>(tris, n, off, M, w.tb, w.ids_a, w.root_ord, w.ctl);
    }
    with_chunk(n, [&](auto chunk) {
        constexpr uint32_t CHUNK = decltype(chunk)::value;
        k_root_tasks_seg<CHUNK><<<(M + 3) / 4, 128, 0, s>>>(w.root_ord, off, M, leaf_size, root0, (int)nb, w.lists[0],
                                                            w.parts, w.done());
        enqueue_root_bins<CHUNK>(w, (int)nb, s);
        enqueue_levels<CHUNK>(w, 0, kBatchLargeLevels, (int)nb, 0u, leaf_size, nodes, s);
    });
    launch_subtrees(w, (int)nb, leaf_size, 0u, nodes, leaf0, s);
    k_small_big<<<sm * 8u, 128, 0, s>>>(w.lists[kBatchLargeLevels & 1].tasks, &w.ctl->level[kBatchLargeLevels % 3],
                                        w.ids_a, w.ids_b, w.tb, (int)nb, leaf_size, 0u, nodes, leaf0, err);
    k_emit_leaves<<<sm * 8u, 256, 0, s>>>(w.leaves, w.ctl, w.ids_a, w.ids_b, w.tb, nodes, leaf0, err);
    return (int)cudaGetLastError();
#undef SQ_TRY
}

}  // namespace sqk
