// sq_coherent.cu -- the reference's packet and bundle tracers on the GPU.
//
// trace_packet<k> (src/tracer.cpp:232-281, traverse_packet_stack 88-123):
// the k = kx * ky rays of a kx x ky pixel block (kx = floor(sqrt(k)), rays in
// row order) traverse together: a node's children are visited when any ray
// of the packet hits the node's box, and the packet counts one test per node
// box.  Every pixel of the packet gets (tests / k) / 200 in the heatmap.  On
// the GPU a warp walks 4 to 32 packets from one pool (sq_walk_dev.cuh): a lane
// tests a node against the rays of the packet that visits it.
//
// trace_bundle<k> (src/tracer.cpp:292-362, traverse_bundle 126-156,
// intersect_bundle_aabb src/tracer.h:37-80): a tile of k = 16 or 64 rays
// (tw x th pixels, tw = floor(sqrt(k))), ray m * 8 + n at tile position
// morton_lut[m * 8 + n], is tested as one bundle against the box with the
// bundle's direction bounds (min, max and midpoint) while the midpoint
// direction hits; where only the bounds can hit, each packet of 8 rays
// continues alone from that node (the packet tracer above).  A pixel of
// packet m gets bundle_tests / k + packet_tests[m] / 8.  A warp walks two
// tiles of 16 rays or one of 64 from one pool, their bundles and packets
// together.
//
// Both counts are independent of the visiting order (nothing terminates
// early), so the stack order need not be the reference's.  The heatmap bytes
// are the reference's exactly.
#include "sq_common.cuh"
#include "sq_walk_dev.cuh"

#include <algorithm>
#include <array>

namespace {

using namespace sq;

// Packets of one warp's pool (sq_walk_dev.cuh).  Four are enough that the pool
// holds a range for every lane most of the time and few enough that the warps
// of a small image or a deep tree end together; an image of many packets in a
// small tree wants 32, since a packet is then soon done and fetching it, its
// rays and the pool's start are what costs.  So above kFewPackets packets a
// resident warp, each takes a share of what is left, from 32 down to 4
// packets; the larger the tree (the longer the packets), the smaller the share
// (packet_share).  1920x1072, packets of 1 / 2 / 4 / 8 rays, us with four each
// time and with shares:
//   200 triangles     355 / 199 / 116 /  80     79 /  59 /  56 /  56
//   1,500             361 / 202 / 118 /  86     86 /  75 /  80 /  76
//   30,000            373 / 212 / 134          138 / 110 / 104
//   2M                581 / 412 / 387          490 / 395 / 376
// Packets of 8, which take longest, have shares in small trees only: in larger
// ones they gain at 3840x2160 (20,000 triangles 338 and 283 us) and lose below
// (1920x1072 126 and 133; 2M at 3840x2160 929 and 1,054).
constexpr int kPoolPackets = 4, kManyPackets = 32;
constexpr uint32_t kFewPackets = 16;
constexpr uint32_t kSmallTree = 4096, kMediumTree = 1u << 15;
uint32_t packet_share(uint32_t tris) { return tris < kSmallTree ? 4u : (tris < kMediumTree ? 8u : 16u); }

// share: a warp takes 1 / share of the packets left, kPoolPackets to PW of them
template <int K, int PW>
__global__ void __launch_bounds__(32) k_trace_packet(const sqk::TraceArgs a, uint32_t share)
{
    constexpr int KX = (K == 1 || K == 2) ? 1 : 2;  // floor(sqrt(k))
    constexpr int KY = K / KX;
    __shared__ WalkPool<K, PW, false> pool;
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t bw = a.width / KX;
    const uint32_t total = bw * (a.height / KY);
    const float org[3] = {a.cam[0], a.cam[1], a.cam[2]};
    uint64_t tests_sum = 0;
    uint32_t base = 0;
    for (;;) {
        const uint32_t take = PW == kPoolPackets ? (uint32_t)PW
                                                 : min(max((total - base) / share, (uint32_t)kPoolPackets), (uint32_t)PW);
        if (lane == 0) base = atomicAdd(a.work, take);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= total) break;
        const uint32_t count = min(take, total - base);
        // ray m of packet p: pixel (m % KX, m / KX) of the packet's block
        for (uint32_t j = lane; j < count * K; j += 32) {
            const uint32_t p = j / K, m = j % K, pk = base + p;
            Ray r;
            gen_reference_camera((pk % bw) * KX + m % KX, (pk / bw) * KY + m / KX, a.width, a.height, a.cam, r);
#pragma unroll
            for (int c = 0; c < 3; ++c) pool.inv[c][m][p] = 1.0f / r.d[c];
        }
        WalkStats st = {0u, false, false};
        walk_pool(pool, count >= 32u ? 0xFFFFFFFFu : (1u << count) - 1u, a.nodes, a.node_count, a.tri_count,
                                a.root, 1u, org, st, [](uint32_t, const float*, const float*) { return false; });
        if (st.overflow || st.bad) raise_error(a.err, SQ_DEVERR_STACK_OVERFLOW);
        for (uint32_t j = lane; j < count * K; j += 32) {
            const uint32_t p = j / K, m = j % K, pk = base + p;
            const uint32_t x = (pk % bw) * KX + m % KX, y = (pk / bw) * KY + m / KX;
            write_heat(a.heat + 3ull * ((size_t)y * a.width + x), (float)pool.cnt[p] / (float)K, a.heat_ramp);
        }
        if (lane < count) tests_sum += pool.cnt[lane];
        __syncwarp();  // the pool is used again for the warp's next packets
    }
    if (a.stats) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tests_sum += __shfl_xor_sync(0xFFFFFFFFu, tests_sum, o);
        if (lane == 0) atomicAdd(a.stats, (unsigned long long)tests_sum);
    }
}

template <int K>
void launch_packets(const sqk::TraceArgs& a, cudaStream_t s)
{
    static PerDevice<std::array<int, 2>> cache;
    const std::array<int, 2> per_sm = cache.get([] {
        return std::array<int, 2>{blocks_per_sm(k_trace_packet<K, kPoolPackets>, 32),
                                  blocks_per_sm(k_trace_packet<K, kManyPackets>, 32)};
    });
    const uint64_t packets = (uint64_t)a.width * a.height / K;
    const uint32_t many = (uint32_t)(per_sm[1] * sm_count());
    if (packets > (uint64_t)kFewPackets * many && (K < 8 || a.tri_count < kSmallTree)) {
        k_trace_packet<K, kManyPackets><<<many, 32, 0, s>>>(a, many * packet_share(a.tri_count));
        return;
    }
    const uint64_t need = (packets + kPoolPackets - 1) / kPoolPackets;
    const uint32_t grid = (uint32_t)(per_sm[0] * sm_count());
    k_trace_packet<K, kPoolPackets><<<(uint32_t)std::min<uint64_t>(grid, need ? need : 1), 32, 0, s>>>(a, 1u);
}

// morton_lut (src/tracer.cpp:18-23): k with bits 1 and 2 exchanged
__device__ __forceinline__ uint32_t bundle_lut(uint32_t k) { return (k & ~6u) | ((k & 2u) << 1) | ((k & 4u) >> 1); }

// Bundles of one warp's pool: one of 64 rays is eight packets already (two:
// 300k terrain at 1280x720, build included, 970 us against 635), of 16 rays
// one, two, three and four took 436, 454, 540 and 610 us there and 935, 833,
// 838 and 858 us on a 300k soup at 1920x1072.  A bundle at a time, its walk
// repeated on every lane, took 1774 us (64 rays) and 1049 us (16) on the
// terrain.
template <int K>
constexpr int kPoolBundles = K == 16 ? 2 : 1;

template <int K>
__global__ void __launch_bounds__(32) k_trace_bundle(const sqk::TraceArgs a)
{
    constexpr int TW = (K == 16) ? 4 : 8;  // floor(sqrt(k))
    constexpr int TH = K / TW;
    constexpr int NB = kPoolBundles<K>, PK = K / 8, PW = NB * PK;
    __shared__ WalkPool<8, PW, false, NB> pool;
    __shared__ float s_d[3][NB][K];
    const uint32_t lane = threadIdx.x & 31u;
    const uint32_t tiles_x = a.width / TW;
    const uint32_t total = tiles_x * (a.height / TH);
    const float org[3] = {a.cam[0], a.cam[1], a.cam[2]};
    uint64_t tests_sum = 0;
    for (;;) {
        uint32_t base = 0;
        if (lane == 0) base = atomicAdd(a.work, (uint32_t)NB);
        base = __shfl_sync(0xFFFFFFFFu, base, 0);
        if (base >= total) break;
        const uint32_t count = min((uint32_t)NB, total - base);
        // ray r of bundle g: packet r / 8, pixel bundle_lut(r) of the tile
        for (uint32_t j = lane; j < count * K; j += 32) {
            const uint32_t g = j / K, r = j % K, tile = base + g, v = bundle_lut(r);
            Ray ray;
            gen_reference_camera((tile % tiles_x) * TW + v % TW, (tile / tiles_x) * TH + v / TW, a.width, a.height,
                                 a.cam, ray);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                s_d[c][g][r] = ray.d[c];
                pool.inv[c][r % 8][g * PK + r / 8] = 1.0f / ray.d[c];
            }
        }
        __syncwarp();
        // the bundle's direction bounds, accumulated in ray order as the
        // reference does (src/tracer.cpp:331-336)
        if (lane < 3u * count) {
            const uint32_t g = lane / 3u, c = lane % 3u;
            float dmin = FLT_MAX, dmax = -FLT_MAX;
            for (int r = 0; r < K; ++r) {
                dmin = ref_min(dmin, s_d[c][g][r]);
                dmax = ref_max(dmax, s_d[c][g][r]);
            }
            pool.bun[c][g] = 1.0f / dmin;
            pool.bun[3 + c][g] = 1.0f / dmax;
            pool.bun[6 + c][g] = 1.0f / ((dmin + dmax) * 0.5f);
        }
        WalkStats st = {0u, false, false};
        walk_pool(pool, ((1u << count) - 1u) << PW, a.nodes, a.node_count, a.tri_count, a.root, 1u, org, st,
                  [](uint32_t, const float*, const float*) { return false; });
        if (st.overflow || st.bad) raise_error(a.err, SQ_DEVERR_STACK_OVERFLOW);
        for (uint32_t j = lane; j < count * K; j += 32) {
            const uint32_t g = j / K, r = j % K, tile = base + g, v = bundle_lut(r);
            const uint32_t x = (tile % tiles_x) * TW + v % TW, y = (tile / tiles_x) * TH + v / TW;
            const float t = (float)pool.cnt[PW + g] / (float)K + (float)pool.cnt[g * PK + r / 8] / 8.0f;
            write_heat(a.heat + 3ull * ((size_t)y * a.width + x), t, a.heat_ramp);
        }
        if (lane < count * PK) tests_sum += pool.cnt[lane];
        if (lane < count) tests_sum += pool.cnt[PW + lane];
        __syncwarp();  // the pool is used again for the warp's next bundles
    }
    if (a.stats) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) tests_sum += __shfl_xor_sync(0xFFFFFFFFu, tests_sum, o);
        if (lane == 0) atomicAdd(a.stats, (unsigned long long)tests_sum);
    }
}

template <int K>
void launch_bundles(const sqk::TraceArgs& a, cudaStream_t s)
{
    static PerDevice<int> cache;
    const uint32_t grid = (uint32_t)(cache.get([] { return blocks_per_sm(k_trace_bundle<K>, 32); }) * sm_count());
    const uint64_t tiles = (uint64_t)a.width * a.height / K, need = (tiles + kPoolBundles<K> - 1) / kPoolBundles<K>;
    k_trace_bundle<K><<<(uint32_t)std::min<uint64_t>(grid, need ? need : 1), 32, 0, s>>>(a);
}

}  // namespace

namespace sqk {

bool coherent_shape_ok(uint32_t bundle, uint32_t k, uint32_t w, uint32_t h)
{
    if (bundle) {
        if (k != 16 && k != 64) return false;
        const uint32_t tw = k == 16 ? 4u : 8u;
        return w % tw == 0 && h % (k / tw) == 0;
    }
    if (k != 1 && k != 2 && k != 4 && k != 8) return false;
    const uint32_t kx = k <= 2 ? 1u : 2u;
    return w % kx == 0 && h % (k / kx) == 0;
}

void trace_coherent(const TraceArgs& a, uint32_t bundle, uint32_t k, cudaStream_t s)
{
    if (bundle) {
        if (k == 16) launch_bundles<16>(a, s);
        else launch_bundles<64>(a, s);
        return;
    }
    switch (k) {
    case 1: launch_packets<1>(a, s); break;
    case 2: launch_packets<2>(a, s); break;
    case 4: launch_packets<4>(a, s); break;
    default: launch_packets<8>(a, s); break;
    }
}

}  // namespace sqk
