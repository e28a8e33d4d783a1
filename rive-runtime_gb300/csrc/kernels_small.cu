// The passes around the binner for frames whose launches cost more than their
// work: one kernel that prepares every buffer a flush starts from, and a scan
// and a stable sort of one thread-block cluster each, which exchange through
// distributed shared memory what the library's versions pass through global
// memory and further launches.
#include "rive_cuda_internal.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace rivecuda
{
// FlushUniforms fields the passes use (gpu.hpp:1466-1537: pathIDGranularity
// at byte 72, ditherScale at 88, ditherBias at 92), read on the device so no
// pass waits for the host, one thread per flush of the batch; and what must
// start at zero: the gradient texture (texels no span covers are never sampled;
// zeroed so the texture is deterministic), the tile heads, the wide triangles'
// counter. One launch in the place of four.
__global__ void __launch_bounds__(256) flush_start_kernel(FlushStart F)
{
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t stride = gridDim.x * blockDim.x;
    for (uint32_t i = first; i < F.sceneCount; i += stride)
    {
        FlushParams& P = F.scenes[i];
        const uint8_t* u = P.uniforms;
        const uint32_t granularity = *reinterpret_cast<const uint32_t*>(u + 72);
        P.pathIDGranularity = granularity ? granularity : 1u;
        P.ditherScale = *reinterpret_cast<const float*>(u + 88);
        P.ditherBias = *reinterpret_cast<const float*>(u + 92);
        P.mipLodBias = *reinterpret_cast<const float*>(u + 80);
    }
    if (first == 0 && F.wide)
        *F.wide = 0;
    if (first == 0 && F.error)
        *F.error = 0;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    for (uint32_t i = first; i < F.gradVectors; i += stride)
        F.grad[i] = zero;
    for (uint32_t i = first; i < F.tiles; i += stride)
    {
        const uint32_t scene = find_range(F.tileBase, F.sceneCount, i);
        const uint2 st = F.sceneTiles[scene]; // (tileBase, tilesX)
        const uint32_t y = (i - st.x) / st.y;
        F.ranges[i] = TileHead{0u, 0u, scene, (i - st.x - y * st.y) | (y << 16)};
    }
}

// Exclusive scan of up to kSmallScanSlots tile counts (offsets[slots] = the
// total, also stored where the host reads it), by one cluster: each CTA sums
// its share, the CTAs before it give it its start, and a second walk over the
// share (from L1 or L2) writes the offsets. Bound by latency: 5 us for 115 k
// slots, against 8 us and two launches of a decoupled look-back scan.
__global__ void __cluster_dims__(kSmallCluster, 1, 1) __launch_bounds__(1024, 1)
    small_scan_kernel(uint32_t slots,
                      const uint32_t* __restrict__ counts,
                      uint32_t* __restrict__ offsets,
                      uint32_t* __restrict__ hostTotal)
{
    __shared__ uint32_t sums[32];
    __shared__ uint32_t share;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t vectors = (slots + 3) / 4;
    const uint32_t per = (vectors + kSmallCluster - 1) / kSmallCluster;
    const uint32_t lo = min(rank * per, vectors), hi = min(lo + per, vectors);
    auto load = [&](uint32_t v) {
        if (4 * v + 4 <= slots)
            return reinterpret_cast<const uint4*>(counts)[v];
        uint4 c = make_uint4(0u, 0u, 0u, 0u);
        c.x = counts[4 * v];
        if (4 * v + 1 < slots)
            c.y = counts[4 * v + 1];
        if (4 * v + 2 < slots)
            c.z = counts[4 * v + 2];
        return c;
    };
    uint32_t total = 0;
    for (uint32_t v = lo + threadIdx.x; v < hi; v += 1024)
    {
        const uint4 c = load(v);
        total += c.x + c.y + c.z + c.w;
    }
    total = __reduce_add_sync(0xffffffffu, total);
    if (lane == 0)
        sums[warp] = total;
    __syncthreads();
    if (warp == 0)
    {
        const uint32_t t = __reduce_add_sync(0xffffffffu, sums[lane]);
        if (lane == 0)
            share = t;
    }
    cluster.sync();
    uint32_t before = 0, all = 0;
    for (uint32_t r = 0; r < kSmallCluster; ++r)
    {
        const uint32_t t = *cluster.map_shared_rank(&share, r);
        before += r < rank ? t : 0u;
        all += t;
    }
    if (rank == 0 && threadIdx.x == 0)
    {
        offsets[slots] = all;
        if (hostTotal)
            *hostTotal = all;
    }
    for (uint32_t v0 = lo; v0 < hi; v0 += 1024)
    {
        const uint32_t v = v0 + threadIdx.x;
        const uint4 c = v < hi ? load(v) : make_uint4(0u, 0u, 0u, 0u);
        const uint32_t mine = c.x + c.y + c.z + c.w;
        uint32_t scan = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1)
        {
            const uint32_t x = __shfl_up_sync(0xffffffffu, scan, o);
            scan += lane >= o ? x : 0u;
        }
        __syncthreads(); // the last round's sums are read
        if (lane == 31)
            sums[warp] = scan;
        __syncthreads();
        const uint32_t w = sums[lane];
        const uint32_t at = before + __reduce_add_sync(0xffffffffu, lane < warp ? w : 0u) + scan - mine;
        before += __reduce_add_sync(0xffffffffu, w);
        if (v < hi)
        {
            const uint4 o = make_uint4(at, at + c.x, at + c.x + c.y, at + c.x + c.y + c.z);
            if (4 * v + 4 <= slots)
            {
                reinterpret_cast<uint4*>(offsets)[v] = o;
            }
            else
            {
                offsets[4 * v] = o.x;
                if (4 * v + 1 < slots)
                    offsets[4 * v + 1] = o.y;
                if (4 * v + 2 < slots)
                    offsets[4 * v + 2] = o.z;
            }
        }
    }
    cluster.sync(); // no CTA leaves while another reads its share
}

// Stable sort of up to kSmallSortEntries bin entries by 16-bit tile key, and the
// tiles' ranges, by one cluster: one counting pass per key byte. A warp ranks 32
// entries at a time among equal digits (match), per-warp counters and the
// CTAs' totals give every entry its place; the first pass moves entries through
// the owners' shared memory, the last one writes them out. The number of
// entries is read on the device. When they are more than `capacity`, the binner
// has dropped the rest; `guarded` (a speculative flush, which then runs again)
// leaves every range empty.
// Bound by latency: 50 k entries in 12 us, against 45 us and seven launches and
// fills for the library's sort and a pass for the ranges.
constexpr int kSortWarps = 32, kSortItems = kSmallSortEntries / (kSmallCluster * 1024);
constexpr int kSortStride = kSortWarps + 2; // counters of a digit, padded against bank conflicts
struct SmallSortShared
{
    uint32_t vals[kSortItems * 1024];
    uint16_t keys[kSortItems * 1024];
    uint16_t count[256 * kSortStride];
    uint32_t totals[2][256]; // per pass: this CTA's entries of each digit
    uint32_t base[256];
    uint32_t sums[8];
};
static_assert(sizeof(SmallSortShared) <= kSmallSortSmemBytes, "kSmallSortSmemBytes");

__global__ void __cluster_dims__(kSmallCluster, 1, 1) __launch_bounds__(1024, 1)
    small_sort_kernel(const uint32_t* __restrict__ entryTotal,
                      uint32_t capacity,
                      bool guarded,
                      int keyBits,
                      const uint16_t* __restrict__ keys,
                      const uint32_t* __restrict__ vals,
                      uint16_t* __restrict__ sortedKeys,
                      uint32_t* __restrict__ sortedVals,
                      TileHead* __restrict__ ranges)
{
    extern __shared__ uint4 dyn[];
    SmallSortShared& sh = *reinterpret_cast<SmallSortShared*>(dyn);
    const uint32_t n = min(*entryTotal, capacity);
    if (n == 0 || (guarded && *entryTotal > capacity))
        return; // the whole cluster
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t ltMask = (1u << lane) - 1u;
    // `per` entries a thread: CTA r holds [r chunk, (r + 1) chunk), a warp a run
    // of it, 32 entries a round. Past the last entry: key 0xffff, which sorts
    // behind every tile.
    const uint32_t per = (n + kSmallCluster * 1024 - 1) / (kSmallCluster * 1024);
    const uint32_t chunk = per * 1024, run = (uint32_t)warp * per * 32 + lane;
    const uint32_t perInverse = (65536 + per - 1) / per;
    const int passes = keyBits > 8 ? 2 : 1;
    for (int p = 0; p < passes; ++p)
    {
        const bool last = p + 1 == passes;
        for (int i = threadIdx.x; i < 256 * kSortStride / 2; i += 1024)
            reinterpret_cast<uint32_t*>(sh.count)[i] = 0;
        __syncthreads();
        auto key_of = [&](uint32_t r) -> uint32_t {
            const uint32_t i = run + 32 * r;
            if (p)
                return sh.keys[i];
            return rank * chunk + i < n ? keys[rank * chunk + i] : 0xffffu;
        };
        uint16_t within[kSortItems]; // place among the warp's entries of the digit
#pragma unroll
        for (int r = 0; r < kSortItems; ++r)
        {
            if (r >= (int)per)
                break;
            const uint32_t digit = (key_of(r) >> (8 * p)) & 0xffu;
            volatile uint16_t* const c = sh.count + digit * kSortStride + warp;
            const uint32_t peers = __match_any_sync(0xffffffffu, digit);
            const uint32_t old = *c;
            within[r] = (uint16_t)(old + __popc(peers & ltMask));
            __syncwarp();
            if (!(peers & ltMask))
                *c = (uint16_t)(old + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        if (threadIdx.x < 256)
        {
            uint32_t sum = 0;
            for (int w = 0; w < kSortWarps; ++w)
            {
                uint16_t* const c = sh.count + threadIdx.x * kSortStride + w;
                const uint32_t v = *c;
                *c = (uint16_t)sum;
                sum += v;
            }
            sh.totals[p][threadIdx.x] = sum;
        }
        cluster.sync();
        uint32_t before = 0, all = 0, scan = 0;
        if (threadIdx.x < 256)
        {
            for (uint32_t c = 0; c < kSmallCluster; ++c)
            {
                const uint32_t t = *cluster.map_shared_rank(&sh.totals[p][threadIdx.x], c);
                before += c < rank ? t : 0u;
                all += t;
            }
            scan = all;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1)
            {
                const uint32_t x = __shfl_up_sync(0xffffffffu, scan, o);
                scan += lane >= o ? x : 0u;
            }
            if (lane == 31)
                sh.sums[warp] = scan;
        }
        __syncthreads();
        if (threadIdx.x < 256)
        {
            const uint32_t earlier =
                __reduce_add_sync(0xffffffffu, lane < warp ? sh.sums[lane & 7] : 0u);
            sh.base[threadIdx.x] = earlier + scan - all + before;
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSortItems; ++r)
        {
            if (r >= (int)per)
                break;
            const uint32_t i = run + 32 * r;
            const uint32_t key = key_of(r), digit = (key >> (8 * p)) & 0xffu;
            const uint32_t to = sh.base[digit] + sh.count[digit * kSortStride + warp] + within[r];
            if (last)
            {
                if (key != 0xffffu)
                {
                    sortedKeys[to] = (uint16_t)key;
                    sortedVals[to] = p ? sh.vals[i] : vals[rank * chunk + i];
                }
            }
            else
            {
                const uint32_t owner = ((to >> 10) * perInverse) >> 16, at = to - owner * chunk;
                *cluster.map_shared_rank(&sh.keys[at], owner) = (uint16_t)key;
                if (key != 0xffffu)
                    *cluster.map_shared_rank(&sh.vals[at], owner) = vals[rank * chunk + i];
            }
        }
        cluster.sync(); // entries are where the next pass, or the ranges, read them
    }
    for (uint32_t i = rank * 1024 + threadIdx.x; i < n; i += kSmallCluster * 1024)
    {
        const uint32_t k = __ldcg(sortedKeys + i);
        if (i == 0 || __ldcg(sortedKeys + i - 1) != k)
            ranges[k].first = i;
        if (i == n - 1 || __ldcg(sortedKeys + i + 1) != k)
            ranges[k].end = i + 1;
    }
}
} // namespace rivecuda
