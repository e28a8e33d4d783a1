// The passes around the binner for frames whose launches cost more than their
// work: one kernel that prepares every buffer a flush starts from, and a scan
// and a stable sort of one thread-block cluster each, which exchange through
// distributed shared memory what the library's versions pass through global
// memory and further launches.
#include "rive_cuda_internal.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <mutex>

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
    const uint32_t first = blockIdx.x * blockDim.x + threadIdx.x + chain_wait();
    chain_next();
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
// share (from L1 or L2) writes the offsets. Bound by latency: 7 us for 46 k
// slots, 8.5 for 109 k (cold), in one launch. With the library's scan (two launches, a
// fill and a copy) scan and binner of a 240x180 widget take 25 us, not 18, of a 1080x1080
// recorded feathered frame 27, not 21.
__global__ void __launch_bounds__(1024, 1)
    small_scan_kernel(uint32_t slots,
                      const uint32_t* __restrict__ counts,
                      uint32_t* __restrict__ offsets,
                      uint32_t* __restrict__ hostTotal)
{
    __shared__ uint32_t sums[32];
    __shared__ uint32_t share;
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(), ctas = cluster.num_blocks();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    counts += chain_wait();
    const uint32_t vectors = (slots + 3) / 4;
    const uint32_t per = (vectors + ctas - 1) / ctas;
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
    for (uint32_t r = 0; r < ctas; ++r)
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

// Stable sort of up to small_sort_capacity bin entries by 16-bit tile key, and the
// tiles' ranges, by one cluster: one counting pass per key byte. A warp ranks 32
// entries at a time among equal digits (match), per-warp counters and the
// CTAs' totals give every entry its place; the first pass moves entries through
// the owners' shared memory, the last one writes them out. The number of
// entries is read on the device. When they are more than `capacity`, the binner
// has dropped the rest; `guarded` (a speculative flush, which then runs again)
// leaves every range empty.
// 512 threads and 76 KB a CTA leave room beside another stream's raster; a thread
// holds its up to 16 entries in registers while their places are found. Bound by
// latency and the exchange. Sort and ranges with it and with the library's sort, in seven
// launches and fills: 240x180 widget, 1.9 k entries, 10 and 13 us; 1080x1080 recorded
// feathered frame, 38 k, 19 and 45; 1080x1920 UI screen, 88 k, 27 and 45.
constexpr int kSortThreads = 512, kSortWarps = kSortThreads / 32;
constexpr int kSortItems = 16;
constexpr int kSortStride = kSortWarps + 2; // counters of a digit, padded against bank conflicts
struct SmallSortShared
{
    uint2 items[kSortItems * kSortThreads]; // (key, value)
    uint16_t count[256 * kSortStride];
    uint32_t totals[2][256]; // per pass: this CTA's entries of each digit
    uint32_t base[256];
    uint32_t sums[8];
};

__global__ void __launch_bounds__(kSortThreads)
    small_sort_kernel(const uint32_t* __restrict__ entryTotal,
                      uint32_t capacity,
                      bool guarded,
                      int keyBits,
                      const uint16_t* __restrict__ keys,
                      const uint32_t* __restrict__ vals,
                      uint32_t* __restrict__ sortedVals,
                      TileHead* __restrict__ ranges)
{
    extern __shared__ uint4 dyn[];
    SmallSortShared& sh = *reinterpret_cast<SmallSortShared*>(dyn);
    const uint32_t zero = chain_wait();
    entryTotal += zero;
    keys += zero;
    vals += zero;
    const uint32_t n = min(*entryTotal, capacity);
    if (n == 0 || (guarded && *entryTotal > capacity))
        return; // the whole cluster
    cg::cluster_group cluster = cg::this_cluster();
    const uint32_t rank = cluster.block_rank(), ctas = cluster.num_blocks();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t ltMask = (1u << lane) - 1u;
    // `per` entries a thread: CTA r holds [r chunk, (r + 1) chunk), a warp a run
    // of it, 32 entries a round. Past the last entry: key 0xffff, which sorts
    // behind every tile.
    const uint32_t per = (n + ctas * kSortThreads - 1) / (ctas * kSortThreads);
    const uint32_t chunk = per * kSortThreads, run = (uint32_t)warp * per * 32 + lane;
    const uint32_t perInverse = (65536 + per - 1) / per;
    uint2 item[kSortItems];
#pragma unroll
    for (int r = 0; r < kSortItems; ++r)
    {
        const uint32_t i = rank * chunk + run + 32 * r;
        item[r] = make_uint2(0xffffu, 0u);
        if (r < (int)per && i < n)
            item[r] = make_uint2(keys[i], vals[i]);
    }
    const int passes = keyBits > 8 ? 2 : 1;
    for (int p = 0; p < passes; ++p)
    {
        for (int i = threadIdx.x; i < 256 * kSortStride / 2; i += kSortThreads)
            reinterpret_cast<uint32_t*>(sh.count)[i] = 0;
        if (p)
        {
#pragma unroll
            for (int r = 0; r < kSortItems; ++r)
                if (r < (int)per)
                    item[r] = sh.items[run + 32 * r];
        }
        __syncthreads();
        uint16_t within[kSortItems]; // place among the warp's entries of the digit
#pragma unroll
        for (int r = 0; r < kSortItems; ++r)
        {
            if (r >= (int)per)
                break;
            const uint32_t digit = (item[r].x >> (8 * p)) & 0xffu;
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
        {
            // kParts threads a digit, eight warps' counters each: their prefix
            // within the CTA, and the CTA's total.
            constexpr int kParts = kSortWarps / 8;
            static_assert(kParts * 256 == kSortThreads, "a thread per digit and part");
            const int digit = threadIdx.x / kParts, part = threadIdx.x % kParts;
            uint16_t* const c = sh.count + digit * kSortStride + part * 8;
            uint32_t v[8], sum = 0;
#pragma unroll
            for (int w = 0; w < 8; ++w)
            {
                v[w] = sum;
                sum += c[w];
            }
            uint32_t scan = sum;
#pragma unroll
            for (int o = 1; o < kParts; o <<= 1)
            {
                const uint32_t x = __shfl_up_sync(0xffffffffu, scan, o, kParts);
                scan += part >= o ? x : 0u;
            }
#pragma unroll
            for (int w = 0; w < 8; ++w)
                c[w] = (uint16_t)(v[w] + scan - sum);
            if (part == kParts - 1)
                sh.totals[p][digit] = scan;
        }
        cluster.sync(); // totals are there; every CTA has its entries in registers
        uint32_t before = 0, all = 0, scan = 0;
        if (threadIdx.x < 256)
        {
            for (uint32_t c = 0; c < ctas; ++c)
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
            const uint32_t digit = (item[r].x >> (8 * p)) & 0xffu;
            const uint32_t to = sh.base[digit] + sh.count[digit * kSortStride + warp] + within[r];
            const uint32_t owner = ((to / kSortThreads) * perInverse) >> 16;
            *cluster.map_shared_rank(&sh.items[to - owner * chunk], owner) = item[r];
        }
        cluster.sync(); // entries are where the next pass, or the ranges, read them
    }
    for (uint32_t j = threadIdx.x; j < chunk; j += kSortThreads)
    {
        const uint32_t i = rank * chunk + j;
        if (i >= n)
            break;
        const uint2 e = sh.items[j];
        sortedVals[i] = e.y;
        const uint32_t prev = j ? sh.items[j - 1].x
                              : i ? cluster.map_shared_rank(&sh.items[chunk - 1], rank - 1)->x
                                  : 0xffffu;
        if (prev != e.x)
        {
            ranges[e.x].first = i;
            if (prev != 0xffffu)
                ranges[prev].end = i;
        }
        if (i == n - 1)
            ranges[e.x].end = n;
    }
    cluster.sync(); // no CTA leaves while the next one reads its last key
}

namespace
{
template <typename... P, typename... A>
cudaError_t launch_cluster(void (*kernel)(P...), uint32_t ctas, int threads, size_t smem,
                           cudaStream_t stream, bool overlap, const A&... args)
{
    cudaLaunchAttribute attr[2] = {};
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = ctas;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c = {};
    c.gridDim = dim3(ctas);
    c.blockDim = dim3(threads);
    c.dynamicSmemBytes = smem;
    c.stream = stream;
    c.attrs = attr;
    c.numAttrs = overlap ? 2 : 1;
    return cudaLaunchKernelEx(&c, kernel, P(args)...);
}

// CTAs of a cluster for `items` of work at `perCta` each: the smallest cluster
// (lower latency: a 240x180 widget 41 us, 42 with 16) where it has room for a few
// rounds, the device's largest above (38 k entries sorted by 16 CTAs 20 us, by 8 24).
uint32_t cluster_for(uint32_t items, uint32_t perCta, uint32_t largest)
{
    return items <= 8 * perCta ? std::min(8u, largest) : largest;
}
} // namespace

cudaError_t small_passes_init(int device, uint32_t* largest)
{
    static std::mutex m;
    static uint32_t found[64] = {};
    std::lock_guard<std::mutex> lock(m);
    if (device < 0 || device >= 64)
        return cudaErrorInvalidDevice;
    if (!found[device])
    {
        // 16 CTAs need a GPC with as many free SMs (not every partition of the
        // device has one); 8 are portable.
        cudaError_t e = cudaFuncSetAttribute(
            small_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, sizeof(SmallSortShared));
        for (auto fn : {(const void*)small_sort_kernel, (const void*)small_scan_kernel})
            if (e == cudaSuccess)
                e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        if (e != cudaSuccess)
            return e;
        cudaLaunchAttribute attr = {};
        attr.id = cudaLaunchAttributeClusterDimension;
        attr.val.clusterDim.x = 16;
        attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
        cudaLaunchConfig_t c = {};
        c.gridDim = dim3(16);
        c.attrs = &attr;
        c.numAttrs = 1;
        int sorts = 0, scans = 0;
        c.blockDim = dim3(kSortThreads);
        c.dynamicSmemBytes = sizeof(SmallSortShared);
        e = cudaOccupancyMaxActiveClusters(&sorts, small_sort_kernel, &c);
        c.blockDim = dim3(1024);
        c.dynamicSmemBytes = 0;
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveClusters(&scans, small_scan_kernel, &c);
        if (e != cudaSuccess)
            cudaGetLastError(); // a failed query only leaves the portable size
        found[device] = e == cudaSuccess && sorts > 0 && scans > 0 ? 16 : 8;
    }
    *largest = found[device];
    return cudaSuccess;
}

uint32_t small_sort_capacity(uint32_t largest) { return largest * kSortThreads * kSortItems; }

cudaError_t launch_small_scan(uint32_t largest, uint32_t slots, const uint32_t* counts,
                              uint32_t* offsets, uint32_t* hostTotal, cudaStream_t stream,
                              bool overlap)
{
    return launch_cluster(small_scan_kernel, cluster_for(slots, 8192, largest), 1024, 0, stream,
                          overlap, slots, counts, offsets, hostTotal);
}

cudaError_t launch_small_sort(uint32_t largest, uint32_t entries, const uint32_t* entryTotal,
                              bool guarded, int keyBits, const uint16_t* keys, const uint32_t* vals,
                              uint32_t* sortedVals, TileHead* ranges, cudaStream_t stream,
                              bool overlap)
{
    return launch_cluster(small_sort_kernel, cluster_for(entries, 2048, largest), kSortThreads,
                          sizeof(SmallSortShared), stream, overlap, entryTotal, entries, guarded, keyBits, keys,
                          vals, sortedVals, ranges);
}
} // namespace rivecuda
