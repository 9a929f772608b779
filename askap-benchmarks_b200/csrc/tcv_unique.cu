// tcv_unique.cu -- binning of variable-width plans by distinct footprint.
//
// Samples of a track repeat footprints: a baseline moves by less than an oversampling step between
// many of its integrations, so several samples have the same first column and row, table offset and
// width (the 12 h track of current/tConvolveMPI/Benchmark.cc:61-165: 3.83 M samples have 0.93 M
// distinct footprints in the spectral run, 5.44 M have 1.57 M in the continuum run).  Gridding is
// linear in the data, so a footprint is gridded once with the sum of its samples' data, and
// degridding gives all its samples one value.  Plans of many samples whose both passes are
// sample-parallel are binned so (kUniqSamples); the passes then work on footprints ("uniques", numbered 0 .. n_uniq - 1) where they
// worked on samples.
//
// One radix sort orders the samples by (work cell of the footprint's first point, table offset, row
// and column in the tile, width), which is the footprint, so equal footprints are neighbours (in
// sample order: the sort is stable) and a scan numbers them.  There is no sort of (sample, tile)
// pairs (15 per sample in the continuum run, most of them fillers): a cell's list is gathered from the
// first-point cells whose footprints can reach it, which are contiguous in the sorted order; a
// counting pass sizes the lists, a second writes them.  Within a cell footprints of one kernel are
// neighbours, so their table entries are read from L1.
// No atomics on sums, the same order on every run.
// Measured (all samples, c64): spectral gridding 0.910 -> 0.338 ms, degridding 0.784 -> 0.290 ms, continuum
// gridding 3.50 -> 1.98 ms, degridding 3.41 -> 1.63 ms; binning 0.46 -> 0.63 ms (spectral) and, with the
// pairs of 15 tiles a sample no longer sorted, 1.64 -> 1.00 ms (continuum).
#include "tcv_internal.cuh"

#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <thrust/iterator/counting_iterator.h>
#include <thrust/iterator/transform_iterator.h>

#include <algorithm>

namespace tcv {
namespace {

constexpr int kTX = 6, kTY = 5;  // log2 of the tile sides (64 x 32 tiles of 8-row plans)
static_assert((1 << kTX) == kTileW && (1 << kTY) == tile_height(8), "key fields");
constexpr uint32_t kNone = 0xffffffffu;

// The samples of one footprint are summed in order by one thread, so a footprint of more than this is taken
// as several: a sorted sample at a multiple of it starts another.  Gridding 2^18 samples of one footprint took
// 9.8 ms and was 1.7e-5 off (relative L2), 2^20 39 ms; now 0.17 each and within 1e-5; the tracks' sums cost
// the same.
constexpr uint32_t kRun = 512;

struct Head {  // 1 where a footprint starts (fillers of left-out samples: 0)
    const uint64_t* keys;
    uint64_t sentinel;
    __host__ __device__ __forceinline__ uint32_t operator()(uint32_t i) const
    {
        const uint64_t k = keys[i];
        return k < sentinel && (i % kRun == 0 || keys[i - 1] != k) ? 1u : 0u;
    }
};

__global__ void uniq_keys_kernel(PlanGeom g, const int32_t* __restrict__ iu, const int32_t* __restrict__ iv,
                                 const int32_t* __restrict__ coff, const int32_t* __restrict__ wplane,
                                 const int32_t* __restrict__ plane_s, const int32_t* __restrict__ plane_grp,
                                 const int32_t* __restrict__ plane_rank, uint64_t* keys, uint32_t* vals,
                                 unsigned long long* rejected)
{
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= g.n) return;
    const int plane = wplane[k];
    const bool plane_ok = plane >= 0 && plane < g.n_planes;
    const int64_t s = plane_ok ? plane_s[plane] : 1;
    const int64_t fx = (int64_t)iu[k] - s / 2, fy = iv[k], co = coff[k];
    const bool ok = plane_ok && fx >= 0 && fx + s <= g.g_size && fy >= 0 && fy + s <= g.g_size && co >= 0 &&
                    co + s * s <= g.c_len;
    vals[k] = uint32_t(k);
    if (!ok) {
        atomicAdd(rejected, 1ull);
        keys[k] = uint64_t(1) << g.u_bits;
        return;
    }
    const uint64_t cell = uint64_t(plane_grp[plane]) * uint64_t(g.ntiles) + uint64_t(fy >> kTY) * uint64_t(g.ntx) +
                          uint64_t(fx >> kTX);
    uint64_t key = cell << g.u_coff_bits | uint64_t(co);
    key = key << (kTY + kTX) | uint64_t(fy & ((1 << kTY) - 1)) << kTX | uint64_t(fx & ((1 << kTX) - 1));
    keys[k] = key << g.u_rank_bits | uint64_t(plane_rank[plane]);
}

// Per sorted sample: its footprint's number; per footprint (its first sample): the record, the tiles
// it touches (counted per cell: whole numbers, so in any order; neighbours share cells, so a warp
// adds each cell once), where its samples start; per first-point cell: its footprints.
__global__ void uniq_records_kernel(PlanGeom g, const uint64_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                                    const uint32_t* __restrict__ usum, const int32_t* __restrict__ iu,
                                    const int32_t* __restrict__ iv, const int32_t* __restrict__ coff,
                                    const int32_t* __restrict__ wplane, const int32_t* __restrict__ plane_s, int4* urec,
                                    uint32_t* ustart, uint32_t* repu, uint16_t* ntl, uint32_t* count,
                                    uint32_t* cell_first, uint32_t* cell_end, uint32_t* n_uniq)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    const uint64_t sentinel = uint64_t(1) << g.u_bits, key = i < g.n ? keys[i] : sentinel;
    const uint32_t k = i < g.n ? vals[i] : 0u;
    if (i < g.n && key >= sentinel) repu[k] = kNone;
    const int shift = g.u_coff_bits + kTY + kTX + g.u_rank_bits;
    uint32_t cell = 0;
    int nx = 0, ny = 0;  // tiles of a footprint that starts here
    if (key < sentinel) {
        const uint32_t u = usum[i] - 1u;
        repu[k] = u;
        cell = uint32_t(key >> shift);
        const uint64_t before = i ? keys[i - 1] : sentinel, after = i + 1 < g.n ? keys[i + 1] : sentinel;
        if (before != key || i % kRun == 0) {  // as Head has it
            const int s = plane_s[wplane[k]], fx = iu[k] - s / 2, fy = iv[k];
            urec[u] = make_int4(fx, fy, coff[k], s);
            ustart[u] = uint32_t(i);
            nx = ((fx + s - 1) >> kTX) - (fx >> kTX) + 1;
            ny = ((fy + s - 1) >> kTY) - (fy >> kTY) + 1;
            ntl[u] = uint16_t(nx * ny);
            if (i == 0 || uint32_t(before >> shift) != cell) cell_first[cell] = u;
        }
        if (after >= sentinel || uint32_t(after >> shift) != cell) cell_end[cell] = u + 1u;
        if (after >= sentinel) {
            ustart[u + 1u] = uint32_t(i + 1);
            *n_uniq = u + 1u;
        }
    }
    const int most = __reduce_max_sync(0xffffffffu, nx * ny);
    for (int t = 0; t < most; ++t) {
        const bool has = t < nx * ny;
        const uint32_t c = has ? cell + uint32_t(t / nx) * uint32_t(g.ntx) + uint32_t(t % nx) : kNone;
        const uint32_t same = __match_any_sync(0xffffffffu, c);
        if (has && (threadIdx.x & 31) == __ffs(same) - 1) atomicAdd(&count[c], uint32_t(__popc(same)));
    }
}

// One CTA per cell (strided): the cell's list, the footprints that reach it from the first-point cells
// up to reach_x, reach_y tiles before it, in that order.
template <int kThreads>
__global__ void __launch_bounds__(kThreads)
uniq_lists_kernel(PlanGeom g, uint32_t cells, int reach_x, int reach_y, const int4* __restrict__ urec,
                  const uint32_t* __restrict__ cell_first, const uint32_t* __restrict__ cell_end,
                  const uint32_t* __restrict__ start, uint32_t* tile_end, uint32_t* order, int4* grec)
{
    constexpr int kWarps = kThreads / 32;
    __shared__ uint32_t ws[2][kWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    int par = 0;
    for (uint32_t c = blockIdx.x; c < cells; c += gridDim.x) {
        const uint32_t grp = c / uint32_t(g.ntiles), t = c % uint32_t(g.ntiles);
        const int tx = int(t % uint32_t(g.ntx)), ty = int(t / uint32_t(g.ntx));
        uint32_t at = start[c];
        for (int dy = 0; dy <= reach_y && dy <= ty; ++dy)
            for (int dx = 0; dx <= reach_x && dx <= tx; ++dx) {
                const uint32_t a = grp * uint32_t(g.ntiles) + uint32_t(ty - dy) * uint32_t(g.ntx) + uint32_t(tx - dx);
                const uint32_t u1 = cell_end[a];
                for (uint32_t u0 = cell_first[a]; u0 < u1; u0 += kThreads) {  // the same for the whole CTA
                    const uint32_t u = u0 + threadIdx.x;
                    int4 r = make_int4(0, 0, 0, 0);
                    if (u < u1) r = urec[u];
                    const bool in = u < u1 && r.x + r.w > (tx << kTX) && r.y + r.w > (ty << kTY);
                    const uint32_t b = __ballot_sync(0xffffffffu, in);
                    if (lane == 0) ws[par][warp] = __popc(b);
                    __syncthreads();
                    // before this warp's, and the CTA's: lane w holds warp w's
                    uint32_t v = lane < kWarps ? ws[par][lane] : 0u;
                    const uint32_t total = __reduce_add_sync(0xffffffffu, v);
                    uint32_t mine = at + __reduce_add_sync(0xffffffffu, lane < warp ? v : 0u);
                    at += total;
                    par ^= 1;  // the next round's counts go to the other row: one barrier between its uses
                    if (in) {
                        mine += __popc(b & ((1u << lane) - 1u));
                        order[mine] = u;
                        grec[mine] = r;
                    }
                }
            }
        if (threadIdx.x == 0) tile_end[c] = at;
    }
}

// the work-unit sizes in footprints
__global__ void uniq_split_kernel(PlanGeom g, uint32_t cells, const uint32_t* __restrict__ count,
                                  const uint32_t* __restrict__ start, uint32_t* sizes)
{
    unit_sizes(g, start[cells - 1u] + count[cells - 1u], sizes);
}

// the sums of the footprints' data, in sample order
__global__ void uniq_sum_kernel(const float2* __restrict__ data, const uint32_t* __restrict__ vals,
                                const uint32_t* __restrict__ ustart, const uint32_t* __restrict__ n_uniq,
                                float2* __restrict__ sum)
{
    const uint32_t n = *n_uniq;
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < n; u += gridDim.x * blockDim.x) {
        uint32_t i = ustart[u];
        const uint32_t i1 = ustart[u + 1u];
        float2 v = data[vals[i++]];
        for (; i + 4 <= i1; i += 4) {  // four loads in flight
            float2 w[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) w[e] = data[vals[i + e]];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                v.x += w[e].x;
                v.y += w[e].y;
            }
        }
        for (; i < i1; ++i) {
            const float2 w = data[vals[i]];
            v.x += w.x;
            v.y += w.y;
        }
        sum[u] = v;
    }
}

// every sample's value: its footprint's tile slots in tile order (left-out samples: 0)
__global__ void uniq_slots_kernel(const float2* __restrict__ slots, const uint16_t* __restrict__ ntl,
                                  const uint32_t* __restrict__ repu, int64_t n, int max_tiles, float c_scale,
                                  float2* __restrict__ out)
{
    const int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (k >= n) return;
    const uint32_t u = repu[k];
    float2 v = make_float2(0.f, 0.f);
    if (u != kNone) {
        const int nt = ntl[u];
        const float2* sl = slots + size_t(u) * max_tiles;
        for (int t = 0; t < nt; ++t) {
            v.x += sl[t].x;
            v.y += sl[t].y;
        }
    }
    out[k] = make_float2(v.x * c_scale, v.y * c_scale);
}

thrust::transform_iterator<Head, thrust::counting_iterator<uint32_t>> heads(const uint64_t* keys, const PlanGeom& g)
{
    return {thrust::counting_iterator<uint32_t>(0), Head{keys, uint64_t(1) << g.u_bits}};
}

int list_ctas(uint32_t cells)
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return int(std::min<uint32_t>(cells, uint32_t(sms) * 8u));
}

}  // namespace

size_t uniq_temp_bytes(const PlanGeom& g)
{
    size_t a = 0, b = 0, c = 0;
    cub::DoubleBuffer<uint64_t> kb(nullptr, nullptr);
    cub::DoubleBuffer<uint32_t> vb(nullptr, nullptr);
    cub::DeviceRadixSort::SortPairs(nullptr, a, kb, vb, g.n, 0, g.u_bits + 1);
    cub::DeviceScan::InclusiveSum(nullptr, b, heads(nullptr, g), static_cast<uint32_t*>(nullptr), g.n);
    cub::DeviceScan::ExclusiveSum(nullptr, c, static_cast<uint32_t*>(nullptr), static_cast<uint32_t*>(nullptr),
                                  int64_t(g.n_groups) * g.ntiles);
    return std::max(a, std::max(b, c));
}

// Cell lists of the plan's distinct footprints: fills vals[0] (order), grec, ntl, tile_start (starts)
// and tile_count (ends) of every cell, and the unit sizes in footprints.  g.n > 0.
tcv_status uniq_bin(tcv_plan* p, cudaStream_t st)
{
    const PlanGeom& g = p->g;
    const uint32_t cells = uint32_t(g.n_groups) * uint32_t(g.ntiles);
    const unsigned blocks = unsigned((g.n + 255) / 256);
    TCV_CUDA(cudaMemsetAsync(p->ucell, 0, size_t(cells) * 3 * sizeof(uint32_t), st));
    uniq_keys_kernel<<<blocks, 256, 0, st>>>(g, p->iu, p->iv, p->coff, p->wplane, p->plane_s, p->plane_grp, p->plane_rank,
                                             p->ukeys[0], p->uvals[0], p->rejected);
    TCV_CUDA(cudaGetLastError());
    cub::DoubleBuffer<uint64_t> kb(p->ukeys[0], p->ukeys[1]);
    cub::DoubleBuffer<uint32_t> vb(p->uvals[0], p->uvals[1]);
    size_t tb = p->cub_bytes;
    TCV_CUDA(cub::DeviceRadixSort::SortPairs(p->cub_temp, tb, kb, vb, g.n, 0, g.u_bits + 1, st));
    p->usel = vb.selector;
    tb = p->cub_bytes;
    TCV_CUDA(cub::DeviceScan::InclusiveSum(p->cub_temp, tb, heads(kb.Current(), g), p->usum, g.n, st));
    uint32_t *count = p->ucell, *first = p->ucell + cells, *end = p->ucell + 2 * size_t(cells);
    uniq_records_kernel<<<blocks, 256, 0, st>>>(g, kb.Current(), vb.Current(), p->usum, p->iu, p->iv, p->coff, p->wplane,
                                                p->plane_s, p->urec, p->ufirst, p->repu, p->ntl, count, first, end,
                                                p->n_uniq);
    TCV_CUDA(cudaGetLastError());
    const int rx = (g.s + g.tw - 2) / g.tw, ry = (g.s + g.th - 2) / g.th;  // tiles past its first that one can touch
    const int ctas = list_ctas(cells);
    tb = p->cub_bytes;
    TCV_CUDA(cub::DeviceScan::ExclusiveSum(p->cub_temp, tb, count, p->tile_start, int64_t(cells), st));
    uniq_split_kernel<<<1, 1, 0, st>>>(g, cells, count, p->tile_start, p->sizes);
    TCV_CUDA(cudaGetLastError());
    // few cells have long lists (spectral run: 561 cells, up to 37 k footprints): large CTAs there
    if (cells < 4096)
        uniq_lists_kernel<1024><<<ctas, 1024, 0, st>>>(g, cells, rx, ry, p->urec, first, end, p->tile_start, p->tile_count,
                                                       p->vals[0], p->grec);
    else
        uniq_lists_kernel<256><<<ctas, 256, 0, st>>>(g, cells, rx, ry, p->urec, first, end, p->tile_start, p->tile_count,
                                                     p->vals[0], p->grec);
    TCV_CUDA(cudaGetLastError());
    p->sel = 0;
    return TCV_OK;
}

tcv_status uniq_sum(const tcv_plan* p, const float2* data, cudaStream_t st)
{
    const PlanGeom& g = p->g;
    const unsigned blocks = unsigned(std::min<int64_t>((g.n + 255) / 256, int64_t(list_ctas(kNone))));
    uniq_sum_kernel<<<blocks, 256, 0, st>>>(data, p->uvals[p->usel], p->ufirst, p->n_uniq, p->usums);
    TCV_CUDA(cudaGetLastError());
    return TCV_OK;
}

tcv_status uniq_slots(const tcv_plan* p, float c_scale, float2* out, cudaStream_t st)
{
    const PlanGeom& g = p->g;
    uniq_slots_kernel<<<unsigned((g.n + 255) / 256), 256, 0, st>>>(p->slots, p->ntl, p->repu, g.n, g.max_tiles, c_scale, out);
    TCV_CUDA(cudaGetLastError());
    return TCV_OK;
}

}  // namespace tcv
