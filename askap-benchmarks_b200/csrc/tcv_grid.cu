// tcv_grid.cu -- launchers of the output-stationary tile kernels (tcv_device.cuh): gridding
// (Benchmark::gridKernel, attic/tConvolveMPI/Benchmark.cc:125-155) and its adjoint degridding
// (Benchmark::degridKernel, :158-195), one persistent launch per plane group.  Each launch uses
// the copy of the kernel specialised on the footprint width when one is available (tcv_jit.cu)
// and the generic copy otherwise.
#include "tcv_internal.cuh"

namespace tcv {
namespace {

// CTAs of a persistent launch: every SM filled to the kernel's occupancy
int resident_of(const void* kernel)
{
    int dev = 0, sms = 148, per_sm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kTileThreads, 0) != cudaSuccess || per_sm < 1)
        per_sm = 1;
    return per_sm * sms;
}

// CTAs of a fold launch: a few per SM, each walking the group's cells
int fold_ctas()
{
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return 4 * sms;
}

GridArgs make_args(const tcv_plan* p, int grp, float c_scale, float2* grid)
{
    const PlanGeom& g = p->g;
    GridArgs a{};
    a.support = g.support;
    a.s = g.s;
    a.ntiles = int(g.ntiles);
    a.group = grp;
    a.c_scale = c_scale;
    a.grid = grid;
    a.jobs = p->jobs;
    a.tinfo = p->tinfo;
    a.partial = p->partial;
    a.ssz = p->ssz;
    a.sched = p->status + kSchedWord;
    return a;
}

// Gridding of a plan with few busy tiles.  A CTA of grid_tile_kernel walks its unit's samples one after
// another, and with one CTA on an SM each sample costs a warp a full L2 latency (16 k samples of a
// 45^2 footprint on 25 tiles, cells whole: 0.71 ms, 1.3 k cycles a sample and warp).  Here a tile is
// shared out in slices of 8 rows to as many CTAs, a warp's block is 32 columns x 2 rows, and the
// table rows of six samples are loaded before the first is added.  Every point still has one owner
// that adds its samples in order, group after group, so the sums are the same, bit for bit; per
// update it costs more instructions, which a device that is mostly idle has to spare.
// Whole-cell plans take it when every plane group has at most 1.2 busy tiles per SM (plan_mode_kernel):
// 169 tiles gain (0.72 -> 0.49 ms; 60 k samples of 65^2 on 144, a bfloat16 table, 0.45 -> 0.39), 289 do not
// (0.38 and 0.51 ms).  The samples above take 0.162 ms, 160 k samples of 29^2 on 9 tiles 4.3 ms (18.8 whole).  Six samples at four CTAs an SM: eight at three
// take 0.165 and 4.1 ms but 0.55 ms on 169 tiles, four at four 0.19, 4.7 and 0.52.
// A kernel of its own: inside grid_tile_kernel it cost the other path 1.4 % (registers).  It is launched
// behind the tile kernels, whose ranges are then empty, without the usual gap (it waits for them
// itself): where it is not taken that costs about 1 us a pass (65 k samples of 45^2 157.3 -> 158.4 us, 160 k
// of 129^2 1238.1 -> 1239.3), an ordinary launch before them 4 us.
template <class Tab, int kR, bool kVar>
__global__ void __launch_bounds__(kTileThreads, 4)
grid_slice_kernel(const float2* __restrict__ data, const typename Tab::elem* __restrict__ ctab,
                  const int* __restrict__ iu, const int* __restrict__ iv, const int* __restrict__ coff,
                  const u32* __restrict__ order, const u32* __restrict__ tile_start, const u32* __restrict__ tile_count,
                  const unsigned int* __restrict__ taken, int n_groups, GridArgs a)
{
    constexpr int kTH = tile_height(kR), kRows = 2, kDeep = 6;
    constexpr u32 kSlices = kTH / (4 * kRows);  // a slice: four pairs of warps
    constexpr u32 kLook = 4 * kTileThreads;     // tiles looked over at a time
    cudaGridDependencySynchronize();  // launched ahead of the tile kernels' end
    if (!*taken) return;
    __shared__ float4 sm_rec[2][kTileChunk];  // (data.re, data.im, first column, first row)
    __shared__ int sm_coff[2][kTileChunk];
    __shared__ int sm_w[kVar ? 2 : 1][kVar ? kTileChunk : 1];
    __shared__ unsigned char sm_mask[2][kTileChunk];  // per sample: the warps whose blocks it meets
    __shared__ u32 busy[kLook], sm_n[4 * kTileWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int s0 = a.s;
    u32 before = 0;  // busy tiles of the looks before
    for (u32 look = 0; look < u32(a.ntiles); look += kLook) {
        // the busy tiles, in order (every CTA finds the same list)
        bool on[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const u32 t = look + u32(e) * kTileThreads + threadIdx.x;
            on[e] = false;
            if (t < u32(a.ntiles))
                for (int g = 0; g < n_groups; ++g) on[e] |= tile_count[u32(g) * u32(a.ntiles) + t] != 0u;
        }
        __syncthreads();  // the last look's list is used
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const u32 b = __ballot_sync(0xffffffffu, on[e]);
            if (lane == 0) sm_n[e * kTileWarps + warp] = __popc(b);
        }
        __syncthreads();
        const u32 mine = sm_n[lane];  // lane e * kTileWarps + w: 32 counts
        static_assert(4 * kTileWarps == 32, "one count per lane");
        const u32 n = __reduce_add_sync(0xffffffffu, mine);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const u32 b = __ballot_sync(0xffffffffu, on[e]);
            const u32 at = __reduce_add_sync(0xffffffffu, lane < e * kTileWarps + warp ? mine : 0u) + __popc(b & ((1u << lane) - 1u));
            if (on[e]) busy[at] = look + u32(e) * kTileThreads + threadIdx.x;
        }
        __syncthreads();
        // items (busy tile, slice), numbered over all looks, dealt to the CTAs in turn
        const u32 first = before * kSlices, rest = first % gridDim.x;
        for (u32 item = rest <= blockIdx.x ? blockIdx.x - rest : gridDim.x - rest + blockIdx.x; item < n * kSlices;
             item += gridDim.x) {
            const u32 tile = busy[item / kSlices], ti = a.tinfo[tile];
            const int x0 = rec_tx(ti) * kTileW, y0 = rec_ty(ti) * kTH + int(item % kSlices) * (4 * kRows);
            const int gx = x0 + (warp & 1) * 32 + lane, gy0 = y0 + (warp >> 1) * kRows;
            const JobDesc& jd = a.jobs[rec_job(ti)];
            const int gs = jd.g_size;
            float2* grid = a.grid ? a.grid : jd.grid;
            for (int g = 0; g < n_groups; ++g) {
                const u32 c = u32(g) * u32(a.ntiles) + tile, start = tile_start[c], cnt = tile_count[c];
                if (cnt == 0) continue;  // the same for the whole CTA
                float2 acc[kRows];
#pragma unroll
                for (int r = 0; r < kRows; ++r) acc[r] = make_float2(0.f, 0.f);
                auto stage = [&](u32 base, int buf) {
                    if (base + threadIdx.x >= cnt) return;
                    const u32 k = order[start + base + threadIdx.x];
                    const float2 d = data[k];
                    const int sk = kVar ? int(a.ssz[k]) : s0;
                    const int fx = iu[k] - (kVar ? sk / 2 : a.support), fy = iv[k];
                    sm_rec[buf][threadIdx.x] =
                        make_float4(d.x * a.c_scale, d.y * a.c_scale, __int_as_float(fx), __int_as_float(fy));
                    sm_coff[buf][threadIdx.x] = coff[k];
                    if (kVar) sm_w[kVar ? buf : 0][kVar ? threadIdx.x : 0] = sk;
                    const int bx = x0 - fx, by = y0 - fy;
                    u32 m = 0;
#pragma unroll
                    for (int w = 0; w < kTileWarps; ++w) {
                        const int cx = bx + (w & 1) * 32, cy = by + (w >> 1) * kRows;
                        m |= u32(cx < sk && cx + 32 > 0 && cy < sk && cy + kRows > 0) << w;
                    }
                    sm_mask[buf][threadIdx.x] = (unsigned char)m;
                };
                __syncthreads();  // the records before are used
                stage(0, 0);
                int buf = 0;
                for (u32 base = 0; base < cnt; base += u32(kTileChunk), buf ^= 1) {
                    __syncthreads();  // this chunk is staged, the one before is used
                    stage(base + u32(kTileChunk), buf ^ 1);
                    const int m = int(cnt - base < u32(kTileChunk) ? cnt - base : u32(kTileChunk));
                    for (int e = 0; e < m; e += 32) {
                        u32 bits = __ballot_sync(0xffffffffu, e + lane < m && ((sm_mask[buf][e + lane] >> warp) & 1u));
                        while (bits) {
                            // entries as they are stored: converting one would wait for its load
                            typename Tab::elem cv[kDeep][kRows];
                            float2 dv[kDeep];
                            u32 has = 0;  // rows that this lane's column of the footprint has, kRows bits per sample
#pragma unroll
                            for (int b = 0; b < kDeep; ++b) {
                                if (!bits) break;
                                const int j = e + __ffs(bits) - 1;
                                bits &= bits - 1;
                                const float4 q = sm_rec[buf][j];
                                const int s = kVar ? sm_w[kVar ? buf : 0][kVar ? j : 0] : s0;
                                const int dx = gx - __float_as_int(q.z), dy = gy0 - __float_as_int(q.w);
                                const int ci = sm_coff[buf][j] + dy * s + dx;
                                dv[b] = make_float2(q.x, q.y);
#pragma unroll
                                for (int r = 0; r < kRows; ++r)
                                    if (unsigned(dx) < unsigned(s) && unsigned(dy + r) < unsigned(s)) {
                                        has |= 1u << (b * kRows + r);
                                        cv[b][r] = __ldg(ctab + (ci + r * s));
                                    }
                            }
#pragma unroll
                            for (int b = 0; b < kDeep; ++b)
#pragma unroll
                                for (int r = 0; r < kRows; ++r)
                                    if ((has >> (b * kRows + r)) & 1u) cmac<Tab::kReal>(acc[r], dv[b], Tab::value(cv[b][r]));
                        }
                    }
                }
#pragma unroll
                for (int r = 0; r < kRows; ++r)
                    if (gx < gs && gy0 + r < gs) {
                        float2* gp = grid + ((unsigned long long)(gy0 + r) * gs + gx);
                        float2 v = *gp;
                        v.x += acc[r].x;
                        v.y += acc[r].y;
                        *gp = v;
                    }
            }
        }
        before += n;
    }
}

// One persistent launch per plane group, in group order on the stream: launches of one stream
// run one after another, so a tile's read-modify-write never races with another group's.
template <class Tab, int kR, bool kVar = false>
tcv_status launch(const tcv_plan* p, const float2* data, const void* c, float c_scale, float2* grid,
                  cudaStream_t st, int c_type)
{
    const PlanGeom& g = p->g;
    if (g.n == 0) return TCV_OK;
    const void* spec = kVar ? nullptr
                       : p->jit_cached_only ? jit_tile_kernel_cached(0, c_type, g.s, kR)
                                            : jit_tile_kernel(0, c_type, g.s, kR);
    const void* generic = reinterpret_cast<const void*>(&grid_tile_kernel<Tab, 0, kR, kVar>);
    const void* kernel = spec ? spec : generic;
    const int ctas = resident_of(kernel);
    const typename Tab::elem* tab = static_cast<const typename Tab::elem*>(c);
    const unsigned int* order = p->vals[p->sel];
    for (int grp = 0; grp < g.n_groups; ++grp) {
        GridArgs a = make_args(p, grp, c_scale, grid);
        const uint32_t* range = p->grid_range ? p->grid_range + grp : p->group_ustart;  // [grp], [grp + 1]: first, end unit
        void* args[] = {&data, &tab, const_cast<const int32_t**>(&p->iu), const_cast<const int32_t**>(&p->iv),
                        const_cast<const int32_t**>(&p->coff), &order, const_cast<uint4**>(&p->units), &range, &a};
        TCV_CUDA(cudaLaunchKernel(kernel, dim3(ctas), dim3(kTileThreads), args, 0, st));
        if (g.split) {
            // the split cells' partial tiles into the grid, before the next group touches it
            fold_kernel<kR><<<fold_ctas(), kTileThreads, 0, st>>>(p->items, p->group_start, p->group_ustart, p->nunits,
                                                                  p->pstart, a);
            TCV_CUDA(cudaGetLastError());
        }
    }
    if (p->grid_range) {  // plans of few busy tiles: the launches above found no units
        const void* slices = reinterpret_cast<const void*>(&grid_slice_kernel<Tab, kR, kVar>);
        const GridArgs a = make_args(p, 0, c_scale, grid);
        TCV_CHECK(launch_behind(&grid_slice_kernel<Tab, kR, kVar>, unsigned(resident_of(slices)), kTileThreads, st, data, tab,
                                p->iu, p->iv, p->coff, order, p->tile_start, p->tile_count, p->status + kSliceWord,
                                g.n_groups, a));
    }
    return TCV_OK;
}

template <class Tab, int kR, bool kVar = false>
tcv_status launch_adjoint(const tcv_plan* p, const float2* grid, const void* c, float c_scale, float2* out,
                          cudaStream_t st, int c_type)
{
    const PlanGeom& g = p->g;
    if (g.n == 0) return TCV_OK;
    const void* spec = kVar ? nullptr
                       : p->jit_cached_only ? jit_tile_kernel_cached(1, c_type, g.s, kR)
                                            : jit_tile_kernel(1, c_type, g.s, kR);
    const void* generic = reinterpret_cast<const void*>(&degrid_tile_kernel<Tab, 0, kR, kVar>);
    const void* kernel = spec ? spec : generic;
    const int ctas = resident_of(kernel);
    const typename Tab::elem* tab = static_cast<const typename Tab::elem*>(c);
    const unsigned int* order = p->vals[p->sel];
    int max_tiles = g.max_tiles;
    float2* gridp = const_cast<float2*>(grid);
    for (int grp = 0; grp < g.n_groups; ++grp) {
        GridArgs a = make_args(p, grp, c_scale, gridp);
        void* args[] = {&tab, const_cast<const int32_t**>(&p->iu), const_cast<const int32_t**>(&p->iv),
                        const_cast<const int32_t**>(&p->coff), &order, const_cast<uint4**>(&p->d_units),
                        const_cast<uint32_t**>(&p->d_group_ustart), const_cast<float2**>(&p->slots), &max_tiles, &a};
        TCV_CUDA(cudaLaunchKernel(kernel, dim3(ctas), dim3(kTileThreads), args, 0, st));
    }
    return slot_reduce(p, c_scale, out, st);
}

}  // namespace

tcv_status launch_fold8(const tcv_plan* p, const GridArgs& a, cudaStream_t st)
{
    fold_kernel<8><<<fold_ctas(), kTileThreads, 0, st>>>(p->items, p->group_start, p->group_ustart, p->nunits,
                                                         p->pstart, a);
    TCV_CUDA(cudaGetLastError());
    return TCV_OK;
}

namespace {

template <class Tab>
tcv_status grid_rows(const tcv_plan* p, const float2* data, const void* c, float c_scale, float2* grid,
                     cudaStream_t st, int c_type)
{
    if (p->g.var) {  // per-sample widths: complex tables (the w-term is complex), 64 x 64 or 64 x 32 tiles
        if constexpr (!Tab::kReal) {
            if (p->g.dense) return launch_dense_grid<Tab>(p, data, c, c_scale, grid, st);
            if (p->g.rows == 16) return launch<Tab, 16, true>(p, data, c, c_scale, grid, st, c_type);
            if (p->g.rows == 8) return launch<Tab, 8, true>(p, data, c, c_scale, grid, st, c_type);
        }
        return TCV_ERR_UNSUPPORTED;
    }
    if (p->g.dense) return launch_dense_grid<Tab>(p, data, c, c_scale, grid, st);
    switch (p->g.rows) {
        case 8: return launch<Tab, 8>(p, data, c, c_scale, grid, st, c_type);
        case 16: return launch<Tab, 16>(p, data, c, c_scale, grid, st, c_type);
        case 32: return launch<Tab, 32>(p, data, c, c_scale, grid, st, c_type);
        default: return TCV_ERR_UNSUPPORTED;
    }
}

template <class Tab>
tcv_status degrid_rows(const tcv_plan* p, const float2* grid, const void* c, float c_scale, float2* out,
                       cudaStream_t st, int c_type)
{
    if (p->g.var) {
        if constexpr (!Tab::kReal) {
            if (p->g.ddense) return launch_dense_degrid<Tab>(p, grid, c, c_scale, out, st);
            if (p->g.rows == 16) return launch_adjoint<Tab, 16, true>(p, grid, c, c_scale, out, st, c_type);
            if (p->g.rows == 8) return launch_adjoint<Tab, 8, true>(p, grid, c, c_scale, out, st, c_type);
        }
        return TCV_ERR_UNSUPPORTED;
    }
    if (p->g.ddense) return launch_dense_degrid<Tab>(p, grid, c, c_scale, out, st);
    switch (p->g.rows) {
        case 8: return launch_adjoint<Tab, 8>(p, grid, c, c_scale, out, st, c_type);
        case 16: return launch_adjoint<Tab, 16>(p, grid, c, c_scale, out, st, c_type);
        case 32: return launch_adjoint<Tab, 32>(p, grid, c, c_scale, out, st, c_type);
        default: return TCV_ERR_UNSUPPORTED;
    }
}

}  // namespace

tcv_status launch_degrid_tiles(const tcv_plan* p, const float2* grid, const void* c, int c_type,
                               float c_scale, float2* out, cudaStream_t st)
{
    switch (c_type) {
        case TCV_C_C64: return degrid_rows<TabC64>(p, grid, c, c_scale, out, st, c_type);
        case TCV_C_R32: return degrid_rows<TabR32>(p, grid, c, c_scale, out, st, c_type);
        case TCV_C_CBF16: return degrid_rows<TabCBF16>(p, grid, c, c_scale, out, st, c_type);
        case TCV_C_RBF16: return degrid_rows<TabRBF16>(p, grid, c, c_scale, out, st, c_type);
        case TCV_C_CF16: return degrid_rows<TabCF16>(p, grid, c, c_scale, out, st, c_type);
        case TCV_C_RF16: return degrid_rows<TabRF16>(p, grid, c, c_scale, out, st, c_type);
        default: return TCV_ERR_ARG;
    }
}

tcv_status launch_grid(const tcv_plan* p, const float2* data, const void* c, int c_type,
                       float c_scale, float2* grid, cudaStream_t st)
{
    switch (c_type) {
        case TCV_C_C64: return grid_rows<TabC64>(p, data, c, c_scale, grid, st, c_type);
        case TCV_C_R32: return grid_rows<TabR32>(p, data, c, c_scale, grid, st, c_type);
        case TCV_C_CBF16: return grid_rows<TabCBF16>(p, data, c, c_scale, grid, st, c_type);
        case TCV_C_RBF16: return grid_rows<TabRBF16>(p, data, c, c_scale, grid, st, c_type);
        case TCV_C_CF16: return grid_rows<TabCF16>(p, data, c, c_scale, grid, st, c_type);
        case TCV_C_RF16: return grid_rows<TabRF16>(p, data, c, c_scale, grid, st, c_type);
        default: return TCV_ERR_ARG;
    }
}

}  // namespace tcv
