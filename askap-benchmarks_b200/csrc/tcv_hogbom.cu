// tcv_hogbom.cu -- Hogbom CLEAN (the minor cycle) on the device.
//
// Reference: current/tHogbomCleanOMP/HogbomGolden.cc:47-141 (HogbomGolden::deconvolve, findPeak,
// subtractPSF) and the same steps inside current/tMajorACC/tMajorACC.cc:689-877 (deconvolve).  Each
// iteration takes the pixel of largest |residual| (the first such index, as the reference's strict
// '>' scan in index order does), adds gain * peak to the model there, and subtracts
// (gain * peak) * psf, shifted so that the PSF's own peak lands on that pixel, over the overlap of
// the two images.  The arithmetic is the reference's, rounding by rounding: t = gain * peak,
// u = t * psf, r = r - u, each rounded to float (no contraction into fused multiply-adds), so the
// model and the residual are bit-identical to the reference's.
//
// The reference computes the PSF row as y - (ry - px) (its diffy uses the PSF peak's x,
// HogbomGolden.cc:108); that is kept.  Where it points outside the PSF (only when the PSF peak is
// off the diagonal) the reference reads out of bounds; here those rows are skipped and counted.
//
// Four forms, chosen by size and image (tcv_hogbom_deconvolve); all give the same bits.
//
// Up to 1792 x 1792 (as many clusters as the device holds decide it; hog_resident_kernel): the residual
// stays in registers, one cooperative launch.
//
// Larger images: updates are put off.  The image is cut into blocks of at least 32 x 32 pixels, and
// a block's updates wait until the block could hold the next peak:
//   * per block, a bound on its |residual|: its largest |value| when last brought up to date, plus
//     |t| x the largest |psf| over the part of the PSF each update since has laid on it (from a table
//     of the PSF's block maxima), rounded up;
//   * the updated value at the peak itself, |peak - t psf(peak)|, is a lower limit of the next peak:
//     blocks whose bound is below it cannot hold that and are left alone; the others ("hot", ~25 per
//     iteration around the brightest pixels, of 16384 at 4096^2) apply their pending updates in
//     order and give their largest value, which is exact.
// hog_lead_kernel runs kLeadIters iterations in one cluster, whose CTAs share out the blocks and
// exchange candidates through distributed shared memory: an iteration is a chain of latencies
// (bounds, the hot blocks' loads, the exchange: 5 us at 4096^2), not a pass over the image.
// hog_apply_kernel follows on the whole device: it brings blocks near the peak up to date, and
// every kRing iterations and at the end all blocks (7.7 us an iteration at 4096^2, most of it the PSF
// windows from L2).  A pixel's updates are applied in iteration order with the reference's roundings
// whenever they are applied, so the bits do not depend on the schedule.
//
// Where many blocks are near the peak, as in an image that an earlier cycle has cleaned, and for a few
// iterations: a pass over the image per iteration in cooperative launches (hog_pass_kernel).
//
// Beyond the block table's size, for one or two iterations (or with TCV_HOGBOM_PER_LAUNCH): a launch per
// iteration, which subtracts the PSF over its blocks' slices of the image and scans the updated values for the
// next peak in the same pass, so an iteration reads the residual once, reads the PSF's overlap
// once and writes the overlap once.  Each block leaves one candidate, a 64-bit key (|value| bits
// << 32 | ~index: the largest key is the largest magnitude at the smallest index) with its signed
// value; the last block to finish (an atomic ticket, no waiting) reduces the candidates to the
// winner that the next launch reads.  The stop test (|peak| < threshold) is taken on the device:
// later launches see the flag and return.
//
// Measured on one B200, us an iteration of 1000 (20 sources), and in brackets with one pass over the image per
// iteration (in one cooperative launch up to 48 MiB of images, a launch each beyond): 128^2 1.11 (10.1), 223^2
// 1.5 (7.9), 1024^2 3.2 (4.7), 1700^2 7.4 (7.4), 1900^2 6.3 (8.35), 2600^2 7.9 (15.9), 4096^2 12.8 (28.0); 5 sources cleaned
// to noise 1900^2 8.0 (8.1), 4096^2 20.7 (26.6); an image cleaned before 1900^2 8.3 (8.05), 2048^2 8.5 (8.1), 2600^2
// 11.7 (14.2), 4096^2 19.4 (21.9).
#include "tcv_internal.cuh"

#include <cooperative_groups.h>
#include <cuda_pipeline.h>

#include <algorithm>
#include <cstdint>

namespace tcv {
namespace {

constexpr int kHogThreads = 256;
constexpr int kHogMaxBlocks = 592;  // 4 x 148: one wave of four 256-thread CTAs per SM

// device state of one deconvolution (start of the caller's workspace; zeroed by the host)
struct HogState {
    unsigned long long win_key[3];  // winners: [0], [1] by iteration parity, [2] the PSF's
    float win_val[3];
    unsigned int arrived;           // blocks finished in the current launch
    int stopped;                    // 1 + the iteration whose |peak| fell below the threshold; 0 = running
    int done;                       // iterations carried out
    unsigned int psf_pos;           // PSF peak index
    unsigned long long skipped_rows;  // PSF rows outside the PSF (reference out-of-bounds reads)
    int error;                        // a wait for other CTAs gave up
    int batch, used;                  // put-off updates: the ring's last batch and its PSF windows
    unsigned int nwarm;               // and the blocks of the list for hog_apply_kernel
    unsigned int visits;              // most hot blocks that a leading CTA had in the last launch
    int pass;                         // 1: hog_pass_kernel has taken over
    int pass_end;                     // iterations that it has done
    unsigned int meet;                // its CTAs' arrivals in the current launch
    unsigned int win_next;            // and the winner that its last launch left
    float val_next;
    unsigned int near, tops;          // blocks of the dirty image that reach half its peak; its second peak's limit
};

struct HogArgs {
    const float* psf;
    float* residual;
    float* model;
    unsigned long long* keys;  // one candidate per block
    float* vals;
    HogState* state;
    float* hist_val;         // per iteration: peak value (may be null)
    unsigned int* hist_pos;  // per iteration: peak index (may be null)
    int width, psf_width, nblocks;
    long long n;  // width * width
    float gain, threshold;
};

__device__ __forceinline__ unsigned int key_index(unsigned long long k) { return ~static_cast<unsigned int>(k); }

// Block-wide maximum of (key, value); the winner is returned to every thread.
__device__ unsigned long long block_max(unsigned long long k, float& v)
{
    __shared__ unsigned long long sk[kHogThreads / 32];
    __shared__ float sv[kHogThreads / 32];
    for (int o = 16; o > 0; o >>= 1) {
        const unsigned long long ko = __shfl_down_sync(0xffffffffu, k, o);
        const float vo = __shfl_down_sync(0xffffffffu, v, o);
        if (ko > k) {
            k = ko;
            v = vo;
        }
    }
    const int w = threadIdx.x >> 5;
    __syncthreads();  // earlier readers of sk/sv are done
    if ((threadIdx.x & 31) == 0) {
        sk[w] = k;
        sv[w] = v;
    }
    __syncthreads();
    k = sk[0];
    v = sv[0];
    for (int i = 1; i < kHogThreads / 32; ++i)
        if (sk[i] > k) {
            k = sk[i];
            v = sv[i];
        }
    return k;
}

// Leave this block's candidate; the last block of the launch reduces all of them into
// state->win_key/win_val[slot] (and for the PSF slot, the PSF peak position).
__device__ void finish_scan(unsigned long long best, float bv, unsigned long long* keys, float* vals, int nblocks,
                            HogState* st, int slot)
{
    best = block_max(best, bv);
    __shared__ bool last;
    if (threadIdx.x == 0) {
        keys[blockIdx.x] = best;
        vals[blockIdx.x] = bv;
        __threadfence();
        last = atomicAdd(&st->arrived, 1u) == unsigned(nblocks - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    unsigned long long k = 0;
    float v = 0.f;
    for (int i = threadIdx.x; i < nblocks; i += kHogThreads) {
        const unsigned long long ki = __ldcg(keys + i);
        if (ki > k) {
            k = ki;
            v = __ldcg(vals + i);
        }
    }
    k = block_max(k, v);
    if (threadIdx.x == 0) {
        const bool zero = (k >> 32) == 0;  // an all-zero image: the reference keeps maxPos = 0, maxVal = 0
        st->win_key[slot] = zero ? static_cast<unsigned long long>(~0u) : k;
        st->win_val[slot] = zero ? 0.f : v;
        if (slot == 2) st->psf_pos = zero ? 0u : key_index(k);
        st->arrived = 0;
    }
}

// Scan an image (copying it to copy_to when given) for its peak.
__global__ void __launch_bounds__(kHogThreads) hog_scan_kernel(const float* __restrict__ img, float* __restrict__ copy_to,
                                                               long long n, int nblocks, unsigned long long* keys,
                                                               float* vals, HogState* st, int slot)
{
    const long long per = (n + nblocks - 1) / nblocks;
    const long long lo = per * blockIdx.x, hi = min(n, lo + per);
    float best_abs = -1.f, bv = 0.f;
    unsigned int bi = 0;
    for (long long i = lo + threadIdx.x; i < hi; i += kHogThreads) {
        const float v = img[i];
        if (copy_to) copy_to[i] = v;
        if (fabsf(v) > best_abs) {  // strict '>' in index order keeps the first index
            best_abs = fabsf(v);
            bv = v;
            bi = static_cast<unsigned int>(i);
        }
    }
    const unsigned long long best =
        best_abs < 0.f ? 0ull : (static_cast<unsigned long long>(__float_as_uint(best_abs)) << 32) | (~bi & 0xffffffffu);
    finish_scan(best, bv, keys, vals, nblocks, st, slot);
}

// subtractPSF (HogbomGolden.cc:99-124) over this CTA's share of the image, and the scan of the
// updated values: returns the CTA-thread's candidate key (0 if it saw no pixel) and value.
// kVec: width a multiple of 4 and the residual 16-byte aligned (float4 residual I/O).  Whole rows per CTA.
template <bool kVec>
__device__ __forceinline__ unsigned long long iter_body(const HogArgs& a, unsigned int ppos, float peak,
                                                        unsigned int psf_pos, float& bv_out,
                                                        unsigned long long& skipped_out)
{
    const int W = a.width, P = a.psf_width;
    const int rx = int(ppos % unsigned(W)), ry = int(ppos / unsigned(W));
    const int px = int(psf_pos % unsigned(P)), py = int(psf_pos / unsigned(P));
    const int diffx = rx - px, diffy = ry - px;  // diffy uses px, as the reference does
    const int startx = max(0, rx - px), starty = max(0, ry - py);
    const int stopx = min(W - 1, rx + (P - px - 1)), stopy = min(W - 1, ry + (P - py - 1));
    const float t = __fmul_rn(a.gain, peak);

    // running maximum of |value| in index order: strict '>' keeps the first index (findPeak's rule)
    float best_abs = -1.f, bv = 0.f;
    unsigned int bi = 0;
    unsigned long long skipped = 0;
    auto track = [&](float v, unsigned int idx) {
        const float av = fabsf(v);
        if (av > best_abs) {
            best_abs = av;
            bv = v;
            bi = idx;
        }
    };
    if (kVec) {
        // whole rows per block, walked as items (row, column chunk of 256 float4) in index order;
        // every thread loads the float4s of U items (of one or several rows) before any store
        constexpr int U = 4;
        const int rows_per = (W + a.nblocks - 1) / a.nblocks;
        const int r0 = int(blockIdx.x) * rows_per, r1 = min(W, r0 + rows_per);
        const int nch = (W / 4 + kHogThreads - 1) / kHogThreads;  // chunks per row
        if (threadIdx.x == 0)
            for (int y = r0; y < r1; ++y)
                if (y >= starty && y <= stopy && !(y - diffy >= 0 && y - diffy < P)) ++skipped;
        int y = r0, c = 0;
        while (y < r1) {
            float4 r[U];
            float pv[U][4];
            bool sub[U], val[U];
            int xs[U], ys[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                ys[u] = y;
                xs[u] = 4 * (int(threadIdx.x) + kHogThreads * c);
                val[u] = y < r1 && xs[u] < W;
                if (++c == nch) {
                    c = 0;
                    ++y;
                }
                sub[u] = false;
                r[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (val[u]) {
                    r[u] = __ldcg(reinterpret_cast<const float4*>(a.residual + ((long long)ys[u] * W + xs[u])));
                    const int prow = ys[u] - diffy;
                    sub[u] = ys[u] >= starty && ys[u] <= stopy && prow >= 0 && prow < P && xs[u] + 3 >= startx &&
                             xs[u] <= stopx;
                    const long long pbase = (long long)prow * P - diffx;  // + x: inside the PSF row for x in range
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int x = xs[u] + j;
                        pv[u][j] = (sub[u] && x >= startx && x <= stopx) ? __ldg(a.psf + (pbase + x)) : 0.f;
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (!val[u]) continue;
                if (sub[u]) {
                    float* rv = reinterpret_cast<float*>(&r[u]);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int x = xs[u] + j;
                        if (x >= startx && x <= stopx) rv[j] = __fsub_rn(rv[j], __fmul_rn(t, pv[u][j]));
                    }
                    __stcg(reinterpret_cast<float4*>(a.residual + ((long long)ys[u] * W + xs[u])), r[u]);
                }
                const unsigned int i0 = unsigned(ys[u]) * unsigned(W) + unsigned(xs[u]);
                track(r[u].x, i0);
                track(r[u].y, i0 + 1);
                track(r[u].z, i0 + 2);
                track(r[u].w, i0 + 3);
            }
        }
    } else {
        // the same by single pixels
        constexpr int U = 8;
        const int rows_per = (W + a.nblocks - 1) / a.nblocks;
        const int r0 = int(blockIdx.x) * rows_per, r1 = min(W, r0 + rows_per);
        const int nch = (W + kHogThreads - 1) / kHogThreads;
        if (threadIdx.x == 0)
            for (int y = r0; y < r1; ++y)
                if (y >= starty && y <= stopy && !(y - diffy >= 0 && y - diffy < P)) ++skipped;
        int y = r0, c = 0;
        while (y < r1) {
            float r[U], pv[U];
            bool sub[U], val[U];
            unsigned int at[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int x = int(threadIdx.x) + kHogThreads * c, prow = y - diffy;
                val[u] = y < r1 && x < W;
                sub[u] = val[u] && y >= starty && y <= stopy && prow >= 0 && prow < P && x >= startx && x <= stopx;
                at[u] = unsigned(y) * unsigned(W) + unsigned(x);  // n < 2^32
                r[u] = val[u] ? __ldcg(a.residual + at[u]) : 0.f;
                pv[u] = sub[u] ? __ldg(a.psf + ((long long)prow * P + (x - diffx))) : 0.f;
                if (++c == nch) {
                    c = 0;
                    ++y;
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                if (sub[u]) {
                    r[u] = __fsub_rn(r[u], __fmul_rn(t, pv[u]));
                    __stcg(a.residual + at[u], r[u]);
                }
                if (val[u]) track(r[u], at[u]);
            }
        }
    }
    const unsigned long long best =
        best_abs < 0.f ? 0ull : (static_cast<unsigned long long>(__float_as_uint(best_abs)) << 32) | (~bi & 0xffffffffu);
    bv_out = bv;
    skipped_out = skipped;
    return best;
}

// model[absPeakPos] += absPeakVal * g_gain (HogbomGolden.cc:93), by one thread
__device__ __forceinline__ void model_update(const HogArgs& a, int it, unsigned int ppos, float peak)
{
    a.model[ppos] = __fadd_rn(a.model[ppos], __fmul_rn(peak, a.gain));
    if (a.hist_val) a.hist_val[it] = peak;
    if (a.hist_pos) a.hist_pos[it] = ppos;
}

// One launch per iteration: the previous scan's winner, the model update, the PSF subtraction and
// the scan of this CTA's rows.
template <bool kVec>
__global__ void __launch_bounds__(kHogThreads, 4) hog_iter_kernel(HogArgs a, int it)
{
    HogState* st = a.state;
    if (st->stopped) return;  // an earlier launch stopped the loop
    const int par = it & 1;
    const unsigned int ppos = key_index(st->win_key[par]);
    const float peak = st->win_val[par];
    if (fabsf(peak) < a.threshold) {  // HogbomGolden.cc:86-89
        if (blockIdx.x == 0 && threadIdx.x == 0) st->stopped = it + 1;
        return;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        model_update(a, it, ppos, peak);
        st->done = it + 1;
    }
    if (it > 0) {
        // rows wholly outside this iteration's PSF overlap do not change: the CTA's candidate from
        // an earlier iteration (same row partition; iteration 0 always scans, after the image
        // scan's pixel partition) still holds, so it is left as it is without reading the rows
        const int W = a.width, P = a.psf_width;
        const int ry = int(ppos / unsigned(W)), py = int(st->psf_pos / unsigned(P));
        const int starty = max(0, ry - py), stopy = min(W - 1, ry + (P - py - 1));
        const int rows_per = (W + a.nblocks - 1) / a.nblocks;
        const int r0 = int(blockIdx.x) * rows_per, r1 = min(W, r0 + rows_per);
        if (r1 <= starty || r0 > stopy) {
            const unsigned long long old = __ldcg(a.keys + blockIdx.x);
            const float oldv = __ldcg(a.vals + blockIdx.x);
            finish_scan(old, oldv, a.keys, a.vals, a.nblocks, st, par ^ 1);
            return;
        }
    }
    float bv;
    unsigned long long skipped;
    const unsigned long long best = iter_body<kVec>(a, ppos, peak, st->psf_pos, bv, skipped);
    if (skipped) atomicAdd(&st->skipped_rows, skipped);
    finish_scan(best, bv, a.keys, a.vals, a.nblocks, st, par ^ 1);
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

constexpr int kLeadThreads = 512;
constexpr int kLeadWarps = kLeadThreads / 32;
constexpr int kLeadCtas = 16;        // CTAs of the leading cluster (8 where 16 do not fit)
constexpr int kBlkSide = 128;        // image and PSF blocks per side, at most
constexpr int kBlkMax = kBlkSide * kBlkSide;
constexpr int kDeferMaxWidth = 128 * kBlkSide;  // blocks of up to 128 x 128 pixels
constexpr int kOwned = kBlkMax / 8;  // blocks per CTA of the cluster, at most
constexpr int kLeadIters = 16;       // iterations per launch of the cluster (even)
constexpr int kRing = 128;           // iterations whose updates may be pending (a multiple of kLeadIters)
constexpr int kApplyThreads = 128;
constexpr int kApplyRows = 4;        // rows per warp: a CTA works on 32 x 16 pixels at a time
constexpr int kApplyDeep = 4;        // windows whose copies are issued together
constexpr int kSlots = 52;           // PSF windows of that size an applying CTA holds
constexpr int kStrips = 32 / (kApplyThreads / 32 * kApplyRows);  // parts of 32 columns a 32 x 32 square is worked on in
constexpr int kWindow = kApplyThreads * kApplyRows;  // pixels of a window

// A candidate as one word: larger |value| first, then the smaller index (row << 16 | column, so that
// no division is needed to get at them); the sign last.
__device__ __forceinline__ unsigned long long cand_key(float v, int x, int y)
{
    const unsigned int b = __float_as_uint(v), idx = unsigned(y) << 16 | unsigned(x);
    return (static_cast<unsigned long long>(b & 0x7fffffffu) << 33) | (static_cast<unsigned long long>(~idx) << 1) | (b >> 31);
}
__device__ __forceinline__ float cand_abs(unsigned long long k) { return __uint_as_float(unsigned(k >> 33)); }
__device__ __forceinline__ float cand_value(unsigned long long k)
{
    return __uint_as_float(unsigned(k >> 33) | (unsigned(k & 1u) << 31));
}
__device__ __forceinline__ unsigned int cand_index(unsigned long long k) { return ~unsigned(k >> 1); }
__device__ __forceinline__ unsigned long long warp_max(unsigned long long k)
{
    const unsigned int hi = unsigned(k >> 32), top = __reduce_max_sync(0xffffffffu, hi);
    const unsigned int lo = __reduce_max_sync(0xffffffffu, hi == top ? unsigned(k) : 0u);
    return (static_cast<unsigned long long>(top) << 32) | lo;
}

// ------------------------------------------------------------------------------------------
// Images that fit the register files: the residual stays in registers for all iterations.  Each CTA
// owns whole rows, a thread up to kRowsT x kChunks pixels of them; an iteration loads the PSF (from
// L2), updates, and finds the CTA's candidate; the CTAs of a cluster send theirs to its first CTA
// through distributed shared memory, the first CTAs exchange theirs through global memory (a
// word a cluster instead of one per CTA: all CTAs polling all CTAs' words kept the few L2 lines they lie on
// busy and took 4 us), and each hands the winner to its cluster.
// ------------------------------------------------------------------------------------------
constexpr int kResThreads = 512;
constexpr int kResChunks = 4;       // columns per thread, at most: widths up to 2048
constexpr int kResClusters = 31;    // clusters of a launch, at most: a lane each, and one for a withheld one

struct ResArgs {
    HogArgs h;
    unsigned long long* post;  // [2][kResClusters][2]: the clusters' candidates, by iteration parity
    int rows;                  // rows per CTA
};

__device__ __forceinline__ unsigned smem_addr(const void* p) { return unsigned(__cvta_generic_to_shared(p)); }

// one candidate to CTA `cta` of the cluster, counted there by its barrier
__device__ __forceinline__ void send_key(const unsigned long long* slot, const unsigned long long* bar, int cta,
                                         unsigned long long key)
{
    unsigned dst, mb;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(dst) : "r"(smem_addr(slot)), "r"(cta));
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(mb) : "r"(smem_addr(bar)), "r"(cta));
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.u64 [%0], %1, [%2];" ::"r"(dst), "l"(key), "r"(mb)
                 : "memory");
}
__device__ __forceinline__ void expect_bytes(const unsigned long long* bar, int bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
// waits for the barrier's phase; false after wait_ns (or the iteration cap)
__device__ __forceinline__ bool wait_phase(const unsigned long long* bar, unsigned phase, unsigned long long wait_ns)
{
    unsigned long long t0 = 0;
    for (unsigned spin = 0; spin < (1u << 24); ++spin) {
        unsigned ok;
        asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
                     " selp.u32 %0, 1, 0, p;\n}" : "=r"(ok) : "r"(smem_addr(bar)), "r"(phase) : "memory");
        if (ok) return true;
        if ((spin & 63u) == 63u) {
            if (!t0)
                t0 = global_ns();
            else if (global_ns() - t0 >= wait_ns)
                return false;
        }
    }
    return false;
}

// rows whose PSF values are loaded into registers: 32 values a thread at most, beside up to 64 pixels
__host__ __device__ constexpr int res_direct(int rows, int chunks) { return rows * chunks <= 32 ? rows : 32 / chunks; }

template <int kRowsT, int kChunks, bool kOne>
__global__ void __launch_bounds__(kResThreads, 1) hog_resident_kernel(ResArgs a, int niters, unsigned long long wait_ns,
                                                                      unsigned int withheld)
{
    constexpr int kDirect = res_direct(kRowsT, kChunks);
    extern __shared__ __align__(16) float later[];  // [(kRowsT - kDirect) * kChunks][kResThreads]
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    __shared__ unsigned long long got[2][16], win[2];    // by iteration parity: the cluster's candidates; the winner
    __shared__ unsigned long long bar_got[2], bar_win[2];
    __shared__ unsigned long long key;
    __shared__ unsigned wk[kResThreads / 32];
    HogState* st = a.h.state;
    const int tid = int(threadIdx.x), warp = tid >> 5, lane = tid & 31;
    const int W = a.h.width, P = a.h.psf_width;
    const int ctas = int(cluster.num_blocks()), rank = int(cluster.block_rank()), cl = int(blockIdx.x) / ctas;
    const int ncl = int(gridDim.x) / ctas;
    const int y0 = int(blockIdx.x) * a.rows, ye = min(W, y0 + a.rows);
    if (tid == 0) {
        for (int p = 0; p < 2; ++p) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bar_got[p])) : "memory");
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&bar_win[p])) : "memory");
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    float r[kRowsT][kChunks];
#pragma unroll
    for (int i = 0; i < kRowsT; ++i)
#pragma unroll
        for (int j = 0; j < kChunks; ++j) {
            const int x = tid + j * kResThreads, y = y0 + i;
            r[i][j] = x < W && y < ye ? a.h.residual[size_t(y) * W + x] : __int_as_float(0x7fffffff);  // never a peak
        }
    const int px = int(st->psf_pos % unsigned(P)), py = int(st->psf_pos / unsigned(P));
    const unsigned int flat = key_index(st->win_key[0]);  // the dirty image's scan
    int rx = int(flat % unsigned(W)), ry = int(flat / unsigned(W));
    float peak = st->win_val[0];
    // the model update of the last iteration, its load left in flight (one thread of the first CTA)
    const bool models = blockIdx.x == 0 && tid == kResThreads - 1;
    float m_old = 0.f, m_add = 0.f;
    size_t m_pos = 0;
    bool m_open = false;
    unsigned long long skipped = 0;
    cluster.sync();  // every CTA runs (its shared memory is written to)
    for (int it = 0; it < niters; ++it) {
        const int par = it & 1;
        const unsigned phase = unsigned(it >> 1) & 1u;
        if (fabsf(peak) < a.h.threshold) {  // every CTA holds the same winner: all stop here (HogbomGolden.cc:86-89)
            if (models) st->stopped = it + 1;
            break;
        }
        const int diffx = rx - px, diffy = ry - px;  // diffy uses px, as the reference does
        const int startx = max(0, diffx), stopx = min(W - 1, rx + (P - px - 1));
        const int starty = max(0, ry - py), stopy = min(W - 1, ry + (P - py - 1));
        // rows whose PSF row lies inside the PSF (all of them unless its peak is off the diagonal)
        const int ya = max(starty, diffy), yb = min(stopy, diffy + P - 1);
        const float t = __fmul_rn(a.h.gain, peak);
        if (tid == 0) {
            if (kOne || rank == 0) expect_bytes(&bar_got[par], (ctas + (kOne ? int(withheld) : 0)) * 8);
            if (!kOne) expect_bytes(&bar_win[par], 8);
        }
        if (models) {  // model[absPeakPos] += absPeakVal * g_gain (HogbomGolden.cc:93)
            if (m_open) a.h.model[m_pos] = __fadd_rn(m_old, m_add);
            m_pos = size_t(ry) * W + rx;
            m_add = __fmul_rn(peak, a.h.gain);
            m_old = *reinterpret_cast<volatile float*>(a.h.model + m_pos);
            m_open = true;
            if (a.h.hist_val) a.h.hist_val[it] = peak;
            if (a.h.hist_pos) a.h.hist_pos[it] = unsigned(m_pos);
            st->done = it + 1;
            skipped += (unsigned long long)(stopy - starty + 1 - max(0, yb - ya + 1));
        }
        const float* __restrict__ p0 = a.h.psf + (ptrdiff_t(y0 - diffy) * P + (tid - diffx));
        // per chunk, what the update covers of the thread's column: all its rows (2; the common case,
        // without a test per pixel), some (1) or none (0).  Rows past the image count as covered: they
        // hold NaN.  A test per row and pixel cost 32 rows 1 us.
        const int lasty = min(ry + (P - py - 1), diffy + P - 1);
        const int rows = y0 >= ya && y0 + kRowsT - 1 <= lasty ? 2 : ya < ye && yb >= y0 ? 1 : 0;
        int state[kChunks];
#pragma unroll
        for (int j = 0; j < kChunks; ++j) {
            const int x = tid + j * kResThreads;
            state[j] = x >= startx && x <= stopx ? rows : 0;
        }
        auto on = [&](int i) { return y0 + i >= ya && y0 + i <= yb; };
        // the whole iteration's PSF values in flight at once: the later rows' by asynchronous copies to
        // this thread's own places in shared memory, the first rows' in registers
        // (half of them loaded after the other half cost a fifth more at 16 rows of four columns)
        float pv[kDirect][kChunks], top = -1.f;  // only the largest |value| is kept here
#pragma unroll
        for (int j = 0; j < kChunks; ++j) {
            const float* __restrict__ q = p0 + j * kResThreads;
            if (state[j] == 2) {
#pragma unroll
                for (int i = kDirect; i < kRowsT; ++i)
                    __pipeline_memcpy_async(later + ((i - kDirect) * kChunks + j) * kResThreads + tid, q + ptrdiff_t(i) * P, 4);
#pragma unroll
                for (int i = 0; i < kDirect; ++i) pv[i][j] = __ldg(q + ptrdiff_t(i) * P);
            } else if (state[j] == 1) {
#pragma unroll
                for (int i = kDirect; i < kRowsT; ++i)
                    if (on(i))
                        __pipeline_memcpy_async(later + ((i - kDirect) * kChunks + j) * kResThreads + tid, q + ptrdiff_t(i) * P, 4);
#pragma unroll
                for (int i = 0; i < kDirect; ++i)
                    if (on(i)) pv[i][j] = __ldg(q + ptrdiff_t(i) * P);
            }
        }
        if (kDirect < kRowsT) __pipeline_commit();
        auto value = [&](int i, int j) {
            return i < kDirect ? pv[i < kDirect ? i : 0][j] : later[((i < kDirect ? 0 : i - kDirect) * kChunks + j) * kResThreads + tid];
        };
#pragma unroll
        for (int i0 = 0; i0 < kRowsT; i0 += kDirect) {
            if (i0) __pipeline_wait_prior(0);
#pragma unroll
            for (int j = 0; j < kChunks; ++j) {
                if (state[j] == 2) {
#pragma unroll
                    for (int i = i0; i < i0 + kDirect && i < kRowsT; ++i) r[i][j] = __fsub_rn(r[i][j], __fmul_rn(t, value(i, j)));
                } else if (state[j] == 1) {
#pragma unroll
                    for (int i = i0; i < i0 + kDirect && i < kRowsT; ++i)
                        if (on(i)) r[i][j] = __fsub_rn(r[i][j], __fmul_rn(t, value(i, j)));
                }
            }
        }
#pragma unroll
        for (int i = 0; i < kRowsT; ++i)
#pragma unroll
            for (int j = 0; j < kChunks; ++j) top = fmaxf(top, fabsf(r[i][j]));  // (places past the image hold NaN)
        // the CTA's largest |value|, then its first place (only threads that hold that value look)
        const unsigned mine = top < 0.f ? 0u : __float_as_uint(top) + 1u;
        const unsigned most = __reduce_max_sync(0xffffffffu, mine);
        if (lane == 0) wk[warp] = most;
        if (tid == 0) key = 0;
        __syncthreads();
        const unsigned all = __reduce_max_sync(0xffffffffu, lane < kResThreads / 32 ? wk[lane] : 0u);
        if (mine == all && all) {
            int at = 0;
            float tv = 0.f;
#pragma unroll
            for (int e = kRowsT * kChunks - 1; e >= 0; --e)  // rows, then columns in order: the thread's first
                if (fabsf(r[e / kChunks][e % kChunks]) == top) {
                    at = e;
                    tv = r[e / kChunks][e % kChunks];
                }
            atomicMax(&key, cand_key(tv, tid + at % kChunks * kResThreads, y0 + at / kChunks));
        }
        __syncthreads();
        unsigned long long c;
        bool ok = true;
        if (kOne) {  // one cluster: every CTA sends its candidate to every other
            if (warp == 0 && lane < ctas) send_key(&got[par][rank], &bar_got[par], lane, key);
        } else if (warp == 0) {
            c = key;
            if (lane == 0) send_key(&got[par][rank], &bar_got[par], 0, c);
            if (rank == 0) {
                ok = wait_phase(&bar_got[par], phase, wait_ns);
                c = warp_max(lane < ctas ? got[par][lane] : 0ull);
                volatile unsigned long long* w = a.post + size_t(par) * kResClusters * 2;
                const unsigned long long tag = unsigned(it + 1);
                // two words, each with the iteration: a reader takes them when both are there.  Two
                // buffers suffice: a cluster posts iteration it + 2's after it has all of it + 1's.
                if (lane == 0) {
                    w[cl * 2] = (c & 0xffffffff00000000ull) | tag;
                    w[cl * 2 + 1] = (c << 32) | tag;
                }
                c = 0;
                if (lane < ncl + int(withheld)) {
                    bool here = false;
                    unsigned long long t0 = 0;
                    for (unsigned spin = 0; spin < (1u << 26) && ok; ++spin) {
                        const unsigned long long k0 = w[min(lane, ncl - 1) * 2], k1 = w[min(lane, ncl - 1) * 2 + 1];
                        if (lane < ncl && unsigned(k0) == unsigned(tag) && unsigned(k1) == unsigned(tag)) {
                            c = (k0 & 0xffffffff00000000ull) | (k1 >> 32);
                            here = true;
                            break;
                        }
                        if ((spin & 63u) == 63u) {
                            if (*reinterpret_cast<volatile int*>(&st->error)) break;
                            if (!t0) t0 = global_ns();
                            if (global_ns() - t0 >= wait_ns) break;
                        }
                    }
                    ok = here;
                }
                ok = __all_sync(0xffffffffu, ok);
                c = warp_max(c);
                if (!ok) st->error = 1;
                if (ok && lane < ctas) send_key(&win[par], &bar_win[par], lane, c);
            }
        }
        if (ok) ok = wait_phase(kOne ? &bar_got[par] : &bar_win[par], phase, wait_ns);
        if (!__syncthreads_and(ok)) {
            st->error = 1;
            break;
        }
        c = kOne ? warp_max(lane < ctas ? got[par][lane] : 0ull) : win[par];
        const bool zero = (c >> 33) == 0;  // an all-zero residual: the reference keeps maxPos = 0, maxVal = 0
        const unsigned int idx = zero ? 0u : cand_index(c);
        rx = int(idx & 0xffffu);
        ry = int(idx >> 16);
        peak = zero ? 0.f : cand_value(c);
    }
#pragma unroll
    for (int i = 0; i < kRowsT; ++i)
#pragma unroll
        for (int j = 0; j < kChunks; ++j) {
            const int x = tid + j * kResThreads, y = y0 + i;
            if (x < W && y < ye) a.h.residual[size_t(y) * W + x] = r[i][j];
        }
    if (models && m_open) a.h.model[m_pos] = __fadd_rn(m_old, m_add);
    if (models && skipped) st->skipped_rows = skipped;
    cluster.sync();  // no CTA leaves while another's store to it may be under way
}

// ------------------------------------------------------------------------------------------
// Larger images: put-off updates (see the top of the file).
// ------------------------------------------------------------------------------------------
// One update as the blocks apply it: residual[y][x] -= t * psf[y * P + x + off] for the pixels
// (x, y) of the image that the PSF's rows and columns cover.
struct Update {
    float t;
    int off;
    unsigned int xr, yr;  // first | last << 16
};

// How the applying CTAs share PSF windows among updates at one peak: the ring is walked in batches
// of at most kSlots windows; an update's window is loaded unless an update of the batch already
// has (prev: the last earlier update in the ring at the same place, or -1).
struct UpdateSlot {
    short prev, slot, batch, pad;  // batch: ring index its batch starts at
};

// Where passes over the image take over from put-off updates (hog_pass_kernel): with more blocks than these
struct PassLimits {
    int near, tops;    // at the start: near half the peak (-1: always); above the second peak's limit
    int warm, visits;  // later: of the last launch's list for hog_apply_kernel; hot in a leading CTA
};

struct DeferArgs {
    HogArgs h;
    float* bound;           // per image block: limit of its |residual| as of the last update
    int* applied;           // per image block: iterations whose updates it has
    unsigned int* warm;     // st->nwarm blocks that hog_apply_kernel is to bring up to date
    const float* pmax;      // per PSF block: its largest |value|
    Update* ring;           // [kRing] updates of the iterations from base on
    UpdateSlot* slots;      // [kRing]
    int lb, nbx;            // log2 of the block side; blocks per image side
    int lbp, npx;           // the same of the PSF
    unsigned long long wait_ns;  // limit of a wait
    unsigned int withheld;       // candidates or arrivals more than are made (tcv_hogbom_set_wait)
};

// An update's cover of the 32 columns from x0 and `rows` rows from y0: whole (2; they then lie
// inside the image), in part (1) or none (0).
__device__ __forceinline__ int cover_of(const Update& u, int x0, int y0, int rows)
{
    const int xa = int(u.xr & 0xffffu), xb = int(u.xr >> 16), ya = int(u.yr & 0xffffu), yb = int(u.yr >> 16);
    if (xa <= x0 && xb >= x0 + 31 && ya <= y0 && yb >= y0 + rows - 1) return 2;
    return xa > x0 + 31 || xb < x0 || ya > y0 + rows - 1 || yb < y0 ? 0 : 1;
}

// Block b of an image by one warp: its largest |value| into top[b], the key returned; copies the
// block when copy_to is given.
__device__ __forceinline__ unsigned long long scan_block(const float* __restrict__ img, float* __restrict__ copy_to, int W,
                                                         int lb, int nbx, int b, float* top)
{
    const int lane = threadIdx.x & 31;
    const int x0 = (b % nbx) << lb, y0 = (b / nbx) << lb, side = 1 << lb;
    const int ye = min(W, y0 + side);
    unsigned long long k = 0;
    for (int x = x0 + lane; x < min(W, x0 + side); x += 32) {
        float t = -1.f, tv = 0.f;
        int ty = 0;
        for (int y = y0; y < ye; y += 8) {
            float v[8];
#pragma unroll
            for (int r = 0; r < 8; ++r) v[r] = y + r < ye ? __ldcs(img + (size_t(y + r) * W + x)) : 0.f;
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                if (y + r >= ye) break;
                if (copy_to) copy_to[size_t(y + r) * W + x] = v[r];
                if (fabsf(v[r]) > t) {  // rows in order: strict '>' keeps the first
                    t = fabsf(v[r]);
                    tv = v[r];
                    ty = y + r;
                }
            }
        }
        if (t >= 0.f) k = max(k, cand_key(tv, x, ty));
    }
    k = warp_max(k);
    if (lane == 0) top[b] = cand_abs(k);
    return k;
}

// The largest of the blocks' candidates, to every thread: its value v, and its flat index returned (an
// all-zero image: 0 and 0, as findPeak has it).
__device__ __forceinline__ unsigned int win_of(const unsigned long long* keys, const float* vals, int n, float& v)
{
    unsigned long long k = 0;
    v = 0.f;
    for (int i = threadIdx.x; i < n; i += kHogThreads) {
        const unsigned long long ki = __ldcg(keys + i);
        if (ki > k) {
            k = ki;
            v = __ldcg(vals + i);
        }
    }
    k = block_max(k, v);
    if ((k >> 32) != 0) return key_index(k);
    v = 0.f;
    return 0u;
}

// Both images' blocks (one warp per block) and peaks, residual = dirty, in one launch; the CTA that
// finishes last finds the peaks and counts the blocks of the dirty image that say whether put-off updates
// pay (a launch for each image and none for the count: as long).
__global__ void __launch_bounds__(kHogThreads) hog_blocks_kernel(DeferArgs a, const float* __restrict__ dirty, float* pmax)
{
    HogState* st = a.h.state;
    const int W = a.h.width, P = a.h.psf_width, nb = a.nbx * a.nbx, np = a.npx * a.npx, ctas = int(gridDim.x);
    const int warp = int(blockIdx.x) * (kHogThreads / 32) + (threadIdx.x >> 5), warps = ctas * (kHogThreads / 32);
    unsigned long long best[2] = {0, 0};  // the image's, the PSF's
    for (int b = warp; b < np + nb; b += warps)
        if (b < np) {
            best[1] = max(best[1], scan_block(a.h.psf, nullptr, P, a.lbp, a.npx, b, pmax));
        } else {
            best[0] = max(best[0], scan_block(dirty, a.h.residual, W, a.lb, a.nbx, b - np, a.bound));
            if ((threadIdx.x & 31) == 0) a.applied[b - np] = 0;
        }
    __shared__ bool last;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        // the one-pass kernels' form of a candidate: a flat index, and the value beside it
        const unsigned int at = cand_index(best[i]), flat = (at >> 16) * unsigned(i ? P : W) + (at & 0xffffu);
        float v = cand_value(best[i]);
        const unsigned long long k = block_max(best[i] ? ((best[i] >> 33) << 32) | unsigned(~flat) : 0ull, v);
        if (threadIdx.x == 0) {
            a.h.keys[i * ctas + blockIdx.x] = k;
            a.h.vals[i * ctas + blockIdx.x] = v;
        }
    }
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(&st->arrived, 1u) == unsigned(ctas - 1);
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    float peak, psf_peak;
    const unsigned int ppos = win_of(a.h.keys, a.h.vals, ctas, peak);
    const unsigned int psf_pos = win_of(a.h.keys + ctas, a.h.vals + ctas, ctas, psf_peak);
    unsigned int near = 0, tops = 0;
    const int px = int(psf_pos % unsigned(P));
    const float half = 0.5f * fabsf(peak);
    // the peak's pixel after the first update, a lower limit of the second peak (see hog_lead_kernel)
    const float least = fabsf(__fsub_rn(peak, __fmul_rn(__fmul_rn(a.h.gain, peak), a.h.psf[size_t(px) * P + px])));
    for (int b = threadIdx.x; b < nb; b += kHogThreads) {
        const float top = __ldcg(a.bound + b);
        near += !(top < half);
        tops += !(top < least);
    }
    near = __reduce_add_sync(0xffffffffu, near);
    tops = __reduce_add_sync(0xffffffffu, tops);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&st->near, near);
        atomicAdd(&st->tops, tops);
    }
    if (threadIdx.x == 0) {
        st->win_key[0] = static_cast<unsigned int>(~ppos);
        st->win_val[0] = peak;
        st->psf_pos = psf_pos;
        st->arrived = 0;
    }
}

constexpr int kLeadRows = 8;  // rows per warp: four warps per hot block, four blocks at a time
constexpr int kLeadGroup = 32 / kLeadRows;

struct LeadShared {
    Update ring[kRing];
    unsigned long long cand[2][kLeadCtas];  // the cluster's candidates, by iteration parity
    unsigned long long arrived[2];          // mbarriers: all of cand[parity] is here
    float bound[kOwned];
    int applied[kOwned];
    unsigned int at[kOwned];                // first row << 16 | first column
    unsigned short hot[kOwned];
    int nhot[2];
};

// The blocks are dealt to the cluster's CTAs in 4 x (CTAs / 4) tiles, so that neighbours, which
// are hot together, are different CTAs'.  Block `own` of CTA `rank`:
struct LeadDeal {
    int nox, noy;  // blocks of a CTA per row and per column (some past the image)
    __host__ __device__ LeadDeal(int nbx, int ctas) : nox((nbx + 3) / 4), noy((nbx + ctas / 4 - 1) / (ctas / 4)) {}
    __device__ int x(int own, int rank) const { return own % nox * 4 + (rank & 3); }
    __device__ int y(int own, int rank, int ctas) const { return own / nox * (ctas / 4) + (rank >> 2); }
};

// The pending updates up to iteration `to` of the CTA's nhot hot blocks, four warps per block, and the
// blocks' candidates.  One short loop for every case (the code of an iteration has to stay in the
// instruction cache: an iteration runs each line once).
__device__ __forceinline__ void lead_apply(const DeferArgs& a, LeadShared& sh, unsigned long long* parts, int nhot, int base,
                                           int to)
{
    constexpr int kRows = kLeadRows, kDeep = 4;  // kDeep updates' loads are in flight together
    const int W = a.h.width, P = a.h.psf_width;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = warp / kLeadGroup; i < nhot; i += kLeadWarps / kLeadGroup) {
        const int own = sh.hot[i], from = sh.applied[own];
        unsigned long long c = 0;
        for (int part = 0; part < 1 << (2 * (a.lb - 5)); ++part) {  // 32 x 32 pixels of the block
            const int x = int(sh.at[own] & 0xffffu) + ((part & ((1 << (a.lb - 5)) - 1)) << 5) + lane;
            const int y = int(sh.at[own] >> 16) + ((part >> (a.lb - 5)) << 5) + (warp % kLeadGroup) * kRows;
            const int rows = x < W ? min(kRows, W - y) : 0;  // none past the image
            float r[kRows];
            float* rp = a.h.residual + (size_t(y) * W + x);
#pragma unroll
            for (int k = 0; k < kRows; ++k) r[k] = k < rows ? rp[size_t(k) * W] : 0.f;
            const float* __restrict__ pp = a.h.psf + (ptrdiff_t(y) * P + x);
#pragma unroll 1
            for (int q = from; q < to; q += kDeep) {
                float pv[kDeep][kRows];
#pragma unroll
                for (int d = 0; d < kDeep; ++d) {
                    if (q + d >= to) break;
                    const Update u = sh.ring[q + d - base];
                    const int ya = int(u.yr & 0xffffu), yb = int(u.yr >> 16);
                    const bool cx = x >= int(u.xr & 0xffffu) && x <= int(u.xr >> 16);
#pragma unroll
                    for (int k = 0; k < kRows; ++k)
                        pv[d][k] = cx && y + k >= ya && y + k <= yb ? __ldg(pp + (u.off + ptrdiff_t(k) * P)) : 0.f;
                }
#pragma unroll
                for (int d = 0; d < kDeep; ++d) {
                    if (q + d >= to) break;
                    const Update u = sh.ring[q + d - base];
                    const int ya = int(u.yr & 0xffffu), yb = int(u.yr >> 16);
                    const bool cx = x >= int(u.xr & 0xffffu) && x <= int(u.xr >> 16);
#pragma unroll
                    for (int k = 0; k < kRows; ++k)
                        if (cx && y + k >= ya && y + k <= yb) r[k] = __fsub_rn(r[k], __fmul_rn(u.t, pv[d][k]));
                }
            }
            float top = -1.f, tv = 0.f;
            int ty = 0;
#pragma unroll
            for (int k = 0; k < kRows; ++k)
                if (k < rows) {
                    rp[size_t(k) * W] = r[k];
                    if (fabsf(r[k]) > top) {
                        top = fabsf(r[k]);
                        tv = r[k];
                        ty = y + k;
                    }
                }
            c = max(c, top < 0.f ? 0ull : cand_key(tv, x, ty));
        }
        c = warp_max(c);
        if (lane == 0) parts[i * kLeadGroup + warp % kLeadGroup] = c;
    }
}


// Iterations [it0, it1) by one cluster; the ring holds the updates from iteration base on.
__global__ void __launch_bounds__(kLeadThreads, 1) hog_lead_kernel(DeferArgs a, int it0, int it1, int base)
{
    extern __shared__ __align__(16) unsigned char lead_smem[];
    LeadShared& sh = *reinterpret_cast<LeadShared*>(lead_smem);
    const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
    HogState* st = a.h.state;
    cudaGridDependencySynchronize();  // launched ahead of the end of the kernel before
    if (st->stopped || st->error) return;  // an earlier launch stopped the loop (the whole cluster returns)
    const int tid = int(threadIdx.x), warp = tid >> 5, lane = tid & 31;
    if (blockIdx.x == 0 && tid == 0) st->meet = 0;  // for the next launch of passes
    if (st->pass) return;
    const int W = a.h.width, P = a.h.psf_width, ctas = int(gridDim.x), rank = int(blockIdx.x);
    const int side = 1 << a.lb;
    const LeadDeal deal(a.nbx, ctas);
    const int owned = deal.nox * deal.noy;
    // the hot blocks' candidates, a part per warp; the PSF blocks' largest |value|
    unsigned long long* parts = reinterpret_cast<unsigned long long*>(lead_smem + sizeof(LeadShared));
    float* pmax = reinterpret_cast<float*>(parts + owned * kLeadGroup);
    for (int i = tid; i < owned; i += kLeadThreads) {
        const int x = deal.x(i, rank), y = deal.y(i, rank, ctas);
        const bool in = x < a.nbx && y < a.nbx;
        sh.bound[i] = in ? a.bound[y * a.nbx + x] : 0.f;
        sh.applied[i] = in ? a.applied[y * a.nbx + x] : 0;
        sh.at[i] = in ? unsigned(y) << (16 + a.lb) | unsigned(x) << a.lb : 0xffffffffu;
    }
    for (int i = tid; i < it0 - base; i += kLeadThreads) sh.ring[i] = a.ring[i];
    for (int i = tid; i < a.npx * a.npx; i += kLeadThreads) pmax[i] = a.pmax[i];
    if (rank == 0 && tid == 0) st->nwarm = st->visits = 0;
    if (tid == 0) {
        sh.nhot[0] = sh.nhot[1] = 0;
        for (int p = 0; p < 2; ++p)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&sh.arrived[p])) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    const int px = int(st->psf_pos % unsigned(P)), py = int(st->psf_pos / unsigned(P));
    const float at_peak = a.h.psf[size_t(px) * P + px];  // what an update takes t times of at its own peak
    const unsigned int flat = key_index(st->win_key[0]);  // the scan's, or the last launch's last
    int rx = int(flat % unsigned(W)), ry = int(flat / unsigned(W));
    float peak = st->win_val[0];
    // the model update of the last iteration, its load left in flight (one thread of the first CTA);
    // the ring's entries are another thread's, both in warps that seldom have a block's bound
    const bool models = rank == 0 && tid == kLeadThreads - 32, rings = tid == kLeadThreads - 64;
    float m_old = 0.f, m_add = 0.f;
    size_t m_pos = 0;
    bool m_open = false;
    unsigned long long skipped = 0;
    unsigned int visits = 0;
    int it = it0;
    cluster.sync();  // every CTA runs (its shared memory is written to) and has read the state
    for (; it < it1; ++it) {
        const int par = it & 1;
        if (fabsf(peak) < a.h.threshold) {  // every CTA holds the same winner: all stop here (HogbomGolden.cc:86-89)
            if (rank == 0 && tid == 0) st->stopped = it + 1;
            break;
        }
        const int diffx = rx - px, diffy = ry - px;  // diffy uses px, as the reference does
        const float t = __fmul_rn(a.h.gain, peak), at = fabsf(t);
        const float least = fabsf(__fsub_rn(peak, __fmul_rn(t, at_peak)));  // the peak's pixel after the update
        if (tid == 0) {
            sh.nhot[par ^ 1] = 0;
            expect_bytes(&sh.arrived[par], (ctas + int(a.withheld)) * 8);
        }
        if (rings) {
            const int startx = max(0, diffx), stopx = min(W - 1, rx + (P - px - 1));
            const int starty = max(0, ry - py), stopy = min(W - 1, ry + (P - py - 1));
            // rows whose PSF row lies inside the PSF (all of them unless its peak is off the diagonal)
            const int ya = max(starty, diffy), yb = min(stopy, diffy + P - 1);
            Update u;
            u.t = t;
            u.off = -(diffy * P + diffx);
            u.xr = unsigned(startx) | (unsigned(stopx) << 16);
            u.yr = yb >= ya ? unsigned(ya) | (unsigned(yb) << 16) : 1u;  // no row: first > last
            sh.ring[it - base] = u;
            if (rank == 0) a.ring[it - base] = u;
            skipped += (unsigned long long)(stopy - starty + 1 - max(0, yb - ya + 1));
        }
        if (models) {  // model[absPeakPos] += absPeakVal * g_gain (HogbomGolden.cc:93)
            if (m_open) a.h.model[m_pos] = __fadd_rn(m_old, m_add);
            m_pos = size_t(ry) * W + rx;
            m_add = __fmul_rn(peak, a.h.gain);
            m_old = *reinterpret_cast<volatile float*>(a.h.model + m_pos);
            m_open = true;
            if (a.h.hist_val) a.h.hist_val[it] = peak;
            if (a.h.hist_pos) a.h.hist_pos[it] = unsigned(m_pos);
            st->done = it + 1;
        }
        for (int i = tid; i < owned; i += kLeadThreads) {
            const unsigned int where = sh.at[i];
            if (where == 0xffffffffu) continue;
            const int bx = int(where & 0xffffu), by = int(where >> 16);
            float bound = sh.bound[i];
            // the PSF under the block (clipped to the PSF: where it ends nothing is subtracted)
            const int u0 = max(0, bx - diffx), u1 = min(P - 1, bx + side - 1 - diffx);
            const int v0 = max(0, by - diffy), v1 = min(P - 1, by + side - 1 - diffy);
            if (u0 <= u1 && v0 <= v1) {
                const int c0 = u0 >> a.lbp, c1 = u1 >> a.lbp;
                const float *p0 = pmax + (v0 >> a.lbp) * a.npx, *p1 = pmax + (v1 >> a.lbp) * a.npx;
                const float top = fmaxf(fmaxf(p0[c0], p0[c1]), fmaxf(p1[c0], p1[c1]));
                bound = __fadd_ru(bound, __fmul_ru(at, top));
                sh.bound[i] = bound;
            }
            if (!(bound < least)) {  // also when either is not a number
                sh.hot[atomicAdd(&sh.nhot[par], 1)] = (unsigned short)(i);
            }
        }
        __syncthreads();
        const int nhot = sh.nhot[par];
        visits += unsigned(nhot);
        lead_apply(a, sh, parts, nhot, base, it + 1);
        __syncthreads();
        if (warp == 0) {
            unsigned long long c = 0;
            for (int i = lane; i < nhot; i += 32) {
                const int own = sh.hot[i];
                unsigned long long k = parts[i * kLeadGroup];
#pragma unroll
                for (int j = 1; j < kLeadGroup; ++j) k = max(k, parts[i * kLeadGroup + j]);
                sh.bound[own] = cand_abs(k);
                sh.applied[own] = it + 1;
                c = max(c, k);
            }
            c = warp_max(c);
            // to every CTA of the cluster, each store counted by that CTA's barrier.  Two buffers
            // suffice: a CTA sends iteration it + 2's after it has all of it + 1's, which the
            // others sent having read it's.
            if (lane < ctas) send_key(&sh.cand[par][rank], &sh.arrived[par], lane, c);
        }
        // this parity's barrier completes once per two iterations of this launch
        const unsigned phase = unsigned((it - it0) >> 1) & 1u;
        if (!__syncthreads_and(wait_phase(&sh.arrived[par], phase, a.wait_ns))) {  // leave (tcv_hogbom_result says so)
            st->error = 1;
            break;
        }
        const unsigned long long c = warp_max(lane < ctas ? sh.cand[par][lane] : 0ull);
        const bool zero = (c >> 33) == 0;  // an all-zero residual: the reference keeps maxPos = 0, maxVal = 0
        const unsigned int idx = zero ? 0u : cand_index(c);
        rx = int(idx & 0xffffu);
        ry = int(idx >> 16);
        peak = zero ? 0.f : cand_value(c);
    }
    cluster.sync();  // no CTA leaves while another's store to it may be under way
    for (int i = tid; i < owned; i += kLeadThreads) {
        if (sh.at[i] == 0xffffffffu) continue;
        const int b = deal.y(i, rank, ctas) * a.nbx + deal.x(i, rank);
        a.bound[b] = sh.bound[i];
        a.applied[b] = sh.applied[i];
        // near the peak: soon to be hot, and better without a long chain of updates to catch up on
        if (sh.applied[i] < it && !(sh.bound[i] < 0.5f * fabsf(peak))) a.warm[atomicAdd(&st->nwarm, 1u)] = unsigned(b);
    }
    if (tid == 0) atomicMax(&st->visits, visits);
    if (rank != 0) return;
    if (models && m_open) a.h.model[m_pos] = __fadd_rn(m_old, m_add);
    if (rings && skipped) st->skipped_rows += skipped;
    if (tid == 0) {
        st->win_key[0] = static_cast<unsigned int>(~(unsigned(ry) * unsigned(W) + unsigned(rx)));
        st->win_val[0] = peak;
    }
    // this launch's updates: the last earlier one at the same place, a warp per update; then the
    // batches and windows, on from the state of the last launch
    __shared__ short prev[kLeadIters];
    for (int j = warp; j < it - it0; j += kLeadWarps) {
        const int q = it0 - base + j;
        const Update u = sh.ring[q];
        int last = -1;
        for (int i = lane; i < q; i += 32) {
            const Update o = sh.ring[i];
            if (o.off == u.off && o.xr == u.xr && o.yr == u.yr) last = i;
        }
        last = __reduce_max_sync(0xffffffffu, last);
        if (lane == 0) prev[j] = short(last);
    }
    __syncthreads();
    if (tid == 0) {
        int batch = it0 == base ? 0 : st->batch, used = it0 == base ? 0 : st->used;
        for (int j = 0; j < it - it0; ++j) {
            const int q = it0 - base + j, p = prev[j];
            int slot;
            if (p >= batch) {
                slot = a.slots[p].slot;
            } else {
                if (used == kSlots) {
                    batch = q;
                    used = 0;
                }
                slot = used++;
            }
            a.slots[q] = UpdateSlot{short(p), short(slot), short(batch), 0};
        }
        st->batch = batch;
        st->used = used;
    }
}

// Apply what is pending to every block when `all`, else to those of the warm list.  A CTA works on
// 32 x 16 pixels at a time; a lane keeps its four in registers and walks the updates in order.  The
// PSF values it needs come from windows in shared memory, in which every lane copies
// (asynchronously) and reads its own places only: updates at one peak share a window, so the
// loads from L2 are one per distinct peak of a batch, not one per update, and an update of a pixel
// costs 4 bytes from shared memory, a product and a difference.  Two CTAs of four warps fit on an SM,
// so the copy loop is a chain of latencies: a window's place and cover come in one 16-byte read, the
// reads of four windows go ahead of their copies, and a warp's places of a row are neighbours (one
// float4 a lane made the copies conflict four ways): 15.9 -> 13.5 us an iteration at 4096^2; 52
// windows, the most that two CTAs hold, 12.9 (48: 13.5; 32 at three CTAs: 15.3).  A pass of 128 updates
// over all blocks takes 0.83 ms; loading each update's 4 bytes a pixel from L2 would take 0.67 alone.
// Copying one batch while computing another (two halves of 25 windows) took 20 us an iteration.
__global__ void __launch_bounds__(kApplyThreads) hog_apply_kernel(DeferArgs a, int base, int all)
{
    constexpr int kRows = kApplyRows;
    static_assert(kRows % 2 == 0, "rows in pairs");
    extern __shared__ __align__(16) float apply_win[];  // [kSlots][kWindow]
    __shared__ Update ring[kRing];
    __shared__ UpdateSlot slots[kRing];
    __shared__ float2 code[kRing];  // of the part's updates in order: -t and, as bits, the window
    __shared__ unsigned short which[kRing];               // the codes' ring entries
    __shared__ int4 load[kSlots + kApplyDeep];            // windows to copy: PSF offset, place, columns, rows
    __shared__ unsigned short batch_end[kRing];
    __shared__ int warps[2][kApplyThreads / 32];
    __shared__ unsigned long long wk[kApplyThreads / 32];
    cudaGridDependencySynchronize();  // launched ahead of the leading cluster's end
    // after a wait that ran out the iteration's windows are not laid out, nor is anything kept
    if (a.h.state->pass || a.h.state->error) return;
    const int to = a.h.state->done;
    const int tid = int(threadIdx.x), warp = tid >> 5, lane = tid & 31;
    const int W = a.h.width, P = a.h.psf_width, q1 = to - base, lsub = a.lb - 5;
    const int count = all ? a.nbx * a.nbx : int(a.h.state->nwarm);
    if (q1 <= 0 || count == 0) return;
    for (int i = tid; i < q1; i += kApplyThreads) {
        ring[i] = a.ring[i];
        slots[i] = a.slots[i];
        if (i + 1 == q1 || a.slots[i + 1].batch != a.slots[i].batch) batch_end[a.slots[i].batch] = (unsigned short)(i + 1);
    }
    float* const mine = apply_win + tid;  // this lane's place in the first window
    for (int item = int(blockIdx.x); item < count; item += int(gridDim.x)) {
        const int b = all ? item : int(a.warm[item]);
        const int q0 = a.applied[b] - base;
        if (q0 >= q1) continue;  // the same for the whole CTA, as all that follows but `rows`
        unsigned long long best = 0;
        for (int part = 0; part < kStrips << (2 * lsub); ++part) {
            const int sub = part / kStrips;
            const int x0 = ((b % a.nbx) << a.lb) + ((sub & ((1 << lsub) - 1)) << 5);
            const int y0 = ((b / a.nbx) << a.lb) + ((sub >> lsub) << 5) + part % kStrips * (32 / kStrips);
            if (x0 >= W || y0 >= W) continue;
            const int x = x0 + lane, y = y0 + warp * kRows;
            const int rows = x < W ? min(kRows, W - y) : 0;  // this lane's (none past the image)
            float* rp = a.h.residual + (size_t(y) * W + x);
            float r[kRows];
#pragma unroll
            for (int k = 0; k < kRows; ++k) r[k] = k < rows ? __ldcs(rp + size_t(k) * W) : 0.f;
            const float* __restrict__ pp = a.h.psf + (ptrdiff_t(y) * P + x);
            for (int first = q0; first < q1;) {
                __syncthreads();  // ring and slots are there; the last batch's codes are used
                const int end = batch_end[slots[first].batch];
                // the batch's updates that reach these pixels, in order, and those whose window is to
                // be copied (no earlier one of the batch has it)
                int n = 0, nc = 0;
                bool partial = false;
                for (int i0 = first; i0 < end; i0 += kApplyThreads) {
                    const int i = i0 + tid;
                    const int cover = i < end ? cover_of(ring[i], x0, y0, 32 / kStrips) : 0;
                    const bool copy = cover && slots[i].prev < first;
                    const unsigned bu = __ballot_sync(0xffffffffu, cover != 0), bc = __ballot_sync(0xffffffffu, copy);
                    if (lane == 0) {
                        warps[0][warp] = __popc(bu);
                        warps[1][warp] = __popc(bc);
                    }
                    partial |= __syncthreads_or(cover == 1) != 0;
                    int at = n, atc = nc;
#pragma unroll
                    for (int w = 0; w < kApplyThreads / 32; ++w) {
                        if (w == warp) {
                            at = n;
                            atc = nc;
                        }
                        n += warps[0][w];
                        nc += warps[1][w];
                    }
                    if (cover) {
                        at += __popc(bu & ((1u << lane) - 1u));
                        code[at] = make_float2(-ring[i].t, __int_as_float(int(slots[i].slot) * kWindow));
                        which[at] = (unsigned short)(i);
                    }
                    if (copy)
                        load[atc + __popc(bc & ((1u << lane) - 1u))] =
                            make_int4(ring[i].off, int(slots[i].slot) * kWindow, int(ring[i].xr), int(ring[i].yr));
                    __syncthreads();
                }
                for (int i0 = 0; i0 < nc; i0 += kApplyDeep) {
                    int4 e[kApplyDeep];
#pragma unroll
                    for (int d = 0; d < kApplyDeep; ++d) e[d] = load[i0 + d];
#pragma unroll
                    for (int d = 0; d < kApplyDeep; ++d) {
                        if (i0 + d >= nc) break;
                        const float* __restrict__ src = pp + e[d].x;
                        float* w = mine + e[d].y;
                        const int ya = e[d].w & 0xffff, yb = int(unsigned(e[d].w) >> 16);
                        const bool cx = x >= (e[d].z & 0xffff) && x <= int(unsigned(e[d].z) >> 16);
#pragma unroll
                        for (int k = 0; k < kRows; ++k)
                            if (!partial || (cx && y + k >= ya && y + k <= yb))
                                __pipeline_memcpy_async(w + k * kApplyThreads, src + ptrdiff_t(k) * P, 4);
                    }
                }
                __pipeline_commit();
                __pipeline_wait_prior(0);  // a lane reads only what it copied: no barrier
                if (!partial) {
                    // r + (-t) p is r - t p, bit for bit (the sums one by one: a paired product and a
                    // paired sum would be contracted into one rounding)
#pragma unroll 8
                    for (int i = 0; i < n; ++i) {
                        const float2 cd = code[i], nt = make_float2(cd.x, cd.x);
                        const float* w = mine + __float_as_int(cd.y);
#pragma unroll
                        for (int k = 0; k < kRows; k += 2) {
                            const float2 s = __fmul2_rn(nt, make_float2(w[k * kApplyThreads], w[(k + 1) * kApplyThreads]));
                            r[k] = __fadd_rn(r[k], s.x);
                            r[k + 1] = __fadd_rn(r[k + 1], s.y);
                        }
                    }
                } else {
                    for (int i = 0; i < n; ++i) {
                        const float2 cd = code[i];
                        const Update u = ring[which[i]];
                        const float* w = mine + __float_as_int(cd.y);
                        const int ya = int(u.yr & 0xffffu), yb = int(u.yr >> 16);
                        const bool cx = x >= int(u.xr & 0xffffu) && x <= int(u.xr >> 16);
#pragma unroll
                        for (int k = 0; k < kRows; ++k)
                            if (cx && y + k >= ya && y + k <= yb) r[k] = __fadd_rn(r[k], __fmul_rn(cd.x, w[k * kApplyThreads]));
                    }
                }
                first = end;
            }
            float top = -1.f, tv = 0.f;
            int ty = 0;
#pragma unroll
            for (int k = 0; k < kRows; ++k)
                if (k < rows) {
                    __stcs(rp + size_t(k) * W, r[k]);
                    if (fabsf(r[k]) > top) {
                        top = fabsf(r[k]);
                        tv = r[k];
                        ty = y + k;
                    }
                }
            best = max(best, top < 0.f ? 0ull : cand_key(tv, x, ty));
        }
        best = warp_max(best);
        if (lane == 0) wk[warp] = best;
        __syncthreads();
        if (tid == 0) {
            for (int i = 1; i < kApplyThreads / 32; ++i) best = max(best, wk[i]);
            a.bound[b] = cand_abs(best);
            a.applied[b] = to;
        }
    }
}

// Iterations [it0, it1) with a pass over the image each, all CTAs meeting in between, where put-off
// updates do not pay: where the residual is flat, as a cleaned one is, the next peak may be in thousands of
// blocks, the leading cluster takes most of the time and the applying launches find most blocks near the
// peak.  Takes over for good, at the start of a ring (all blocks are up to date then); until then a launch
// ends at once (3 us each).  From the start for an image with more blocks near half its peak, or above the
// limit of its second peak, than lim says; later by the last launch's list of blocks near the peak and its
// hot blocks (PassLimits pass_limits()).  us for 100 iterations, and in brackets with put-off updates up to
// the first ring's end: an image cleaned before 1900^2 881 (1270), 2600^2 1232 (1819), 4096^2 2342 (3862);
// noise 883 (1655), 1233 (1930), 2504 (3420).
// Two CTAs an SM where the images stay in L2, three beyond (4096^2 26.8 -> 24.5 us an iteration; 2048^2
// 8.4 -> 9.2; they meet at 2800^2).  Two candidate buffers suffice: a CTA cannot write iteration it + 1's
// before every CTA has arrived at barrier it, i.e. has read iteration it - 1's.
template <bool kVec, int kCtas>
__global__ void __launch_bounds__(kHogThreads, kCtas) hog_pass_kernel(HogArgs a, PassLimits lim, int it0, int it1,
                                                                      unsigned long long wait_ns, unsigned int withheld)
{
    HogState* st = a.state;
    // set by an earlier launch, or behind a fence when this one is done
    const bool own = *reinterpret_cast<volatile int*>(&st->pass) != 0;
    if (st->stopped || st->error) return;
    if (!own && (it0 == 0 ? int(st->near) <= lim.near && int(st->tops) <= lim.tops
                          : int(st->nwarm) <= lim.warm && int(st->visits) <= lim.visits))
        return;
    if (own) it0 = max(it0, *reinterpret_cast<volatile int*>(&st->pass_end));
    if (it0 >= it1) return;
    const unsigned int psf_pos = st->psf_pos;
    __shared__ int ok;
    unsigned int ppos = own ? __ldcg(&st->win_next) : key_index(__ldcg(&st->win_key[0]));
    float peak = own ? __ldcg(&st->val_next) : __ldcg(&st->win_val[0]);
    // the CTA's rows (iter_body's): beyond L2, where an update does not reach them its candidate stays as it is
    // and they are not read (4096^2 with a PSF of half the width 21.0 -> 18.8 us an iteration; the test alone
    // costs 2048^2 0.15)
    const int W = a.width, P = a.psf_width, py = int(psf_pos / unsigned(P));
    const int rows = (W + a.nblocks - 1) / a.nblocks, r0 = int(blockIdx.x) * rows, r1 = min(W, r0 + rows);
    unsigned long long best = 0;
    float bv = 0.f;
    int it = it0;
    for (; it < it1; ++it) {
        if (fabsf(peak) < a.threshold) {  // every CTA holds the same winner: all stop here
            if (blockIdx.x == 0 && threadIdx.x == 0) st->stopped = it + 1;
            break;
        }
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            model_update(a, it, ppos, peak);
            st->done = it + 1;
        }
        const int ry = kCtas > 2 ? int(ppos / unsigned(W)) : 0;
        if (kCtas == 2 || it == it0 || (r1 > ry - py && r0 <= ry + (P - py - 1))) {
            unsigned long long skipped;
            best = iter_body<kVec>(a, ppos, peak, psf_pos, bv, skipped);
            if (skipped) atomicAdd(&st->skipped_rows, skipped);
            best = block_max(best, bv);
        }
        unsigned long long* keys = a.keys + (it & 1) * a.nblocks;
        float* vals = a.vals + (it & 1) * a.nblocks;
        if (threadIdx.x == 0) {
            keys[blockIdx.x] = best;
            vals[blockIdx.x] = bv;
            __threadfence();
            atomicAdd(&st->meet, 1u);
            const unsigned int target = unsigned(it - it0 + 1) * unsigned(a.nblocks) + withheld;
            ok = 0;
            const unsigned long long t0 = global_ns();
            for (unsigned int spin = 0; spin < (1u << 24); ++spin) {
                if (*reinterpret_cast<volatile unsigned int*>(&st->meet) >= target) {
                    ok = 1;
                    break;
                }
                if (*reinterpret_cast<volatile int*>(&st->error)) break;
                __nanosleep(32);
                if ((spin & 63u) == 63u && global_ns() - t0 >= wait_ns) break;
            }
            if (!ok) st->error = 1;
            __threadfence();
        }
        __syncthreads();
        if (!ok) return;
        ppos = win_of(keys, vals, a.nblocks, peak);
    }
    // for the next launch.  A CTA that starts only now (all stopped at once) finds what it would have
    // found before.
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->win_next = ppos;
        st->val_next = peak;
        st->pass_end = it;
        __threadfence();
        st->pass = 1;
    }
}

size_t align256(size_t b) { return (b + 255) & ~size_t(255); }

int g_hog_strategy = TCV_HOGBOM_AUTO;
constexpr unsigned long long kDefaultWaitNs = 2000000000ull;  // 2 s
unsigned long long g_wait_ns = kDefaultWaitNs;
unsigned int g_withheld = 0;

int hog_blocks(long long n)
{
    const long long want = (n + 4095) / 4096;  // at least ~4096 pixels per block
    return int(std::max<long long>(1, std::min<long long>(kHogMaxBlocks, want)));
}

// log2 of the block side that covers `width` pixels with at most kBlkSide blocks (32 at least)
int log2_side(int width)
{
    int lb = 5;
    while ((width + (1 << lb) - 1) >> lb > kBlkSide) ++lb;
    return lb;
}

// the workspace: state and the clusters' posted candidates (zeroed per call), candidates of the
// scans, then what put-off updates need
struct HogWork {
    HogState* state;
    unsigned long long *keys, *post;
    float* vals;
    float *bound, *pmax;
    int* applied;
    unsigned int* warm;
    Update* ring;
    UpdateSlot* slots;
    size_t zeroed, total;
    explicit HogWork(void* w)
    {
        char* q = static_cast<char*>(w);
        auto take = [&](size_t bytes) {
            char* r = q;
            q += align256(bytes);
            return static_cast<void*>(r);
        };
        state = static_cast<HogState*>(take(sizeof(HogState)));
        post = static_cast<unsigned long long*>(take(size_t(2) * kResClusters * 2 * 8));
        zeroed = size_t(q - static_cast<char*>(w));
        keys = static_cast<unsigned long long*>(take(size_t(2) * kHogMaxBlocks * 8));  // two sets
        vals = static_cast<float*>(take(size_t(2) * kHogMaxBlocks * 4));
        bound = static_cast<float*>(take(size_t(kBlkMax) * 4));
        pmax = static_cast<float*>(take(size_t(kBlkMax) * 4));
        applied = static_cast<int*>(take(size_t(kBlkMax) * 4));
        warm = static_cast<unsigned int*>(take(size_t(kBlkMax) * 4));
        ring = static_cast<Update*>(take(size_t(kRing) * sizeof(Update)));
        slots = static_cast<UpdateSlot*>(take(size_t(kRing) * sizeof(UpdateSlot)));
        total = size_t(q - static_cast<char*>(w));
    }
};

// Scans of the PSF and of the dirty image that the one-pass kernels and the resident kernel start from:
// the PSF's peak (HogbomGolden.cc:73-76), then residual = dirty with the first scan (:70).
tcv_status first_scans(const HogArgs& a, const float* dirty, cudaStream_t st)
{
    const long long np = (long long)a.psf_width * a.psf_width;
    const int pb = hog_blocks(np), nb = hog_blocks(a.n);
    hog_scan_kernel<<<pb, kHogThreads, 0, st>>>(a.psf, nullptr, np, pb, a.keys, a.vals, a.state, 2);
    TCV_CUDA(cudaGetLastError());
    hog_scan_kernel<<<nb, kHogThreads, 0, st>>>(dirty, a.residual, a.n, nb, a.keys, a.vals, a.state, 0);
    TCV_CUDA(cudaGetLastError());
    return TCV_OK;
}

using ResKernel = void (*)(ResArgs, int, unsigned long long, unsigned int);

template <int kRowsT>
ResKernel resident_of(int chunks)
{
    switch (chunks) {
        case 1: return hog_resident_kernel<kRowsT, 1, false>;
        case 2: return hog_resident_kernel<kRowsT, 2, false>;
        case 3: return hog_resident_kernel<kRowsT, 3, false>;
        default: return hog_resident_kernel<kRowsT, 4, false>;
    }
}

// All iterations with the residual in registers, in one cooperative launch of clusters.  ran = false:
// the image does not fit (or the device cannot hold the clusters), nothing launched.
tcv_status deconvolve_resident(const HogArgs& h, const HogWork& w, const float* dirty, int niters, cudaStream_t st, bool& ran)
{
    ran = false;
    const int W = h.width;
    if (W > kResChunks * kResThreads || h.psf_width > 65535) return TCV_OK;
    int dev = 0, coop = 0, sms = 0;
    TCV_CUDA(cudaGetDevice(&dev));
    TCV_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    TCV_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    if (!coop) return TCV_OK;
    const int chunks = (W + kResThreads - 1) / kResThreads;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeCooperative;
    attr[1].val.cooperative = 1;
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(kResThreads);
    cfg.attrs = attr;
    cfg.stream = st;
    // up to 256 wide in one cluster, which meets in its shared memory alone (128^2: 1.23 us an
    // iteration, 1.75 in clusters that meet through L2; 256^2 1.62 and 1.8; 300^2, with 32 rows a
    // CTA, 2.5 and 1.75)
    for (int rows_t : {-8, -16, 4, 8, 16}) {  // negative: one cluster
        const bool one = rows_t < 0;
        rows_t = std::abs(rows_t);
        if (W > (one ? 16 : sms) * rows_t) continue;  // too few CTAs (asking the device takes 5 us)
        const ResKernel kernel = one ? (rows_t == 8 ? ResKernel(hog_resident_kernel<8, 1, true>)
                                                    : ResKernel(hog_resident_kernel<16, 1, true>))
                                 : rows_t == 4 ? resident_of<4>(chunks)
                                 : rows_t == 8 ? resident_of<8>(chunks)
                                               : resident_of<16>(chunks);
        // clusters of 16 where they fit: half as many meet as of 8 (300^2: 1.80 us an iteration, not 1.91)
        int size = 16, most = 0;
        cfg.dynamicSmemBytes = size_t(rows_t - res_direct(rows_t, chunks)) * chunks * kResThreads * sizeof(float);
        if (cfg.dynamicSmemBytes)
            TCV_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(cfg.dynamicSmemBytes)));
        for (; size >= 8; size /= 2) {
            attr[0].val.clusterDim.x = unsigned(size);
            cfg.gridDim = dim3(unsigned(size));
            cfg.numAttrs = 1;
            if ((size == 8 || cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) &&
                cudaOccupancyMaxActiveClusters(&most, kernel, &cfg) == cudaSuccess && most > 0)
                break;
            cudaGetLastError();
            most = 0;
        }
        most = std::min(most, one ? 1 : kResClusters);
        // rows per CTA: at least four, so that small images meet in few clusters
        const int rows = std::max(4, (W + most * size - 1) / std::max(1, most * size));
        if (most < 1 || rows > rows_t) continue;
        TCV_CHECK(first_scans(h, dirty, st));
        ran = true;
        if (niters == 0) return TCV_OK;
        ResArgs a{h, w.post, rows};
        const int ctas = (W + rows - 1) / rows;
        cfg.gridDim = dim3(unsigned((ctas + size - 1) / size * size));
        cfg.numAttrs = 2;
        TCV_CUDA(cudaLaunchKernelEx(&cfg, kernel, a, niters, g_wait_ns, g_withheld));
        return TCV_OK;
    }
    return TCV_OK;
}

// CTAs of the leading cluster: 16 where one such cluster can be resident, else 8, else 0
int lead_ctas(cudaLaunchConfig_t& cfg, cudaLaunchAttribute& attr, const DeferArgs& a)
{
    constexpr size_t kMost =
        sizeof(LeadShared) + size_t(kBlkMax) / 8 * kLeadGroup * sizeof(unsigned long long) + size_t(kBlkMax) * sizeof(float);
    static_assert(kMost <= 227 * 1024, "shared memory of a CTA");
    attr.id = cudaLaunchAttributeClusterDimension;
    attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
    cfg = cudaLaunchConfig_t{};
    cfg.blockDim = dim3(kLeadThreads);
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    if (cudaFuncSetAttribute(hog_lead_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        cudaGetLastError();
    if (cudaFuncSetAttribute(hog_lead_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kMost)) != cudaSuccess)
        return 0;
    for (int n : {kLeadCtas, 8}) {
        const LeadDeal deal(a.nbx, n);
        cfg.dynamicSmemBytes = sizeof(LeadShared) + size_t(deal.nox) * deal.noy * kLeadGroup * sizeof(unsigned long long) +
                               size_t(a.npx) * a.npx * sizeof(float);
        attr.val.clusterDim.x = unsigned(n);
        cfg.gridDim = dim3(unsigned(n));
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, hog_lead_kernel, &cfg) == cudaSuccess && clusters > 0) return n;
        cudaGetLastError();
    }
    return 0;
}

// At the start: more than 4 % of the blocks near half the peak (sources and their sidelobes: 0.2 to 2 %; an
// extended source of a twelfth of the side 3.5, where both are as fast; 400 sources 5 to 8, cleaned images 25
// to 60, noise 100), or more above the second peak's limit than an iteration may have hot (equal sources).
// Later: two fifths near the peak (4096^2, 300 sources, 300 iterations 9.6 -> 7.4 ms; 20 sources cleaned by
// 100, 1000 more 15.8 -> 14.5; a twelfth switched 3 sources too early, 200 iterations 2.72 -> 3.01), or hot
// blocks of a leading CTA in one launch: 6 an iteration at 2048^2, 18 at 4096^2.  us an iteration of 1000 by
// the hot blocks (0: never; nothing else): 2048^2, 5 sources 0 13.0, 12 8.24, 6 8.22; 60 sources 0 9.07, 12
// 9.05, 6 8.30, 4 8.42; 40 sources, 300 iterations 0 7.36, 6 7.40, 4 8.0.  2600^2, 20 sources 0 9.03, 8 9.02,
// 6 11.5.  4096^2, 5 sources 0 35.9, 24 21.9, 12 21.9; 60 sources 0 19.5, 24 19.5, 12 21.4, 8 27.5.
// By single pixels (an odd width) a pass takes nearly twice as long: where blocks are small only twice as many
// hot blocks count (ms of 1000 iterations by that number times 1, 2, 3, never: 60 sources 2049^2 12.9, 9.4,
// 9.4, 9.4, 2601^2 19.8, 12.4, 12.4, 12.4; noise 2049^2 15.1, 15.1, 15.0, 33.0, 4095^2 44.1, 44.0, 44.0, 59.1).
PassLimits pass_limits(long long n, int blocks, bool singles)
{
    const int hot = int(2 + (n >> 20)), most = 0x7fffffff;
    if (singles) return PassLimits{most, most, most, 2 * hot * kLeadIters};
    return PassLimits{blocks / 25, hot * kLeadCtas, blocks * 2 / 5, hot * kLeadIters};
}

// The kernel of passes for an image: as many CTAs as are resident; ctas 0 where it cannot run.
struct Passes {
    const void* kernel;
    HogArgs h;
    int ctas;
};
bool whole_float4s(const HogArgs& h) { return h.width % 4 == 0 && reinterpret_cast<uintptr_t>(h.residual) % 16 == 0; }

tcv_status passes_of(const HogArgs& h, Passes& p)
{
    const bool vec = whole_float4s(h);
    const bool large = (h.n + (long long)h.psf_width * h.psf_width) * 4 > (64ll << 20);
    p.kernel = large ? (vec ? reinterpret_cast<const void*>(hog_pass_kernel<true, 3>)
                            : reinterpret_cast<const void*>(hog_pass_kernel<false, 3>))
                     : (vec ? reinterpret_cast<const void*>(hog_pass_kernel<true, 2>)
                            : reinterpret_cast<const void*>(hog_pass_kernel<false, 2>));
    int dev = 0, sms = 0, per_sm = 0, coop = 0;
    TCV_CUDA(cudaGetDevice(&dev));
    TCV_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TCV_CUDA(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    TCV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p.kernel, kHogThreads, 0));
    p.ctas = coop ? std::min({sms * std::min(per_sm, large ? 3 : 2), kHogMaxBlocks, hog_blocks(h.n), h.width}) : 0;
    p.h = h;
    p.h.nblocks = p.ctas;
    return TCV_OK;
}
tcv_status launch_passes(Passes& p, PassLimits lim, int from, int to, cudaStream_t st)
{
    void* args[] = {&p.h, &lim, &from, &to, &g_wait_ns, &g_withheld};
    TCV_CUDA(cudaLaunchCooperativeKernel(p.kernel, dim3(unsigned(p.ctas)), dim3(kHogThreads), args, 0, st));
    return TCV_OK;
}

// Iterations up to which a call is passes from the start: bringing all blocks up to date at its end costs as
// much as several (us a call as passes, and in brackets with put-off updates: 1 iteration 1900^2 41 (71),
// 4096^2 100 (217); 8 iterations 98 (103) and 280 (317), 10 116 (112) and 333 (333)).
// By single pixels up to three (2049^2 76 and 91, 2601^2 123 and 127; four 143 and 130).  One or two are a
// launch each: the cooperative launch alone takes 3 us more.
constexpr int kFewIters = 8, kFewSingle = 3, kLeastPasses = 3;

// From this width on a single iteration is a launch at the resident sizes too (alone, us: 1024^2 34 and 37 in the
// resident form, 1500^2 38 and 41; 512^2 32 and 31).
constexpr int kSingleWidth = 1024;

// All iterations as passes, in one cooperative launch.  ran = false: nothing launched.
tcv_status deconvolve_passes(const HogArgs& h, const float* dirty, int niters, cudaStream_t st, bool& ran)
{
    ran = false;
    Passes p;
    TCV_CHECK(passes_of(h, p));
    // the arrivals reach niters x CTAs (and those withheld): within 32 bits
    if (p.ctas < 1 || uint64_t(niters) * uint64_t(p.ctas) + g_withheld >= 1ull << 32) return TCV_OK;
    TCV_CHECK(first_scans(h, dirty, st));
    ran = true;
    return niters > 0 ? launch_passes(p, PassLimits{-1, -1, -1, -1}, 0, niters, st) : TCV_OK;
}

// All iterations with put-off updates.  false: the device cannot hold the cluster, nothing launched.
tcv_status deconvolve_deferred(const HogArgs& h, const HogWork& w, const float* dirty, int niters, cudaStream_t st, bool& ran)
{
    ran = false;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attr;
    DeferArgs a{};
    a.h = h;
    a.bound = w.bound;
    a.applied = w.applied;
    a.warm = w.warm;
    a.pmax = w.pmax;
    a.ring = w.ring;
    a.slots = w.slots;
    a.wait_ns = g_wait_ns;
    a.withheld = g_withheld;
    a.lb = log2_side(h.width);
    a.nbx = (h.width + (1 << a.lb) - 1) >> a.lb;
    a.lbp = std::max(a.lb, log2_side(h.psf_width));  // a block then lies on at most 2 x 2 of the PSF's
    a.npx = (h.psf_width + (1 << a.lbp) - 1) >> a.lbp;
    if (!lead_ctas(cfg, attr, a)) return TCV_OK;
    cfg.stream = st;
    const int nb = a.nbx * a.nbx;
    // the PSF's peak (HogbomGolden.cc:73-76), residual = dirty with the first scan (:70)
    const int scans = std::min(kHogMaxBlocks, (nb + a.npx * a.npx + kHogThreads / 32 - 1) / (kHogThreads / 32));
    hog_blocks_kernel<<<scans, kHogThreads, 0, st>>>(a, dirty, w.pmax);
    TCV_CUDA(cudaGetLastError());
    const size_t win = size_t(kSlots) * kWindow * sizeof(float);
    TCV_CUDA(cudaFuncSetAttribute(hog_apply_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, int(win)));
    int dev = 0, sms = 0, per_sm = 0;
    TCV_CUDA(cudaGetDevice(&dev));
    TCV_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    TCV_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, hog_apply_kernel, kApplyThreads, win));
    const int most = std::min(nb, sms * std::max(1, per_sm));
    Passes passes;  // may take over
    TCV_CHECK(passes_of(h, passes));
    const PassLimits lim = pass_limits(h.n, nb, !whole_float4s(h) && a.lb == 5);
    cudaLaunchAttribute attrs[2] = {attr, {}};
    attrs[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attrs[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attrs;
    cfg.numAttrs = 2;
    cudaLaunchConfig_t apply{};
    apply.gridDim = dim3(unsigned(most));
    apply.blockDim = dim3(kApplyThreads);
    apply.dynamicSmemBytes = win;
    apply.stream = st;
    apply.attrs = attrs + 1;
    apply.numAttrs = 1;
    for (int it = 0, base = 0; it < niters; it += kLeadIters) {
        const int to = std::min(niters, it + kLeadIters);
        // all blocks are up to date; from the start to the end (the arrivals have to fit 32 bits)
        if (passes.ctas && it == base)
            TCV_CHECK(launch_passes(passes, lim, it, std::min(niters, it == 0 ? 1 << 20 : it + kRing), st));
        TCV_CUDA(cudaLaunchKernelEx(&cfg, hog_lead_kernel, a, it, to, base));
        const int all = to == niters || to - base == kRing;
        TCV_CUDA(cudaLaunchKernelEx(&apply, hog_apply_kernel, a, base, all));
        if (all) base = to;
    }
    ran = true;
    return TCV_OK;
}


}  // namespace
}  // namespace tcv

using namespace tcv;

extern "C" {

size_t tcv_hogbom_workspace_bytes(int width)
{
    if (width < 1) return 0;
    return HogWork(nullptr).total;
}

tcv_status tcv_hogbom_deconvolve(const float* d_dirty, int width, const float* d_psf, int psf_width, float* d_model,
                                 float* d_residual, int niters, float gain, float threshold, float* d_hist_val,
                                 uint32_t* d_hist_pos, void* d_work, size_t work_bytes, void* stream)
{
    if (!d_dirty || !d_psf || !d_model || !d_residual || !d_work || width < 1 || psf_width < 1 || niters < 0)
        return TCV_ERR_ARG;
    if (uint64_t(width) * uint64_t(width) >= 0xffffffffull || uint64_t(psf_width) * uint64_t(psf_width) >= 0xffffffffull)
        return TCV_ERR_UNSUPPORTED;
    if (work_bytes < tcv_hogbom_workspace_bytes(width)) return TCV_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const HogWork w(d_work);
    HogArgs a{};
    a.state = w.state;
    a.keys = w.keys;
    a.vals = w.vals;
    a.psf = d_psf;
    a.residual = d_residual;
    a.model = d_model;
    a.hist_val = d_hist_val;
    a.hist_pos = d_hist_pos;
    a.width = width;
    a.psf_width = psf_width;
    a.n = (long long)width * width;
    a.nblocks = hog_blocks(a.n);
    a.gain = gain;
    a.threshold = threshold;
    TCV_CUDA(cudaMemsetAsync(a.state, 0, w.zeroed, st));
    bool ran = false;
    tcv_status s = TCV_OK;
    const int few = whole_float4s(a) ? kFewIters : kFewSingle;
    const bool any = g_hog_strategy == TCV_HOGBOM_AUTO, passes = g_hog_strategy == TCV_HOGBOM_PERSISTENT;
    const bool single = any && niters == 1 && width >= kSingleWidth;
    if ((any || passes) && !single) s = deconvolve_resident(a, w, d_dirty, niters, st, ran);
    if (s == TCV_OK && !ran && (passes || (any && niters >= kLeastPasses && niters <= few)))
        s = deconvolve_passes(a, d_dirty, niters, st, ran);
    if (s == TCV_OK && !ran && any && niters > few && width <= kDeferMaxWidth && psf_width <= kDeferMaxWidth)
        s = deconvolve_deferred(a, w, d_dirty, niters, st, ran);
    if (s != TCV_OK || ran) return s;
    TCV_CHECK(first_scans(a, d_dirty, st));
    const bool vec = whole_float4s(a);
    for (int it = 0; it < niters; ++it) {
        if (vec)
            hog_iter_kernel<true><<<a.nblocks, kHogThreads, 0, st>>>(a, it);
        else
            hog_iter_kernel<false><<<a.nblocks, kHogThreads, 0, st>>>(a, it);
    }
    TCV_CUDA(cudaGetLastError());
    return TCV_OK;
}

void tcv_hogbom_set_strategy(int strategy)
{
    if (strategy >= TCV_HOGBOM_AUTO && strategy <= TCV_HOGBOM_PERSISTENT) g_hog_strategy = strategy;
}

tcv_status tcv_hogbom_set_wait(uint64_t limit_ns, uint32_t withheld_arrivals)
{
    if (limit_ns > kDefaultWaitNs || withheld_arrivals > 1024u) return TCV_ERR_ARG;
    g_wait_ns = limit_ns;
    g_withheld = withheld_arrivals;
    return TCV_OK;
}

tcv_status tcv_hogbom_result(const void* d_work, int* iters_done, int* stopped_at, int64_t* skipped_rows,
                             int64_t* psf_peak_pos, void* stream)
{
    if (!d_work) return TCV_ERR_ARG;
    HogState h{};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    TCV_CUDA(cudaMemcpyAsync(&h, d_work, sizeof(h), cudaMemcpyDeviceToHost, st));
    TCV_CUDA(cudaStreamSynchronize(st));
    if (iters_done) *iters_done = h.done;
    if (stopped_at) *stopped_at = h.stopped - 1;
    if (skipped_rows) *skipped_rows = int64_t(h.skipped_rows);
    if (psf_peak_pos) *psf_peak_pos = int64_t(h.psf_pos);
    return h.error ? TCV_ERR_TIMEOUT : TCV_OK;
}

tcv_status tcv_find_peak(const float* d_image, int64_t n, float* val_out, int64_t* pos_out, void* d_work,
                         size_t work_bytes, void* stream)
{
    if (!d_image || n < 1 || !d_work || n >= int64_t(0xffffffffll)) return TCV_ERR_ARG;
    // the state and one set of candidates: less than a deconvolution's workspace
    const size_t at_keys = align256(sizeof(HogState)), at_vals = at_keys + align256(size_t(kHogMaxBlocks) * 8);
    if (work_bytes < at_vals + align256(size_t(kHogMaxBlocks) * 4)) return TCV_ERR_WORKSPACE;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    char* w = static_cast<char*>(d_work);
    HogState* state = reinterpret_cast<HogState*>(w);
    unsigned long long* keys = reinterpret_cast<unsigned long long*>(w + at_keys);
    float* vals = reinterpret_cast<float*>(w + at_vals);
    TCV_CUDA(cudaMemsetAsync(state, 0, sizeof(HogState), st));
    const int nb = hog_blocks(n);
    hog_scan_kernel<<<nb, kHogThreads, 0, st>>>(d_image, nullptr, n, nb, keys, vals, state, 0);
    TCV_CUDA(cudaGetLastError());
    HogState h{};
    TCV_CUDA(cudaMemcpyAsync(&h, state, sizeof(h), cudaMemcpyDeviceToHost, st));
    TCV_CUDA(cudaStreamSynchronize(st));
    if (val_out) *val_out = h.win_val[0];
    if (pos_out) *pos_out = int64_t(~static_cast<unsigned int>(h.win_key[0]));
    return TCV_OK;
}

}  // extern "C"
