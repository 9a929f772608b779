// tcv_init.cu -- device set-up of the tConvolve problem: sample coordinates, the W-projection
// table C, and per-sample grid/table offsets.  These are the untimed parts of Benchmark::init
// (attic/tConvolveMPI/Benchmark.cc:60-96, 206-324); every floating-point step uses the same
// IEEE operations in the same order as the reference so that the results agree with its CPU
// output (offsets bit for bit; the table up to the last-bit behaviour of the FP64 cos/exp).
#include "tcv_internal.cuh"

#include <atomic>
#include <climits>
#include <cmath>
#include <thread>
#include <vector>

namespace tcv {
namespace {

constexpr double kMaxInt = 2147483647.0;

__device__ __forceinline__ double lcg_coord(uint64_t& state, double baseline, double half)
{
    // Benchmark::randomInt (Benchmark.cc:53-58), then baseline * r / maxint - baseline/2 (:72-74)
    state = state * kLcgA + kLcgC;
    const unsigned int r = (unsigned int)(state / 65536ull) % 2147483647u;
    return __dsub_rn(__ddiv_rn(__dmul_rn(baseline, (double)(int)r), kMaxInt), half);
}

__global__ void uvw_kernel(int64_t n, int baseline, uint64_t state0, double* u, double* v, double* w)
{
    const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    uint64_t A, C;
    lcg_jump(3ull * (uint64_t)i, A, C);
    uint64_t s = A * state0 + C;
    const double b = (double)baseline, h = (double)(baseline / 2);
    u[i] = lcg_coord(s, b, h);
    v[i] = lcg_coord(s, b, h);
    w[i] = lcg_coord(s, b, h);
}

struct CParams {
    int s, os, w_size, c_center;
    double w_cell_size, freq0, cell_size;
};

// Benchmark.cc:236-258 in FP64, stored as float (imaginary part 0).  One thread per entry of the
// planes w >= 0: plane -w has the same |w|, so the same values, and the thread stores them there
// too (half the double-precision cosines, which bound this kernel: 378 -> 243 us at 33 planes of
// 64 x 129^2 entries).
__global__ void init_c_kernel(CParams p, float2* c)
{
    const int64_t per_plane = int64_t(p.s) * p.s * p.os * p.os;
    const int64_t cind = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (cind >= per_plane * (p.w_size / 2 + 1)) return;
    int64_t t = cind;
    const int i = int(t % p.s); t /= p.s;
    const int j = int(t % p.s); t /= p.s;
    const int osi = int(t % p.os); t /= p.os;
    const int osj = int(t % p.os); t /= p.os;
    const int above = p.w_size / 2 + int(t), below = p.w_size / 2 - int(t);
    const double w = (double)int(t);
    const double f_scale = __ddiv_rn(sqrt(__dmul_rn(__dmul_rn(fabs(w), p.w_cell_size), p.freq0)), p.cell_size);
    const double os = (double)p.os;
    const double dj = __dadd_rn((double)(j - p.c_center), __ddiv_rn((double)osj, os));
    const double di = __dadd_rn((double)(i - p.c_center), __ddiv_rn((double)osi, os));
    const double r2 = __dadd_rn(__dmul_rn(dj, dj), __dmul_rn(di, di));
    double val;
    if (w != 0.0)
        val = cos(__ddiv_rn(r2, __dmul_rn(w, f_scale)));  // cos is even: also plane -w's value
    else
        val = exp(-r2);
    const int64_t in_plane = cind - t * per_plane;
    const float2 z = make_float2((float)val, 0.0f);
    if (above < p.w_size) c[above * per_plane + in_plane] = z;
    if (below != above) c[below * per_plane + in_plane] = z;
}

__device__ __forceinline__ float cabs_ref(float2 z)
{
    // std::abs(std::complex<float>) is hypotf(re, im); exact |re| when im == 0
    return z.y == 0.0f ? fabsf(z.x) : hypotf(z.x, z.y);
}

// ------------------------------------------------------------------------------------------
// The reference normalises with a sequential float sum of |C| over the flat table
// (Benchmark.cc:261-265).  The order of a float sum decides its value (it saturates at 2^24 for
// the default 35 M entry table), and one thread adding in that order took 117.6 ms there.  The
// same value in parallel: while the sum s = m * u stays in one binade (u its last place, m in
// [2^23, 2^24)), adding x >= 0 takes m to m + round(x / u) whatever m is, except that a tie is
// rounded by the parity of m + floor(x / u).  So an entry is a pair of whole-number increments,
// for an even and an odd m (Inc2), a run of entries composes into one such pair, and composition
// is associative: it can be summed in any grouping.  Where m would reach 2^24 the binade ends:
// the entries around that place are added one by one in float, and the sum goes on with the next
// binade's u.
//   sum_blocks_kernel   per block of entries, its sum in double (an estimate of where s stands)
//   sum_incs_kernel     per block, its increments for the two binades s may be in there
//   sum_walk_kernel     one CTA walks the blocks, 1024 composed at a time; a block in which the
//                       binade ends, or whose two binades do not hold s, is walked entry by entry
// Both block kernels read the table once (281 MB at the default size: bandwidth); the walk is a
// chain of a dozen binades of a few microseconds.  117.6 -> 0.38 ms at the default size.
// ------------------------------------------------------------------------------------------
constexpr int kSumChunk = 4096;       // entries a CTA of the block kernels handles per round
constexpr int kSumMaxBlocks = 4096;
constexpr unsigned kIncCap = 1u << 26;  // increments from 2^24 on only say "the binade ends"

struct Inc2 {
    unsigned even, odd;  // increment of m from an even and from an odd m
};

struct SumBlocks {
    int64_t n, per;  // entries, entries per block (a multiple of kSumChunk)
    int nb;
    double* sum;     // per block
    Inc2* incs;      // per block: increments at exponent exps[b], then at exps[b] + 1
    int* exps;
};

__device__ __forceinline__ Inc2 inc_then(const Inc2 a, const Inc2 b)  // a's entries, then b's
{
    return Inc2{min(kIncCap, a.even + ((a.even & 1u) ? b.odd : b.even)),
                min(kIncCap, a.odd + ((a.odd & 1u) ? b.even : b.odd))};
}

__device__ __forceinline__ Inc2 inc_of(float x, float per_u)  // per_u = 1 / u, a power of two
{
    const float q = fminf(x * per_u, float(kIncCap)), f = floorf(q), r = q - f;
    const unsigned n = unsigned(f);
    const unsigned up = r > 0.5f, tie = r == 0.5f;
    return Inc2{n + (up | (tie & n)), n + (up | (tie & ~n & 1u))};
}

__device__ __forceinline__ int exponent_of(float s) { return int((__float_as_uint(s) >> 23) & 0xffu) - 127; }
__device__ __forceinline__ float pow2f(int e) { return __uint_as_float(unsigned(e + 127) << 23); }

// inclusive scan over the warp's lanes in lane order
__device__ __forceinline__ Inc2 inc_warp_scan(Inc2 v, int lane)
{
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const Inc2 o{__shfl_up_sync(0xffffffffu, v.even, d), __shfl_up_sync(0xffffffffu, v.odd, d)};
        if (lane >= d) v = inc_then(o, v);
    }
    return v;
}

__global__ void __launch_bounds__(256) sum_blocks_kernel(const float2* __restrict__ c, SumBlocks b)
{
    __shared__ double ws[8];
    const int64_t lo = b.per * blockIdx.x, hi = min(b.n, lo + b.per);
    double s = 0.0;
    for (int64_t i = lo + threadIdx.x; i < hi; i += 256) s += double(cabs_ref(c[i]));
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < 8; ++w) s += ws[w];
        b.sum[blockIdx.x] = s;
    }
}

__global__ void __launch_bounds__(256) sum_incs_kernel(const float2* __restrict__ c, SumBlocks b)
{
    __shared__ double ws[8];
    __shared__ Inc2 wi[2][8];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the sum before this block, as the double sums have it; the float sum lags or leads it by its
    // accumulated roundings, so the binade is taken from a little below
    double s = 0.0;
    for (int k = threadIdx.x; k < int(blockIdx.x); k += 256) s += b.sum[k];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) ws[warp] = s;
    __syncthreads();
    s = 0.0;
    for (int w = 0; w < 8; ++w) s += ws[w];
    const int e = max(-64, min(100, exponent_of(float(0.9 * s))));
    const float q0 = pow2f(23 - e), q1 = pow2f(22 - e);
    Inc2 t0{0, 0}, t1{0, 0};  // thread 0: of the block so far
    const int64_t lo = b.per * blockIdx.x, hi = min(b.n, lo + b.per);
    for (int64_t base = lo; base < hi; base += kSumChunk) {
        constexpr int kPer = kSumChunk / 256;  // consecutive entries per thread
        const int64_t at = base + int64_t(threadIdx.x) * kPer;
        Inc2 v0{0, 0}, v1{0, 0};
#pragma unroll
        for (int k = 0; k < kPer; ++k) {
            if (at + k >= hi) break;
            const float x = cabs_ref(c[at + k]);
            v0 = inc_then(v0, inc_of(x, q0));
            v1 = inc_then(v1, inc_of(x, q1));
        }
        v0 = inc_warp_scan(v0, lane);
        v1 = inc_warp_scan(v1, lane);
        __syncthreads();  // thread 0 is done with the last round's warps
        if (lane == 31) {
            wi[0][warp] = v0;
            wi[1][warp] = v1;
        }
        __syncthreads();
        if (threadIdx.x == 0)
            for (int w = 0; w < 8; ++w) {
                t0 = inc_then(t0, wi[0][w]);
                t1 = inc_then(t1, wi[1][w]);
            }
    }
    if (threadIdx.x == 0) {
        b.exps[blockIdx.x] = e;
        b.incs[2 * blockIdx.x] = t0;
        b.incs[2 * blockIdx.x + 1] = t1;
    }
}

constexpr int kWalkThreads = 1024;
constexpr float kSumTiny = 1e-18f;  // below this the entries are added one by one

struct WalkShared {
    Inc2 warp[kWalkThreads / 32];
    unsigned first;  // first thread whose part the binade ends in
    float s;         // the sum so far
};

// Add the threads' parts (inc each, in thread order) to sh.s as far as the binade reaches: returns
// the first thread whose part was not added (kWalkThreads: none), and with m_out that thread's m
// at its part's start (all threads get their own).
__device__ unsigned walk_parts(WalkShared& sh, Inc2 inc, bool stop, unsigned m, float u, unsigned& m_out)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const Inc2 in = inc_warp_scan(inc, lane);
    if (lane == 31) sh.warp[warp] = in;
    if (threadIdx.x == 0) sh.first = kWalkThreads;
    __syncthreads();
    Inc2 pre{0, 0};
    if (warp == 0) {
        const Inc2 w = inc_warp_scan(sh.warp[lane], lane);
        __syncwarp();
        sh.warp[lane] = w;
    }
    __syncthreads();
    if (warp) pre = sh.warp[warp - 1];
    Inc2 before{__shfl_up_sync(0xffffffffu, in.even, 1), __shfl_up_sync(0xffffffffu, in.odd, 1)};
    if (lane == 0) before = Inc2{0, 0};
    before = inc_then(pre, before);
    const Inc2 after = inc_then(before, inc);
    const unsigned m0 = m + ((m & 1u) ? before.odd : before.even), m1 = m + ((m & 1u) ? after.odd : after.even);
    if (stop || m1 >= (1u << 24)) atomicMin(&sh.first, threadIdx.x);
    m_out = m0;
    __syncthreads();
    const unsigned first = sh.first;
    if (first == kWalkThreads && threadIdx.x == kWalkThreads - 1) sh.s = float(m1) * u;
    return first;
}

// The entries [lo, hi) added to sh.s.  A sum that is not a number (entries of a table set up with a
// negative baseline are not) stays so, as it does added in order: it has no place in a binade.
__device__ void walk_entries(WalkShared& sh, const float2* __restrict__ c, int64_t lo, int64_t hi)
{
    constexpr int kPer = 4;
    while (lo < hi) {
        __syncthreads();
        const float s = sh.s;
        if (s != s) break;  // the same for the whole CTA
        const int64_t at = lo + int64_t(threadIdx.x) * kPer;
        float x[kPer];
#pragma unroll
        for (int k = 0; k < kPer; ++k) x[k] = at + k < hi ? cabs_ref(c[at + k]) : 0.f;
        unsigned first, m0 = 0;
        float u = 1.f;
        if (s < kSumTiny) {  // no binade yet: on to the first entries that are not zero
            const bool any = x[0] != 0.f || x[1] != 0.f || x[2] != 0.f || x[3] != 0.f;
            first = walk_parts(sh, Inc2{0, 0}, any, 0u, 0.f, m0);
            if (first == kWalkThreads) {
                __syncthreads();
                if (threadIdx.x == 0) sh.s = s;
            } else if (threadIdx.x == first) {
                float t = s;
#pragma unroll
                for (int k = 0; k < kPer; ++k) t = __fadd_rn(t, x[k]);
                sh.s = t;
            }
        } else {
            const int e = exponent_of(s);
            u = pow2f(e - 23);
            const float per_u = pow2f(23 - e);
            Inc2 inc{0, 0};
#pragma unroll
            for (int k = 0; k < kPer; ++k) inc = inc_then(inc, inc_of(x[k], per_u));
            first = walk_parts(sh, inc, false, unsigned(s * per_u), u, m0);
            if (threadIdx.x == first) {
                float t = float(m0) * u;
#pragma unroll
                for (int k = 0; k < kPer; ++k) t = __fadd_rn(t, x[k]);
                sh.s = t;
            }
        }
        lo += first == kWalkThreads ? int64_t(kWalkThreads) * kPer : (int64_t(first) + 1) * kPer;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(kWalkThreads) sum_walk_kernel(const float2* __restrict__ c, SumBlocks b, float* out)
{
    __shared__ WalkShared sh;
    // the first binades are short, and a round of all threads per binade (3.5 us each, a dozen in the
    // first 4096 entries) costs more than one thread's 4096 additions (9 us)
    __shared__ __align__(16) float head[kSumChunk];
    const int64_t nh = min(b.n, int64_t(kSumChunk));
    for (int i = threadIdx.x; i < kSumChunk; i += kWalkThreads) head[i] = i < nh ? cabs_ref(c[i]) : 0.f;
    __syncthreads();
    if (threadIdx.x == 0) {
        float s = 0.f;
#pragma unroll 8
        for (int i = 0; i < (int(nh) + 3) / 4; ++i) {  // (the places past the table add 0)
            const float4 v = reinterpret_cast<const float4*>(head)[i];
            s = __fadd_rn(__fadd_rn(__fadd_rn(__fadd_rn(s, v.x), v.y), v.z), v.w);
        }
        sh.s = s;
    }
    walk_entries(sh, c, nh, min(b.n, b.per));
    int k = 1;
    while (k < b.nb) {
        const float s = sh.s;
        if (s != s) break;
        const int mine = k + int(threadIdx.x);
        unsigned first = 0, m0 = 0;
        if (s >= kSumTiny) {
            const int e = exponent_of(s);
            Inc2 inc{0, 0};
            bool stop = false;
            if (mine < b.nb) {
                const int d = e - b.exps[mine];
                stop = d < 0 || d > 1;
                if (!stop) inc = b.incs[2 * mine + d];
            }
            const float u = pow2f(e - 23);
            first = walk_parts(sh, inc, stop, unsigned(s * pow2f(23 - e)), u, m0);
            if (threadIdx.x == first) sh.s = float(m0) * u;
        }
        if (first == kWalkThreads) {
            k += kWalkThreads;
            __syncthreads();
            continue;
        }
        k += int(first);
        __syncthreads();  // the sum before block k
        walk_entries(sh, c, int64_t(k) * b.per, min(b.n, (int64_t(k) + 1) * b.per));
        ++k;
    }
    if (threadIdx.x == 0) out[0] = sh.s;
}

// C *= float(wSize*os*os) / sumC, as a complex multiply by (scale, 0) (Benchmark.cc:267-269).
__global__ void scale_c_kernel(float2* c, int64_t n, float numer, const float* sum_c)
{
    const float scale = __fdiv_rn(numer, sum_c[0]);
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        float2 z = c[i];
        z.x = __fmul_rn(z.x, scale);
        z.y = __fmul_rn(z.y, scale);
        c[i] = z;
    }
}

struct OffParams {
    int64_t n_samples;
    int n_chan, w_size, g_size, s, os;
    double cell_size, w_cell_size;
};

// Benchmark.cc:293-323, one thread per (sample, channel).
__global__ void offsets_kernel(OffParams p, const double* u, const double* v, const double* w,
                               const double* freq, int32_t* iu_out, int32_t* iv_out, int32_t* co_out)
{
    const int64_t d = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (d >= p.n_samples * p.n_chan) return;
    const int64_t i = d / p.n_chan;
    const int chan = int(d % p.n_chan);
    const double f = freq[chan];
    const double os = (double)p.os;
    const double us = __ddiv_rn(__dmul_rn(f, u[i]), p.cell_size);
    int iu = (int)us;
    if (us < (double)iu) iu -= 1;
    const int fracu = (int)__dmul_rn(os, __dsub_rn(us, (double)iu));
    iu += p.g_size / 2;
    const double vs = __ddiv_rn(__dmul_rn(f, v[i]), p.cell_size);
    int iv = (int)vs;
    if (vs < (double)iv) iv -= 1;
    const int fracv = (int)__dmul_rn(os, __dsub_rn(vs, (double)iv));
    iv += p.g_size / 2;
    const double ws = __ddiv_rn(__dmul_rn(f, w[i]), p.w_cell_size);
    const int woff = p.w_size / 2 + (int)ws;
    iu_out[d] = iu;
    iv_out[d] = iv;
    co_out[d] = p.s * p.s * (fracu + p.os * (fracv + p.os * woff));
}

// ---- table storage conversions ----
// What a conversion reads back: a slot of a fixed device array per call in flight (taken and given
// back on the host, so calls of several threads do not meet).  Allocating 16 bytes for it instead
// took 0.6-1.4 ms a call, most of a small table's set-up.
struct ConvCount {
    unsigned long long imag_nonzero;
    unsigned int absmax_bits, pad;
};
constexpr int kConvSlots = 64;
__device__ ConvCount g_conv[kConvSlots];
std::atomic<uint64_t> g_conv_taken{0};

int take_conv_slot()  // waits while all are in use (each is given back when its call returns)
{
    for (;;) {
        uint64_t m = g_conv_taken.load();
        while (~m) {
            const int i = __builtin_ctzll(~m);
            if (g_conv_taken.compare_exchange_weak(m, m | uint64_t(1) << i)) return i;
        }
        std::this_thread::yield();
    }
}
struct ConvSlot {
    const int i = take_conv_slot();
    ~ConvSlot() { g_conv_taken.fetch_and(~(uint64_t(1) << i)); }
};

__global__ void conv_clear_kernel(int slot) { g_conv[slot] = ConvCount{0ull, 0u, 0u}; }

// The FP16 forms are scaled by the largest |value|, so they need a pass before the conversion: it counts
// the imaginary parts as well, and the conversion is left running when the call returns (35 M entries to
// rf16: 181 us; 231 with the count in the conversion, which the call then has to wait for).
__global__ void absmax_imag_kernel(const float2* c, int64_t n, int slot)
{
    float m = 0.f;
    unsigned long long nz = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float2 z = c[i];
        m = fmaxf(m, fmaxf(fabsf(z.x), fabsf(z.y)));
        nz += (z.y != 0.f);
    }
    for (int o = 16; o; o >>= 1) {
        m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
        nz += __shfl_xor_sync(0xffffffffu, nz, o);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&g_conv[slot].absmax_bits, __float_as_uint(m));  // non-negative floats order like their bits
        if (nz) atomicAdd(&g_conv[slot].imag_nonzero, nz);
    }
}

// One entry per thread and step; kCount: counts the entries with an imaginary part as it goes (for
// the forms without a scale this is the only pass over the table: 35 M entries to r32 in 175 us with a
// counting pass before it, 107 us in one).
template <bool kCount>
__global__ void convert_kernel(const float2* c, int64_t n, int c_type, float pre_scale, void* out, int slot)
{
    unsigned long long nz = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float2 z = c[i];
        if (kCount) nz += (z.y != 0.f);
        switch (c_type) {
            case TCV_C_R32: static_cast<float*>(out)[i] = z.x; break;
            case TCV_C_CBF16: {
                const __nv_bfloat16 re = __float2bfloat16_rn(z.x), im = __float2bfloat16_rn(z.y);
                const uint32_t u = (uint32_t)__bfloat16_as_ushort(re) | ((uint32_t)__bfloat16_as_ushort(im) << 16);
                static_cast<uint32_t*>(out)[i] = u;
                break;
            }
            case TCV_C_RBF16: static_cast<__nv_bfloat16*>(out)[i] = __float2bfloat16_rn(z.x); break;
            case TCV_C_CF16:
                static_cast<__half2*>(out)[i] = __halves2half2(__float2half_rn(z.x * pre_scale), __float2half_rn(z.y * pre_scale));
                break;
            case TCV_C_RF16: static_cast<__half*>(out)[i] = __float2half_rn(z.x * pre_scale); break;
            default: break;
        }
    }
    if (kCount) {
        for (int o = 16; o; o >>= 1) nz += __shfl_xor_sync(0xffffffffu, nz, o);
        if ((threadIdx.x & 31) == 0 && nz) atomicAdd(&g_conv[slot].imag_nonzero, nz);
    }
}

inline int grid_blocks(int64_t n, int threads)
{
    int64_t b = (n + threads - 1) / threads;
    return int(b > 148 * 64 ? 148 * 64 : (b < 1 ? 1 : b));
}

}  // namespace
}  // namespace tcv

using namespace tcv;

extern "C" {

tcv_status tcv_c_geometry(double freq0, double cell_size, int baseline, int w_size, int* support,
                          int* over_sample, double* w_cell_size, int64_t* c_len)
{
    if (!(cell_size > 0.0) || !(freq0 > 0.0) || w_size < 1) return TCV_ERR_ARG;
    // Benchmark.cc:212-217
    const int sup = static_cast<int>(1.5 * std::sqrt(double(std::abs(baseline)) * cell_size * freq0) / cell_size);
    const int os = 8;
    const double wcs = double(2 * baseline) * freq0 / double(w_size);
    const int64_t s = 2 * int64_t(sup) + 1;
    if (support) *support = sup;
    if (over_sample) *over_sample = os;
    if (w_cell_size) *w_cell_size = wcs;
    if (c_len) *c_len = s * s * os * os * w_size;
    return TCV_OK;
}

// the sum, then the per-block sums, increments and exponents of the parallel sum
size_t tcv_init_c_scratch_bytes(void)
{
    return 256 + size_t(kSumMaxBlocks) * (sizeof(double) + 2 * sizeof(Inc2) + sizeof(int));
}

tcv_status tcv_init_c_raw(double freq0, double cell_size, int baseline, int w_size, float* d_c,
                          void* d_scratch, float* sum_c_out, void* stream)
{
    if (!d_c || !d_scratch) return TCV_ERR_ARG;
    int support, os;
    double wcs;
    int64_t n;
    tcv_status st = tcv_c_geometry(freq0, cell_size, baseline, w_size, &support, &os, &wcs, &n);
    if (st != TCV_OK) return st;
    if (n > INT_MAX) return TCV_ERR_UNSUPPORTED;  // cOffset is a 32-bit int in the reference
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    CParams p{2 * support + 1, os, w_size, support, wcs, freq0, cell_size};
    const int64_t half = n / w_size * (w_size / 2 + 1);  // entries of the planes w >= 0
    init_c_kernel<<<unsigned((half + 255) / 256), 256, 0, s>>>(p, reinterpret_cast<float2*>(d_c));
    TCV_CUDA(cudaGetLastError());
    float* d_sum = static_cast<float*>(d_scratch);
    SumBlocks sb{};
    sb.n = n;
    const int64_t chunks = (n + kSumChunk - 1) / kSumChunk;
    sb.per = (chunks + kSumMaxBlocks - 1) / kSumMaxBlocks * kSumChunk;
    sb.nb = int((n + sb.per - 1) / sb.per);
    sb.sum = reinterpret_cast<double*>(static_cast<char*>(d_scratch) + 256);
    sb.incs = reinterpret_cast<Inc2*>(sb.sum + kSumMaxBlocks);
    sb.exps = reinterpret_cast<int*>(sb.incs + 2 * kSumMaxBlocks);
    const float2* table = reinterpret_cast<const float2*>(d_c);
    if (sb.nb > 1) {  // the walk takes the first block entry by entry
        sum_blocks_kernel<<<unsigned(sb.nb), 256, 0, s>>>(table, sb);
        TCV_CUDA(cudaGetLastError());
        sum_incs_kernel<<<unsigned(sb.nb), 256, 0, s>>>(table, sb);
        TCV_CUDA(cudaGetLastError());
    }
    sum_walk_kernel<<<1, kWalkThreads, 0, s>>>(table, sb, d_sum);
    TCV_CUDA(cudaGetLastError());
    scale_c_kernel<<<grid_blocks(n, 256), 256, 0, s>>>(reinterpret_cast<float2*>(d_c), n,
                                                       float(w_size * os * os), d_sum);
    TCV_CUDA(cudaGetLastError());
    if (sum_c_out) {
        TCV_CUDA(cudaMemcpyAsync(sum_c_out, d_sum, sizeof(float), cudaMemcpyDeviceToHost, s));
        TCV_CUDA(cudaStreamSynchronize(s));
    }
    return TCV_OK;
}

size_t tcv_ctype_bytes(int c_type)
{
    switch (c_type & 0xff) {
        case TCV_C_C64: return 8;
        case TCV_C_R32: return 4;
        case TCV_C_CBF16: return 4;
        case TCV_C_RBF16: return 2;
        case TCV_C_CF16: return 4;
        case TCV_C_RF16: return 2;
        default: return 0;
    }
}

tcv_status tcv_convert_c(const float* d_c64, int64_t c_len, int c_type, void* d_out,
                         float* c_scale_out, int64_t* imag_nonzero_out, void* stream)
{
    if (!d_c64 || c_len <= 0 || tcv_ctype_bytes(c_type) == 0 || (c_type & TCV_C_PADDED)) return TCV_ERR_ARG;
    if (c_type == TCV_C_C64) {
        if (!d_out) return TCV_ERR_ARG;
        if (d_out != d_c64)
            TCV_CUDA(cudaMemcpyAsync(d_out, d_c64, size_t(c_len) * 8, cudaMemcpyDeviceToDevice,
                                     static_cast<cudaStream_t>(stream)));
        if (c_scale_out) *c_scale_out = 1.0f;
        if (imag_nonzero_out) *imag_nonzero_out = 0;
        return TCV_OK;
    }
    if (!d_out) return TCV_ERR_ARG;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const float2* c = reinterpret_cast<const float2*>(d_c64);
    const ConvSlot slot;
    conv_clear_kernel<<<1, 1, 0, s>>>(slot.i);
    cudaError_t e = cudaGetLastError();
    auto read_back = [&](ConvCount& h) {
        if (e == cudaSuccess)
            e = cudaMemcpyFromSymbolAsync(&h, g_conv, sizeof(h), size_t(slot.i) * sizeof(h), cudaMemcpyDeviceToHost, s);
        const cudaError_t w = cudaStreamSynchronize(s);  // also after an error: nothing uses the slot from here on
        if (e == cudaSuccess) e = w;
    };
    ConvCount h{};
    float pre = 1.0f, post = 1.0f;
    const bool scaled = c_type == TCV_C_CF16 || c_type == TCV_C_RF16;
    if (e == cudaSuccess && scaled) {
        // power-of-two scale putting max |C| in [2^14, 2^15): the table keeps FP16's full
        // precision without approaching its 65504 limit; kernels undo it exactly with c_scale.
        absmax_imag_kernel<<<grid_blocks(c_len, 256), 256, 0, s>>>(c, c_len, slot.i);
        e = cudaGetLastError();
        read_back(h);
        const float amax = __builtin_bit_cast(float, h.absmax_bits);
        int ex = 0;
        if (amax > 0.f) {
            std::frexp(amax, &ex);  // amax = m * 2^ex, m in [0.5, 1)
            const int shift = 15 - ex;
            pre = std::ldexp(1.0f, shift);
            post = std::ldexp(1.0f, -shift);
        }
    }
    if (e == cudaSuccess) {
        const int blocks = grid_blocks(c_len, 256);
        if (scaled)
            convert_kernel<false><<<blocks, 256, 0, s>>>(c, c_len, c_type, pre, d_out, slot.i);
        else
            convert_kernel<true><<<blocks, 256, 0, s>>>(c, c_len, c_type, pre, d_out, slot.i);
        e = cudaGetLastError();
    }
    if (!scaled || e != cudaSuccess) read_back(h);
    TCV_CUDA(e);
    if (c_scale_out) *c_scale_out = post;
    if (imag_nonzero_out) *imag_nonzero_out = int64_t(h.imag_nonzero);
    return TCV_OK;
}

tcv_status tcv_init_uvw_raw(int64_t n_samples, int baseline, uint64_t state0, double* d_u,
                            double* d_v, double* d_w, void* stream)
{
    if (n_samples < 0 || (n_samples > 0 && (!d_u || !d_v || !d_w))) return TCV_ERR_ARG;
    if (n_samples == 0) return TCV_OK;
    uvw_kernel<<<unsigned((n_samples + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        n_samples, baseline, state0, d_u, d_v, d_w);
    TCV_CUDA(cudaGetLastError());
    return TCV_OK;
}

tcv_status tcv_init_offsets_raw(const double* d_u, const double* d_v, const double* d_w,
                                int64_t n_samples, const double* d_freq, int n_chan,
                                double cell_size, double w_cell_size, int w_size, int g_size,
                                int support, int over_sample, int32_t* d_iu, int32_t* d_iv,
                                int32_t* d_coff, void* stream)
{
    if (n_samples < 0 || n_chan < 1 || support < 0 || over_sample < 1 || g_size < 1 || w_size < 1)
        return TCV_ERR_ARG;
    if (n_samples == 0) return TCV_OK;
    if (!d_u || !d_v || !d_w || !d_freq || !d_iu || !d_iv || !d_coff) return TCV_ERR_ARG;
    OffParams p{n_samples, n_chan, w_size, g_size, 2 * support + 1, over_sample, cell_size, w_cell_size};
    const int64_t n = n_samples * n_chan;
    offsets_kernel<<<unsigned((n + 255) / 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(
        p, d_u, d_v, d_w, d_freq, d_iu, d_iv, d_coff);
    TCV_CUDA(cudaGetLastError());
    return TCV_OK;
}

}  // extern "C"
