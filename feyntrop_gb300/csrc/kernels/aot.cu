// Topology-independent kernels, compiled ahead of time with nvcc for sm_103a.
//
//  ft_stride_matrices  powers of a stride's skip matrix (T^S)^n over GF(2), T the xoshiro256+
//                      step: the matrices the sampling kernels reach their threads' start
//                      states with.
//  ft_batch_start_states  stream state of each of a batch's integrals' first samples (one
//                      warp per integral, GF(2) skip-ahead).
//  ft_batch_finalize   per-integral sums of a batch's work items and FP64 pass.
#include <cuda_runtime.h>

#include <mutex>

#include "aot.hpp"

typedef unsigned long long u64;

namespace {

// Block b < 32 writes the images under (T^S)^b of every nibble n of the state and value v of
// it at out[((16 n + v) * 32 + b) * 4 ..] (with `lanes`), the next
// ones (T^S)^(f 8^d v), v = 1 .. 7, f = 32 with `lanes`, else 1, 1024 words each.  Every
// matrix is the product of the T^(2^j) of its exponent's set bits, so the blocks are
// independent (a chain of squarings in one block took 190 us).  A product M <- A M by 1024
// threads: thread (w, c) adds the columns of A in rows' word w for column c of M, all lanes
// of a warp reading the same column of A (broadcasts), then the four words' parts meet.
__global__ void __launch_bounds__(1024) ft_stride_matrices(const u64* __restrict__ tpow, u64 S, int lanes,
                                                           u64* __restrict__ out)
{
    __shared__ __align__(16) u64 A[1024];   // read in 16-byte words
    __shared__ u64 M[1024];
    __shared__ ulonglong2 part[4][256][2];
    const int w = threadIdx.x >> 8, c = threadIdx.x & 255;
    int b = (int)blockIdx.x;
    u64 n, *dst;
    const bool nibbles = lanes && b < 32;
    if (nibbles) {
        n = S * (u64)b;
        dst = out + b * 4;
    } else {
        if (lanes) b -= 32;
        n = (lanes ? 32ull : 1ull) * S * (u64)(b % 7 + 1) << (3 * (b / 7));
        dst = out + (lanes ? 131072 : 0) + (size_t)b * 1024;
    }
    // the identity, or the first factor: each word written once before the first barrier
    if (n == 0) M[c * 4 + w] = (w == (c >> 6)) ? (1ull << (c & 63)) : 0ull;
    bool first = true;
    for (; n; n &= n - 1) {
        const u64* P = tpow + (size_t)(__ffsll((long long)n) - 1) * 1024;
        if (first) {
            M[threadIdx.x] = P[threadIdx.x];
            first = false;
            continue;
        }
        A[threadIdx.x] = P[threadIdx.x];
        __syncthreads();
        const u64 bits = M[c * 4 + w];
        const ulonglong2* col = (const ulonglong2*)(A + w * 256);
        u64 r0 = 0, r1 = 0, r2 = 0, r3 = 0;
#pragma unroll 8
        for (int k = 0; k < 64; k++) {
            const u64 mask = 0ull - ((bits >> k) & 1ull);
            const ulonglong2 lo = col[2 * k], hi = col[2 * k + 1];
            r0 ^= lo.x & mask;
            r1 ^= lo.y & mask;
            r2 ^= hi.x & mask;
            r3 ^= hi.y & mask;
        }
        part[w][c][0] = make_ulonglong2(r0, r1);
        part[w][c][1] = make_ulonglong2(r2, r3);
        __syncthreads();
        const u64* p = (const u64*)part;
        M[threadIdx.x] = p[threadIdx.x] ^ p[1024 + threadIdx.x] ^ p[2048 + threadIdx.x] ^ p[3072 + threadIdx.x];
        __syncthreads();
    }
    __syncthreads();
    if (!nibbles) {
        dst[threadIdx.x] = M[threadIdx.x];
        return;
    }
    const int nib = threadIdx.x >> 4, v = threadIdx.x & 15;
    u64 r[4] = {0, 0, 0, 0};
    for (int k = 0; k < 4; k++)
        for (int i = 0; i < 4; i++) r[i] ^= (v >> k) & 1 ? M[(nib * 4 + k) * 4 + i] : 0ull;
    ulonglong2* q = (ulonglong2*)(dst + (size_t)threadIdx.x * 128);
    q[0] = make_ulonglong2(r[0], r[1]);
    q[1] = make_ulonglong2(r[2], r[3]);
}

__device__ __forceinline__ void dd_add(double& ah, double& al, double bh, double bl)
{
    const double s = ah + bh;
    const double bb = s - ah;
    double err = (ah - (s - bb)) + (bh - bb);
    err += al + bl;
    ah = s + err;
    al = err - (ah - s);
}

// ------------------------------------------------------------------ batches
// Device views of the batch descriptors (layouts shared with the batch kernels of the
// sampling module and with batch.cpp).
struct batch_inst_view {
    const void* prm;
    const void* tab;
    u64 nsamples, first_item, nitems, pad[3];
};
struct item_prep {
    u64 s[4];         // seed state of the instance's stream
    u64 skip;         // draws before its first sample
    u64 pad[3];
};

__device__ __forceinline__ u64 word_of(const u64 (&g)[4], int w)
{
    return w == 0 ? g[0] : w == 1 ? g[1] : w == 2 ? g[2] : g[3];
}

// g <- M g over GF(2) by one warp: lane l owns input bits 8l .. 8l+7 (column c of M is
// the four words M[4c .. 4c+3]); the partial results are XOR-reduced across the warp
__device__ __forceinline__ void warp_gf2_apply(const u64* __restrict__ M, u64 (&g)[4], int lane)
{
    u64 r0 = 0, r1 = 0, r2 = 0, r3 = 0;
    const u64 sw = word_of(g, lane >> 3);
#pragma unroll
    for (int k = 0; k < 8; k++) {
        const int c = lane * 8 + k;
        const u64 mask = 0ull - ((sw >> (((lane & 7) << 3) + k)) & 1ull);
        const ulonglong2 lo = __ldg((const ulonglong2*)(M + 4 * c)), hi = __ldg((const ulonglong2*)(M + 4 * c + 2));
        r0 ^= lo.x & mask;
        r1 ^= lo.y & mask;
        r2 ^= hi.x & mask;
        r3 ^= hi.y & mask;
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        r0 ^= __shfl_xor_sync(0xffffffffu, r0, off);
        r1 ^= __shfl_xor_sync(0xffffffffu, r1, off);
        r2 ^= __shfl_xor_sync(0xffffffffu, r2, off);
        r3 ^= __shfl_xor_sync(0xffffffffu, r3, off);
    }
    g[0] = r0;
    g[1] = r1;
    g[2] = r2;
    g[3] = r3;
}

// one warp per instance: the stream state of its first sample
__global__ void __launch_bounds__(128) ft_batch_start_states(const item_prep* __restrict__ d, int n,
                                                            const u64* __restrict__ tpow, u64* __restrict__ out)
{
    const int w = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = (int)(threadIdx.x & 31u);
    if (w >= n) return;   // the whole warp
    u64 g[4] = {d[w].s[0], d[w].s[1], d[w].s[2], d[w].s[3]};
    const u64 skip = d[w].skip;
    for (int b = 0; b < 64; b++)
        if ((skip >> b) & 1ull) warp_gf2_apply(tpow + (size_t)b * 1024, g, lane);
    if (lane < 4) out[(size_t)w * 4 + lane] = word_of(g, lane);
}

// An exact fixed-point accumulator (kExactDigits signed 64-bit digits of weight
// 2^(32 j - 1074)) as a double-double: carries normalised from the lowest digit up
// (digits in [0, 2^32), the sign in the final carry), a negative total negated, then
// the digits added from the most significant down.
__device__ void exact_to_dd(const u64* __restrict__ dig, double& h, double& l)
{
    unsigned int d[ft::kExactDigits];
    long long carry = 0;
    for (int j = 0; j < ft::kExactDigits; j++) {
        const long long t = (long long)dig[j] + carry;
        d[j] = (unsigned int)(unsigned long long)t;
        carry = t >> 32;
    }
    const bool neg = carry < 0;
    if (neg) {
        // two's complement of the digit vector: invert, add one
        unsigned long long c = 1;
        for (int j = 0; j < ft::kExactDigits; j++) {
            const unsigned long long t = (unsigned long long)(~d[j]) + c;
            d[j] = (unsigned int)t;
            c = t >> 32;
        }
    }
    h = 0.0;
    l = 0.0;
    for (int j = ft::kExactDigits - 1; j >= 0; j--)
        if (d[j]) dd_add(h, l, ldexp((double)d[j], 32 * j - 1074), 0.0);
    if (neg) {
        h = -h;
        l = -l;
    }
}

// Per instance: the sums of its work items (double-double for the moment pairs) plus
// the FP64 pass's exact sums (qacc, NULL for FP64 batches).  One warp per (instance,
// moment pair or counter): its lanes take every 32nd item, then meet (one thread per sum
// went through 366 items of a 3e6-sample integral at 0.4 us each).  Slots: 8K moments as
// 4K (hi, lo) pairs, then kept, dropped, queued, exact, robust, 3 spare; qacc: 4K exact
// accumulators, then kept, dropped, robust, spare.
__global__ void __launch_bounds__(128) ft_batch_finalize(const batch_inst_view* __restrict__ inst, int n,
                                                         const double* __restrict__ parts, int K,
                                                         const u64* __restrict__ qacc, double* __restrict__ out)
{
    const int slots = 8 * K + 8, units = 4 * K + 8;
    const u64 qwords = 4ull * (u64)K * ft::kExactDigits + 4ull;   // ft::exact_words(K)
    const long long t = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned lane = threadIdx.x & 31u;
    if (t >= (long long)n * units) return;   // the whole warp
    const int m = (int)(t / units), u = (int)(t % units);
    const u64 f = inst[m].first_item, cnt = inst[m].nitems;
    double* o = out + (size_t)m * slots;
    if (u < 4 * K) {
        double h = 0.0, l = 0.0;
        for (u64 k = lane; k < cnt; k += 32)
            dd_add(h, l, parts[(f + k) * slots + 2 * u], parts[(f + k) * slots + 2 * u + 1]);
        for (int off = 16; off; off >>= 1) {
            const double oh = __shfl_down_sync(0xffffffffu, h, off), ol = __shfl_down_sync(0xffffffffu, l, off);
            dd_add(h, l, oh, ol);
        }
        if (lane) return;
        if (qacc) {
            double qh, ql;
            exact_to_dd(qacc + (size_t)m * qwords + (size_t)u * ft::kExactDigits, qh, ql);
            dd_add(h, l, qh, ql);
        }
        o[2 * u] = h;
        o[2 * u + 1] = l;
    } else {
        const int c = u - 4 * K;
        double v = 0.0;   // whole numbers below 2^53
        for (u64 k = lane; k < cnt; k += 32) v += parts[(f + k) * slots + 8 * K + c];
        for (int off = 16; off; off >>= 1) v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane) return;
        if (qacc) {
            const u64* cnt4 = qacc + (size_t)m * qwords + 4ull * K * ft::kExactDigits;
            if (c == 0) v += (double)cnt4[0];
            if (c == 1) v += (double)cnt4[1];
            if (c == 4) v += (double)cnt4[2];
        }
        o[8 * K + c] = v;
    }
}

// Issue-rate probes for the roofline denominators: every thread runs 8 independent
// FMA chains, so the pipe, not the dependency latency, limits the rate.
template <class T>
__global__ void __launch_bounds__(256) ft_fma_probe(T* __restrict__ out, int iters, T a, T b)
{
    T x[8];
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = (T)(threadIdx.x + k) * (T)1e-3;
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int k = 0; k < 8; k++) x[k] = x[k] * a + b;
    }
    T s = 0;
#pragma unroll
    for (int k = 0; k < 8; k++) s += x[k];
    if (s == (T)12345.678) out[threadIdx.x] = s;   // keeps the chains alive
}

}  // namespace

namespace ft {

// FMA issue rate in TFLOP/s (2 flops per FMA), timed with CUDA events
double fma_peak_tflops(bool fp64)
{
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    void* buf = nullptr;
    cudaMalloc(&buf, 4096);
    const int blocks = sms * 8, iters = fp64 ? 2048 : 65536;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    float best = 1e30f;
    for (int rep = 0; rep < 4; rep++) {
        cudaEventRecord(e0);
        if (fp64)
            ft_fma_probe<double><<<blocks, 256>>>((double*)buf, iters, 0.999999, 1e-7);
        else
            ft_fma_probe<float><<<blocks, 256>>>((float*)buf, iters, 0.999999f, 1e-7f);
        cudaEventRecord(e1);
        cudaEventSynchronize(e1);
        float ms = 0;
        cudaEventElapsedTime(&ms, e0, e1);
        if (rep > 0 && ms < best) best = ms;
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(buf);
    const double flops = 2.0 * 8 * (double)iters * blocks * 256;
    return flops / (best * 1e-3) / 1e12;
}

// ------------------------------------------------------------------ no-allocation scratch
// Scratch of ft_integrate_noalloc, for callers that must not allocate device memory
// during an integration.  It is one file-scope device array per GPU that loads this
// library, held until the process exits:
//   [2 words] FP64 hand-off queue count and the finished blocks' ticket,
//   [NOALLOC_PART_DOUBLES] per-block partial moments, [5 * NOALLOC_QUEUE_ENTRIES]
//   hand-off queue, [NOALLOC_MAT_WORDS] stride matrices.
// Every call shares it (and it keeps the last call's contents), so calls that overlap
// on the GPU race; the queue count is cleared at the start of each call.
constexpr unsigned long long kNoallocParts = 2, kNoallocQueue = kNoallocParts + NOALLOC_PART_DOUBLES,
                             kNoallocMats = kNoallocQueue + 5ull * NOALLOC_QUEUE_ENTRIES;
// the regions end inside the array, and each holds what the host-side checks of
// ft_integrate_noalloc let a call use: 2048 blocks of up to 8K+8 = 136 slots (16 eps
// orders), the matrices of up to 2^24 threads
static_assert(kNoallocMats + NOALLOC_MAT_WORDS <= NOALLOC_TOTAL_WORDS, "no-allocation layout overruns");
static_assert(NOALLOC_PART_DOUBLES >= (NOALLOC_MAX_BLOCKS + 1) * (8 * 16 + 8), "partial sums of 16 eps orders");
static_assert(NOALLOC_MAT_WORDS >= (128 + 7 * ((NOALLOC_MAX_LANE_BITS - 5 + 2) / 3)) * 1024, "stride matrices");
static_assert(kNoallocQueue % 2 == 0 && kNoallocMats % 2 == 0, "16-byte aligned regions (ulonglong2 loads)");
static __device__ __align__(256) u64 g_noalloc_scratch[NOALLOC_TOTAL_WORDS];

cudaError_t noalloc_scratch(noalloc_layout* out)
{
    // In host code g_noalloc_scratch names a host-side stand-in; the device address is
    // looked up once per device, with that device current.
    static std::mutex mu;
    static void* addr[64] = {};
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    void* base = nullptr;
    {
        std::lock_guard<std::mutex> lock(mu);
        if (!addr[dev]) {
            e = cudaGetSymbolAddress(&addr[dev], g_noalloc_scratch);
            if (e != cudaSuccess) {
                addr[dev] = nullptr;
                return e;
            }
        }
        base = addr[dev];
    }
    u64* w = (u64*)base;
    out->qcount = (unsigned int*)w;
    out->ticket = (unsigned int*)w + 1;
    out->parts = (double*)(w + kNoallocParts);
    out->queue = w + kNoallocQueue;
    out->mats = w + kNoallocMats;
    return cudaSuccess;
}

cudaError_t launch_stride_matrices(const u64* tpow, u64 S, int digits, u64* out, cudaStream_t st)
{
    ft_stride_matrices<<<32 + 7 * digits, 1024, 0, st>>>(tpow, S, 1, out);
    return cudaGetLastError();
}

cudaError_t launch_digit_matrices(const u64* tpow, u64 S, int digits, u64* out, cudaStream_t st)
{
    if (digits <= 0) return cudaSuccess;
    ft_stride_matrices<<<7 * digits, 1024, 0, st>>>(tpow, S, 0, out);
    return cudaGetLastError();
}

cudaError_t launch_batch_start_states(const void* prep, int n, const u64* tpow, u64* out, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    ft_batch_start_states<<<(n + 3) / 4, 128, 0, st>>>((const item_prep*)prep, n, tpow, out);
    return cudaGetLastError();
}

cudaError_t launch_batch_finalize(const void* inst, int n, const double* parts, int K,
                                  const unsigned long long* qacc, double* out, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    const long long threads = (long long)n * (4 * K + 8) * 32;
    ft_batch_finalize<<<(unsigned)((threads + 127) / 128), 128, 0, st>>>((const batch_inst_view*)inst, n, parts, K,
                                                                         qacc, out);
    return cudaGetLastError();
}

}  // namespace ft
