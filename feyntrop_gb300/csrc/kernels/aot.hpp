// Host wrappers of the ahead-of-time kernels (aot.cu).
#pragma once

#include <cuda_runtime.h>

namespace ft {

// The matrices that take a sampling kernel's threads to their start states (layout in
// sample_body.cuh): nibble images under (T^S)^l, l < 32, then (T^S)^(32 8^d v), v = 1 .. 7, d <
// digits; tpow = T^(2^j), j < 64 (1024 words per matrix).  stride_words(digits) words.
inline unsigned long long stride_words(int digits) { return (128ull + 7ull * (unsigned long long)digits) * 1024ull; }
// octal digits of a warp index in a launch of 2^bits threads
inline int stride_digits(int bits) { return bits <= 5 ? 0 : (bits - 5 + 2) / 3; }
cudaError_t launch_stride_matrices(const unsigned long long* tpow, unsigned long long S, int digits,
                                   unsigned long long* out, cudaStream_t st);
// (T^S)^(8^d v), v = 1 .. 7, d < digits
cudaError_t launch_digit_matrices(const unsigned long long* tpow, unsigned long long S, int digits,
                                  unsigned long long* out, cudaStream_t st);

// Batches (layouts in aot.cu): the integrals' start states from item_prep records (one warp
// per integral), and the per-instance sums of the work items plus the FP64 pass (qacc may
// be NULL).
cudaError_t launch_batch_start_states(const void* prep, int n, const unsigned long long* tpow,
                                      unsigned long long* out, cudaStream_t st);
cudaError_t launch_batch_finalize(const void* inst, int n, const double* parts, int K,
                                  const unsigned long long* qacc, double* out, cudaStream_t st);

// The FP64 pass of a mixed batch adds each handed-off sample's values exactly into
// per-integral fixed-point accumulators: digit j (a signed 64-bit counter) has weight
// 2^(32 j - 1074), and a double enters as three signed 32-bit digits of its integer
// significand, so the sums are exact and independent of the order of the atomics.
// Per integral: 4K accumulators of kExactDigits words, then 4 counters (kept,
// dropped, robust, spare).  The kernel source gets the same count as FT_XA_DIGITS.
constexpr int kExactDigits = 68;
inline unsigned long long exact_words(int K) { return 4ull * (unsigned long long)K * kExactDigits + 4ull; }

// Limits of the no-allocation path (ft_integrate_noalloc): per-block partial moments
// for up to 2048 blocks of up to 136 slots (16 eps orders), 65536 FP64 hand-off
// entries, stride matrices for up to 2^24 threads.  6.3 MB per device.
#define NOALLOC_MAX_BLOCKS 2048
#define NOALLOC_MAX_SLOTS 136
#define NOALLOC_PART_DOUBLES ((NOALLOC_MAX_BLOCKS + 1) * NOALLOC_MAX_SLOTS)   // one for the sampling launch's sum
#define NOALLOC_QUEUE_ENTRIES 65536
#define NOALLOC_MAX_LANE_BITS 24
#define NOALLOC_MAT_WORDS (177 * 1024)
#define NOALLOC_TOTAL_WORDS (2 + NOALLOC_PART_DOUBLES + 5 * NOALLOC_QUEUE_ENTRIES + NOALLOC_MAT_WORDS)

struct noalloc_layout {
    unsigned int* qcount;
    double* parts;
    unsigned long long* queue;
    unsigned long long* mats;
    unsigned int* ticket;
};

// device addresses inside the static scratch of the current device (first call per
// device looks the symbol up)
cudaError_t noalloc_scratch(noalloc_layout* out);

// FMA issue-rate probe (TFLOP/s, FMA = 2 flops) of the current device
double fma_peak_tflops(bool fp64);

}  // namespace ft
