// Launch shapes of the sampling kernels: defaults from sweeps on GB300 and a tuning
// table filled by the autotuner (ft_autotune), persisted next to the kernel cache.
#pragma once

#include <string>

#include "jit.hpp"

namespace ft {

struct launch_shape {
    int block = 256;               // threads per block
    int minb = 1;                  // minimum resident blocks per SM given to the register allocator
    int variant = 0;               // FT_VARIANT code-size options of the kernel body
    unsigned long long chunk = 0;  // batch work item: samples per thread (0: default)
    double rate = 0;               // samples/s measured when tuned (0: default shape)
};

// tuning class of a kernel: topology, eps orders, regime, precision, table placement
std::string tune_class(const kernel_key& k);

// the shape the sampling kernels of key k use: tuned if the table has the class, else
// the defaults (launch fields of k are ignored); FEYNTROP_GB300_BLOCK / _MINB / _VARIANT
// override, and the block shrinks until the shared memory fits an SM
launch_shape choose_shape(const kernel_key& k);

// default shape (no table, no environment)
launch_shape default_shape(const kernel_key& k);

// default samples per thread of a batch's work items (FP64: the most that a run takes, run_chunk
// of batch.cpp): items of about a millisecond, so that a batch of a few items per block does not
// wait for the last ones (24 mixed box-pentagon points of 1e5 to 3e6 samples: 12.4 ms with 32,
// 15.5 with 128, 13.6 with 8, whose start and sums show; FP64, 8, 16 and 24: a batch of 20 of every
// kind, 1e5 to 1e6, 15.1, 15.3, 16.2; 24 K4 points of 1e5 to 3e6 6.30, 5.88, 5.76, and longer items
// only balance worse: 12 of 1e4 to 3e5 0.41, 0.40, 0.57)
unsigned long long default_chunk(const kernel_key& k);

// record a tuned shape for the class of k (in memory and in the table file)
void record_shape(const kernel_key& k, const launch_shape& s);

// forget tuned shapes (in memory; the file is rewritten by the next record)
void clear_shapes();

// applies shape s to k and shrinks the block until its shared memory fits
void apply_shape(kernel_key& k, const launch_shape& s);

// batch work-item size forced on batches created by this thread (0: none); the
// autotuner sets it while it measures candidates
void set_chunk_override(unsigned long long chunk);
unsigned long long chunk_override();

}  // namespace ft
