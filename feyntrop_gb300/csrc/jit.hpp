// Run-time compilation of the sampling kernels for one graph topology.
//
// The kernel body (kernels/sample_body.cuh, embedded in the library at build
// time) is prefixed with the topology as compile-time constants and compiled by
// NVRTC straight to an sm_103a cubin.  Cubins are cached in memory per device
// and on disk (FEYNTROP_GB300_CACHE, else a _jit_cache folder beside the
// library), keyed by a hash of the full source and options.
#pragma once

#include <cuda.h>

#include <string>
#include <vector>

namespace ft {

struct kernel_key {
    int E = 0, V = 0, K = 1, loops = 0, rank = 1;
    int table_global = 0;   // read the table from global memory instead of staging it
    int prec = 0;       // 0 FP64, 1 mixed
    int mode = 0;       // 0 undeformed, 1 deformed
    int only_psi = 0;
    int record = 0;
    int block = 128;
    int minb = 1;           // minimum resident blocks per SM asked of the register allocator
    int variant = 0;        // code-size options of the kernel body (FT_VARIANT)
    int batch = 0;          // 1: the batch kernels (many integrals of the topology per launch)
    int part = 0;           // 0: the sampling kernel, 1: the FP64 pass over hand-offs (FP64 keys only)
    int scratch = 0;        // mixed: what the threads' shared-memory scratch holds (FT_SCRATCH of the kernel body)
    int q0 = 0;             // reduced vertices [0, q0) carry no external momentum (zero rows of P~)
    std::vector<int> ek, el;   // endpoints in the kernel's vertex labels, ek > el
};

// Graphs of up to 12 edges stage their table in shared memory, with the cut thresholds (E
// 2^(E-1) words: 98 KB of 147 at E = 12, beside the sums); larger ones read it from global
// memory and find cuts by a running-sum scan over Jr/r, 12 times smaller.
inline bool staged_table(int E) { return E <= 12; }

struct kernel_set {
    CUmodule module = nullptr;
    CUfunction sample = nullptr;   // ft_sample, ft_sample_batch (part 0)
    CUfunction queue = nullptr;    // ft_sample_queue, ft_sample_queue_batch (part 1)
    int block = 128;
    int variant = 0;               // FT_VARIANT of the module
    unsigned smem = 0;             // dynamic shared memory per block
    int regs = 0;
    int local_bytes = 0;
    int blocks_per_sm = 0;         // of ft_sample at this block size and smem
    int queue_blocks_per_sm = 0;
    double compile_seconds = 0;
};

std::string kernel_source(const kernel_key& key);

// directory of the compiled-kernel cache (and of the launch-shape tuning table)
std::string cache_dir();

// floats per thread in the shared-memory scratch of the mixed form
unsigned scratch_slots(const kernel_key& key);

// dynamic shared memory of a block: the staged table, the sums, the scratch
unsigned table_smem_bytes(const kernel_key& key);

struct driver_api {
    CUresult (*ModuleLoadData)(CUmodule*, const void*);
    CUresult (*ModuleGetFunction)(CUfunction*, CUmodule, const char*);
    CUresult (*FuncSetAttribute)(CUfunction, CUfunction_attribute, int);
    CUresult (*FuncGetAttribute)(int*, CUfunction_attribute, CUfunction);
    CUresult (*OccupancyMaxActiveBlocksPerMultiprocessor)(int*, CUfunction, int, size_t);
    CUresult (*LaunchKernel)(CUfunction, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned,
                             CUstream, void**, void**);
    CUresult (*GetErrorString)(CUresult, const char**);
};
driver_api& drv();
void check(CUresult r, const char* what);

// compiled and loaded on the current device (throws std::runtime_error)
const kernel_set& get_kernels(const kernel_key& key);

// already loaded on the current device, else nullptr (never compiles or loads)
const kernel_set* find_kernels(const kernel_key& key);

// compile only (no device needed); returns the cubin size
size_t compile_only(const kernel_key& key, std::string* log = nullptr);

// compile into the on-disk cache unless it is there already
void precompile(const kernel_key& key);
// the cubins of several keys, compiled concurrently on the host's threads
void precompile_all(const std::vector<kernel_key>& keys);

}  // namespace ft
