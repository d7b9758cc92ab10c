// Internal to the library: plans, device state and error plumbing shared by the
// single-integral path (runtime.cpp) and the batch path (batch.cpp).
#pragma once

#include <cuda_runtime.h>

#include <exception>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/feyntrop_gb300.h"
#include "jit.hpp"
#include "problem.hpp"
#include "tune.hpp"
#include "xoshiro.hpp"

namespace ftrt {

extern thread_local std::string g_error;

struct cuda_error : std::runtime_error {
    using std::runtime_error::runtime_error;
};

inline void cu(cudaError_t e, const char* what)
{
    if (e == cudaSuccess) return;
    cudaGetLastError();   // reported here, not again by the next launch's check
    throw cuda_error(std::string(what) + ": " + cudaGetErrorString(e));
}

// status code of the exception in flight (sets g_error)
int status_of(const std::exception_ptr& ep);

// throws std::logic_error when there is no CUDA device
void require_device();

// per-device constants: the 64 skip matrices T^(2^b), the SM count
struct device_state {
    unsigned long long* tpow = nullptr;
    int sms = 0;
};
device_state& dev_state();

// the device parameter block of a plan: the FP64 values, then the same as floats,
// then in two-float as (hi, hi, lo, lo) quadruples (the layout the kernel body reads)
std::vector<double> param_block(const std::vector<double>& prm);

// sums of one integration (8K+8 slots) into the caller's result
void fill_result(const ft::prepared& P, const std::vector<double>& acc, ft_result* r);

}  // namespace ftrt

// What a plan's runs need beside its data: a stream, events, pinned words, scratch.  Sets
// are handed from plan to plan (acquire, release in runtime.cpp): making one takes 200 us
// and freeing it 90, more than a small integration.
struct run_scratch {
    // parameter block and table: device, pinned staging (NULL above kStagedBytes)
    unsigned char *d_in = nullptr, *h_in = nullptr;
    size_t in_cap = 0;
    static constexpr size_t kStagedBytes = 12u << 20;
    double* d_parts = nullptr;
    size_t parts_cap = 0;
    double* h_final = nullptr;   // pinned, written by the last block of a launch
    size_t final_cap = 0;
    unsigned long long* d_queue = nullptr;
    unsigned int* d_qcount = nullptr;   // hand-offs, finished blocks: both zero between launches
    size_t qcap = 0;
    // stride matrices for the last few per-thread strides S (alternating precisions or sample
    // counts reuse them): 1.3 MB per entry
    struct stride_entry {
        unsigned long long* d = nullptr;
        unsigned long long S = 0;
        int digits = -1, cap = -1;
        unsigned long long used = 0;
    };
    stride_entry strides[4];
    unsigned long long stride_clock = 0;
    cudaStream_t stream = nullptr;
    cudaEvent_t ev0 = nullptr, ev1 = nullptr;
};

namespace ftrt {
// a set for the current device: an idle one, or a new one
run_scratch acquire_scratch(int device);
// back to the idle ones (at most 8 per device of at most 32 MB each, else freed); `dirty`: its
// last run did not complete, so it is freed
void release_scratch(int device, run_scratch& s, bool dirty);
// frees the idle sets of every device
void free_idle_scratch();
// cudaMalloc; where the device has no room, once more without the idle sets
void device_alloc(void** p, size_t bytes, const char* what);
}  // namespace ftrt

struct ft_plan : run_scratch {
    ft::prepared P;
    // the kernels' vertex labels: vertices without external momentum first, the external
    // ones last, the last of them the deleted (ground) vertex; kek/kel the edges in these
    // labels and kP the scalar products; reduced vertices [0, q0) carry no momentum
    std::vector<int> kek, kel;
    std::vector<double> kP;
    int q0 = 0;
    std::vector<double> sigma, q, prm;
    std::vector<unsigned char> tab;
    int device = 0;
    double* d_prm = nullptr;   // in d_in
    unsigned char* d_tab = nullptr;
    size_t queue_entries = 0;  // hand-offs that this plan's mixed runs may queue
    bool uploading = false;    // the copy to d_in may still be in flight on `stream`
    bool running = false;      // a run was started and did not complete
    bool detached = false;     // ft_integrate_noalloc ran: work of this plan may be in flight
    std::mutex mu;
    // a launch shape under measurement by the autotuner (for one precision)
    bool forced = false;
    int forced_prec = 0;
    ft::launch_shape forced_shape;

    ft::kernel_key key(int prec, int record, int batch = 0, int part = 0) const
    {
        ft::kernel_key k;
        k.E = P.E;
        k.V = P.V;
        k.K = P.K;
        k.loops = P.loops;
        k.rank = (int)sigma.size();
        k.prec = prec;
        k.mode = P.deformed() ? 1 : 0;
        k.only_psi = P.only_psi() ? 1 : 0;
        k.record = record;
        k.batch = batch;
        k.part = part;
        k.ek = kek;
        k.el = kel;
        k.q0 = q0;
        // tables are staged per block in shared memory up to E = 12 (147 KB, beside one
        // block's sums: the cube's mixed kernel ran 8 % faster than reading its table through
        // L1); from E = 13 on they are read through L1
        k.table_global = ft::staged_table(P.E) ? 0 : 1;
        // launch shape: a shape being measured by the autotuner, else the tuning table's
        // (or the default) for this kernel class
        ft::apply_shape(k, (forced && forced_prec == prec) ? forced_shape : ft::choose_shape(k));
        return k;
    }

    int slots() const { return 8 * P.K + 8; }

    ~ft_plan()
    {
        if (!stream) return;
        if (uploading) cudaStreamSynchronize(stream);
        if (detached) {   // on whichever stream
            int cur = 0;
            cudaGetDevice(&cur);
            cudaSetDevice(device);
            cudaDeviceSynchronize();
            cudaSetDevice(cur);
        }
        ftrt::release_scratch(device, *this, running);
    }
};
