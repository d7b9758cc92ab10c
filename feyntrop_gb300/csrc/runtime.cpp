// Plans, launches and the C ABI (include/feyntrop_gb300.h).
//
// A plan holds one integral: the host preprocessing result, its parameter block
// and J(gamma) table in device memory, and the scratch its launches reuse.  An
// integration is
//   1. skip matrices for the launch's stride (cached per stride),
//   2. the sampling kernel (one thread per contiguous block of samples),
//   3. in mixed precision, the FP64 pass over the samples the FP32 kernel queued,
// all on one stream; the last launch's last block adds the blocks' sums into pinned host
// memory.
#include <cuda_runtime.h>

#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <sstream>
#include <stdexcept>
#include <string>
#include <vector>
#include <atomic>
#include <thread>

#include "../../include/feyntrop_gb300.h"
#include "jit.hpp"
#include "json.hpp"
#include "kernels/aot.hpp"
#include "problem.hpp"
#include "xoshiro.hpp"

#include "plan.hpp"

namespace ftrt {

thread_local std::string g_error;

int status_of(const std::exception_ptr& ep)
{
    try {
        std::rethrow_exception(ep);
    } catch (const std::invalid_argument& e) {
        g_error = e.what();
        return FT_ERR_INVALID_ARGUMENT;
    } catch (const std::domain_error& e) {
        g_error = e.what();
        return FT_ERR_DOMAIN;
    } catch (const cuda_error& e) {
        g_error = e.what();
        return FT_ERR_CUDA;
    } catch (const std::runtime_error& e) {
        g_error = e.what();
        return FT_ERR_RUNTIME;
    } catch (const std::exception& e) {
        g_error = e.what();
        return FT_ERR_RUNTIME;
    } catch (...) {
        g_error = "unknown error";
        return FT_ERR_RUNTIME;
    }
}

void require_device()
{
    int n = 0;
    if (cudaGetDeviceCount(&n) != cudaSuccess || n < 1) {
        cudaGetLastError();
        throw std::logic_error("no CUDA device: the feyntrop_gb300 sampling path runs on the GPU only");
    }
}

// idle scratch sets per device; never destroyed, so that a plan may outlive it at exit
struct scratch_pool {
    std::mutex mu;
    std::map<int, std::vector<run_scratch>> idle;
};
static scratch_pool& idle_scratch()
{
    static scratch_pool* p = new scratch_pool;
    return *p;
}

static void free_scratch(run_scratch& s)
{
    if (s.d_in) cudaFree(s.d_in);
    if (s.h_in) cudaFreeHost(s.h_in);
    if (s.d_parts) cudaFree(s.d_parts);
    if (s.h_final) cudaFreeHost(s.h_final);
    if (s.d_queue) cudaFree(s.d_queue);
    if (s.d_qcount) cudaFree(s.d_qcount);
    for (run_scratch::stride_entry& e : s.strides)
        if (e.d) cudaFree(e.d);
    if (s.ev0) cudaEventDestroy(s.ev0);
    if (s.ev1) cudaEventDestroy(s.ev1);
    if (s.stream) cudaStreamDestroy(s.stream);
    s = run_scratch();
}

void free_idle_scratch()
{
    std::map<int, std::vector<run_scratch>> sets;
    {
        scratch_pool& pool = idle_scratch();
        std::lock_guard<std::mutex> lock(pool.mu);
        sets.swap(pool.idle);
    }
    for (auto& d : sets)
        for (run_scratch& s : d.second) free_scratch(s);
}

void device_alloc(void** p, size_t bytes, const char* what)
{
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        free_idle_scratch();
        e = cudaMalloc(p, bytes);
    }
    cu(e, what);
}

run_scratch acquire_scratch(int device)
{
    {
        scratch_pool& pool = idle_scratch();
        std::lock_guard<std::mutex> lock(pool.mu);
        std::vector<run_scratch>& idle = pool.idle[device];
        if (!idle.empty()) {
            const run_scratch s = idle.back();
            idle.pop_back();
            return s;
        }
    }
    run_scratch s;
    try {
        cu(cudaStreamCreateWithFlags(&s.stream, cudaStreamNonBlocking), "cudaStreamCreate");
        cu(cudaEventCreate(&s.ev0), "cudaEventCreate");
        cu(cudaEventCreate(&s.ev1), "cudaEventCreate");
        device_alloc((void**)&s.d_qcount, 16, "cudaMalloc(queue count)");
        cu(cudaMemset(s.d_qcount, 0, 16), "cudaMemset(queue count)");
    } catch (...) {
        release_scratch(device, s, true);
        throw;
    }
    return s;
}

void release_scratch(int device, run_scratch& s, bool dirty)
{
    if (s.qcap * 40 > (8u << 20)) {   // a long mixed run's hand-off queue
        cudaFree(s.d_queue);
        s.d_queue = nullptr;
        s.qcap = 0;
    }
    size_t bytes = (s.h_in ? 2 : 1) * s.in_cap + s.parts_cap * 8 + s.final_cap * 8 + s.qcap * 40;
    for (const run_scratch::stride_entry& e : s.strides)
        if (e.d) bytes += ft::stride_words(e.cap) * 8;
    if (!dirty && bytes <= (32u << 20)) {
        scratch_pool& pool = idle_scratch();
        std::lock_guard<std::mutex> lock(pool.mu);
        std::vector<run_scratch>& idle = pool.idle[device];
        if (idle.size() < 8) {
            idle.push_back(s);
            s = run_scratch();
            return;
        }
    }
    free_scratch(s);
}

device_state& dev_state()
{
    static std::mutex mu;
    static device_state st[64];
    int dev = 0;
    cu(cudaGetDevice(&dev), "cudaGetDevice");
    std::lock_guard<std::mutex> lock(mu);
    device_state& d = st[dev & 63];
    if (!d.tpow) {
        const std::vector<uint64_t>& P = ft::power_table();
        cu(cudaMalloc(&d.tpow, P.size() * 8), "cudaMalloc(skip matrices)");
        cu(cudaMemcpy(d.tpow, P.data(), P.size() * 8, cudaMemcpyHostToDevice), "cudaMemcpy(skip matrices)");
        cu(cudaDeviceGetAttribute(&d.sms, cudaDevAttrMultiProcessorCount, dev), "cudaDeviceGetAttribute");
    }
    return d;
}

std::vector<double> param_block(const std::vector<double>& prm)
{
    const size_t n = prm.size();
    const size_t pair = (n + (n + 1) / 2 + 1) & ~(size_t)1;   // 16-byte aligned
    std::vector<double> blk(pair + 2 * n, 0.0);
    std::memcpy(blk.data(), prm.data(), n * 8);
    float* f = (float*)(blk.data() + n);
    for (size_t i = 0; i < n; i++) f[i] = (float)prm[i];
    float* pd = (float*)(blk.data() + pair);
    for (size_t i = 0; i < n; i++) {
        pd[4 * i] = pd[4 * i + 1] = (float)prm[i];
        pd[4 * i + 2] = pd[4 * i + 3] = (float)(prm[i] - (double)pd[4 * i]);
    }
    return blk;
}

}  // namespace ftrt

using namespace ftrt;

namespace {

// The kernels' vertex labels (any labelling gives the same integrand; the reference
// deletes a vertex chosen per sample, srcs/feynman_integral.hpp:166-194): vertices whose
// row of P is zero first, in their order, then the external ones, the last external
// vertex being the deleted one.  The eliminations then remove the internal vertices
// first, and the quadratic forms of P~ only involve the external rows [q0, V-1).
void relabel(ft_plan& pl)
{
    const ft::prepared& p = pl.P;
    const int V = p.V;
    std::vector<int> ext(V, 0), lab(V, -1);
    for (int v = 0; v < V; v++)
        for (int w = 0; w < V; w++) ext[v] |= p.P[(size_t)v * V + w] != 0.0;
    int next = 0;
    for (int pass = 0; pass < 2; pass++)
        for (int v = 0; v < V; v++)
            if (ext[v] == pass) lab[v] = next++;
    int nint = 0;
    for (int v = 0; v < V; v++) nint += !ext[v];
    pl.q0 = nint == V ? V - 1 : nint;
    pl.kek.resize(p.E);
    pl.kel.resize(p.E);
    for (int e = 0; e < p.E; e++) {
        const int a = lab[p.ek[e]], b = lab[p.el[e]];
        pl.kek[e] = a > b ? a : b;
        pl.kel[e] = a > b ? b : a;
    }
    pl.kP.assign((size_t)V * V, 0.0);
    for (int v = 0; v < V; v++)
        for (int w = 0; w < V; w++) pl.kP[(size_t)lab[v] * V + lab[w]] = p.P[(size_t)v * V + w];
}

// P~ = kP restricted to vertices 0..V-2 (vertex V-1 is the deleted one), split as
// sum_r sigma_r q_r q_r^T; eigenpairs with |sigma| <= 1e-14 max|sigma| are dropped
void low_rank(const std::vector<double>& P, int V, std::vector<double>& sigma, std::vector<double>& q)
{
    const int n = V - 1;
    std::vector<double> A((size_t)n * n), Vv((size_t)n * n, 0.0);
    for (int i = 0; i < n; i++)
        for (int j = 0; j < n; j++) A[i * n + j] = P[i * V + j];
    for (int i = 0; i < n; i++) Vv[i * n + i] = 1.0;
    for (int sweep = 0; sweep < 100; sweep++) {
        double off = 0;
        for (int i = 0; i < n; i++)
            for (int j = i + 1; j < n; j++) off += A[i * n + j] * A[i * n + j];
        if (off < 1e-300) break;
        for (int a = 0; a < n; a++)
            for (int b = a + 1; b < n; b++) {
                double apq = A[a * n + b];
                if (apq == 0.0) continue;
                double theta = (A[b * n + b] - A[a * n + a]) / (2.0 * apq);
                double t = (theta >= 0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
                double c = 1.0 / std::sqrt(t * t + 1.0), s = t * c;
                for (int k = 0; k < n; k++) {
                    double akp = A[k * n + a], akq = A[k * n + b];
                    A[k * n + a] = c * akp - s * akq;
                    A[k * n + b] = s * akp + c * akq;
                }
                for (int k = 0; k < n; k++) {
                    double apk = A[a * n + k], aqk = A[b * n + k];
                    A[a * n + k] = c * apk - s * aqk;
                    A[b * n + k] = s * apk + c * aqk;
                }
                for (int k = 0; k < n; k++) {
                    double vka = Vv[k * n + a], vkb = Vv[k * n + b];
                    Vv[k * n + a] = c * vka - s * vkb;
                    Vv[k * n + b] = s * vka + c * vkb;
                }
            }
    }
    double mx = 0;
    for (int i = 0; i < n; i++) mx = std::max(mx, std::fabs(A[i * n + i]));
    sigma.clear();
    q.clear();
    for (int r = 0; r < n; r++) {
        double ev = A[r * n + r];
        if (mx == 0.0 || std::fabs(ev) <= 1e-14 * mx) continue;
        sigma.push_back(ev);
        for (int i = 0; i < n; i++) q.push_back(Vv[i * n + r]);
    }
    if (sigma.empty()) {   // P~ = 0: one zero term keeps the arrays non-empty
        sigma.push_back(0.0);
        q.assign(n, 0.0);
    }
}


}  // namespace

namespace {

// parameter block and table bytes in the layout the kernel body expects
void build_blocks(ft_plan& pl)
{
    const ft::prepared& p = pl.P;
    const int E = p.E, n = p.V - 1, R = (int)pl.sigma.size(), ne = n - pl.q0;
    pl.prm.assign(8 + 2 * E + R + R * n + ne * (ne + 1) / 2, 0.0);
    pl.prm[0] = p.D;
    pl.prm[1] = p.W;
    pl.prm[2] = p.IGtr;
    pl.prm[3] = p.def_ref;
    pl.prm[4] = 1. / (p.D / 2. * p.loops + p.W);
    pl.prm[5] = p.Jr[(1ULL << E) - 1];
    pl.prm[6] = -pl.prm[4] * (p.D / 2.);
    pl.prm[7] = -pl.prm[4] * p.W;
    for (int e = 0; e < E; e++) {
        pl.prm[8 + e] = p.m2[e];
        pl.prm[8 + E + e] = p.nu[e];
    }
    for (int r = 0; r < R; r++) {
        pl.prm[8 + 2 * E + r] = pl.sigma[r];
        for (int i = 0; i < n; i++) pl.prm[8 + 2 * E + R + r * n + i] = pl.q[r * n + i];
    }
    // P~ on the external rows [q0, n): upper triangle row by row, off-diagonal doubled
    // (the mixed form's deformed integrand contracts it with L(y)^-1 directly)
    for (int j = 0, o = 8 + 2 * E + R + R * n; j < ne; j++)
        for (int k = j; k < ne; k++) pl.prm[o++] = (j == k ? 1.0 : 2.0) * pl.kP[(size_t)(pl.q0 + j) * p.V + pl.q0 + k];
    const size_t N = 1ULL << E;
    const size_t f32 = (24 * N + 15) & ~(size_t)15;
    const bool cut = ft::staged_table(E);
    pl.tab.assign(f32 + (cut ? 12 + 2 * (size_t)E : 20) * N, 0);
    double* w64 = (double*)pl.tab.data();
    double* Jr64 = w64 + N;
    double* ri64 = w64 + 2 * N;
    float* rh = (float*)(pl.tab.data() + f32);
    float* rl = rh + N;
    unsigned* meta = (unsigned*)(rl + N);
    unsigned* q = meta + N;
    float* w32 = (float*)(meta + N);
    float* Jr32 = w32 + N;
    unsigned off = 0;
    for (size_t s = 0; s < N; s++) {
        // the scan adds Jr/r and the X update raises to 1./r (srcs/tropical_sampling.hpp:487,558)
        w64[s] = p.Jr[s] / p.r[s];
        Jr64[s] = p.Jr[s];
        ri64[s] = 1. / p.r[s];
        rh[s] = (float)ri64[s];   // 1/r as two floats (hi, lo)
        rl[s] = (float)(ri64[s] - (double)rh[s]);
        meta[s] = (p.mm[s] ? 0x80u : 0u) | (unsigned)(p.L[s] & 0x7f);
        if (!cut) {
            w32[s] = (float)w64[s];
            Jr32[s] = (float)Jr64[s];
            continue;
        }
        // cut thresholds: floor(2^28 T_k / Jr(s)) << 4 | edge, T_k the running sum of Jr/r over
        // the subgraph's edges in the reference's order (srcs/tropical_sampling.hpp:482-490);
        // smaller subgraphs (those with an edge less) have smaller masks, so w64 is complete
        meta[s] |= off << 16;
        const double scale = 268435456.0 / Jr64[s];
        double T = 0.0;
        for (size_t left = s; left; left &= left - 1) {
            const int c = __builtin_ctzll(left);
            T += w64[s ^ ((size_t)1 << c)];
            const double v = T * scale;
            q[off++] = (v < 268435455.0 ? (unsigned)v : 268435455u) << 4 | (unsigned)c;
        }
    }
}

// device copies and scratch of a plan, made on its first integration (a plan used only
// through batches never has its own)
void upload(ft_plan& pl)
{
    if (pl.d_prm) return;
    if (!pl.stream) static_cast<run_scratch&>(pl) = acquire_scratch(pl.device);
    const std::vector<double> blk = param_block(pl.prm);
    const size_t off = (blk.size() * 8 + 255) & ~(size_t)255, bytes = off + pl.tab.size();
    // up to 12 MB (E = 18) through pinned staging, which the next plans of the set use again.  Larger
    // tables go from the plan's own memory: pinning as much again, for sets too large to be kept,
    // cost more than it saved (E = 19, 23 MB: first integration of a plan 2.3 -> 0.45 ms, closing it
    // 0.61 -> 0.004, as its set now fits the 32 MB)
    const bool staged = bytes <= pl.kStagedBytes;
    if (bytes > pl.in_cap || (staged && !pl.h_in)) {
        if (pl.d_in) cudaFree(pl.d_in);
        if (pl.h_in) cudaFreeHost(pl.h_in);
        pl.d_in = pl.h_in = nullptr;
        pl.in_cap = 0;
        const size_t cap = std::max<size_t>(bytes, 64 * 1024);
        device_alloc((void**)&pl.d_in, cap, "cudaMalloc(parameters and table)");
        if (staged) cu(cudaMallocHost(&pl.h_in, cap), "cudaMallocHost(parameters and table)");
        pl.in_cap = cap;
    }
    if ((size_t)pl.slots() > pl.final_cap) {
        if (pl.h_final) cudaFreeHost(pl.h_final);
        pl.h_final = nullptr;
        pl.final_cap = 0;
        cu(cudaMallocHost(&pl.h_final, pl.slots() * 8), "cudaMallocHost(final)");
        pl.final_cap = pl.slots();
    }
    pl.uploading = true;
    if (staged) {
        std::memcpy(pl.h_in, blk.data(), blk.size() * 8);
        std::memcpy(pl.h_in + off, pl.tab.data(), pl.tab.size());
        cu(cudaMemcpyAsync(pl.d_in, pl.h_in, bytes, cudaMemcpyHostToDevice, pl.stream), "cudaMemcpyAsync(parameters)");
    } else {   // pageable: read before the calls return
        cu(cudaMemcpyAsync(pl.d_in, blk.data(), blk.size() * 8, cudaMemcpyHostToDevice, pl.stream),
           "cudaMemcpyAsync(parameters)");
        cu(cudaMemcpyAsync(pl.d_in + off, pl.tab.data(), pl.tab.size(), cudaMemcpyHostToDevice, pl.stream),
           "cudaMemcpyAsync(table)");
    }
    pl.d_prm = (double*)pl.d_in;
    pl.d_tab = pl.d_in + off;
}

// before work of the plan on stream st
void order_after_upload(ft_plan& pl, cudaStream_t st)
{
    if (!pl.uploading || st == pl.stream) return;
    cu(cudaStreamSynchronize(pl.stream), "upload");
    pl.uploading = false;
}

void ensure_parts(ft_plan& pl, size_t nparts)
{
    size_t need = nparts * pl.slots();
    if (need <= pl.parts_cap) return;
    if (pl.d_parts) cudaFree(pl.d_parts);
    pl.d_parts = nullptr;
    pl.parts_cap = 0;
    device_alloc((void**)&pl.d_parts, need * 8, "cudaMalloc(partial sums)");
    pl.parts_cap = need;
}

void ensure_queue(ft_plan& pl, size_t entries)
{
    if (entries <= pl.qcap) return;
    if (pl.d_queue) cudaFree(pl.d_queue);
    pl.d_queue = nullptr;
    pl.qcap = 0;
    device_alloc((void**)&pl.d_queue, entries * 5 * 8, "cudaMalloc(FP64 queue)");
    pl.qcap = entries;
}

// the stride's matrices; *made is set when they had to be computed (one launch)
const unsigned long long* stride_matrices(ft_plan& pl, unsigned long long S, int digits, cudaStream_t st, bool* made)
{
    pl.stride_clock++;
    run_scratch::stride_entry* victim = &pl.strides[0];
    for (run_scratch::stride_entry& e : pl.strides) {
        if (e.d && e.S == S && e.digits >= digits) {
            e.used = pl.stride_clock;
            *made = false;
            return e.d;
        }
        if (e.used < victim->used) victim = &e;
    }
    victim->digits = -1;
    if (victim->cap < digits) {
        if (victim->d) cudaFree(victim->d);
        victim->d = nullptr;
        victim->cap = -1;
        device_alloc((void**)&victim->d, ft::stride_words(digits) * 8, "cudaMalloc(stride matrices)");
        victim->cap = digits;
    }
    cu(ft::launch_stride_matrices(dev_state().tpow, S, digits, victim->d, st), "stride matrices");
    victim->S = S;
    victim->digits = digits;
    victim->used = pl.stride_clock;
    *made = true;
    return victim->d;
}

struct launch_geometry {
    unsigned blocks;
    unsigned long long chunk;
    int lanebits;
};

// Threads of a launch and samples per thread.  Kernels without the per-sample block
// barrier (the FP64 form) get at most 128 samples per thread, in whole waves of resident
// blocks (a multiple of the SM count): with long static chunks the warps of a block
// drift apart and the block waits at its final reduction for its slowest warp (the
// 5-loop cube ran 6x slower at 2570 samples per thread than at 128).  Kernels with the
// barrier keep their warps together and run one wave of long chunks (more waves cost
// them 1-2 % per halving of the chunk).  max_blocks bounds the waves (the
// no-allocation path, whose scratch holds a bounded number of blocks).
launch_geometry geometry(const ft::kernel_set& ks, unsigned long long N, unsigned long long max_blocks = ~0ull)
{
    const unsigned long long wave_blocks = (unsigned long long)dev_state().sms * ks.blocks_per_sm;
    const unsigned long long per_wave = wave_blocks * ks.block;
    unsigned long long w = 1;
    if (N > 0 && !(ks.variant & 4)) {
        static const unsigned long long cap = [] {
            const char* e = std::getenv("FEYNTROP_GB300_CHUNK_CAP");
            const unsigned long long v = e ? std::strtoull(e, nullptr, 10) : 128ull;
            return v ? v : 128ull;
        }();
        w = std::max(1ull, (N + per_wave * cap - 1) / (per_wave * cap));
        w = std::min(w, std::max(1ull, max_blocks / wave_blocks));
    }
    const unsigned long long max_threads = per_wave * w;
    launch_geometry g;
    g.chunk = N == 0 ? 1 : (N + max_threads - 1) / max_threads;
    const unsigned long long threads = N == 0 ? 1 : (N + g.chunk - 1) / g.chunk;
    g.blocks = (unsigned)((threads + ks.block - 1) / ks.block);
    g.lanebits = 1;
    while ((1ULL << g.lanebits) < (unsigned long long)g.blocks * ks.block) g.lanebits++;
    return g;
}

struct records {
    uint8_t* order = nullptr;
    double* X = nullptr;
    double* R = nullptr;
    uint8_t* flags = nullptr;
};

struct run_out {
    std::vector<double> acc;   // slots
    double kernel_ms = 0;
    int launches = 0;
};

// the launches of one integration (or one record run) on stream st
run_out run(ft_plan& pl, const ft_run_options& o, cudaStream_t st, const records* rec)
{
    const int prec = o.precision == FT_PRECISION_MIXED ? 1 : 0;
    const int record = rec ? 1 : 0;
    if (prec && !ft::find_kernels(pl.key(prec, record))) {
        // with the FP64 sampling kernel, for a run that hands over more than its queue holds
        ft::precompile_all({pl.key(prec, record), pl.key(0, record), pl.key(0, record, 0, 1)});
        ft::get_kernels(pl.key(0, record));
    }
    const ft::kernel_set& ks = ft::get_kernels(pl.key(prec, record));
    const ft::kernel_set* k64 = prec ? &ft::get_kernels(pl.key(0, record, 0, 1)) : nullptr;
    const unsigned long long N = o.num_samples;
    const launch_geometry g = geometry(ks, N);
    const unsigned long long draws = 2ULL * pl.P.E - 1;
    run_out out;
    out.acc.assign(pl.slots(), 0.0);
    if (N == 0) return out;

    order_after_upload(pl, st);
    if (pl.running) {
        // the last run failed: its work may be in flight on another stream, its stride
        // matrices unwritten, its counters not back at zero
        cu(cudaDeviceSynchronize(), "after a failed run");
        for (run_scratch::stride_entry& e : pl.strides) e.digits = -1;
        cu(cudaMemsetAsync(pl.d_qcount, 0, 16, st), "cudaMemsetAsync");
    }
    pl.running = true;
    bool made = false;
    int digits = ft::stride_digits(g.lanebits);
    const unsigned long long* mats = stride_matrices(pl, g.chunk * draws, digits, st, &made);
    if (made) out.launches++;
    const unsigned qblocks = prec ? (unsigned)(dev_state().sms * std::max(1, k64->queue_blocks_per_sm)) : 0;
    ensure_parts(pl, g.blocks + qblocks + 1);
    if (prec) {
        size_t want = (size_t)std::min<unsigned long long>(N, N / 16 + 65536);
        ensure_queue(pl, want);
        pl.queue_entries = std::max(pl.queue_entries, want);   // not qcap: a pooled queue may be longer
    }
    ft::xstate base = ft::advance(ft::seed_state(o.seed), o.first_sample * draws);
    cu(cudaEventRecord(pl.ev0, st), "cudaEventRecord");
    unsigned long long nsamples = N, chunk = g.chunk;
    unsigned int qcap = (unsigned int)pl.queue_entries;
    unsigned long long* queue = pl.d_queue;
    unsigned int *qcount = pl.d_qcount, *ticket = pl.d_qcount + 1;
    double *parts = pl.d_parts, *final_out = pl.h_final, *none = nullptr;
    const double* prm = pl.d_prm;
    const unsigned char* tab = pl.d_tab;
    uint8_t* r_order = nullptr;
    double* r_X = nullptr;
    double* r_R = nullptr;
    uint8_t* r_flags = nullptr;
    if (rec) {
        r_order = rec->order;
        r_X = rec->X;
        r_R = rec->R;
        r_flags = rec->flags;
    }
    void* args[] = {&prm, &tab, &mats, &digits, &base.s[0], &base.s[1], &base.s[2], &base.s[3], &nsamples, &chunk,
                    &parts, &queue, &qcount, &qcap, &ticket, prec ? &none : &final_out, &r_order, &r_X, &r_R, &r_flags};
    ft::check(ft::drv().LaunchKernel(ks.sample, g.blocks, 1, 1, ks.block, 1, 1, ks.smem, (CUstream)st, args, nullptr),
              "launch ft_sample");
    out.launches++;
    if (prec) {
        unsigned int nparts = g.blocks;
        void* qargs[] = {&prm, &tab, &queue, &qcount, &qcap, &parts, &nparts, &ticket, &final_out,
                         &r_order, &r_X, &r_R, &r_flags};
        ft::check(ft::drv().LaunchKernel(k64->queue, qblocks, 1, 1, k64->block, 1, 1, k64->smem, (CUstream)st, qargs,
                                         nullptr),
                  "launch ft_sample_queue");
        out.launches++;
    }
    cu(cudaEventRecord(pl.ev1, st), "cudaEventRecord");
    cu(cudaStreamSynchronize(st), "sampling");
    pl.running = false;
    if (st == pl.stream) pl.uploading = false;
    float ms = 0;
    cu(cudaEventElapsedTime(&ms, pl.ev0, pl.ev1), "cudaEventElapsedTime");
    out.kernel_ms = ms;
    out.acc.assign(pl.h_final, pl.h_final + pl.slots());
    const unsigned long long queued = (unsigned long long)out.acc[8 * pl.P.K + 2];
    if (prec && queued > qcap) {
        // more samples needed FP64 than the queue holds: redo the whole range in FP64
        ft_run_options o64 = o;
        o64.precision = FT_PRECISION_FP64;
        run_out r = run(pl, o64, st, rec);
        r.acc[8 * pl.P.K + 2] = (double)queued;
        r.launches += out.launches;
        r.kernel_ms += out.kernel_ms;
        return r;
    }
    return out;
}


}  // namespace

namespace ftrt {

void fill_result(const ft::prepared& P, const std::vector<double>& acc, ft_result* r)
{
    const int K = P.K;
    r->num_eps_terms = K;
    r->kept = (uint64_t)acc[8 * K];
    r->dropped = (uint64_t)acc[8 * K + 1];
    r->fp64_fallback = (uint64_t)acc[8 * K + 2];
    r->exact_steps = (uint64_t)acc[8 * K + 3];
    r->robust = (uint64_t)acc[8 * K + 4];
    std::vector<ft_moments> m(2 * K);
    for (int j = 0; j < K; j++)
        for (int part = 0; part < 2; part++) {
            ft_moments& x = m[2 * j + part];
            x.n = (double)r->kept;
            x.s1_hi = acc[8 * j + 4 * part + 0];
            x.s1_lo = acc[8 * j + 4 * part + 1];
            x.s2_hi = acc[8 * j + 4 * part + 2];
            x.s2_lo = acc[8 * j + 4 * part + 3];
        }
    if (r->moments) std::memcpy(r->moments, m.data(), m.size() * sizeof(ft_moments));
    ft_finalize_moments(m.data(), K, P.deformed() ? 0 : 1, r);
}

}  // namespace ftrt

static ft::problem_input input_of(const ft_problem* pb)
{
    if (!pb || pb->num_edges < 1 || !pb->edges || !pb->nu || !pb->masses_sqr || !pb->scalarproducts)
        throw std::invalid_argument("empty or incomplete problem");
    ft::problem_input in;
    int Vmax = 0;
    for (int e = 0; e < pb->num_edges; e++) {
        in.v.push_back(pb->edges[2 * e]);
        in.w.push_back(pb->edges[2 * e + 1]);
        in.nu.push_back(pb->nu[e]);
        in.m2.push_back(pb->masses_sqr[e]);
        Vmax = std::max(Vmax, std::max(pb->edges[2 * e], pb->edges[2 * e + 1]) + 1);
    }
    const int V = pb->num_vertices >= 0 ? pb->num_vertices : Vmax;
    if (V != Vmax) throw std::invalid_argument("input scalarproducts must be a (V x V)-matrix");
    in.P.assign(pb->scalarproducts, pb->scalarproducts + (size_t)V * V);
    in.D = pb->dimension;
    in.K = pb->num_eps_terms;
    in.lambda = pb->lambda;
    if (in.K < 1) throw std::invalid_argument("num_eps_terms must be at least 1");
    return in;
}

static void info_of(const ft::prepared& P, size_t table_bytes, ft_plan_info* info)
{
    info->W = P.W;
    info->IGtr = P.IGtr;
    info->loops = P.loops;
    info->euclidean = P.euclidean;
    info->pseudo_euclidean = P.pseudo_euclidean;
    info->generic = P.generic;
    info->gp_property = P.gp;
    info->deformed = P.deformed();
    info->lambda_used = P.lambda;
    info->seconds_preprocessing = P.seconds_preprocessing;
    info->table_bytes = table_bytes;
    info->num_log_lines = (int)P.log.size();
}

// ------------------------------------------------------------------ C ABI
extern "C" {

const char* ft_last_error(void) { return g_error.c_str(); }
const char* ft_version(void) { return "feyntrop_gb300 0.1 (sm_103a)"; }
void ft_free(void* p) { std::free(p); }

// host part of a plan (preprocessing, parameter block, table); threads for the table
static std::unique_ptr<ft_plan> make_plan(const ft_problem* pb, int threads, int device)
{
    ft::problem_input in = input_of(pb);
    std::unique_ptr<ft_plan> pl(new ft_plan());
    pl->P = ft::prepare(in, threads);
    if (pl->P.E > 24) throw std::domain_error("graphs with more than 24 edges are not supported by the GPU sampler");
    relabel(*pl);
    low_rank(pl->kP, pl->P.V, pl->sigma, pl->q);
    build_blocks(*pl);
    pl->device = device;
    return pl;
}

// status of a failed plan creation: input errors keep their codes, a missing device
// (std::logic_error from require_device) is FT_ERR_NO_DEVICE
static int create_status(const std::exception_ptr& ep)
{
    try {
        std::rethrow_exception(ep);
    } catch (const std::invalid_argument&) {
        return status_of(ep);
    } catch (const std::domain_error&) {
        return status_of(ep);
    } catch (const std::logic_error& e) {
        g_error = e.what();
        return FT_ERR_NO_DEVICE;
    } catch (...) {
        return status_of(ep);
    }
}

int ft_plan_create(const ft_problem* pb, ft_plan** out)
{
    *out = nullptr;
    try {
        std::unique_ptr<ft_plan> pl = make_plan(pb, 0, 0);
        require_device();
        dev_state();
        cu(cudaGetDevice(&pl->device), "cudaGetDevice");
        *out = pl.release();
        return FT_OK;
    } catch (...) {
        return create_status(std::current_exception());
    }
}

int ft_plans_create(const ft_problem* problems, int32_t count, ft_plan** out, int32_t* status)
{
    if (!out || (count > 0 && !problems)) {
        g_error = "ft_plans_create: NULL argument";
        return FT_ERR_INVALID_ARGUMENT;
    }
    for (int i = 0; i < count; i++) {
        out[i] = nullptr;
        if (status) status[i] = FT_ERR_RUNTIME;
    }
    int device = 0;
    try {
        require_device();
        dev_state();
        cu(cudaGetDevice(&device), "cudaGetDevice");
    } catch (...) {
        const int rc = create_status(std::current_exception());
        if (status)
            for (int i = 0; i < count; i++) status[i] = rc;
        return rc;
    }
    // one problem per task on all host threads (each table single-threaded)
    std::vector<int> rcs(count, FT_OK);
    std::vector<std::string> msgs(count);
    std::atomic<int> next{0};
    auto work = [&]() {
        for (int i = next.fetch_add(1); i < count; i = next.fetch_add(1)) {
            try {
                out[i] = make_plan(&problems[i], 1, device).release();
            } catch (...) {
                rcs[i] = create_status(std::current_exception());
                msgs[i] = g_error;
            }
        }
    };
    const int nth = (int)std::min<unsigned>(std::max(1u, std::thread::hardware_concurrency()), (unsigned)std::max(1, count));
    std::vector<std::thread> pool;
    for (int t = 1; t < nth; t++) pool.emplace_back(work);
    work();
    for (auto& th : pool) th.join();
    int first = FT_OK;
    for (int i = 0; i < count; i++) {
        if (status) status[i] = rcs[i];
        if (rcs[i] != FT_OK && first == FT_OK) {
            first = rcs[i];
            g_error = "problem " + std::to_string(i) + ": " + msgs[i];
        }
    }
    return first;
}

void ft_plan_destroy(ft_plan* p) { delete p; }

void ft_release_scratch(void) { free_idle_scratch(); }

int ft_plan_get_info(const ft_plan* pl, ft_plan_info* info)
{
    info_of(pl->P, pl->tab.size(), info);
    return FT_OK;
}

const char* ft_plan_log_line(const ft_plan* pl, int32_t i)
{
    if (i < 0 || i >= (int)pl->P.log.size()) return "";
    return pl->P.log[i].c_str();
}

int ft_subgraph_table(const ft_problem* pb, double* Jr, double* r, uint8_t* mm, uint8_t* L, ft_plan_info* info)
{
    try {
        ft::prepared P = ft::prepare(input_of(pb));
        const size_t n = P.Jr.size();
        if (Jr) std::memcpy(Jr, P.Jr.data(), n * 8);
        if (r) std::memcpy(r, P.r.data(), n * 8);
        if (mm) std::memcpy(mm, P.mm.data(), n);
        if (L) std::memcpy(L, P.L.data(), n);
        if (info) info_of(P, 0, info);
        return FT_OK;
    } catch (...) {
        return status_of(std::current_exception());
    }
}

int ft_precompile(const ft_problem* pb, int32_t precision, double* seconds)
{
    try {
        ft::problem_input in = input_of(pb);
        ft_plan pl;
        pl.P = ft::prepare(in);
        relabel(pl);
        low_rank(pl.kP, pl.P.V, pl.sigma, pl.q);
        auto t0 = std::chrono::steady_clock::now();
        const int prec = precision & 0xff;
        const bool batch = (precision & FT_PRECOMPILE_BATCH) != 0;
        std::vector<ft::kernel_key> keys;
        for (int bt = 0; bt <= (batch ? 1 : 0); bt++) {
            keys.push_back(pl.key(0, 0, bt));
            if (prec != FT_PRECISION_MIXED) continue;
            keys.push_back(pl.key(1, 0, bt));
            keys.push_back(pl.key(0, 0, bt, 1));
        }
        ft::precompile_all(keys);
        if (seconds) *seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        return FT_OK;
    } catch (...) {
        return status_of(std::current_exception());
    }
}

int ft_device_peaks(double* fp32, double* fp64)
{
    try {
        require_device();
        if (fp32) *fp32 = ft::fma_peak_tflops(false);
        if (fp64) *fp64 = ft::fma_peak_tflops(true);
        cu(cudaGetLastError(), "probe kernels");
        return FT_OK;
    } catch (const std::logic_error& e) {
        g_error = e.what();
        return FT_ERR_NO_DEVICE;
    } catch (...) {
        return status_of(std::current_exception());
    }
}

int ft_finalize_moments(const ft_moments* m, int32_t K, int32_t real_only, ft_result* r)
{
    // srcs/stats.hpp:86-104 on the merged sums (long double for the final arithmetic)
    for (int j = 0; j < K; j++) {
        for (int part = 0; part < 2; part++) {
            const ft_moments& x = m[2 * j + part];
            double avg, acc;
            if (part == 1 && real_only) {
                avg = 0.0;   // two zero updates per thread in the reference (srcs/feynman_integral.hpp:130-140)
                acc = 0.0;
            } else {
                const long double N = x.n;
                const long double S1 = (long double)x.s1_hi + x.s1_lo, S2 = (long double)x.s2_hi + x.s2_lo;
                const long double a = S1 / N;
                const long double var = (N / (N - 1)) * (S2 / N - a * a);
                avg = (double)a;
                acc = (double)std::sqrt(var / N);
            }
            if (part == 0) {
                if (r->re_avg) r->re_avg[j] = avg;
                if (r->re_acc) r->re_acc[j] = acc;
            } else {
                if (r->im_avg) r->im_avg[j] = avg;
                if (r->im_acc) r->im_acc[j] = acc;
            }
        }
    }
    return FT_OK;
}

int ft_integrate(ft_plan* pl, const ft_run_options* o, ft_result* r)
{
    try {
        std::lock_guard<std::mutex> lock(pl->mu);
        auto t0 = std::chrono::steady_clock::now();
        cu(cudaSetDevice(pl->device), "cudaSetDevice");
        upload(*pl);
        cudaStream_t st = o->stream ? (cudaStream_t)o->stream : pl->stream;
        run_out ro = run(*pl, *o, st, nullptr);
        fill_result(pl->P, ro.acc, r);
        r->kernel_ms = ro.kernel_ms;
        r->kernel_launches = ro.launches;
        r->seconds_sampling = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
        return FT_OK;
    } catch (...) {
        return status_of(std::current_exception());
    }
}

int ft_integrate_noalloc(ft_plan* pl, const ft_run_options* o, double* d_slots)
{
    try {
        std::lock_guard<std::mutex> lock(pl->mu);
        cu(cudaSetDevice(pl->device), "cudaSetDevice");
        if (!d_slots) throw std::invalid_argument("ft_integrate_noalloc: output pointer is NULL");
        const int prec = o->precision == FT_PRECISION_MIXED ? 1 : 0;
        if (pl->slots() > NOALLOC_MAX_SLOTS)
            throw std::invalid_argument("ft_integrate_noalloc: more than 16 eps orders exceed the static scratch");
        const ft::kernel_set* ks = ft::find_kernels(pl->key(prec, 0));
        const ft::kernel_set* k64 = prec ? ft::find_kernels(pl->key(0, 0, 0, 1)) : nullptr;
        if (!ks || (prec && !k64) || !pl->d_prm)
            throw std::invalid_argument(
                "ft_integrate_noalloc: this plan's kernels are not loaded; call ft_integrate once with the same "
                "precision first (loading them allocates)");
        const unsigned long long N = o->num_samples;
        if (N == 0) throw std::invalid_argument("ft_integrate_noalloc: num_samples must be positive");
        const unsigned qblocks = prec ? (unsigned)(dev_state().sms * std::max(1, k64->queue_blocks_per_sm)) : 0;
        // ft_integrate's launch shape, its waves capped to the blocks the scratch holds
        const launch_geometry g =
            geometry(*ks, N,
                     qblocks < NOALLOC_MAX_BLOCKS ? (unsigned long long)(NOALLOC_MAX_BLOCKS - qblocks) : 1ull);
        if (g.blocks + qblocks > NOALLOC_MAX_BLOCKS || g.lanebits > NOALLOC_MAX_LANE_BITS)
            throw std::invalid_argument("ft_integrate_noalloc: launch exceeds the static scratch (2048 blocks)");
        ft::noalloc_layout sc;
        cu(ft::noalloc_scratch(&sc), "cudaGetSymbolAddress(no-allocation scratch)");
        cudaStream_t st = o->stream ? (cudaStream_t)o->stream : pl->stream;
        order_after_upload(*pl, st);
        pl->detached = true;
        const unsigned long long draws = 2ULL * pl->P.E - 1;
        int digits = ft::stride_digits(g.lanebits);
        cu(ft::launch_stride_matrices(dev_state().tpow, g.chunk * draws, digits, sc.mats, st), "stride matrices");
        cu(cudaMemsetAsync(sc.qcount, 0, 8, st), "cudaMemsetAsync");   // hand-offs and ticket
        ft::xstate base = ft::advance(ft::seed_state(o->seed), o->first_sample * draws);
        unsigned long long nsamples = N, chunk = g.chunk;
        unsigned int qcap = NOALLOC_QUEUE_ENTRIES;
        unsigned long long* queue = sc.queue;
        unsigned int *qcount = sc.qcount, *ticket = sc.ticket;
        double *parts = sc.parts, *none = nullptr;
        const double* prm = pl->d_prm;
        const unsigned char* tab = pl->d_tab;
        const unsigned long long* mats = sc.mats;
        uint8_t* r_order = nullptr;
        double* r_X = nullptr;
        double* r_R = nullptr;
        uint8_t* r_flags = nullptr;
        void* args[] = {&prm, &tab, &mats, &digits, &base.s[0], &base.s[1], &base.s[2], &base.s[3], &nsamples,
                        &chunk, &parts, &queue, &qcount, &qcap, &ticket, prec ? &none : &d_slots, &r_order, &r_X,
                        &r_R, &r_flags};
        ft::check(ft::drv().LaunchKernel(ks->sample, g.blocks, 1, 1, ks->block, 1, 1, ks->smem, (CUstream)st, args,
                                         nullptr),
                  "launch ft_sample");
        if (prec) {
            unsigned int nparts = g.blocks;
            void* qargs[] = {&prm, &tab, &queue, &qcount, &qcap, &parts, &nparts, &ticket, &d_slots,
                             &r_order, &r_X, &r_R, &r_flags};
            ft::check(ft::drv().LaunchKernel(k64->queue, qblocks, 1, 1, k64->block, 1, 1, k64->smem, (CUstream)st,
                                             qargs, nullptr),
                      "launch ft_sample_queue");
        }
        return FT_OK;
    } catch (...) {
        return status_of(std::current_exception());
    }
}

int ft_autotune(ft_plan* pl, int32_t precision, uint64_t samples, ft_tune_result* out)
{
    try {
        if (!pl || !out) throw std::invalid_argument("ft_autotune: NULL argument");
        if (samples < 1000) throw std::invalid_argument("ft_autotune: at least 1000 samples per trial");
        std::lock_guard<std::mutex> lock(pl->mu);
        cu(cudaSetDevice(pl->device), "cudaSetDevice");
        upload(*pl);
        const int prec = precision == FT_PRECISION_MIXED ? 1 : 0;
        const bool deformed = pl->P.deformed();
        // candidates: launch shapes (threads per block x blocks per SM) and code variants
        std::vector<ft::launch_shape> cands;
        auto add = [&](int block, int minb, int variant) {
            ft::launch_shape s;
            s.block = block;
            s.minb = minb;
            s.variant = variant;
            cands.push_back(s);
        };
        if (prec == 1 && deformed) {
            // out-of-line two-float routines (bits 3, 4) and shapes from 128 registers (16 warps
            // per SM) to 255 (8 warps, no spills)
            // (four 128-thread blocks won one-integral trials by noise and ran the
            // persistent batch kernel 9 % slower: not a candidate)
            add(512, 1, 20);
            add(512, 1, 29);
            add(256, 2, 29);
            add(256, 2, 21);
            add(256, 2, 5);
            add(256, 1, 29);
        } else if (prec == 1) {
            for (int var : {4, 0}) {
                add(256, 1, var);
                add(256, 2, var);
                add(512, 1, var);
            }
        } else {
            for (int var : {4, 0}) {
                add(256, 1, var);
                add(256, 2, var);
                add(384, 1, var);
                add(512, 1, var);
            }
        }
        {
            // every candidate's kernels compiled concurrently before the timing
            std::vector<ft::kernel_key> keys;
            for (const ft::launch_shape& c : cands) {
                ft::kernel_key k = pl->key(prec, 0);
                ft::apply_shape(k, c);
                keys.push_back(k);
            }
            if (prec == 1) {
                keys.push_back(pl->key(0, 0));
                keys.push_back(pl->key(0, 0, 0, 1));
            }
            ft::precompile_all(keys);
        }
        // trials long enough for the steady state: at least 256 samples per thread of a
        // full 512-thread-per-SM launch (shorter trials favour small blocks, which only
        // balance the tail better)
        const uint64_t tsamples = std::max<uint64_t>(samples, (uint64_t)dev_state().sms * 512ull * 256ull);
        ft_run_options o{};
        o.num_samples = tsamples;
        o.precision = precision;
        double best_rate = -1, default_rate = -1;
        ft::launch_shape best;
        const ft::launch_shape dflt = ft::default_shape(pl->key(prec, 0));
        int tried = 0;
        for (const ft::launch_shape& c : cands) {
            pl->forced = true;
            pl->forced_prec = prec;
            pl->forced_shape = c;
            double rate = 0;
            try {
                ft_run_options w = o;
                w.num_samples = std::max<uint64_t>(1000, tsamples / 8);
                run(*pl, w, pl->stream, nullptr);   // loads the candidate
                for (int rep = 0; rep < 2; rep++) {
                    o.seed = (uint64_t)rep;
                    run_out ro = run(*pl, o, pl->stream, nullptr);
                    rate = std::max(rate, (double)tsamples / (ro.kernel_ms * 1e-3));
                }
            } catch (...) {
                pl->forced = false;
                throw;
            }
            pl->forced = false;
            tried++;
            const ft::kernel_key kc = [&] {
                ft::kernel_key k = pl->key(prec, 0);
                ft::apply_shape(k, c);
                return k;
            }();
            ft::kernel_key kd = pl->key(prec, 0);
            ft::apply_shape(kd, dflt);
            if (kc.block == kd.block && kc.minb == kd.minb && kc.variant == kd.variant)
                default_rate = std::max(default_rate, rate);
            if (rate > best_rate) {
                best_rate = rate;
                best = c;
            }
        }
        // a candidate replaces the default only when clearly faster: trials of close
        // shapes differ by run-to-run noise, and a one-integral trial does not rank close
        // shapes reliably for the persistent batch kernel
        const double kMargin = 1.03;
        if (default_rate > 0 && best_rate < kMargin * default_rate) {
            best = dflt;
            best_rate = default_rate;
        }
        best.rate = best_rate;
        ft::record_shape(pl->key(prec, 0), best);
        // the batch work item (samples per thread) of the class, under the chosen shape:
        // a batch of this one integral per candidate, with enough samples that even the
        // largest item leaves every SM four items
        double best_batch = -1, default_batch = -1;
        unsigned long long best_chunk = 0;
        const unsigned long long default_chunk = ft::default_chunk(pl->key(prec, 0));
        const uint64_t bsamples =
            std::max<uint64_t>(tsamples, (uint64_t)dev_state().sms * (uint64_t)pl->key(prec, 0).block * 256ull * 4ull);
        for (unsigned long long c : {8ull, 16ull, 32ull, 64ull, 128ull, 256ull}) {
            if (prec ? c < 32 : c > 64) continue;   // outside the precision's range
            ft::set_chunk_override(c);
            ft_batch* b = nullptr;
            int rc = ft_batch_create(&pl, 1, prec, &b);
            ft::set_chunk_override(0);
            if (rc != FT_OK) throw std::runtime_error(std::string("ft_autotune: batch: ") + g_error);
            std::vector<double> avg(4 * pl->P.K);
            ft_result r{};
            r.num_eps_terms = pl->P.K;
            r.re_avg = avg.data();
            r.re_acc = avg.data() + pl->P.K;
            r.im_avg = avg.data() + 2 * pl->P.K;
            r.im_acc = avg.data() + 3 * pl->P.K;
            double rate = 0;
            for (int rep = 0; rep < 3 && rc == FT_OK; rep++) {
                ft_run_options bo = o;
                bo.num_samples = bsamples;
                bo.seed = (uint64_t)rep;
                bo.stream = nullptr;
                rc = ft_batch_run(b, &bo, &r);
                ft_batch_info bi{};
                ft_batch_get_info(b, &bi);
                if (rep > 0 && bi.kernel_ms > 0) rate = std::max(rate, (double)bsamples / (bi.kernel_ms * 1e-3));
            }
            ft_batch_destroy(b);
            if (rc != FT_OK) throw std::runtime_error(std::string("ft_autotune: batch run: ") + g_error);
            if (rate > best_batch) {
                best_batch = rate;
                best_chunk = c;
            }
            if (c == default_chunk) default_batch = rate;
        }
        if (default_batch > 0 && best_batch < kMargin * default_batch) {
            best_batch = default_batch;
            best_chunk = default_chunk;
        }
        best.chunk = best_chunk;
        ft::record_shape(pl->key(prec, 0), best);
        out->batch_chunk = best_chunk;
        out->batch_samples_per_second = best_batch;
        ft::kernel_key kb = pl->key(prec, 0);
        out->block = kb.block;
        out->min_blocks_per_sm = kb.minb;
        out->variant = kb.variant;
        out->samples_per_second = best_rate;
        out->default_samples_per_second = default_rate;
        out->candidates = tried;
        return FT_OK;
    } catch (...) {
        if (pl) pl->forced = false;
        return status_of(std::current_exception());
    }
}

int ft_sample_records(ft_plan* pl, const ft_run_options* o, uint8_t* order, double* X, double* R, uint8_t* flags)
{
    try {
        std::lock_guard<std::mutex> lock(pl->mu);
        cu(cudaSetDevice(pl->device), "cudaSetDevice");
        upload(*pl);
        const size_t N = o->num_samples, E = pl->P.E, K = pl->P.K;
        records d;
        device_alloc((void**)&d.order, N * E + 1, "cudaMalloc(records)");
        device_alloc((void**)&d.X, N * E * 8 + 8, "cudaMalloc(records)");
        device_alloc((void**)&d.R, N * K * 16 + 16, "cudaMalloc(records)");
        device_alloc((void**)&d.flags, N + 1, "cudaMalloc(records)");
        cu(cudaMemset(d.flags, 0, N + 1), "cudaMemset");
        run(*pl, *o, pl->stream, &d);
        if (order) cu(cudaMemcpy(order, d.order, N * E, cudaMemcpyDeviceToHost), "cudaMemcpy");
        if (X) cu(cudaMemcpy(X, d.X, N * E * 8, cudaMemcpyDeviceToHost), "cudaMemcpy");
        if (R) cu(cudaMemcpy(R, d.R, N * K * 16, cudaMemcpyDeviceToHost), "cudaMemcpy");
        if (flags) cu(cudaMemcpy(flags, d.flags, N, cudaMemcpyDeviceToHost), "cudaMemcpy");
        cudaFree(d.order);
        cudaFree(d.X);
        cudaFree(d.R);
        cudaFree(d.flags);
        return FT_OK;
    } catch (...) {
        return status_of(std::current_exception());
    }
}

}  // extern "C"
