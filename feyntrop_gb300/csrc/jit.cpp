#include "jit.hpp"
#include "kernels/aot.hpp"

#include <cuda_runtime.h>
#include <dlfcn.h>
#include <nvrtc.h>
#include <sys/stat.h>

#include <algorithm>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <map>
#include <mutex>
#include <sstream>
#include <stdexcept>
#include <thread>
#include <vector>

extern const char* ft_sample_body_source;   // generated at build time from kernels/sample_body.cuh

namespace ft {

static const char* kArch = "--gpu-architecture=sm_103a";

unsigned scratch_slots(const kernel_key& k)
{
    const unsigned E = (unsigned)k.E;
    if (k.mode == 0) return 4u * E;   // two samples
    return 2u * E + (k.scratch >= 1 ? 2u * E : 0u) + (k.scratch >= 2 ? E * (E + 1u) / 2u : 0u);
}

unsigned table_smem_bytes(const kernel_key& k)
{
    // staged table (unless read from global memory): 1/r (FP64, or two floats), a word per
    // subgraph and the cut thresholds (E 2^(E-1)); then the sums: FP64 form two doubles per
    // slot and thread, mixed form two floats per slot and thread, two doubles per slot and
    // warp, and the threads' scratch
    const unsigned entries = 1u << k.E;
    const unsigned tab = k.table_global ? 0u : (12u + 2u * (unsigned)k.E) * entries;
    const unsigned slots = (k.mode == 1 ? 4u : 2u) * (unsigned)k.K, block = (unsigned)k.block;
    const unsigned acc = k.prec == 0 ? 16u * slots * block
                                     : 8u * slots * block + 16u * slots * (block / 32u) + 4u * block * scratch_slots(k);
    return ((tab + 15u) & ~15u) + acc + 16u;
}

// Tables of the two-float logarithm, exponential and sine / cosine of the mixed kernels
// (FP32 values written exactly as hexadecimal literals):
//   FT_LOGTAB[i] = r_i = fl(1 / (1 + (i + 1/2)/64)), -log(r_i) as hi, lo, 0 (i < 64)
//   FT_EXPTAB[j] = 2^(j/32) as hi, lo (j < 32)
//   FT_ATANTAB[i] = atan(i/64) as hi, lo (i <= 64; 128 entries, as its index is masked)
//   FT_SCTAB[j] = sin(j pi/64) as hi, lo, cos(j pi/64) as hi, lo (j < 128)
static std::string tables_source()
{
    static const std::string text = [] {
        std::ostringstream s;
        char buf[64];
        s << "__device__ const float4 FT_LOGTAB[64] = {";
        for (int i = 0; i < 64; i++) {
            const float r = (float)(1.0 / (1.0 + (i + 0.5) / 64.0));
            const double nl = -std::log((double)r);
            const float hi = (float)nl, lo = (float)(nl - (double)hi);
            s << "{";
            for (float v : {r, hi, lo, 0.0f}) {
                std::snprintf(buf, sizeof buf, "%af,", (double)v);
                s << buf;
            }
            s << "},";
        }
        s << "};\n__device__ const float2 FT_EXPTAB[32] = {";
        for (int j = 0; j < 32; j++) {
            const double t = std::exp2(j / 32.0);
            const float hi = (float)t, lo = (float)(t - (double)hi);
            s << "{";
            for (float v : {hi, lo}) {
                std::snprintf(buf, sizeof buf, "%af,", (double)v);
                s << buf;
            }
            s << "},";
        }
        s << "};\n__device__ const float2 FT_ATANTAB[128] = {";
        for (int i = 0; i < 128; i++) {
            const double t = std::atan(i / 64.0);
            const float hi = (float)t, lo = (float)(t - (double)hi);
            s << "{";
            for (float v : {hi, lo}) {
                std::snprintf(buf, sizeof buf, "%af,", (double)v);
                s << buf;
            }
            s << "},";
        }
        s << "};\n__device__ const float4 FT_SCTAB[128] = {";
        const double pi = 3.14159265358979323846;
        for (int j = 0; j < 128; j++) {
            const double sn = std::sin(j * pi / 64.0), cs = std::cos(j * pi / 64.0);
            const float sh = (float)sn, sl = (float)(sn - (double)sh), ch = (float)cs, cl = (float)(cs - (double)ch);
            s << "{";
            for (float v : {sh, sl, ch, cl}) {
                std::snprintf(buf, sizeof buf, "%af,", (double)v);
                s << buf;
            }
            s << "},";
        }
        s << "};\n";
        return s.str();
    }();
    return text;
}

// Tables and constants of the FP64 form's functions, in fixed point (Qn: units of 2^-n; from the
// host's long double, to a unit or so) and as exact hexadecimal literals:
//   FT_LOG64[i] = r, -log2(r / 1024) in Q62, r = ceil(1024 / (1 + i/256)) (i < 256)
//   FT_EXP64[j] = 2^(j/256) in Q63 (j < 256)
//   FT_SC64[k] = sin(k pi/128), cos(k pi/128) in Q63 (k < 64)
//   FT_ATAN64[2i], [2i+1] = {i/128, hi}, {lo, 0}, atan(i/128) = hi + lo (i <= 128)
//   log2 e in Q63, ln 2 in Q64, 128/pi in Q58 and the next 64 bits, pi/128 in Q69
static std::string tables64_source()
{
    static const std::string text = [] {
        std::ostringstream s;
        char buf[64];
        auto fixed = [&](long double v, int q) {
            std::snprintf(buf, sizeof buf, "0x%llxull,", (unsigned long long)(std::ldexp(v, q) + 0.5L));
            s << buf;
        };
        const long double pi = std::acos(-1.0L);
        s << "__device__ const ulonglong2 FT_LOG64[256] = {";
        for (int i = 0; i < 256; i++) {
            const int r = (1024 * 256 + 255 + i) / (256 + i);
            s << "{" << r << "ull,";
            fixed(-std::log2(r / 1024.0L), 62);
            s << "},";
        }
        s << "};\n__device__ const unsigned long long FT_EXP64[256] = {";
        for (int j = 0; j < 256; j++) fixed(std::exp2(j / 256.0L), 63);
        s << "};\n__device__ const ulonglong2 FT_SC64[64] = {";
        for (int k = 0; k < 64; k++) {
            s << "{";
            fixed(std::sin(k * pi / 128.0L), 63);
            fixed(std::cos(k * pi / 128.0L), 63);
            s << "},";
        }
        s << "};\n__device__ const double2 FT_ATAN64[258] = {";
        for (int i = 0; i <= 128; i++) {
            const long double t = std::atan(i / 128.0L);
            std::snprintf(buf, sizeof buf, "{%a,%a},", i / 128.0, (double)t);
            s << buf;
            std::snprintf(buf, sizeof buf, "{%a,0.0},", (double)(t - (double)t));
            s << buf;
        }
        s << "};\n#define FT_LOG2E_Q63 0xb8aa3b295c17f0bcull\n#define FT_LN2_Q64 0xb17217f7d1cf79acull\n"
             "#define FT_STEPS_Q58 0xa2f9836e4e441529ull\n#define FT_STEPS_LO 0xfc2757d1f534ddc0ull\n"
             "#define FT_STEP_Q69 0xc90fdaa22168c235ull\n";
        return s.str();
    }();
    return text;
}

// Structural pattern of the conductance-form elimination of the reduced Laplacian (the
// deleted vertex is V-1): nz[i*n+j] (i < j) marks a conductance between i and j that is
// non-zero when vertex i is eliminated (an edge, or fill from an earlier elimination),
// nzg[i] a conductance to ground, nzm[i*n+j] an entry of M^-1 (M the unit upper
// triangular factor) that can be non-zero.  The kernels skip every update on a
// structural zero (a compiler cannot drop x + 0 * y in IEEE arithmetic).
static void elimination_pattern(const kernel_key& k, std::vector<int>& nz, std::vector<int>& nzg,
                                std::vector<int>& nzm)
{
    const int n = k.V - 1;
    nz.assign((size_t)n * n, 0);
    nzg.assign(n, 0);
    nzm.assign((size_t)n * n, 0);
    for (int e = 0; e < k.E; e++) {
        const int a = k.ek[e], b = k.el[e];   // a > b
        if (a == k.V - 1)
            nzg[b] = 1;
        else
            nz[b * n + a] = 1;
    }
    for (int kk = 0; kk < n; kk++)
        for (int i = kk + 1; i < n; i++) {
            if (!nz[kk * n + i]) continue;
            if (nzg[kk]) nzg[i] = 1;
            for (int j = i + 1; j < n; j++)
                if (nz[kk * n + j]) nz[i * n + j] = 1;
        }
    for (int i = n - 1; i >= 0; i--)
        for (int j = i + 1; j < n; j++) {
            int v = nz[i * n + j];
            for (int m = i + 1; m < j && !v; m++) v = nz[i * n + m] && nzm[m * n + j];
            nzm[i * n + j] = v;
        }
}

std::string kernel_source(const kernel_key& k)
{
    std::ostringstream s;
    s << "// generated: one topology of the tropical sampling kernel\n";
    s << "#define FT_E " << k.E << "\n#define FT_V " << k.V << "\n#define FT_K " << k.K << "\n";
    s << "#define FT_LOOPS " << k.loops << "\n#define FT_RANK " << k.rank << "\n";
    s << "#define FT_PREC " << k.prec << "\n#define FT_MODE " << k.mode << "\n";
    s << "#define FT_ONLY_PSI " << k.only_psi << "\n#define FT_RECORD " << k.record << "\n";
    s << "#define FT_BLOCK " << k.block << "\n#define FT_TABLE_GLOBAL " << k.table_global << "\n";
    s << "#define FT_MINB " << k.minb << "\n#define FT_VARIANT " << k.variant << "\n";
    s << "#define FT_BATCH " << k.batch << "\n#define FT_XA_DIGITS " << kExactDigits << "\n";
    s << "#define FT_PART " << k.part << "\n";
    s << "#define FT_SCRATCH " << k.scratch << "\n";
    s << "#define FT_Q0 " << k.q0 << "\n";
    s << "__device__ constexpr int FT_EK[" << k.E << "] = {";
    for (int e = 0; e < k.E; e++) s << (e ? "," : "") << k.ek[e];
    s << "};\n__device__ constexpr int FT_EL[" << k.E << "] = {";
    for (int e = 0; e < k.E; e++) s << (e ? "," : "") << k.el[e];
    s << "};\n";
    {
        std::vector<int> nz, nzg, nzm;
        elimination_pattern(k, nz, nzg, nzm);
        const int n = k.V - 1;
        auto matrix = [&](const char* name, const std::vector<int>& m) {
            s << "__device__ constexpr signed char " << name << "[" << n << "][" << n << "] = {";
            for (int i = 0; i < n; i++) {
                s << "{";
                for (int j = 0; j < n; j++) s << (j ? "," : "") << m[i * n + j];
                s << "},";
            }
            s << "};\n";
        };
        // contributions to each conductance (edges, then fill by eliminated vertices)
        std::vector<int> cf((size_t)n * n, n), cs((size_t)n * n, 0), gf(n, n), gs(n, 0);
        for (int e = 0; e < k.E; e++) {
            const int a = k.ek[e], b = k.el[e];
            (a == k.V - 1 ? gf[b] : cf[b * n + a]) = -1;
            (a == k.V - 1 ? gs[b] : cs[b * n + a])++;
        }
        for (int m = 0; m < n; m++)
            for (int i = m + 1; i < n; i++) {
                if (!nz[m * n + i]) continue;
                if (nzg[m]) {
                    gf[i] = std::min(gf[i], m);
                    gs[i]++;
                }
                for (int j = i + 1; j < n; j++)
                    if (nz[m * n + j]) {
                        cf[i * n + j] = std::min(cf[i * n + j], m);
                        cs[i * n + j]++;
                    }
            }
        for (int& x : cs) x = x > 1;
        for (int& x : gs) x = x > 1;
        auto row = [&](const char* name, const std::vector<int>& m) {
            s << "__device__ constexpr signed char " << name << "[" << n << "] = {";
            for (int i = 0; i < n; i++) s << (i ? "," : "") << m[i];
            s << "};\n";
        };
        matrix("FT_CF", cf);
        matrix("FT_CS", cs);
        row("FT_GF", gf);
        row("FT_GS", gs);
        matrix("FT_NZC", nz);
        matrix("FT_NZM", nzm);
        row("FT_NZG", nzg);
    }
    s << (k.prec == 0 ? tables64_source() : tables_source());
    s << ft_sample_body_source;
    return s.str();
}

static uint64_t fnv1a(const std::string& s)
{
    uint64_t h = 1469598103934665603ULL;
    for (unsigned char c : s) {
        h ^= c;
        h *= 1099511628211ULL;
    }
    return h;
}

std::string cache_dir()
{
    if (const char* env = std::getenv("FEYNTROP_GB300_CACHE")) return env;
    Dl_info info;
    if (dladdr((void*)&cache_dir, &info) && info.dli_fname) {
        std::string p = info.dli_fname;
        size_t slash = p.rfind('/');
        if (slash != std::string::npos) return p.substr(0, slash) + "/../_jit_cache";
    }
    return "_jit_cache";
}

static std::vector<std::string> options()
{
    return {kArch, "--std=c++17", "-lineinfo", "--extra-device-vectorization"};
}

static std::string compile(const std::string& src, std::string* log_out)
{
    nvrtcProgram prog;
    if (nvrtcCreateProgram(&prog, src.c_str(), "ft_sample.cu", 0, nullptr, nullptr) != NVRTC_SUCCESS)
        throw std::runtime_error("nvrtcCreateProgram failed");
    std::vector<std::string> opts = options();
    std::vector<const char*> o;
    for (auto& x : opts) o.push_back(x.c_str());
    if (std::getenv("FEYNTROP_GB300_PTXAS_VERBOSE")) o.push_back("--ptxas-options=-v");
    nvrtcResult rc = nvrtcCompileProgram(prog, (int)o.size(), o.data());
    size_t logn = 0;
    nvrtcGetProgramLogSize(prog, &logn);
    std::string log(logn, '\0');
    if (logn) nvrtcGetProgramLog(prog, &log[0]);
    if (log_out) *log_out = log;
    if (rc != NVRTC_SUCCESS) {
        nvrtcDestroyProgram(&prog);
        throw std::runtime_error("kernel compilation failed:\n" + log);
    }
    if (std::getenv("FEYNTROP_GB300_PTXAS_VERBOSE")) std::fprintf(stderr, "%s\n", log.c_str());
    size_t n = 0;
    nvrtcGetCUBINSize(prog, &n);
    std::string cubin(n, '\0');
    nvrtcGetCUBIN(prog, &cubin[0]);
    nvrtcDestroyProgram(&prog);
    return cubin;
}

static std::string cubin_for(const kernel_key& key, double* seconds)
{
    const std::string src = kernel_source(key);
    std::string tag = src;
    for (auto& o : options()) tag += o;
    int major = 0, minor = 0;
    nvrtcVersion(&major, &minor);
    tag += std::to_string(major) + "." + std::to_string(minor);
    char name[64];
    std::snprintf(name, sizeof name, "%016llx.cubin", (unsigned long long)fnv1a(tag));
    const std::string dir = cache_dir();
    const std::string path = dir + "/" + name;
    {
        std::ifstream f(path, std::ios::binary);
        if (f) {
            std::stringstream b;
            b << f.rdbuf();
            std::string s = b.str();
            if (!s.empty()) {
                *seconds = 0;
                return s;
            }
        }
    }
    auto t0 = std::chrono::steady_clock::now();
    std::string cubin = compile(src, nullptr);
    *seconds = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    mkdir(dir.c_str(), 0755);
    const std::string tmp = path + ".tmp" + std::to_string((unsigned long long)fnv1a(std::to_string((long)&tag)));
    {
        std::ofstream f(tmp, std::ios::binary);
        f.write(cubin.data(), (std::streamsize)cubin.size());
    }
    std::rename(tmp.c_str(), path.c_str());
    return cubin;
}

size_t compile_only(const kernel_key& key, std::string* log) { return compile(kernel_source(key), log).size(); }

void precompile(const kernel_key& key)
{
    double s = 0;
    cubin_for(key, &s);
}

void precompile_all(const std::vector<kernel_key>& keys)
{
    if (keys.size() < 2) {
        for (const kernel_key& k : keys) precompile(k);
        return;
    }
    // at most 8 at a time: a compile of the larger kernels takes about a gigabyte
    const unsigned hw = std::max(1u, std::min(8u, std::thread::hardware_concurrency()));
    const size_t nthreads = std::min<size_t>(keys.size(), hw);
    std::atomic<size_t> next{0};
    std::vector<std::exception_ptr> errs(nthreads);
    std::vector<std::thread> pool;
    for (size_t t = 0; t < nthreads; t++)
        pool.emplace_back([&, t] {
            try {
                for (size_t i; (i = next++) < keys.size();) precompile(keys[i]);
            } catch (...) {
                errs[t] = std::current_exception();
            }
        });
    for (auto& th : pool) th.join();
    for (auto& e : errs)
        if (e) std::rethrow_exception(e);
}

// Driver entry points are fetched through the runtime (no link-time dependency on
// the driver library, so the library also loads on machines without a GPU).
driver_api& drv()
{
    static driver_api d;
    static std::once_flag once;
    std::call_once(once, [] {
        auto get = [](const char* name, void** fn) {
            cudaDriverEntryPointQueryResult q;
            if (cudaGetDriverEntryPointByVersion(name, fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
                q != cudaDriverEntryPointSuccess || !*fn)
                throw std::runtime_error(std::string("driver entry point unavailable: ") + name);
        };
        get("cuModuleLoadData", (void**)&d.ModuleLoadData);
        get("cuModuleGetFunction", (void**)&d.ModuleGetFunction);
        get("cuFuncSetAttribute", (void**)&d.FuncSetAttribute);
        get("cuFuncGetAttribute", (void**)&d.FuncGetAttribute);
        get("cuOccupancyMaxActiveBlocksPerMultiprocessor", (void**)&d.OccupancyMaxActiveBlocksPerMultiprocessor);
        get("cuLaunchKernel", (void**)&d.LaunchKernel);
        get("cuGetErrorString", (void**)&d.GetErrorString);
    });
    return d;
}

void check(CUresult r, const char* what)
{
    if (r != CUDA_SUCCESS) {
        const char* msg = nullptr;
        drv().GetErrorString(r, &msg);
        throw std::runtime_error(std::string(what) + ": " + (msg ? msg : "unknown driver error"));
    }
}

static std::string key_string(const kernel_key& k)
{
    std::ostringstream s;
    s << k.E << "," << k.V << "," << k.K << "," << k.loops << "," << k.rank << "," << k.prec << "," << k.mode << ","
      << k.only_psi << "," << k.record << "," << k.block << "," << k.table_global << "," << k.minb << "," << k.variant
      << "," << k.batch << "," << k.q0 << "," << k.scratch << "," << k.part;
    for (int e = 0; e < k.E; e++) s << ";" << k.ek[e] << "-" << k.el[e];
    return s.str();
}

static std::mutex g_mu;
static std::map<std::pair<int, std::string>, kernel_set> g_loaded;

const kernel_set* find_kernels(const kernel_key& key)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    std::lock_guard<std::mutex> lock(g_mu);
    auto it = g_loaded.find(std::make_pair(dev, key_string(key)));
    return it == g_loaded.end() ? nullptr : &it->second;
}

const kernel_set& get_kernels(const kernel_key& key)
{
    auto& mu = g_mu;
    auto& loaded = g_loaded;
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) throw std::runtime_error("no CUDA device");
    auto k = std::make_pair(dev, key_string(key));
    {
        std::lock_guard<std::mutex> lock(mu);
        auto it = loaded.find(k);
        if (it != loaded.end()) return it->second;
    }
    // compile (or read the disk cache) outside the lock, so that threads loading
    // different kernels compile them concurrently
    kernel_set ks;
    ks.block = key.block;
    ks.variant = key.variant;
    const std::string cubin = cubin_for(key, &ks.compile_seconds);
    std::lock_guard<std::mutex> lock(mu);
    auto it = loaded.find(k);
    if (it != loaded.end()) return it->second;   // another thread loaded it meanwhile
    cudaFree(0);   // make the runtime's primary context current for the driver calls
    check(drv().ModuleLoadData(&ks.module, cubin.data()), "cuModuleLoadData");
    const char* sname = key.batch ? "ft_sample_batch" : "ft_sample";
    const char* qname = key.batch ? "ft_sample_queue_batch" : "ft_sample_queue";
    CUfunction& f = key.part ? ks.queue : ks.sample;
    check(drv().ModuleGetFunction(&f, ks.module, key.part ? qname : sname), "cuModuleGetFunction");
    ks.smem = table_smem_bytes(key);
    check(drv().FuncSetAttribute(f, CU_FUNC_ATTRIBUTE_MAX_DYNAMIC_SHARED_SIZE_BYTES, (int)ks.smem),
          "cuFuncSetAttribute(smem)");
    check(drv().FuncGetAttribute(&ks.regs, CU_FUNC_ATTRIBUTE_NUM_REGS, f), "cuFuncGetAttribute");
    check(drv().FuncGetAttribute(&ks.local_bytes, CU_FUNC_ATTRIBUTE_LOCAL_SIZE_BYTES, f), "cuFuncGetAttribute");
    check(drv().OccupancyMaxActiveBlocksPerMultiprocessor(key.part ? &ks.queue_blocks_per_sm : &ks.blocks_per_sm, f,
                                                          ks.block, ks.smem),
          "cuOccupancyMaxActiveBlocksPerMultiprocessor");
    if (!key.part && ks.blocks_per_sm < 1) throw std::runtime_error("sampling kernel does not fit on an SM");
    return loaded.emplace(k, ks).first->second;
}

}  // namespace ft
