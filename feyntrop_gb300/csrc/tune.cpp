#include "tune.hpp"

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <map>
#include <mutex>
#include <sstream>

#include "json.hpp"

namespace ft {

namespace {

std::mutex g_mu;
std::map<std::string, launch_shape> g_table;
bool g_loaded = false;

const unsigned kSmemLimit = 227 * 1024;

std::string table_path() { return cache_dir() + "/tuning.json"; }

void load_locked()
{
    if (g_loaded) return;
    g_loaded = true;
    std::ifstream f(table_path());
    if (!f) return;
    std::stringstream b;
    b << f.rdbuf();
    try {
        const ftj::value v = ftj::parse(b.str());
        if (!v.is_object()) return;
        for (const auto& kv : v.obj) {
            const ftj::value& e = kv.second;
            if (!e.is_object()) continue;
            launch_shape s;
            s.block = (int)e["block"].num;
            s.minb = (int)e["minb"].num;
            s.variant = (int)e["variant"].num;
            s.chunk = (unsigned long long)e["chunk"].num;
            s.rate = e["rate"].num;
            if (s.block >= 32 && s.block <= 1024 && s.minb >= 1 && s.minb <= 32) g_table[kv.first] = s;
        }
    } catch (...) {
        // an unreadable table is ignored (defaults apply)
    }
}

void save_locked()
{
    std::ostringstream o;
    o << "{\n";
    bool first = true;
    for (const auto& kv : g_table) {
        const launch_shape& s = kv.second;
        o << (first ? "" : ",\n") << "  \"" << kv.first << "\": {\"block\": " << s.block << ", \"minb\": " << s.minb
          << ", \"variant\": " << s.variant << ", \"chunk\": " << s.chunk << ", \"rate\": " << s.rate << "}";
        first = false;
    }
    o << "\n}\n";
    const std::string path = table_path();
    const std::string tmp = path + ".tmp";
    {
        std::ofstream f(tmp);
        f << o.str();
    }
    std::rename(tmp.c_str(), path.c_str());
}

}  // namespace

std::string tune_class(const kernel_key& k)
{
    std::ostringstream s;
    s << "E" << k.E << "V" << k.V << "K" << k.K << "m" << k.mode << "p" << k.prec << "t" << k.table_global << "o"
      << k.only_psi << ":";
    for (size_t e = 0; e < k.ek.size(); e++) s << (e ? "," : "") << k.ek[e] << "-" << k.el[e];
    return s.str();
}

launch_shape default_shape(const kernel_key& k)
{
    // GB300 sweeps.  The per-sample barrier (variant bit 2) makes the warps of a block share
    // their instruction fetches.
    // Mixed, undeformed (two samples per thread): 16 warps of 128 registers in one block (1e9
    // samples/s against 256 threads with up to 255 registers: K4 24.4 / 19.8, wheel 19.2 /
    // 16.0, undeformed box-pentagon 18.0 / 15.1, 3-loop ladder 14.2 / 12.1, triangle 43.8 / 44.8;
    // two blocks of 256 3 to 6 % below the one).  The cube's table leaves one block of 256 threads
    // whatever is asked for (apply_shape): 10.05 held to 128 registers, 9.66 with up to 255.
    // Mixed, deformed: 16 warps of 128 registers per SM.  Single integrals: one block, which
    // keeps all of them together, with one out-of-line copy of the complex two-float product
    // (bit 4; also of the FP32 transcendentals and the larger two-float routines, bits 0 and 3:
    // double box 16.4 ms against 15.9, ladder 7.96 against 7.07; without any 18.3 and 8.6).
    // Batches, where a block also waits for its slowest warp at every item's end: two blocks,
    // with all three (24 box-pentagon points 12.2 ms, one block 12.5; bit 4 alone 12.35).
    // FP64 form, bound by the FP64 pipe: 12 to 16 warps per SM keep it busy.  Deformed, ms with
    // 256, 384 and 512 threads: double box, 3e6 samples, 7.4, 7.1; 12 box-pentagon points of 1e4
    // to 3e5 3.70, 3.41, 3.47; 4-loop ladder (E = 13), 6e6, 51.4, 47.4, 47.4; 5-loop (E = 16),
    // 3e6, 39.9, 39.1, 37.6 (the spills that fewer registers add cost less than the warps give).
    // Undeformed with 256 x 2, 256, 384 and 512: 24 K4 points of 1e5 to 3e6 5.87, 7.96, 7.30,
    // 7.13; 24 triangles 3.53, 5.08, 4.70, 4.54; where the table leaves no room for two blocks
    // (above E = 10), 12 cubes of 1e5 to 1e6 3.35, 3.34, 2.96, 2.85; 4-loop ladder, 1e7, 13.28,
    // 11.45, 10.54 (256, 384, 512).
    launch_shape s;
    if (k.prec == 1) {
        s.block = k.batch && k.mode == 1 ? 256 : 512;
        s.minb = k.batch && k.mode == 1 ? 2 : 1;
    } else if (k.mode == 1) {
        s.block = 384;
        s.minb = 1;
    } else {
        s.block = k.E > 10 ? 512 : 256;
        s.minb = k.E > 10 ? 1 : 2;
    }
    s.variant = k.prec == 1 && k.mode == 1 ? (k.batch ? 29 : 20) : 4;
    return s;
}

unsigned long long default_chunk(const kernel_key& k)
{
    if (k.prec == 1) return k.mode == 1 ? 32 : 128;
    return k.mode == 1 ? 8 : 16;
}

// Shared memory of one block: the dynamic part (staged table, sums) plus the kernel
// body's static variables, in the batch kernels with the staged parameter block (its
// doubles, floats and two-float quadruples) and the work item.
static unsigned block_smem_bytes(const kernel_key& k)
{
    unsigned prm = 0;
    if (k.batch) {
        const unsigned n = (unsigned)(k.V - 1), ne = n - (unsigned)k.q0, r = (unsigned)k.rank;
        const unsigned p = 8u + 2u * (unsigned)k.E + r + r * n + ne * (ne + 1u) / 2u;
        prm = (p + (p + 1u) / 2u + 1u + 2u * p) * 8u + 64u;
    }
    return table_smem_bytes(k) + 64u + prm;
}

void apply_shape(kernel_key& k, const launch_shape& s)
{
    k.block = std::max(32, s.block & ~31);   // whole warps: their collective operations name all lanes
    k.minb = s.minb;
    k.variant = s.variant;
    // as much of the deformed integrand's scratch in shared memory as fits beside minb blocks.
    // Not raised again for a block that is halved below: what its table and sums leave serves the
    // spilled frames as L1 (a cube above threshold, E = 12, 1e7 samples: 13.0 ms with 3 eps orders,
    // 14.1 with the angles in shared memory; in a batch 14.2 and 16.8).
    k.scratch = k.prec == 1 && k.mode == 1 ? 2 : 0;
    while (k.scratch > 0 && block_smem_bytes(k) * (unsigned)k.minb > kSmemLimit) k.scratch--;
    // keep the warps per SM while halving the block until the shared memory fits (with a staged
    // table of E = 12 only one block does: minb then only bounds the registers)
    // (many eps orders: 12 edges and 14 orders halve the FP64 form's 384 threads three times)
    while (k.block > 32 && block_smem_bytes(k) > kSmemLimit) {
        k.block = (k.block / 2 + 31) & ~31;
        k.minb = k.minb * 2 > 32 ? 32 : k.minb * 2;
    }
}

launch_shape choose_shape(const kernel_key& k)
{
    launch_shape s = default_shape(k);
    {
        std::lock_guard<std::mutex> lock(g_mu);
        load_locked();
        auto it = g_table.find(tune_class(k));
        if (it != g_table.end()) {
            // a class whose default won its trials (one integral each) keeps the batch default too
            kernel_key single = k;
            single.batch = 0;
            const launch_shape d = default_shape(single), &t = it->second;
            if (k.batch && t.block == d.block && t.minb == d.minb && t.variant == d.variant)
                s.chunk = t.chunk;
            else
                s = t;
        }
    }
    if (const char* e = std::getenv("FEYNTROP_GB300_BLOCK")) s.block = std::atoi(e);
    if (const char* e = std::getenv("FEYNTROP_GB300_MINB")) s.minb = std::atoi(e);
    if (const char* e = std::getenv("FEYNTROP_GB300_VARIANT")) s.variant = std::atoi(e);
    return s;
}

void record_shape(const kernel_key& k, const launch_shape& s)
{
    std::lock_guard<std::mutex> lock(g_mu);
    load_locked();
    g_table[tune_class(k)] = s;
    save_locked();
}

static thread_local unsigned long long t_chunk_override = 0;
void set_chunk_override(unsigned long long chunk) { t_chunk_override = chunk; }
unsigned long long chunk_override() { return t_chunk_override; }

void clear_shapes()
{
    std::lock_guard<std::mutex> lock(g_mu);
    g_table.clear();
    g_loaded = true;
}

}  // namespace ft
