// plan.cuh -- a plan's levels and launch bookkeeping, shared by the C ABI
// (slak_abi.cu) and the closed-form levels' launches (levels.cu).
#pragma once

#include <string>
#include <type_traits>
#include <vector>

#include "slak_b200.h"
#include "fast.cuh"

namespace slak {

struct Level {
    int64_t F = 0, V = 0, N = 0, B = 0, E = 0;
    int64_t Fo = 0, Vo = 0, No = 0;
    bool quad = true;       // implicit 4-corner faces
    bool poly_fn = false;   // the reference's first-level (polygon) functions
    bool fast = false;      // closed-form refinement from the parent level's state
    bool closed0 = false;        // general level 0 of a closed mesh (closed0.cuh)
    bool cap0 = false;           // ... none of whose vertices is above valence kC0Cap
    bool export_state = false;   // general level whose state feeds a fast level
    bool make_state = false;     // fast level whose state feeds the next fast level
    // fast level whose parent's parent is a closed quad mesh (GQ, fast.cuh):
    // k_g1 sums most of the parent's vertex columns; that mesh's sizes
    bool gq = false;
    int64_t gN = 0, gV = 0, gF = 0;
    // the last GQ level: it takes its parent's state in closed form from the
    // grandparent's (SG, fast.cuh), so the level before writes none
    bool sg = false;
    // closed level with a grandparent (grand.cuh): refined from the
    // grandparent's state and the parent's quads
    bool pp = false;
    bool longcol = false;        // the input has vertices above valence 15 (long columns at every level)
    bool skip_ids = false;       // its refined quads are read by no later level
    // k_g3 with bulk-copied slot records (SLAK_PLAN_BULK_RECORDS, closed parents)
    bool bulk3 = false;
    int bulk_polls = 0;
    DevStatus* st = nullptr;
    QState in_state{}, out_state{};
    SlotScratch slots{};    // fast level: slot-ordered records from k_g1 to k_g3
    const int* ptr = nullptr;
    const int* ids = nullptr;
    const float* verts = nullptr;
    int* o_ids = nullptr;
    float* o_verts = nullptr;
    int* o_ptr = nullptr;
    int* o_vals = nullptr;
    int* scan_tmp = nullptr;       // fast level with a boundary (SLAK, state): scan of C's boundary edges
    // fast level: block size of k_g1, k_g2, k_g3 (chosen by the autotuner)
    int bs[3] = {256, 256, 256};
    int tuned = 0;                 // 0 default, 1 measured now, 2 from the tuning cache
    float tune_ms[3][3] = {};      // measured ms of each kernel at block 128 / 256 / 512
    std::string tune_key;
};

constexpr int kTuneBlocks[3] = {128, 256, 512};

// Calls f with the block size as a compile-time constant.
template <class F>
void with_block(int bs, F&& f)
{
    if (bs == 128) f(std::integral_constant<int, 128>{});
    else if (bs == 512) f(std::integral_constant<int, 512>{});
    else f(std::integral_constant<int, 256>{});
}

// Launch bookkeeping: counts launches and, in debug mode (SLAK_DEBUG_SYNC=1 in
// the environment when the plan is created), synchronises after every launch
// and records which kernel failed.
inline thread_local std::string g_detail;

struct KernelRec {
    const char* name;
    int level;
    int64_t bytes;
};

struct Lc {
    cudaStream_t s;
    int64_t* nl;
    bool debug;
    int level;
    int err = 0;
    std::vector<cudaEvent_t>* ev = nullptr;   // timing: one event after every launch (ev[0] before the first)
    std::vector<KernelRec>* recs = nullptr;
    // independent kernels of a level on side streams (fork / join by events);
    // off while timing (per-launch events need one stream) and when debugging
    bool conc = false;
    cudaStream_t side[2] = {nullptr, nullptr};
    cudaEvent_t cev[4] = {nullptr, nullptr, nullptr, nullptr};
    // side stream k waits for the work enqueued so far on s
    void fork(int k)
    {
        cudaEventRecord(cev[k], s);
        cudaStreamWaitEvent(side[k], cev[k], 0);
    }
    // s waits for side stream k
    void join(int k)
    {
        cudaEventRecord(cev[2 + k], side[k]);
        cudaStreamWaitEvent(s, cev[2 + k], 0);
    }
    void after(const char* name, int n = 1, int64_t bytes = 0)
    {
        *nl += n;
        if (ev && recs->size() + 1 < ev->size()) {
            cudaEventRecord((*ev)[recs->size() + 1], s);
            recs->push_back(KernelRec{name, level, bytes});
        }
        if (!debug || err) return;
        cudaError_t e = cudaGetLastError();
        if (e == cudaSuccess) e = cudaStreamSynchronize(s);
        if (e != cudaSuccess) {
            err = e == cudaErrorMemoryAllocation ? SLAK_ERR_OOM : SLAK_ERR_CUDA;
            g_detail = std::string(name) + " (level " + std::to_string(level) + "): " + cudaGetErrorString(e);
        }
    }
};

// the closed-form levels by parent kind (levels.cu; `cface` / `pf`: the polygon
// parent's or grandparent's corner -> face map / faces)
void launch_fast_quad(const Level& Pl, const Level& L, bool lak, bool comp, Lc& lc);
void launch_fast_quad_open(const Level& Pl, const Level& L, bool lak, bool comp, Lc& lc);
void launch_fast_gq(const Level& Pl, const Level& L, bool lak, bool comp, Lc& lc);
void launch_p1(const Level& Pl, const Level& L, Faces<false> pf, bool lak, bool comp, Lc& lc);
void launch_fast_poly_open(const Level& Pl, const Level& L, const int* cface, bool lak, bool comp, Lc& lc);
void launch_pp_quad(const Level& PPl, const Level& Pl, const Level& L, bool lak, bool comp, Lc& lc);
void launch_pp_poly(const Level& PPl, const Level& Pl, const Level& L, Faces<false> pf, bool lak, bool comp, Lc& lc);

// exclusive scan of n counts (n + 1 outputs; scan.cuh), returns its launches
int scan_launch(const int* in, int* out, int64_t n, int* tmp, cudaStream_t s);

}  // namespace slak
