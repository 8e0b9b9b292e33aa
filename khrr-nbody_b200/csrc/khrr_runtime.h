// Host-side context of libkhrr (the object behind the opaque khrr_ctx*).
#pragma once

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include <cstdint>
#include <map>
#include <string>
#include <tuple>
#include <utility>
#include <vector>

#include "khrr.h"
#include "host_words.h"
#include "khrr_internal.h"

namespace khrr {

// An NVTX range over one library call, shown by Nsight Systems as a named
// phase (header-only NVTX v3; without a tool attached it costs a few ns).
struct NvtxRange {
    explicit NvtxRange(const char* name) { nvtxRangePushA(name); }
    ~NvtxRange() { nvtxRangePop(); }
    NvtxRange(const NvtxRange&) = delete;
    NvtxRange& operator=(const NvtxRange&) = delete;
};

// Grow-only device allocation.
template <class T>
struct DevBuf {
    T* p = nullptr;
    size_t n = 0;
    DevBuf() = default;
    DevBuf(const DevBuf&) = delete;
    DevBuf& operator=(const DevBuf&) = delete;
    ~DevBuf() { release(); }
    cudaError_t ensure(size_t count) {
        if (count <= n && p) return cudaSuccess;
        release();
        cudaError_t e = cudaMalloc(reinterpret_cast<void**>(&p), (count ? count : 1) * sizeof(T));
        if (e != cudaSuccess) {
            p = nullptr;
            n = 0;
            return e;
        }
        n = count;
        return cudaSuccess;
    }
    void release() {
        if (p) cudaFree(p);
        p = nullptr;
        n = 0;
    }
};

// The force-pass work queue for one layout of systems and one kernel shape.
struct ForcePlan {
    bool valid = false;
    int threads = 0, ipt = 0, jt = 0, split_req = -1, ctas = 0;
    std::vector<WorkItem> items;
    std::vector<int> sys_item_begin;  // plain plans: items of system k
    std::vector<int> sys_split;       // j chunks per system
    int chains = 0, ntiles = 0;       // > 0: items leave one partial per j tile, summed in this many runs
    // double4 words of the partials of npad bodies
    size_t partial_words(int64_t npad) const {
        return static_cast<size_t>(chains > 0 ? (ntiles + 1) / 2 : nslots) * static_cast<size_t>(npad);
    }
    int nslots = 1;
    DevBuf<WorkItem> d_items;
    DevBuf<unsigned char> d_nsplit;
    // The symmetric pair kernel's queue (pair plans; FP64 plans with f64_pair).
    bool pair = false;
    bool f64_pair = false;  // FP64 plan: the symmetric FP64 kernel on pair_items
    std::vector<PairItem> pair_items;
    unsigned pair_share = 0;  // an SM's share of the items' weight
    // The same work in the small-layout form, where that is the faster one.
    int small_ki = 0;  // i bodies per thread (0: the pair kernel runs)
    bool small_one_mass = false;  // ... in the block-mass form too
    bool use_small(const ForceVariant* v) const { return small_ki && (small_one_mass || !v->tile_mass); }
    std::vector<SmallItem> small_items;
    DevBuf<SmallItem> d_small_items;
    DevBuf<PairItem> d_pair_items;
    ForcePlan() = default;
    ForcePlan(const ForcePlan&) = delete;
    ForcePlan& operator=(const ForcePlan&) = delete;
};

void plan_force_items(const std::vector<int64_t>& poff, const std::vector<int64_t>& cnt, int itile,
                      int jt, int ctas, int sms, int forced_split, bool plain, ForcePlan& out);
// The symmetric pair kernel's blocks: per system the padded indices
// P_k = b_0 < b_1 < ... < b_nb = P_{k+1}, each block at most kPairBlock
// bodies starting at a multiple of kPad.
using PairBlocks = std::vector<std::vector<int64_t>>;
// 1024-body blocks over each system's padded range (the last may be shorter).
PairBlocks pair_blocks_fixed(const std::vector<int64_t>& poff);
// Runs of 128-body tiles of one mass (tile_mass[tile]), cut at 1024 bodies.
PairBlocks pair_blocks_by_mass(const std::vector<int64_t>& poff, const std::vector<float>& tile_mass);
// The pair kernel's items: block rows cut into chunks of `chunk` blocks (0 =
// chosen from the CTA count), costliest first.
void plan_pair_items(const PairBlocks& blocks, const std::vector<int64_t>& cnt, int ctas, int chunk,
                     ForcePlan& out);
// The pair plan's work in the small-layout form, or small_ki = 0 (the pair
// kernel is faster, or its items are not single block pairs).
void plan_small_items(const PairBlocks& blocks, const std::vector<int64_t>& cnt, int sms, ForcePlan& out);
// Time weights of a pair plan's items, heaviest first, and the share of one of
// `sms` SMs.
void weigh_pair_items(int sms, ForcePlan& out);
// The same pairs cut at 128-body tiles (1024-body i blocks): chunks taper from
// a quarter of a CTA's share of the work down to one tile, so layouts of any
// size fill the persistent grid and its last round.
void plan_pair_tiles(const std::vector<int64_t>& poff, const std::vector<int64_t>& cnt, int ctas, ForcePlan& out);

// Force paths of the state API: the batched FP32 kernels (pair or one-sided,
// per the tuning), the plain one-launch-per-system FP32 baseline (KHRR_PLAIN)
// and the FP64 direct sum (KHRR_FP64).
enum ForceMode { kModeBatched = 0, kModePlain = 1, kModeF64 = 2 };

struct StepGraph {
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t exec = nullptr;
    cudaGraphNode_t ev0 = nullptr, ev1 = nullptr;  // event-record nodes around the force pass
    uint64_t used = 0;  // when it was last asked for (step graphs)
};

// The mesh-force solver (khrr_set_mesh_solver): its mesh, field ring and
// per-body gather slot, and the step graphs per (dt, ring state, phi).
struct MeshSolver {
    bool on = false;
    khrr_mesh_solver cfg{};
    MeshGeom geom{};
    int64_t cells = 0;
    DevBuf<double> cell_mass, phi64, cell_acc;  // C, 4 C (field ring), 3 C
    DevBuf<double> copies;                      // cic_copy_count meshes: zero between deposits
    int ncopies = 0;
    size_t copies_refused = ~size_t(0);         // words that the device had no room for (asked once)
    DevBuf<float> mass32, phi32, tab;           // C, 4 C (field ring), 3 nx
    DevBuf<int2> pci;                           // npad
    DevBuf<double4> part;                       // npad: {acc, -phi} per body
    WaveMaps maps;                              // tensor maps of phi32 / mass32
    DevBuf<unsigned> sync;                      // nx + 1 plane counters of the resident stencil
    DevBuf<unsigned char> ns;                   // npad: 1 for real bodies, 0 for ghosts
    std::vector<int64_t> layout_poff, layout_cnt;  // the layout pci/part/ns were sized for
    int rot = kRingStart;                       // ring state: 4 * (phi^{n-1} buffer) + phi^n buffer
    std::map<std::tuple<uint64_t, int, bool>, StepGraph> graphs;
    void drop_graphs() {
        for (auto& kv : graphs) {
            if (kv.second.exec) cudaGraphExecDestroy(kv.second.exec);
            if (kv.second.graph) cudaGraphDestroy(kv.second.graph);
        }
        graphs.clear();
    }
};

}  // namespace khrr

struct khrr_ctx {
    int device = 0;
    int sm_count = 0;
    cudaStream_t own = nullptr, stream = nullptr;
    std::string err;

    // State layout.
    bool has_state = false;
    int64_t n = 0, npad = 0;
    std::vector<int64_t> off, poff, cnt;  // real offsets, padded offsets, counts per system
    khrr::DevBuf<double> pos, vel, acc, post, velt, acct, mass, eps2, phi;
    khrr::DevBuf<float> shadow_buf;  // SoA FP32 shadow, 5 x npad
    khrr::DevBuf<double4> part;
    khrr::DevBuf<unsigned long long> fx;  // the pair kernel's fixed-point sums, kFxComps x npad
    // What an upload finds out per 128-body tile, in one buffer and one copy (3 us
    // each): the scales of the fixed-point sums, {mass, eps2 / 2} of a tile of 128 real
    // bodies that share both (else {0, -1}), and the first mass in FP32.
    khrr::DevBuf<double> tile_info;
    khrr::FxScale* fx_scale = nullptr;
    double2* tile_class64 = nullptr;
    float* tile_mass = nullptr;
    khrr::DevBuf<double> f64_sums;  // the symmetric FP64 pass's sums, 2 x 4 x npad
    khrr::DevBuf<unsigned> queue, errflag;
    // Page-locked words that small results come back through: 16 doubles of
    // khrr_conservation (the last one the error flag's value), then the error
    // flag of khrr_synchronize.  Read by the host after a synchronisation.
    khrr::HostWords words;
    double* host_words = nullptr;  // words.p
    khrr_status report_flag(unsigned flag);
    khrr::DevBuf<double> cons_blocks, scratch;
    khrr::DevBuf<unsigned> cons_done;  // khrr_conservation's count of finished blocks (zero between calls)
    bool uniform = false;
    float h_uniform = 0.0f;
    bool tile_uniform_mass = false;     // every 128-body tile of the layout has one mass
    bool block_uniform_mass = false;    // every pair block has one mass (the pair kernel's block-mass form)
    khrr::PairBlocks pair_blocks;       // the pair kernel's blocks of the layout
    khrr::FieldConsts field{};
    khrr_tuning tuning{128, 4, 128, 0, 1};
    khrr::ForcePlan plan_batched, plan_plain, plan_fp64;
    bool predicted = false;
    double pred_dt = 0.0;
    // (dt, steps, mode, phi, compat, timed) -> graph: the kMaxGraphs asked for last.  A
    // program that changes dt with every call would keep 0.16 MB of device and of
    // host memory for each of them; one of a constant dt has two to four.
    static constexpr size_t kMaxGraphs = 32;
    std::map<std::tuple<uint64_t, int, int, bool, bool, bool>, khrr::StepGraph> graphs;
    uint64_t graph_clock = 0;
    // Every force pass starts from a zero queue counter and, where its kernel
    // accumulates, zero sums; the kernel that reads the sums zeroes both again.
    // clean: the kind of pass they are zero for (0: unknown).
    enum { kCleanQueue = 1, kCleanFx = 2, kCleanF64 = 3 };
    int clean = 0;
    khrr_status ensure_clean(int mode);

    // Kernel-level entry points: their own shadow, partials, plan and queue
    // words (a graph of the caller's may replay such a pass between the state's
    // passes, whose own words `clean` describes).
    khrr::DevBuf<unsigned> kqueue;
    khrr::DevBuf<float> kshadow, kishadow;
    khrr::DevBuf<double4> kpart;
    khrr::DevBuf<unsigned long long> kfx;  // the pair kernel's sums (pos_i == pos_j under the pair tuning)
    khrr::DevBuf<khrr::FxScale> kscale;    // their tile scales
    khrr::DevBuf<double> ktile_hmin, ktile_msum;  // classification scratch per tile
    khrr::DevBuf<float> ktile_mass;   // per-tile masses (block-mass form)
    khrr::DevBuf<unsigned> kflags;    // classification of the caller's arrays
    float kh_uniform = 0.0f;          // 0.5 eps2[0] when the softenings are all equal
    khrr::ForcePlan kplan;
    int64_t kplan_n = -1;

    // Mesh pipeline (khrr_bin / khrr_wave_solve).
    bool has_bin = false;
    khrr::MeshGeom mesh{};
    int64_t ncells = 0;
    khrr::DevBuf<int2> pci;                              // per padded body: {cell, slot}
    khrr::DevBuf<int> mcount, mstart, maxpbc, mscan, mtmp;  // mscan: scan block/tile totals
    khrr::DevBuf<int> morder;                            // khrr_sort_by_cell: n body indices
    khrr::DevBuf<double> cell_mass, cell_phi, wave_resid;
    khrr::DevBuf<double> cic_copies;                     // khrr_cic_deposit's extra meshes, zero between calls
    khrr::DevBuf<unsigned> cic_crowd;                    // launch_cic_deposit's two words (the mesh solver's too)
    bool cic_deposited = false;                          // a deposit was made without them
    size_t cic_refused = ~size_t(0);                     // words that the device had no room for (asked once)
    int64_t cell_phi_cells = 0;                          // mesh size the cell_phi sums belong to
    khrr::DevBuf<float> wave_phi, wave_mass, wave_tab;   // 4 C (field ring), C, 3 nx
    int wave_nx = 0;
    int wave_rot = khrr::kRingStart;                     // ring state: 4 * (phi^{n-1} buffer) + phi^n buffer
    khrr::WaveMaps wave_maps;                            // tensor maps of wave_phi / wave_mass
    khrr::DevBuf<unsigned> wave_sync;                    // nx + 1 plane counters of the resident stencil
    bool wave_warm = false;
    std::map<std::pair<int, int>, khrr::StepGraph> wave_graphs;  // (chunk, rotation)

    // Mesh-force solver (KHRR_MESH).
    khrr::MeshSolver msolver;

    // Timing.
    bool timing = false;
    cudaEvent_t ph0 = nullptr, ph1 = nullptr;  // placeholders captured in graphs
    std::vector<std::pair<cudaEvent_t, cudaEvent_t>> ev_pool;
    size_t ev_used = 0;
    int64_t timed_launches = 0;
    double timed_pairs = 0.0;
    // Device time of the last synchronising mesh call (khrr_call_timing):
    // events before its first and after its last kernel.
    cudaEvent_t call0 = nullptr, call1 = nullptr;
    bool call_timed = false;
    std::map<const void*, int> occupancy;

    khrr_status fail(khrr_status s, const char* fmt, ...);
    khrr_status cuda(cudaError_t e, const char* what);
    khrr_status check_device_flag();
    int resident_ctas(const khrr::ForceVariant* v);
    const khrr::ForceVariant* variant(bool unif, bool acc, bool phi) const;
    bool pair_mode() const;  // the tuning asks for the pair kernel (any layout of the state admits it)
    khrr::ForcePlan& plan_for(int mode) {
        return mode == khrr::kModePlain ? plan_plain : (mode == khrr::kModeF64 ? plan_fp64 : plan_batched);
    }
    khrr_status ensure_plan(int mode);
    void drop_graphs();
    khrr::ForceArgs force_args(const khrr::ForcePlan& p, int item_begin, int item_end);
    // x: the FP64 positions the forces are wanted at (read by the FP64 kernel;
    // the FP32 kernels read the shadow packed from them).
    khrr_status enqueue_force(int mode, bool acc, bool phi, bool events, const double* x);
    khrr::StepArgs step_args(const khrr::ForcePlan& p, double dt);
    khrr::Shadow shadow() { return khrr::shadow_at(shadow_buf.p, npad); }
    khrr_status enqueue_step(double dt, int mode, bool phi_now, bool compat, bool events);
    khrr_status get_step_graph(double dt, int nsteps, int mode, bool phi_last, bool compat, khrr::StepGraph** out);
    khrr_status timing_pair(cudaEvent_t* e0, cudaEvent_t* e1);
    khrr_status call_start();  // with timing on: event before the call's first kernel
    khrr_status call_stop();   // with timing on: event after its last kernel
    double pairs_per_pass() const;
    khrr_status force_mode(int flags, int* mode);  // KHRR_PLAIN / KHRR_FP64 -> ForceMode
    // Mesh-force solver (mesh_api.cpp).
    khrr_status mesh_ensure_layout();
    khrr_status mesh_enqueue_force(const double* x, int iters, int rot0);
    khrr_status mesh_forces(int flags);
    khrr_status mesh_step(double dt, int nsteps, int flags);
};
