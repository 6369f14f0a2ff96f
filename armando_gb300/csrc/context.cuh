// context.cuh -- the context of one particle system (or batch) and what its state
// implies for the launches, shared by the translation units of the library.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <map>
#include <string>
#include <tuple>
#include <vector>

#include "../../include/armando.h"
#include "kernels.cuh"
#include "adjoint.cuh"
#include "ghosts.cuh"
#include "gpuc.cuh"

using namespace ag;

struct GraphKey {
    float kdt, hdt, dt;
    int heat_on;
    const void* state;  // which of the context's state buffers is current (they swap roles)
    int fused;          // the fused predictor
    int lst;            // neighbour lists in use
    int first;          // a lazily sorting call's first step, which always sorts
    bool operator<(const GraphKey& o) const {
        return std::tie(kdt, hdt, dt, heat_on, state, fused, lst, first) <
               std::tie(o.kdt, o.hdt, o.dt, o.heat_on, o.state, o.fused, o.lst, o.first);
    }
};

struct StepGraph {
    cudaGraphExec_t exec = nullptr;
    int launches = 0;  // kernels outside a conditional body
};

inline int blocks_for(int64_t n, int t) { return (int)((n + t - 1) / t); }

struct armando_ctx {
    int device = 0;
    // The stream the context launches on: its own stream (created blocking, so
    // it is ordered with the legacy default stream both ways), or the caller's
    // (armando_set_stream). Graphs are captured on cap_stream and launched here.
    cudaStream_t stream = nullptr;
    cudaStream_t own_stream = nullptr;
    cudaStream_t cap_stream = nullptr;
    // A device-memory call returned before its work completed: its device
    // status words are being copied to h_flags; armando_sync reports them.
    bool pending = false;
    // Stage the neighbour passes' candidates in shared memory where the
    // variant allows it (ARMANDO_STAGING=1 at creation; otherwise global
    // memory through L1; both give the same bits).
    bool staging = false;
    // Neighbour lists between sorts (ARMANDO_NEIGHBOUR_LISTS=0 at creation:
    // walk the cells every iteration; the GPU-C schemes' results are the same bits, the
    // CERN step's differ by the rounding of its sums: in 2D the split of near and far
    // pairs is another one and a far pair's weight is rounded by itself).
    bool lists = true;
    // Fused predictor on the iterations between sorts (ARMANDO_FUSED_PREDICTOR=0
    // at creation: a reorder copy every iteration; the same bits).
    bool fuse_ok = true;
    // Inside armando_forward_checkpointed or a replay of armando_backward.
    bool reverse_run = false;
    armando_params prm{};
    DevParams dp{};
    int dim = 2;
    int64_t n = 0, nf = 0, nw = 0;
    // Particle slots of the step arrays: n, plus one mirror ghost per fluid
    // particle for contexts created with wall_model 3. n_work: particles of
    // the iteration being launched (n + its ghosts).
    int64_t cap = 0, n_work = 0;
    int mem_kind = ARMANDO_MEM_HOST;
    StateA A{};
    StateB B{};
    unsigned* keys[2] = {nullptr, nullptr};
    int* vals[2] = {nullptr, nullptr};
    // Cell sort: keys[0] the cells by slot, vals[0] the arrival numbers, placed the
    // particles of each cell in order of arrival; keys[1] and vals[1] the sorted
    // cells and the permutation. cell_cnt (zero between sorts), cell_sums: the scan.
    int *placed = nullptr, *cell_cnt = nullptr, *cell_sums = nullptr;
    unsigned* ticket = nullptr;  // k_bbox_grid
    unsigned* hist = nullptr;
    unsigned* dtotal = nullptr;
    int* start = nullptr;
    long long cell_cap = 0;
    float* bbox_part = nullptr;
    DevGrid* grid = nullptr;
    unsigned* flags = nullptr;
    unsigned* h_flags = nullptr;  // pinned
    DevGrid* h_grid = nullptr;    // pinned
    // Device copies of caller arrays (host memory kind).
    float *s_x = nullptr, *s_v = nullptr, *s_m = nullptr, *s_rho = nullptr, *s_p = nullptr,
          *s_u = nullptr, *s_h = nullptr, *s_dvdt = nullptr, *s_dudt = nullptr;
    int* s_itype = nullptr;
    std::vector<void*> owned;
    int* inv = nullptr;  // caller index -> cell-order slot (outputs to mapped host memory)
    std::map<GraphKey, StepGraph> graphs;
    std::string err = "no error";
    int64_t steps_done = 0, launches = 0;
    int launches_per_step = 0;
    int64_t first_sorts = 0;  // sorts of first steps, whose kernels are counted with their graph
    int lazy_body = 0;  // kernels in the conditional body of the lazy step graph (run on sorting steps)
    DevGrid last_grid{};
    bool have_grid = false;
    float last_dt = 0.f;  // dt and next its of the state left on the device
    int next_its = 0;
    // Batches of independent instances (n_inst > 1): packed state, one cell
    // grid per instance, persistent passes over work items.
    int n_inst = 1;
    std::vector<int64_t> inst_n;            // particles per instance
    std::vector<armando_params> prm_inst;   // parameters per instance
    std::vector<float> inst_dt;             // time step per instance
    int* d_inst0 = nullptr;                 // instance of each caller index
    DevParams* d_params = nullptr;          // [n_inst]
    DevGrid* d_grids = nullptr;             // [n_inst]
    int* d_ncells_inst = nullptr;           // [n_inst]
    int* d_inst_items = nullptr;            // [n_inst + 1] first work item per instance
    WorkItem* d_items = nullptr;
    int n_items = 0;
    float* d_part_items = nullptr;          // [n_items * 8] bbox partials
    int* d_total_cells = nullptr;
    int* d_queue = nullptr;                 // [4] work-queue heads, reset every step
    int* d_its = nullptr;
    int any_visc = 0;
    bool batch_lean = false;  // every instance has lean physics: the lean passes
    int grid_density = 0, grid_shear = 0, grid_force = 0;  // persistent CTAs
    cudaGraphExec_t batch_graph = nullptr;
    // Reverse mode (armando_forward_checkpointed / armando_backward).
    std::vector<StateA> ckpts;           // state before iterations its0 + k*K
    armando_tuning tune{1, 1, 128, 0};   // neighbour-pass tuning (armando_set_tuning)
    int64_t sorts_done = 0;              // lazily sorting iterations that sorted (device count)
    int64_t sorts_host = 0;              // iterations that always sort
    cudaStream_t stream2 = nullptr;      // captures the conditional sort body; copies beside the step
    // A host-memory call's copies beside the step (overlapped_call): events
    // {inputs start, rest of the inputs loaded, density done, rho and p written}.
    cudaEvent_t ev_ovl[4] = {nullptr, nullptr, nullptr, nullptr};
    int ovl_ctas = 0;                    // CTAs of the copy kernels beside the step
    bool split_in = false;               // load_inputs left the rest of the inputs on stream2
    bool no_conditional = false;         // conditional graphs failed to build here
    float4* xsort_buf = nullptr;
    std::vector<TapeSlot> tape;          // intermediates of each iteration of one segment
    int tape_seg = -1;                   // the segment the tape holds (-1: none)
    AdjState adjG{}, adjGp{};            // cotangents (output / input slot order)
    float4 *adj_abar = nullptr, *adj_xpart = nullptr, *adj_vpart = nullptr, *adj_xF = nullptr,
           *adj_vhb = nullptr;
    float *adj_rhobar = nullptr, *adj_pbar = nullptr;
    double* adj_blk = nullptr;   // per-block parameter cotangents
    float* adj_divsb = nullptr;  // cotangents of the divergence sums (artificial heat)
    float4 *adj_tbar = nullptr, *adj_tbar2 = nullptr;  // shear-tensor cotangents (viscosity)
    double* adj_pacc = nullptr;
    int adj_its0 = 0, adj_steps = 0, adj_K = 0;
    float adj_dt = 0.f;
    bool adj_ready = false;
    // Mirror ghosts (wall_model 3): the wall grid of the call, the walls in
    // cell order, and per iteration the nearest wall of each particle and the
    // ghosts' owners.
    WallGrid* wgrid = nullptr;
    WallGrid* h_wgrid = nullptr;  // pinned
    int* wstart = nullptr;
    long long wstart_cap = 0;
    int wall_cells = 0;
    float4 *wall_xh = nullptr, *wall_n = nullptr;
    int *wall_id = nullptr, *g_best = nullptr, *g_owner = nullptr, *g_slot = nullptr,
        *d_ng = nullptr, *h_ng = nullptr;
    unsigned *g_tile_count = nullptr, *g_tile_off = nullptr;
    int64_t ghosts_last = 0;
    // Open boundaries of the GPU-C schemes: inlets (with their distances since
    // the last emission), outlets and box, the compaction buffers.
    bool open_set = false;
    std::vector<armando_inlet> inlets;
    std::vector<float> inlet_dist;
    OpenSpec open{};
    StateA A2{};
    // Fused predictor (lazily sorting, lean physics, lists): the force pass
    // writes the next state into A_alt, then the two swap.
    StateA A_alt{};
    bool open_ready = false;
    int *open_keep = nullptr, *d_open_n = nullptr, *h_open_n = nullptr;
    unsigned *open_tc = nullptr, *open_to = nullptr;
    // single_step options: drho/dt carried between calls in caller order
    // (continuity density) and the buffers of the options, allocated on first use.
    float* drho_caller = nullptr;
    bool options_ready = false;
    // GPU-C schemes (scheme 1, 2): the RK3 working state in cell order and the
    // material table (default: Tait with rho0, c0 for every |itype|).
    GpucState gs{};
    bool gs_ready = false;
    DevMaterial* d_mat = nullptr;
    std::vector<armando_material> materials;  // set by armando_set_materials
    DevZones* d_zones = nullptr;               // load and fix zones (armando_set_zones)
    std::vector<armando_load_zone> loads;
    std::vector<armando_fix_zone> fixes;
};

// The context's lazy-sort flags (see sort_skipped); nullptr: always sort.
inline const int* resort_flags(armando_ctx* ctx) { return reinterpret_cast<const int*>(ctx->flags + 1); }

// Whether the context sorts lazily (a sort skin; one particle system).
inline bool lazy(const armando_ctx* ctx) { return ctx->tune.skin > 0 && ctx->n_inst == 1; }

// Neighbour lists: a lazily sorting step with one lane per particle and
// the lists allocated (ensure_lists); the iterations between sorts then read
// the lists instead of walking the cells.
// Not in reverse mode: its iterations sort every time, and the adjoint passes
// decode the neighbour bits that the density pass leaves only for particles
// walking their cells.
inline bool use_lists(const armando_ctx* ctx) {
    return lazy(ctx) && ctx->tune.threads_per_particle == 1 && ctx->B.nlist != nullptr && !ctx->reverse_run;
}

inline bool any_periodic(const DevParams& p) { return p.periodic[0] || p.periodic[1] || p.periodic[2]; }
inline bool lean_physics(const DevParams& p) {
    return !p.visc && !p.heat_art && p.wall_model == 0 && p.density_form == 0 && !p.xsph && !p.sle;
}

// Whether the parameters use a single_step option beyond summation density.
inline bool step_options(const armando_params& p) {
    return p.density_form != 0 || p.average_velocity != 0 || p.sle != 0;
}

// The passes read the state themselves on iterations that do not sort (no
// reorder copy) and write the next state into the other buffer: lists, lean
// physics, no step option.
inline bool fused_wanted(const armando_ctx* ctx) {
    return ctx->fuse_ok && ctx->prm.scheme == 0 && use_lists(ctx) && lean_physics(ctx->dp) && !step_options(ctx->prm);
}
inline bool fused(const armando_ctx* ctx) { return fused_wanted(ctx) && ctx->A_alt.xh != nullptr; }

// The staged passes serve one thread per particle, lean physics, no periodic
// axis, no single_step option and no mirror ghosts (the other variants read
// their candidates from global memory).
inline bool staged_passes(const armando_ctx* ctx) {
    return ctx->staging && !use_lists(ctx) && ctx->tune.threads_per_particle == 1 && lean_physics(ctx->dp) && !any_periodic(ctx->dp) &&
           !step_options(ctx->prm) && ctx->n_inst == 1 && ctx->prm.wall_model != 3;
}
