// nbl_plan.hh -- host-side state of the engine (plans, batches, workspace).
#pragma once

#include <cstdint>
#include <cstring>
#include <vector>

#include <cuda_runtime.h>
#include <nvtx3/nvToolsExt.h>

#include "nbl_b200.h"
#include "nbl_build.cuh"
#include "nbl_internal.cuh"

namespace nbl {

// A batch of independent systems planned on the host.
struct Batch {
    std::vector<SysDev> sys;
    std::vector<int64_t> ncells;
    std::vector<double> pt64;      // concatenated per-type squared cutoffs
    int64_t natoms = 0;
    const double *positions = nullptr;
    bool pos_on_device = false;
    const double *per_atom = nullptr;
    const int32_t *types = nullptr;
    bool aux_on_device = false;
    int grid = kGridDense;         // resolved kGrid*
    int64_t table_size = 1;
    int key_bits = 0;
    bool fp32 = true;
    int quantities = 0;
};

// Sizes of the row passes' neighbour lists (nbl_rows.cu).
struct ListPlan {
    int64_t total = 0, chunks = 0;  // 16-byte groups; first one of the chained chunks
    bool wide = false;              // two-word entries
    int shift = 27;                 // else: bits of the sorted atom
    int64_t row_cap = 0;            // row marks
    double expect = 0.0;            // pairs the density alone would give
    double scale = 1.0, shrink = 1.0;
    int64_t cap(const Batch &b, size_t system) const;  // groups per atom
};

// Device buffers of one call, carved out of the workspace.
struct Bufs {
    double *pos = nullptr;
    double *per_atom = nullptr;
    int32_t *types = nullptr;
    SysDev *sys = nullptr;
    VisitDev *visit = nullptr;     // per-system visit tables (nullptr: none)
    int64_t *sys_atom_base = nullptr;
    double *pt64 = nullptr;
    float *pt32 = nullptr;
    uint32_t *keys = nullptr, *keys2 = nullptr;
    int32_t *vals = nullptr, *vals2 = nullptr;
    int32_t *cell_count = nullptr;  // atoms per cell (counted_cells), or null
    int32_t *hist = nullptr, *hist_scan = nullptr, *scan32 = nullptr;
    int64_t *scan64 = nullptr;
    int2 *table = nullptr;
    unsigned long long *hkey = nullptr;
    double4 *pos64 = nullptr;
    float4 *pos32 = nullptr;
    int4 *aux = nullptr;
    double *radius = nullptr;      // the plan's copy of the caller's device radii
    float *amax = nullptr;
    HomeCell *home = nullptr;
    int32_t *counts = nullptr;
    int64_t *offsets = nullptr;
    int *small = nullptr;  // [0] occupied cells, [1] error bits, [2] matrix
                           // overflow, [3] work items, [4..5] mask-pool cursor
                           // (u64), [6] work-item ticket of the pair passes;
                           // placed right after offsets[N], so one copy of
                           // 32 bytes from offsets + N returns the pair count
                           // and the first six flags
    // The small host tables (systems, their atom bases, per-type cutoffs in
    // FP64 and FP32) lie at these byte offsets from `sys`, one contiguous
    // block of tab_bytes, so that they go up in one copy.
    size_t tab_pos = 0, tab_sab = 0, tab_pt64 = 0, tab_pt32 = 0, tab_bytes = 0;
    uint32_t *mask_pool = nullptr;
    long long mask_cap = 0;
    long long *home_mask = nullptr;
    WorkItem *items = nullptr;
    uint4 *list = nullptr;         // neighbour lists, home cells, sorted indices and
    int4 *hcell = nullptr;         // row marks of the row passes
    int32_t *inv = nullptr;
    int32_t *row_of = nullptr;
    ListPlan list_plan;
    double *lj_part = nullptr;     // force pass: per-atom energies, then block sums
};

struct Workspace {
    void *base = nullptr;
    size_t bytes = 0;
    void *out_base = nullptr;  // device output scratch of nbl_fill_host
    size_t out_bytes = 0;
    void release();
};

// Full waves of resident CTAs in the default grid of a pair pass.
constexpr int kAutoWaves = 2;

// Atoms above which the row of every 128th output slot is marked after the scan
// (k_row_marks), from the second count of the same sizes on; below it, and beyond the
// marks' table, which has room for as many pairs as the lists, the fill's warps search
// the row offsets.  Measured, fill and marks
// with / without, us, uniform gases: a million atoms at 10 / 2 / 0.5 per cell 704 / 713,
// 183 / 182, 74 / 73; 200,000 130 / 133, 37 / 38, 22 / 20; 131,072 81 / 86, 29 / 29,
// 16 / 15; 30,000 30 / 30, 11 / 10, 11 / 10: a launch for little, paid back by long
// lists.
constexpr int64_t kMarkAtoms = 131072;
// Host positions of up to this many atoms are uploaded with the host tables: one
// copy from pinned memory instead of that and one from pageable memory.  The call, with
// the tables / on their own: 1,000 atoms 115 / 117 us, 2,000 126 / 134, 16,000 182 /
// 190, 32,000 250 / 233; the line keeps the pinned staging below 100 KB.
constexpr int64_t kTablePositions = 2048;
// Mean atoms per cell up to which the atoms are counted into cells and ranked there,
// each by reading its cell's atoms; the radix sort above.  Binning to gather, ranked /
// sorted: 2,000 atoms at 150 per cell 15 / 16 us, at 1,000 50 / 18; 20,000 at 150 / 300
// / 1,000 16 / 23, 19 / 20, 60 / 19; 200,000 39 / 47, 63 / 40, 115 / 40; a million
// 109 / 107, 150 / 104, 371 / 105.
constexpr int64_t kRankAtoms = 192;
// Atoms per occupied cell below which the count takes one thread per atom.  Measured,
// k_rows_count / k_count_list, us: 20,000 atoms at 2.2 / 3.1 / 4.1 per occupied cell
// 20 / 26, 21 / 25, 29 / 28; 60,000 at 2.3 / 3.2 / 3.9 41 / 54, 53 / 47, 52 / 46;
// 200,000 at 3.1 / 4.0 / 5.1 99 / 129, 109 / 121, 125 / 113; a million at 4.1 / 6.0 /
// 8.0 392 / 553, 470 / 490, 556 / 469.
constexpr double kSparseAtoms = 4.0;

// Everything that shapes the count phase's launches on a plan: when two
// consecutive single calls have the same key, the second captures the count
// phase into a CUDA graph and later ones replay it (compared bytewise; the
// constructor zeroes the padding).
struct CountKey {
    const void *ws_base, *pos, *per_atom, *types;
    // where the layout put the buffers (their sizes shift one another)
    const void *keys, *table, *pos64, *offsets, *list, *hcell, *row_of, *end;
    int64_t natoms, table_size, mask_cap, list_chunks, row_cap, pt_size, i_lo, i_hi, nvisit;
    int32_t nsys, grid, key_bits, fp32, kind, itile, max_run, nvisit_tab, cull;
    int32_t count_mult, count_warps, count_cand, count_group, count_tickets, atoms, sparse;
    CountKey() { std::memset(this, 0, sizeof(*this)); }
    bool operator==(const CountKey &o) const { return std::memcmp(this, &o, sizeof(*this)) == 0; }
};

constexpr int kOccupiedWord = 4;  // of Plan::host_small

// What a batch is uploaded for.
enum CountUse { kUseLists, kUseOneLaunch, kUseForces };

struct Plan {
    int device = 0;
    int num_sms = 148;
    Workspace ws;
    Bufs bufs;
    TraverseArgs targs{};
    int trav_grid = 0;        // count-pass grid (CTAs)
    int fill_grid = 0;        // fill-pass grid (CTAs)
    // Launch configuration (set by the autotuner for batches, or by
    // nbl_plan_set_launch / nbl_plan_set_launch_config): CTAs per SM of the
    // count and fill passes (0: a whole number of waves of resident CTAs),
    // each pass's launch shape (warps per CTA, staged candidates, atoms per
    // sweep) and the atoms per work item (cell-occupancy tile).
    int count_mult = 0;
    int fill_mult = 0;
    TravShape count_shape;
    TravShape fill_shape = default_fill_shape();
    int itile = 32;
    // Tile chosen per call from the atom count (launch config atoms_per_item
    // 0); itile is then the tile of large systems.
    bool itile_auto = true;
    // Home cells per work item at most (0: chosen on the device from the
    // cells' mean occupancy; 1: one cell per item).  Runs of several cells
    // are only built on the dense grid with the FP32 filter.
    int max_run = 0;
    // Systems of up to this many atoms (at most kSmallMaxAtoms) take the
    // one-CTA count phase; 0: never.
    int small_atoms = kSmallDefaultAtoms;
    // Pair passes with one thread per atom (nbl_trav_atoms.cu): 0 = where the
    // occupied cells hold fewer than two atoms on average, -1 = never, 1 =
    // always (where the systems have visit tables).
    int atom_threads = 0;
    // Occupied cells and pairs counted by the last synchronised count, with the
    // atom count and table size it ran on (steers the default choices).
    int64_t occ_natoms = -1, occ_table = -1, occ_cells = 0, occ_pairs = 0;
    // Work items by atomic ticket (else a fixed warp stride) in each pass.
    bool count_tickets = true;
    bool fill_tickets = true;
    int64_t mask_hint = 0;    // mask-pool words the last count asked for
    // Row passes in use; and what the synchronised counts of these sizes found.
    bool rows = false;
    double cand_atom = 0.0;   // atoms of the cells that an atom visits, on average
    bool forces = false;      // a force pass: no lists planned
    float lj_line = 0.f;      // its choice left to the device (choose_lj)
    bool sparse = false;      // with one thread per atom in the count
    bool spare_ticket = false;  // a cleared work-item ticket is left for one fill
    bool lists_short = true;  // some row may have no list (kErrNoList)
    // (the sizes: atoms, table, row range; groups of chained chunks to plan for)
    int64_t list_natoms = -1, list_table = -1, list_lo = 0, list_hi = 0, list_more = 0;
    double list_pairs = 0.0;
    bool list_stay = false;  // no room for more than the density's estimate
    int64_t most_natoms = -1, most_table = -1, most_lo = 0, most_hi = 0, list_most = 0;
    // Row range of nbl_set_atom_range (global atom indices, [lo, hi)).
    int64_t i_lo = 0;
    int64_t i_hi = INT64_MAX;
    int64_t batch_natoms = 0;
    int batch_nsys = 0;
    bool batch_fp32 = true;
    int batch_kind = kCutScalar;
    int batch_grid = kGridDense;
    bool have_count = false;
    bool count_pending = false;   // a force pass left no counts: made on demand
    int64_t npairs = 0;
    int quantities = 0;
    // pinned: [0] pair count, [1] flags, [kOccupiedWord] occupied cells of the last force
    // pass (low half) and the sizes they belong to
    int64_t *host_small = nullptr;
    void *host_stage = nullptr;     // pinned staging of the small host tables
    size_t host_stage_bytes = 0;
    void *host_out = nullptr;       // pinned landing area of small host fills
    size_t host_out_bytes = 0;
    cudaEvent_t stage_done = nullptr;
    bool stage_in_flight = false;
    // Count-phase graph of the single-call path (see CountKey).
    CountKey last_key, graph_key;
    bool have_last_key = false;
    bool graphs_off = false;        // capture failed once: direct launches only
    cudaStream_t capture_stream = nullptr;
    cudaGraphExec_t count_graph = nullptr;
    long long graph_launches = 0;   // kernels in the graph (launch accounting)
    TraverseArgs graph_targs{};     // host state the capture left behind
    int graph_trav_grid = 0, graph_kind = 0;
};

// Drops the plan's count-phase graph (its pointers refer to the workspace).
void drop_count_graph(Plan &p);

// An NVTX range over one host-side stage (bin, sort, gather, count, scan,
// fill): profilers show the stages of a call by name and can filter their
// kernels by it.  Costs a few nanoseconds when no tool is attached.
struct StageRange {
    explicit StageRange(const char *name) { nvtxRangePushA(name); }
    ~StageRange() { nvtxRangePop(); }
    StageRange(const StageRange &) = delete;
    StageRange &operator=(const StageRange &) = delete;
};

// Stream-ordered scratch pool of device `dev` that keeps its memory between
// calls (cudaMallocFromPoolAsync / cudaFreeAsync on it).
cudaError_t scratch_pool(int dev, cudaMemPool_t *pool);

nbl_status set_error(nbl_status st, const char *fmt, ...);
nbl_status cuda_status(cudaError_t e, const char *where);
nbl_status plan_system(const double origin[3], const double cell[9],
                       const double inv_cell[9], const uint8_t pbc[3], double cutoff,
                       SysDev &S, int64_t &ncells);
nbl_status finish_batch(Batch &b, int grid_req);
nbl_status upload_batch(Plan &p, const Batch &b, cudaStream_t st, CountUse use = kUseLists);
const Plan &batch_plan_of(const nbl_batch *bt);
void note_count(Plan &p, const Batch &b, int64_t npairs, int occupied);
void note_lists(Plan &p, const Batch &b, int64_t npairs, int64_t demand, int flags);
nbl_status enqueue_count(Plan &p, const Batch &b, cudaStream_t st);
nbl_status run_count(Plan &p, const Batch &b, cudaStream_t st, bool sync);
nbl_status run_fill(Plan &p, const nbl_outputs &o, int64_t capacity, cudaStream_t st);
// The device flags of the last count / fill as a status (copy: read them
// first, synchronising st).
nbl_status read_flags(Plan &p, cudaStream_t st, bool copy = true);
void launch_config_of(const Plan &p, nbl_launch_config *cfg);

}  // namespace nbl
