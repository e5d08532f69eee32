// sf_internal.h — shared declarations of the GB300 SPH step (not installed).
#pragma once
#include <cstdint>
#include <vector>
#include <cuda_runtime.h>

#include "../../include/sf_capi.h"

namespace sf {

// Per-step constants, derived once on the host from sf_params (in double,
// rounded to float) and passed to every kernel by value.
struct SimConst {
    float h, h2;          // kernel radius and its square
    float cd;             // m * 315 / (64 pi h^9): density = cd * sum (h^2 - r^2)^3
    float cp;             // m * 45 / (pi h^6) / 2: pressure-force coefficient
    float cv;             // mu * m * 45 / (pi h^6): viscosity-force coefficient
    float k, rho0, inv_rho0;
    float dt, e;          // sub-step, boundary restitution
    float g[3];           // gravity
    float lo[3], hi[3];   // particle-centre clamp box: box_min + r, box_max - r
    float bmin[3];        // grid origin
    float inv_cell[3];    // cells per unit length, per axis
    int n[3];             // cells per axis
    int eos, attractive;
    int reach;            // cells searched on each side: K = cells per kernel radius
    uint32_t ncells;
    float mass;
    // Conservative pruning of the candidate walk (skips only cells that hold
    // no particle within h): cell widths, a slack covering the rounding of
    // cell assignment, and the squared-distance threshold h^2 (1 + 1e-4).
    float cell_w[3];
    float prune_margin;
    float prune_h2;
    uint32_t cell_base;   // first key of this scene's cells (0 outside a batch)
    // adaptive sub-step: dt = min(dt_max, cfl_v h / max|v|, cfl_a sqrt(h / max|a|))
    int adaptive;
    float cfl_v, cfl_a;
    int lists_fit;        // at rest (particles 2r apart) a neighbour list holds all within h
};

// Device-side frame and sub-step state (one per context).
struct FrameState {
    float dt;            // the current sub-step
    uint32_t v2max_bits; // max |v|^2 of the last sub-step (float bits, >= 0)
    uint32_t a2max_bits; // max |a|^2 of the last sub-step
    float frame_acc;     // simulated time of the current frame (float, like frameTime)
    uint32_t iter;       // sub-steps of the current frame
    uint32_t substeps;   // sub-steps since the last reset
    double sim_time;     // simulated time since the last reset: the finished frames' float times, summed
};

// Fill `c` from `p`; returns SF_OK or an error code (with message in `why`).
int derive_constants(const sf_params& p, SimConst* c, const char** why);

// Scene generator (sf_scenes.cpp): AoS float3 positions of `scene`.
int scene_points(const sf_params& p, int scene, uint64_t seed, std::vector<float>& out, const char** why);
// Batched cube workload (sf_scenes.cpp): per-scene parameters, counts and the
// concatenated AoS float3 positions.
int batch_cubes(uint64_t seed, uint32_t nscenes, const sf_params& base, std::vector<sf_params>& params,
                std::vector<uint32_t>& counts, std::vector<float>& pos, const char** why);

// Neighbour lists: up to kNbCap neighbours per particle, in tiles of kNbTile
// particles (see nbr_index in sf_device.cuh).  A buffer for n particles holds
// nbr_entries(n) entries.
constexpr int kNbTile = 128;
constexpr int kNbCap = 64;
// Entries past the last tile: the force pass loads two slots ahead of a list's
// end (and uses none of them).
constexpr int kNbSlack = 2 * kNbTile;
constexpr int kNbWarpTile = 32;  // tiles of SF_LIST_TILE16 lists: one warp's particles
constexpr size_t nbr_entries(size_t n) { return (n + kNbTile - 1) / kNbTile * kNbCap * kNbTile + kNbSlack; }
// list emission modes of the density pass
constexpr int kEmitNone = 0, kEmitStaged = 1, kEmitTile = 2, kEmitTile16 = 3;
// SF_LIST_TILE16: entries hold the neighbour index's low 16 bits, exact when
// |j - i| <= kNear16 (j = i + (int16_t)(entry - i)).
constexpr uint32_t kNear16 = 32767;

// Kernel choices of a context (all give bit-identical results).
struct Tuning {
    bool chosen = false;           // by sf_set_tuning: taken as they are at every size
    int list_mode = SF_LIST_TILE;  // SF_LIST_*: how the density pass records neighbours
    int density_block = 256;       // 128 or 256 threads
    int force_block = 128;         // 128 or 256 threads
    int prefetch = 2;              // neighbours gathered per batch in the force pass: 2 or 4
    int l2_window = 0;             // 1: persisting L2 window over the gather records
    int batch_cluster = 0;         // batches: 0 a launch per stage; 2, 4, 8 one persistent launch of clusters
    int batch_block = 0;           // threads per block of the persistent step: 256, 512, 1024 (0: 256)
};

// Device buffers of one solver context (all owned by the context).
struct DeviceState {
    Tuning tune;
    uint32_t n = 0, cap = 0;
    float4* pos = nullptr;   // sorted positions, w = original index (bit pattern)
    float4* vel = nullptr;   // sorted velocities, w = 0
    float4* pos2 = nullptr;  // integrated positions before the re-sort
    float4* vel2 = nullptr;
    float2* pr = nullptr;    // (pressure, 1/density) of the last density pass
    float* rho = nullptr;    // density of the last density pass
    uint2* key_slot = nullptr;  // (cell key, arrival slot or next of the cell's list) of pos2/vel2 order
    uint32_t* tmp = nullptr;    // scratch; without cell_head, the cell-bucketed unsorted indices
    float* io = nullptr;        // AoS staging, 6 floats per particle
    float4* accel = nullptr;    // optional acceleration output (inspection)
    uint32_t* nbr = nullptr;       // neighbour lists, tile-major (kNbCap * kNbTile per tile)
    uint32_t* nbr_count = nullptr; // neighbours of each particle (may exceed kNbCap)
    uint8_t* nbr_wide = nullptr;   // SF_LIST_TILE16: per warp tile (kNbWarpTile particles), 1 where it holds 32-bit entries
    float4* pv = nullptr;          // 2 per particle (32 bytes): (x, vx, y, vy), (z, vz, p, 1/rho)
    float4* sums = nullptr;        // optional: per particle (AP, 0), (AV, 0) of the force pass (adjoint recording)
    bool shared = false;           // other contexts keep the GPU busy: no team passes
    FrameState* frame = nullptr;   // adaptive sub-steps read dt here and raise the maxima
    // grid
    uint32_t ncells = 0, ncells_pad = 0;
    uint32_t* counts = nullptr;      // ncells_pad, zero between steps
    uint32_t* cell_start = nullptr;  // ncells + 1
    // ncells_pad, or null: the heads of the lists that the particles of a cell
    // form in arrival order (key_slot holds the links), defined where counts
    // is not zero
    uint32_t* cell_head = nullptr;
    // per scan tile (kScanTile cells): particles counted in it, zero between steps
    uint32_t* tile_sums = nullptr;
    uint32_t ntiles = 0;
    // batches of independent scenes (null for a single scene): per-scene
    // constants and the first particle index of each scene (nscenes + 1)
    const SimConst* table = nullptr;
    const uint32_t* scene_off = nullptr;
    uint32_t nscenes = 0;
    // persistent batched step: scenes in decreasing particle count, and the
    // queue counter its clusters take scenes from
    const uint32_t* scene_order = nullptr;
    uint32_t* scene_queue = nullptr;
};

constexpr int kScanTile = 4096;
constexpr int kScanThreads = 128;
constexpr int kScanWarps = kScanThreads / 32;
constexpr int kScanChunks = kScanTile / 4 / kScanThreads;  // groups of four cells per thread
// Uploads of fewer particles count their scan tiles with one atomic per tile
// and warp; larger ones sum the histogram in a launch of its own
// (k_tile_totals).  Upload and sort, atomics / own launch: 16,000 particles
// 13.3 / 15.3 us, 65,536 13.6 / 15.2 in rows but 24.6 / 16.9 in random order,
// where a warp's lanes hit 32 tiles and the atomics contend (236,987: 67 / 29).
constexpr uint32_t kTileAtomics = 32768;
constexpr int kScanBlocksPerSM = 8;  // the scan grid's size

// Persisting L2 (sf_grid.cu).  reserve_persisting_l2(want) grows this
// process's persisting-L2 carve-out on the current device to `want` bytes
// (at most the device's maximum; a limit of the process's context, gone with
// it) and returns it (0 where the device has none); call it outside stream
// capture.  persisting_window() fills an access-policy window over
// [base, base + bytes) (cut to the device's largest window, hit ratio scaled
// to the carve-out) and returns false while no carve-out is reserved.
size_t reserve_persisting_l2(size_t want);
bool persisting_window(const void* base, size_t bytes, cudaAccessPolicyWindow* w);

// ---- kernel launchers (sf_grid.cu, sf_density.cu, sf_force.cu); all enqueue on `s`
// A caller-order AoS state into pos2 and vel (vel3 null: at rest; vel null: the
// velocities come later), its cell keys, histogram and scan-tile totals.
void launch_load_hash(const DeviceState& d, const float* pos3, const float* vel3, float4* vel, const SimConst& c,
                      cudaStream_t s);
void launch_load_vel(const float* vel3, uint32_t n, float4* vel, cudaStream_t s);
void launch_load_sorted(const float* pos3, const float* vel3, const uint32_t* ids, uint32_t n, float4* pos,
                        float4* vel, cudaStream_t s);
void launch_store_sorted(const float4* pos, const float4* vel, uint32_t n, float* pos3, float* vel3, uint32_t* ids,
                         cudaStream_t s);
void launch_store_aos(const float4* pos, const float4* vel, uint32_t n, float* pos3, float* vel3, cudaStream_t s);
// Caller-order AoS output with coalesced stores (for host memory that the
// kernel writes directly); `slot` is n entries of scratch.
void launch_store_caller_order(const float4* pos, const float4* vel, uint32_t n, uint32_t* slot, float* pos3,
                               float* vel3, cudaStream_t s);
// Cell keys, histogram and scan-tile totals of a loaded state.
void launch_hash_count(const DeviceState& d, const float4* pos, uint32_t n, const SimConst& c, uint32_t* counts,
                       uint2* key_slot, cudaStream_t s);
void launch_scan_cells(DeviceState& d, uint32_t n, cudaStream_t s);
// nothing where cells have lists (cell_head)
void launch_scatter(const DeviceState& d, cudaStream_t s);
// also zeroes tile_sums for the next histogram
void launch_rank_gather(const DeviceState& d, cudaStream_t s);
// Cells of this many per kernel radius or more (at rest one particle a cell)
// are sorted through lists, one launch less: a sub-step of 16,000 particles
// 18.2 -> 16.7 us, of 236,987 95 -> 93.  Cells of the kernel radius itself hold
// eight and are bucketed (k_scatter): lists were neither faster nor slower there
// (20 sub-steps of 16,000 particles 681 against 683 us).
constexpr int kListedReach = 2;
// Larger grids keep the bucketing too.  The heads take 4 bytes a cell (16 MB at the
// limit, 32 MB for 1,048,576 particles) and save one launch, about 1.5 us, of steps
// that are long there.  A sub-step in us, bucketing / lists (lattice; disordered):
// 4.5 Mi cells, 300,000 particles 81.6 / 80.8; 110.4 / 110.7, 600,000 147.7 / 146.5;
// 201.8 / 200.2; 7.6 Mi, 1,048,576 221.2 / 219.4; 321.9 / 319.4; 10.2 Mi, 3,345,599
// 659.3 / 653.2; 959.8 / 951.6; three cells per h, 12.2 Mi, 236,987 100.0 / 99.0;
// 123.4 / 123.5, 25.8 Mi, 1,048,576 268.6 / 267.2; 405.4 / 406.8.  Few particles in
// a large grid would gain more (100,000 in 4.9 Mi, three per h: 55.2 / 52.4; 62.6 /
// 57.7).
constexpr uint32_t kListedCells = 4u << 20;
// A list is walked entry by entry, so a crowded cell takes longer than bucketed
// indices do: the sort of 200,000 particles in cells of 16 members 21 us against 25,
// of 64 31 against 26, of 512 107 against 42.  The box keeps the particles of a
// running scene from such crowds (64 members are 60 times the rest density, and
// the passes then take 150 us and more), but an upload may place any number
// outside it, all in a few cells of its border.  Uploads of this many particles or
// more are therefore bucketed.  Upload and sort in us, list / bucketing, with
// none, 1%, 10% and all particles outside: 65,536 particles 31 / 33, 154 / 51,
// 1185 / 185, 6367 / 1526; 4,096 28 / 31, 36 / 32, 95 / 40, 358 / 127; 1,331 28 /
// 31, 29 / 30, 48 / 33, 135 / 63, where the launch counts most and a crowd least.
constexpr uint32_t kListedUpload = 2048;
// The state as the sort of an upload takes it.
inline DeviceState upload_view(DeviceState d) {
    if (d.n >= kListedUpload) d.cell_head = nullptr;
    return d;
}
// Scenes of fewer particles take the team forms (sf_team.cuh) of the two
// passes.  Stage times in us, one thread per particle / the team (jittered
// lattice; disordered), two cells per h: density 18.4 / 10.3; 22.4 / 12.4 at 16,000
// particles, 20.2 / 17.2; 24.4 / 22.6 at 50,000, 24.5 / 20.3; 24.6 / 23.6 at 56,000.
// One cell per h: 24.4 / 14.4; 26.4 / 16.3 at 16,000, 28.4 / 24.4; 31.9 / 27.0 at
// 56,000.  Three: 22.3 / 12.5; 31.0 / 14.2 and 24.6 / 26.9; 34.9 / 31.2.  Force
// 12.3 / 8.5; 14.4 / 10.1 at 16,000, 12.4 / 10.1; 14.5 / 10.9 at 30,000, 12.5 /
// 13.1; 14.4 / 14.7 at 40,000.
// Where a list cannot hold the neighbours at rest (h above 4.9 particle radii)
// both passes walk the candidates anyway and a team only takes room: a sub-step
// of 16,000 to 30,000 particles at 6 radii was 0.72 to 1.0 of one thread's speed.
// Scenes compressed that far with h = 4.5 radii: 0.98 to 1.14 with two or three
// cells per h, about 0.9 with one.
constexpr uint32_t kDensityTeamScene = 57344, kForceTeamScene = 32768;
// Scenes from this size on launch the next pass early (allow_dependents_sized).
constexpr uint32_t kEarlyLaunchScene = 196608;
// Between these sizes the density pass takes blocks of 128 threads: its grid is
// two to seven blocks of 256 per SM there, of which the last are few.  Ten
// sub-steps, 256 / 128 threads (lattice; disordered): 76,000 particles 296 /
// 300, 388 / 389 us; 84,000 321 / 319, 418 / 411; 120,000 456 / 432, 507 / 501;
// 236,987 (disordered) 920 / 909; 300,000 815 / 818, 1095 / 1110.
constexpr uint32_t kSmallBlockFrom = 81920, kSmallBlockTo = 262144;
// Warps per 32 particles in the force pass, and neighbours they take in turn
// (2 x 4; stage times at 16,000 and 32,000 particles 9.5 and 12.3 us, 4 x 4
// 9.6 and 13.7, 3 x 2 9.6 and 13.9, 8 x 2 12.4 and 15.6).
constexpr int kForceTeam = 2, kForceTurn = 4;
// Whether the passes' forms go by the size of the scene: a single scene with lists
// whose kernels the caller did not choose.
bool passes_by_size(const DeviceState& d);
// Whether a pass takes its team form below `limit` particles.
inline bool team_scene(const DeviceState& d, const SimConst& c, uint32_t limit) {
    return d.n < limit && !d.shared && c.lists_fit && passes_by_size(d);
}
const char* density_kernel(const DeviceState& d, const SimConst& c);
const char* force_kernel(const DeviceState& d, const SimConst& c);
void launch_density(const DeviceState& d, const SimConst& c, cudaStream_t s);
// forces + symplectic Euler + box + next-step cell hash into pos2/vel2
void launch_force_integrate(DeviceState& d, const SimConst& c, cudaStream_t s);
// forces only: acceleration into d.accel (inspection)
void launch_force_only(DeviceState& d, const SimConst& c, cudaStream_t s);

// Index-check failures counted by the checked build's kernels, per
// translation unit (always 0 in the release build); `reset` clears them.
uint64_t index_check_failures_density(bool reset);
uint64_t index_check_failures_force(bool reset);
uint64_t index_check_failures_adjoint(bool reset);
uint64_t index_check_failures_grid(bool reset);
void launch_keys(const DeviceState& d, const float4* pos, uint32_t n, const SimConst& c, uint32_t* keys,
                 cudaStream_t s);
// State invariants for sf_check_state: `seen` is n words of scratch, `report`
// kReportWords words (see k_check_state).
constexpr uint32_t kReportWords = 8;
void launch_check_state(const DeviceState& d, const SimConst& c, const uint32_t* nbr_count, uint32_t* seen,
                        uint32_t* report, cudaStream_t s);
void launch_neighbour_stats(const DeviceState& d, const SimConst& c, uint32_t* count, uint32_t* hash,
                            cudaStream_t s);

// The sort tail shared by makeReady and every step: counts -> cell_start,
// bucket (clearing the counters), stable rank, gather pos2/vel2 -> pos/vel.
void enqueue_sort_tail(DeviceState& d, cudaStream_t s, cudaEvent_t before_gather = nullptr);
// One full sub-step on the sorted state.
void enqueue_step(DeviceState& d, const SimConst& c, cudaStream_t s);

// The sub-step as separately launchable stages (for per-stage timing).
constexpr uint32_t kNumStages = 5;
extern const char* const kStageNames[kNumStages];
void enqueue_stage(uint32_t stage, DeviceState& d, const SimConst& c, cudaStream_t s);
// The kernel that the stage launches for this state ("" for none).
const char* stage_kernel(uint32_t stage, const DeviceState& d, const SimConst& c);

// ---- sub-step control (sf_frame.cu) ------------------------------------
// Maxima of the uploaded state: |v|^2 over the particles, |a|^2 = 0.
void launch_init_maxima(const float4* vel, uint32_t n, FrameState* fs, cudaStream_t s);
// A frame runs sub-steps while (double)frame_acc < frame_time and
// iter < max_substeps; none is longer than dt_max.
struct FrameLimits {
    double frame_time;
    float dt_max;
    uint32_t max_substeps;
};
// One of a frame's loops: a while node's handle and the sub-steps of its body
// (0: the frame has no such loop).
struct FrameLoop {
    uint32_t run = 0;
    cudaGraphConditionalHandle h = 0;
};
// Sub-steps per run.  An iteration of a while node drains the GPU and ends in
// the check; a frame of 334 sub-steps of 16,000 particles takes 6715 us in
// single sub-steps, 5280 in runs of 4, 5050 of 8, 4970 of 16.  Long steps fill a
// frame with few (none of 16, some of 4), so there are two lengths.
constexpr uint32_t kFrameRuns[2] = {16, 4};
// Where other threads run frames of this many contexts or more, a frame has the
// loop of single sub-steps alone: more than eight graphs of several while nodes at a time
// get in each other's way.  Frames of 1,331 particles from 8, 10 and 16 threads, ns
// per particle update, runs / single: 2.1 / 2.5, 3.1 / 2.1, 3.2 / 1.4; of 4,000
// 0.83 / 1.07, 1.16 / 0.98, 1.37 / 0.79.
constexpr uint32_t kFrameContexts = 8;
// resets the frame clock; decides whether the loops of runs are entered
void launch_frame_begin(FrameState* fs, const FrameLimits& l, const FrameLoop& first, const FrameLoop& second,
                        cudaStream_t s);
// at the end of a body: decides whether its loop goes on and the next is entered
void launch_frame_check(FrameState* fs, const FrameLimits& l, const FrameLoop& own, const FrameLoop& next,
                        cudaStream_t s);

// ---- adjoint (sf_adjoint.cu) -------------------------------------------
// One recorded forward step, in that step's sorted order.
struct AdjointStep {
    uint32_t n = 0;
    const float4* pos = nullptr;
    const float4* vel = nullptr;
    const float2* pr = nullptr;
    const float* rho = nullptr;
    const uint32_t* nbr = nullptr;
    const uint32_t* cnt = nullptr;
    const uint32_t* cs = nullptr;
    const float4* sums = nullptr;
    const float4* pv = nullptr;  // the step's 32-byte gather records (x, vx, y, vy), (z, vz, p, 1/rho)
};
// Adjoint working buffers (N particles).  Xb/Vb are indexed by particle id.
struct AdjointWork {
    float4* Xb = nullptr;
    float4* Vb = nullptr;
    float4* ab = nullptr;  // 2 per particle (32 bytes): (apb, avb) = (cp tb, cv tb) of the axes, (inv_bar, cv_bar)
    float4* xdir = nullptr;
    float4* vdir = nullptr;
    float4* xf = nullptr;
    float4* vf = nullptr;
    float4* xrb = nullptr;  // per particle (x, y, z, rho_bar): P4's gather record
    double* scalars = nullptr;   // [sum cv_bar, sum k_bar]
};
// The adjoint step's passes: P1 integration and box (adj_integrate), P2 force
// pair terms and density adjoint (adj_forces), P4 poly6 terms (adj_density).
constexpr uint32_t kAdjointPasses = 3;
extern const char* const kAdjointPassNames[kAdjointPasses];
void launch_adjoint_pass(uint32_t pass, const AdjointStep& st, const SimConst& c, AdjointWork& w, double2* partial,
                         cudaStream_t s);
// One step's adjoint (its passes in order); its scalar block partials go to
// `partial` (adjoint_partial_count(N) entries).
void launch_adjoint_step(const AdjointStep& st, const SimConst& c, AdjointWork& w, double2* partial,
                         cudaStream_t s);
uint32_t adjoint_partial_count(uint32_t n);
// scalars += the partials of `nsteps` consecutive steps (last step first).
void launch_adjoint_accumulate(const double2* partial, uint32_t nsteps, uint32_t n, double* scalars, cudaStream_t s);
// CIC histogram loss of the sorted state; dL/dx written to Xb by particle id.
void launch_histogram_loss(const float4* pos, uint32_t n, const SimConst& c, const float box_ext[3], uint32_t res,
                           const float* target, unsigned long long* hist, float* e2, double* partial, float4* Xb,
                           cudaStream_t s);
uint32_t histogram_partial_count(uint32_t res);

// ---- persistent batched step (sf_batch.cu) --------------------------------
struct BatchStep {
    float4* pos;
    float4* vel;
    float4* pos2;
    float4* vel2;
    float2* pr;
    float* rho;
    uint2* key_slot;
    uint32_t* tmp;
    uint32_t* nbr;
    uint32_t* nbr_count;
    float4* pv;
    uint32_t* counts;
    uint32_t* cell_start;
    const SimConst* table;
    const uint32_t* scene_off;
    const uint32_t* order;
    uint32_t* queue;
    uint32_t nscenes;
    uint32_t n;
};
// Clusters of `cluster` blocks (2, 4 or 8) of `block` threads (256, 512 or
// 1024) of the persistent step that the current device keeps resident at
// once (0 if it cannot run them).
int batch_persistent_clusters(int cluster, int block, int reach);
// One sub-step of every scene: a queue reset and one launch of `nclusters`
// clusters.  Scene cell ranges must start at multiples of four cells.
void launch_batch_persistent(const BatchStep& a, int cluster, int block, int nclusters, int reach, cudaStream_t s);

// Density of caller-owned device positions using the library's fixed static
// scratch (sf_noalloc.cu); no device allocation.
int noalloc_density(const sf_params& p, const SimConst& c, const float* d_pos_xyz, uint32_t n, float* d_rho,
                    float* d_pressure, cudaStream_t stream, const char** why);

}  // namespace sf
