// sf_force.cu — force + integration pass of the SPH sub-step (sm_103a).
//
// One thread per cell-sorted particle.  Pressure (spiky gradient, symmetrised
// (p_i + p_j) / (2 rho_j) weight), viscosity (Laplacian) and gravity from the
// neighbour list of the density pass — or from a rescan of the candidate cells
// where the list overflowed or no list was recorded — then, in the stepping
// variant, symplectic Euler, the box clamp with restitution and the next
// step's cell key and arrival slot (the counting sort's histogram).
// A neighbour on the list is one 32-byte record written by the density pass,
// (x, vx, y, vy) and (z, vz, p, 1/rho), fetched with one 256-bit load.
// kPrefetch neighbours are gathered before their terms are added, and the
// next kPrefetch list entries are loaded while they are, so the dependent
// index -> data loads of consecutive batches overlap; the terms are still
// added in list order, which keeps the sum bit-identical.  Lists of 16-bit
// entries (SF_LIST_TILE16) are decoded to indices where they are used.  The
// per-particle pass itself (force_one) is in sf_passes.cuh; small scenes take
// the team form of sf_team.cuh.
#include "sf_team.cuh"

namespace sf {
namespace {

// Raises the frame's maxima of |v'|^2 and |a|^2 to those of the block
// (non-negative floats order like their bits), with one atomic each per block.
template <int kBlockSize>
__device__ __forceinline__ void raise_maxima(FrameState* __restrict__ frame, uint32_t v2, uint32_t a2) {
    __shared__ uint32_t s_max[2][kBlockSize / 32];
    v2 = __reduce_max_sync(0xffffffffu, v2);
    a2 = __reduce_max_sync(0xffffffffu, a2);
    if ((threadIdx.x & 31) == 0) {
        s_max[0][threadIdx.x / 32] = v2;
        s_max[1][threadIdx.x / 32] = a2;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        const bool have = threadIdx.x < kBlockSize / 32;
        const uint32_t mv = __reduce_max_sync(0xffffffffu, have ? s_max[0][threadIdx.x] : 0u);
        const uint32_t ma = __reduce_max_sync(0xffffffffu, have ? s_max[1][threadIdx.x] : 0u);
        if (threadIdx.x == 0) {
            atomicMax(&frame->v2max_bits, mv);
            atomicMax(&frame->a2max_bits, ma);
        }
    }
}

// Registers are capped at 56 (nine blocks of 128 threads per SM; 58 would fit
// only eight: 100 us instead of 95 at 1,048,576 particles) or, with four
// gathers in flight, at 72 (seven blocks).
template <int kList, int kPrefetch, int kBlockSize, bool kIntegrate, int kReach, bool kBatched>
__global__ void __launch_bounds__(kBlockSize, (kPrefetch == 2 ? 1152 : 896) / kBlockSize)
    k_force(const float4* __restrict__ pos, const float4* __restrict__ vel, const float2* __restrict__ pr,
            const uint32_t* __restrict__ cs, const uint32_t* __restrict__ nbr, const uint32_t* __restrict__ nbr_count,
            const uint8_t* __restrict__ nbr_wide, const float4* __restrict__ pv, uint32_t n, SimConst c0, const SimConst* __restrict__ table, const uint32_t* __restrict__ scene_off,
            uint32_t nscenes, float4* __restrict__ pos_out, float4* __restrict__ vel_out,
            uint32_t* __restrict__ counts, uint32_t* __restrict__ cell_head, uint32_t* __restrict__ tile_sums,
            uint2* __restrict__ key_slot, float4* __restrict__ acc_out, float4* __restrict__ sums, FrameState* __restrict__ frame) {
    grid_dependency_wait();
    allow_dependents_sized(n);
    const uint32_t i = blockIdx.x * kBlockSize + threadIdx.x;
    uint32_t v2 = 0u, a2 = 0u;
    if (i < n)
        force_one<kList, kPrefetch, kIntegrate, kReach, kBatched>(i, pos, vel, pr, cs, nbr, nbr_count, nbr_wide, pv, n, c0,
                                                                  table,
                                                                     scene_off, nscenes, pos_out, vel_out, counts,
                                                                     cell_head, tile_sums, key_slot, acc_out, sums, frame, v2, a2);
    if (!kBatched && kIntegrate && frame && c0.adaptive) raise_maxima<kBlockSize>(frame, v2, a2);
}

template <bool kIntegrate, int kReach, int kTeam, int kTurn>
__global__ void __launch_bounds__(kTeam * 32)
    k_force_team(const float4* __restrict__ pos, const float4* __restrict__ vel, const float2* __restrict__ pr,
                 const uint32_t* __restrict__ cs, const uint32_t* __restrict__ nbr,
                 const uint32_t* __restrict__ nbr_count, const float4* __restrict__ pv, uint32_t n, SimConst c,
                 float4* __restrict__ pos_out, float4* __restrict__ vel_out, uint32_t* __restrict__ counts,
                 uint32_t* __restrict__ cell_head, uint32_t* __restrict__ tile_sums, uint2* __restrict__ key_slot,
                 float4* __restrict__ acc_out, float4* __restrict__ sums, FrameState* __restrict__ frame) {
    __shared__ ForceTeamShared sh;
    grid_dependency_wait();
    allow_dependents();
    const uint32_t first = blockIdx.x * kTeamParticles + (threadIdx.x & 31u), i = min(first, n - 1);
    float4 xi, vi;
    float2 pri;
    PairAcc a;
    bool last;
    const bool summed = force_team<kTeam, kTurn>(i, nbr_count, nbr, pv, n, c.h, sh, a, last, [&](bool finishes) {
        if (finishes) {  // the warp that integrates the particles
            xi = ldg4(pos + i);
            vi = ldg4(vel + i);
            pri = __ldg(pr + i);
        }
    });
    uint32_t v2 = 0u, a2 = 0u;
    if (last && first < n) {
        if (!summed) {
            a = PairAcc{};
            force_rescan<kReach, true>(i, c, pos, vel, pr, cs, n, xi, vi, pri.x, a);
        }
        if (sums) {
            sums[2 * (size_t)i] = make_float4(a.apx, a.apy, a.apz, 0.f);
            sums[2 * (size_t)i + 1] = make_float4(a.avx, a.avy, a.avz, 0.f);
        }
        force_finish<kIntegrate>(i, c, xi, vi, pri.y, a, pos_out, vel_out, counts, cell_head, tile_sums, key_slot,
                                 acc_out, frame, v2, a2);
    }
    if (kIntegrate && frame && c.adaptive) raise_maxima<kTeam * 32>(frame, v2, a2);
}

template <bool kIntegrate, int kTeam, int kTurn>
void force_team_as(DeviceState& d, const SimConst& c, cudaStream_t s) {
    with_reach(c.reach, [&](auto R) {
        launch_chained(k_force_team<kIntegrate, decltype(R)::value, kTeam, kTurn>, grid_for(d.n, kTeamParticles),
                       kTeam * 32, s, d.pos, d.vel, d.pr, d.cell_start, d.nbr, d.nbr_count, d.pv, d.n, c,
                       kIntegrate ? d.pos2 : nullptr, kIntegrate ? d.vel2 : nullptr, kIntegrate ? d.counts : nullptr,
                       kIntegrate ? d.cell_head : nullptr, kIntegrate ? d.tile_sums : nullptr, kIntegrate ? d.key_slot : nullptr,
                       kIntegrate ? nullptr : d.accel, d.sums, kIntegrate ? d.frame : nullptr);
    });
}

template <int kList, int kPrefetch, int kBlockSize, bool kIntegrate>
void force_as(DeviceState& d, const SimConst& c, cudaStream_t s) {
    cudaAccessPolicyWindow w{};
    const cudaAccessPolicyWindow* win =
        (kList != 0 && d.tune.l2_window && persisting_window(d.pv, (size_t)d.n * 2 * sizeof(float4), &w)) ? &w
                                                                                                           : nullptr;
    with_reach(c.reach, [&](auto R) {
        constexpr int K = decltype(R)::value;
        float4* po = kIntegrate ? d.pos2 : nullptr;
        float4* vo = kIntegrate ? d.vel2 : nullptr;
        uint32_t* co = kIntegrate ? d.counts : nullptr;
        uint32_t* ch = kIntegrate ? d.cell_head : nullptr;
        uint32_t* ts = kIntegrate ? d.tile_sums : nullptr;
        uint2* ks = kIntegrate ? d.key_slot : nullptr;
        float4* ac = kIntegrate ? nullptr : d.accel;
        if (d.table) {
            if constexpr (K <= 2 && kPrefetch == 2)
                launch_chained_window(win, k_force<kList, kPrefetch, kBlockSize, kIntegrate, K, true>,
                               grid_for(d.n, kBlockSize), kBlockSize, s, d.pos, d.vel, d.pr, d.cell_start, d.nbr,
                               d.nbr_count, d.nbr_wide, d.pv, d.n, c, d.table,
                               d.scene_off, d.nscenes, po, vo, co, ch, ts, ks, ac, d.sums, (FrameState*)nullptr);
        } else {
            launch_chained_window(win, k_force<kList, kPrefetch, kBlockSize, kIntegrate, K, false>,
                           grid_for(d.n, kBlockSize), kBlockSize, s, d.pos, d.vel, d.pr, d.cell_start, d.nbr,
                           d.nbr_count, d.nbr_wide, d.pv, d.n, c,
                           (const SimConst*)nullptr, (const uint32_t*)nullptr, 0u, po, vo, co, ch, ts, ks, ac, d.sums,
                           kIntegrate ? d.frame : nullptr);
        }
    });
}

bool team_force(const DeviceState& d, const SimConst& c) { return team_scene(d, c, kForceTeamScene); }

template <bool kIntegrate>
void launch_force(DeviceState& d, const SimConst& c, cudaStream_t s) {
    if (!d.n) return;
    if (team_force(d, c)) {
        force_team_as<kIntegrate, kForceTeam, kForceTurn>(d, c, s);
        return;
    }
    const bool big = d.tune.force_block == 256;
    if (!d.nbr || d.tune.list_mode == SF_LIST_NONE) {
        big ? force_as<0, 2, 256, kIntegrate>(d, c, s) : force_as<0, 2, 128, kIntegrate>(d, c, s);
    } else if (d.tune.list_mode == SF_LIST_TILE16 && d.nbr_wide) {
        if (d.tune.prefetch == 2)
            big ? force_as<2, 2, 256, kIntegrate>(d, c, s) : force_as<2, 2, 128, kIntegrate>(d, c, s);
        else
            big ? force_as<2, 4, 256, kIntegrate>(d, c, s) : force_as<2, 4, 128, kIntegrate>(d, c, s);
    } else if (d.tune.prefetch == 2) {
        big ? force_as<1, 2, 256, kIntegrate>(d, c, s) : force_as<1, 2, 128, kIntegrate>(d, c, s);
    } else {
        big ? force_as<1, 4, 256, kIntegrate>(d, c, s) : force_as<1, 4, 128, kIntegrate>(d, c, s);
    }
}

}  // namespace

SF_INDEX_CHECK_ACCESSOR(index_check_failures_force)

const char* force_kernel(const DeviceState& d, const SimConst& c) {
    if (team_force(d, c)) return "force_team";
    const bool lists = d.nbr && d.tune.list_mode != SF_LIST_NONE;
    if (lists && d.tune.prefetch == 4) return d.tune.force_block == 256 ? "force_256_gather4" : "force_128_gather4";
    return d.tune.force_block == 256 ? "force_256" : "force_128";
}

void launch_force_integrate(DeviceState& d, const SimConst& c, cudaStream_t s) { launch_force<true>(d, c, s); }

void launch_force_only(DeviceState& d, const SimConst& c, cudaStream_t s) { launch_force<false>(d, c, s); }

}  // namespace sf
