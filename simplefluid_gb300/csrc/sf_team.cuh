// sf_team.cuh — the density and force passes with a team of warps per 32
// particles, for scenes too small to fill the GPU with one thread each.
//
// There a pass takes as long as one thread's chain of dependent loads and
// instructions, with idle issue slots around it (16,000 particles are less
// than one warp per scheduler).  Lane l of every warp of a block works on the
// block's particle l; the warps share its candidate planes (density) or its
// neighbours (force).  What they find is added one term after the other in
// the canonical order, so every result has the same bits as the one-thread
// passes.  Loads stay as coalesced as there, a warp's lanes being consecutive
// particles (teams of 4 to 16 lanes of one warp, whose loads are not, took
// 11.6 to 15.5 us for the density stage below instead of 10.3).  Lists have
// the layout of SF_LIST_TILE.
//
// On the device's clock, 16,000 particles (jittered lattice): density 13.4 ->
// 5.8 us, force 9.7 -> 5.2 us, the step 31.0 -> 20.5 us; 1,331 particles:
// density 11.7 -> 4.1, the step 29.0 -> 18.4 us.
#pragma once
#include "sf_passes.cuh"

namespace sf {

constexpr int kTeamParticles = 32;  // of a block

// Where a particle lies in the grid: its cell and its offset inside it.
struct CellPoint {
    int cx, cy, cz;
    float ox, oy, oz;
};
__device__ __forceinline__ CellPoint cell_point(const SimConst& c, float x, float y, float z) {
    CellPoint p;
    p.cx = cell_coord(x, c.bmin[0], c.inv_cell[0], c.n[0]);
    p.cy = cell_coord(y, c.bmin[1], c.inv_cell[1], c.n[1]);
    p.cz = cell_coord(z, c.bmin[2], c.inv_cell[2], c.n[2]);
    p.ox = (x - c.bmin[0]) - (float)p.cx * c.cell_w[0];
    p.oy = (y - c.bmin[1]) - (float)p.cy * c.cell_w[1];
    p.oz = (z - c.bmin[2]) - (float)p.cz * c.cell_w[2];
    return p;
}

// Density: 2 kReach + 1 warps, one per plane of candidate rows.
template <int kReach>
struct DensityTeamShared {
    float q[kNbCap][kTeamParticles];                       // h^2 - r^2 of the particles' neighbours, in order
    uint32_t count[2 * kReach + 1][kTeamParticles];        // neighbours found in each plane
};
constexpr uint32_t kPlaneOverflow = 1u << 16;  // a plane's count where a row holds more candidates than its mask

// Density of the block's particles (particle i of this lane; live: i < n).  A
// thread keeps a bit per candidate of its plane; once the team's counts are
// known it writes its neighbours to their places, kNbCap places at a time: more
// than a list holds are summed in further rounds.
template <int kReach>
__device__ __forceinline__ void density_team(uint32_t i, bool live, const SimConst& c, const float4* __restrict__ pos,
                                             const uint32_t* __restrict__ cs, uint32_t n, float* __restrict__ rho_out,
                                             float2* __restrict__ pr_out, uint32_t* __restrict__ nbr,
                                             uint32_t* __restrict__ nbr_count, const float4* __restrict__ vel,
                                             float4* __restrict__ pv, DensityTeamShared<kReach>& sh) {
    constexpr int kTeam = 2 * kReach + 1;
    // Words of a row's mask.  At rest a row of one cell per h (2r = h / 2) holds 24
    // candidates and in compressed places more than 64; with two or three per
    // h it holds 5 or 2.
    constexpr int kWords = kReach == 1 ? 3 : 1;
    const int lane = (int)(threadIdx.x & 31u), part = (int)(threadIdx.x / 32u);
    const float4 xi = ldg4(pos + i);
    const CellPoint p = cell_point(c, xi.x, xi.y, xi.z);
    // The plane's row ranges (see for_candidates): end[q] is one past the
    // last candidate, len[q] the number of candidates.
    uint32_t end[kTeam], len[kTeam];
    {
        const int dz = part - kReach, zz = p.cz + dz;
        const uint32_t n0 = (uint32_t)c.n[0];
        const float gz = face_gap(p.oz, dz, c.cell_w[2], c.prune_margin), gz2 = gz * gz;
        const bool plane = zz >= 0 && zz < c.n[2] && gz2 < c.prune_h2;
        const float reach2 = c.prune_h2 - gz2;
        float tlo = reach2, thi = reach2;
        if (kReach > 1) {
            const float gl = face_gap(p.ox, -kReach, c.cell_w[0], c.prune_margin);
            const float gh = face_gap(p.ox, kReach, c.cell_w[0], c.prune_margin);
            tlo -= gl * gl;
            thi -= gh * gh;
        }
        const uint32_t row0 = c.cell_base + ((uint32_t)zz * (uint32_t)c.n[1] + (uint32_t)p.cy) * n0;
        const uint32_t xa = row0 + (uint32_t)max(p.cx - kReach, 0),
                       xb = row0 + (uint32_t)min(p.cx + kReach, c.n[0] - 1) + 1u;
        const uint32_t xa1 = row0 + (uint32_t)max(p.cx - kReach + 1, 0),
                       xb1 = row0 + (uint32_t)min(p.cx + kReach - 1, c.n[0] - 1) + 1u;
#pragma unroll
        for (int q = 0; q < kTeam; ++q) {
            const int dy = q - kReach, yy = p.cy + dy;
            const float gy = face_gap(p.oy, dy, c.cell_w[1], c.prune_margin), g2 = gy * gy;
            const uint32_t* row = cs + (int64_t)dy * (int64_t)n0;  // rows dy are n0 entries apart
            end[q] = len[q] = 0u;
            if (plane && yy >= 0 && yy < c.n[1] && g2 < reach2) {
                end[q] = checked_end(__ldg(row + ((kReach > 1 && g2 >= thi) ? xb1 : xb)), n);
                len[q] = end[q] - checked_end(__ldg(row + ((kReach > 1 && g2 >= tlo) ? xa1 : xa)), n);
            }
        }
    }
    auto r2_of = [&](const float4& xj) {
        const float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
        return fmaf(dz, dz, fmaf(dy, dy, dx * dx));
    };
    // Two candidates of every row at a time, so that the rows' loads are in
    // flight together.  r^2 - h^2 is negative where a candidate is a
    // neighbour: its sign bit is shifted into the row's mask.  Past its row's
    // end a thread tests the particle itself, moved out of reach.
    uint32_t near[kTeam][kWords], past[kWords], mine = 0, most = 0;  // past: one past the candidates in a word
#pragma unroll
    for (int q = 0; q < kTeam; ++q) most = max(most, len[q]);
#pragma unroll
    for (int w = 0; w < kWords; ++w) {
#pragma unroll
        for (int q = 0; q < kTeam; ++q) near[q][w] = 0u;
        uint32_t tested = 32u * w;
#pragma unroll 1
        for (; tested < min(most, 32u * w + 32u); tested += 2) {
            float4 x0[kTeam], x1[kTeam];
#pragma unroll
            for (int q = 0; q < kTeam; ++q) {
                const uint32_t j = end[q] - len[q] + tested;
                x0[q] = ldg4(pos + (tested < len[q] ? j : i));
                x1[q] = ldg4(pos + (tested + 1 < len[q] ? j + 1 : i));
            }
#pragma unroll
            for (int q = 0; q < kTeam; ++q) {
                if (!(tested < len[q])) x0[q].x = __int_as_float(0x7f800000);
                if (!(tested + 1 < len[q])) x1[q].x = __int_as_float(0x7f800000);
                const F2 dx = f2(xi.x - x0[q].x, xi.x - x1[q].x), dy = f2(xi.y - x0[q].y, xi.y - x1[q].y),
                         dz = f2(xi.z - x0[q].z, xi.z - x1[q].z);
                const float2 u = unpack(add2(fma2(dz, dz, fma2(dy, dy, mul2(dx, dx))), f2(-c.h2, -c.h2)));
                near[q][w] = __funnelshift_l(__float_as_uint(u.x), near[q][w], 1);
                near[q][w] = __funnelshift_l(__float_as_uint(u.y), near[q][w], 1);
            }
        }
        past[w] = tested;
#pragma unroll
        for (int q = 0; q < kTeam; ++q) mine += (uint32_t)__popc(near[q][w]);
    }
    sh.count[part][lane] = most > 32u * kWords ? kPlaneOverflow : mine;
    __syncthreads();
    uint32_t at = 0, cnt = 0;
#pragma unroll
    for (int k = 0; k < kTeam; ++k) {
        const uint32_t v = sh.count[k][lane];
        at += k < part ? v : 0u;
        cnt += v;
    }
    const bool masked = cnt < kPlaneOverflow, list = live && cnt <= (uint32_t)kNbCap;
    const uint32_t most_near = __reduce_max_sync(0xffffffffu, masked ? cnt : 0u);  // the same in every warp
    uint32_t* const lst = nbr + nbr_index(i, 0);
    // the thread's neighbours from where it stopped up to place `to`; place `base` is the first of this round
    auto write = [&](uint32_t base, auto bounded, uint32_t to) {
#pragma unroll
        for (int q = 0; q < kTeam; ++q) {
#pragma unroll
            for (int w = 0; w < kWords; ++w) {
                uint32_t m = near[q][w];
#pragma unroll 1
                for (; m && (!decltype(bounded)::value || at < to); ++at) {
                    const uint32_t b = 31u - (uint32_t)__clz((int)m), j = end[q] - len[q] + past[w] - 1u - b;
                    m ^= 1u << b;
                    sh.q[at - base][lane] = c.h2 - r2_of(ldg4(pos + j));
                    if (list) lst[(size_t)at * kNbTile] = j;
                }
                if (decltype(bounded)::value) near[q][w] = m;
            }
        }
    };
    float s = 0.f;
    auto sum = [&](uint32_t terms) {
        for (uint32_t k = 0; k < terms; k += 4) {
#pragma unroll
            for (uint32_t u = 0; u < 4; ++u) {
                const float q = sh.q[k + u][lane];
                s = fmaf(q * q, q, s);
            }
        }
    };
    auto pad = [&](uint32_t terms) {  // zero terms, to a multiple of four
        const uint32_t k = terms + (uint32_t)part;
        if (k < ((terms + 3u) & ~3u)) sh.q[k][lane] = 0.f;
    };
    if (most_near <= (uint32_t)kNbCap) {
        const uint32_t terms = masked ? cnt : 0u;
        if (masked) write(0, std::false_type{}, 0);
        pad(terms);
        __syncthreads();
        if (part == 0) sum(terms);
    } else {
#pragma unroll 1
        for (uint32_t base = 0; base < most_near; base += kNbCap) {
            const uint32_t terms = masked && cnt > base ? min(cnt - base, (uint32_t)kNbCap) : 0u;
            if (terms) write(base, std::true_type{}, base + kNbCap);
            pad(terms);
            __syncthreads();
            if (part == 0) sum(terms);
            __syncthreads();
        }
    }
    if (part != 0 || !live) return;
    if (!masked) {  // a very dense place
        density_one<kEmitTile, kReach>(i, c, xi, pos, cs, n, rho_out, pr_out, nbr, nbr_count, vel, pv, false, nullptr,
                                       0);
        return;
    }
    const float4 v = ldg4(vel + i);
    const float rho = c.cd * s;
    const float pi = pressure_of(c, rho), inv_rho = 1.f / rho;
    rho_out[i] = rho;
    pr_out[i] = make_float2(pi, inv_rho);
    nbr_count[i] = cnt;
    st8(pv + 2 * (size_t)i, make_float4(xi.x, v.x, xi.y, v.y), make_float4(xi.z, v.z, pi, inv_rho));
}

// Force: kTeam warps, which take kTurn neighbours of the list in turn.  A warp
// computes the weights of its neighbours ahead; in its turn it takes the sums
// of all neighbours before from shared memory, adds its own in list order and
// hands them on.
struct ForceTeamShared {
    float2 sum[3][kTeamParticles];   // (AP, AV) of the three axes
    uint32_t small[kTeamParticles];  // PairSums::small so far
};

// Named barriers of the two warps (1 + warp; 0 is __syncthreads): the warp that
// hands on arrives, the next one waits.  Their numbers are constants: with a
// number in a register a block holds all 16 barriers, and fewer blocks fit an SM
// (force stage at 30,000 particles 12.8 -> 10.2 us, disordered 14.4 -> 11.4).
template <int kTeam>
__device__ __forceinline__ void turn_wait(int warp) {
    static_assert(kTeam == 2, "one barrier per warp");
    if (warp == 0)
        asm volatile("bar.sync 1, 64;" ::: "memory");
    else
        asm volatile("bar.sync 2, 64;" ::: "memory");
}
template <int kTeam>
__device__ __forceinline__ void turn_pass(int warp) {
    static_assert(kTeam == 2, "one barrier per warp");
    if (warp == 0)
        asm volatile("bar.arrive 1, 64;" ::: "memory");
    else
        asm volatile("bar.arrive 2, 64;" ::: "memory");
}

// The force sums of particle i (of this lane), and false where the list
// overflowed or a distance lies outside root_quotient's range.  They are those
// of the block's last turn: valid in the warp for which `last` is set.
// Called by the whole block; `idle` is what a warp does while its first
// neighbours are on their way (it is told whether it is the last).
template <int kTeam, int kTurn, typename Idle>
__device__ __forceinline__ bool force_team(uint32_t i, const uint32_t* __restrict__ nbr_count,
                                           const uint32_t* __restrict__ nbr, const float4* __restrict__ pv, uint32_t n,
                                           float h, ForceTeamShared& sh, PairAcc& a, bool& last, Idle&& idle) {
    static_assert(kTurn % 2 == 0, "neighbours are taken in twos");
    const int lane = (int)(threadIdx.x & 31u), part = (int)(threadIdx.x / 32u);
    const int next_part = part + 1 < kTeam ? part + 1 : 0;
    // the first turn's entries, before the count that says which of them are
    // the list's own is there
    const uint32_t* lst = nbr + nbr_index(i, (uint32_t)part * kTurn);
    uint32_t e[kTurn];
#pragma unroll
    for (int u = 0; u < kTurn; ++u) e[u] = __ldg(lst + u * kNbTile);
    const uint32_t cnt = __ldg(nbr_count + i);
    PairRec me, r[kTurn];
    ld_rec<true>(pv + 2 * (size_t)i, me);
    const bool listed = cnt <= (uint32_t)kNbCap;
    const uint32_t used = listed ? cnt : 0u;
    const uint32_t turns = max((__reduce_max_sync(0xffffffffu, used) + kTurn - 1) / kTurn, 1u);  // of every warp
    last = (turns - 1) % kTeam == (uint32_t)part;
    uint32_t k = (uint32_t)part * kTurn;
    // the turn's neighbours, or past the list the particle itself, whose terms are exact zeros
    auto gather = [&]() {
#pragma unroll
        for (int u = 0; u < kTurn; ++u)
            ld_rec<true>(pv + 2 * (size_t)(k + u < used ? checked_index(e[u], n) : i), r[u]);
    };
    auto entries = [&]() {  // of the warp's next turn
        k += kTeam * kTurn;
        lst += kTeam * kTurn * kNbTile;
        if (k < used) {
#pragma unroll
            for (int u = 0; u < kTurn; ++u) e[u] = __ldg(lst + u * kNbTile);
        }
    };
    gather();
    entries();
    idle(last);
    const float2 x = unpack(me.x), y = unpack(me.y), z = unpack(me.z);
    const F2 nx = f2(-x.x, -x.y), ny = f2(-y.x, -y.y), nz = f2(-z.x, -z.y), hh = f2(h, h);
    const float pi = unpack(me.pw).x;
    uint32_t small = 0xffffffffu;
    F2 sx = f2(0.f, 0.f), sy = sx, sz = sx;
#pragma unroll 1
    for (uint32_t t = (uint32_t)part; t < turns; t += kTeam) {
        F2 dx[kTurn], dy[kTurn], dz[kTurn], w[kTurn];
#pragma unroll
        for (int u = 0; u < kTurn; u += 2) {
            const PairRec &ra = r[u], &rb = r[u + 1];
            dx[u] = add2(ra.x, nx), dy[u] = add2(ra.y, ny), dz[u] = add2(ra.z, nz);
            dx[u + 1] = add2(rb.x, nx), dy[u + 1] = add2(rb.y, ny), dz[u + 1] = add2(rb.z, nz);
            const float qa = square3(dx[u], dy[u], dz[u]), qb = square3(dx[u + 1], dy[u + 1], dz[u + 1]);
            small = min(small, min(__float_as_uint(qa) - 1u, __float_as_uint(qb) - 1u));
            const RootQuotient o = root_quotient(hh, qa, qb);
            const float2 hr = unpack(o.hr), pa = unpack(ra.pw), pb = unpack(rb.pw);
            const float wa = hr.x * pa.y, wb = hr.y * pb.y;
            const float sa = ((pi + pa.x) * wa) * o.nq.x, sb = ((pi + pb.x) * wb) * o.nq.y;
            w[u] = f2(qa > 0.f ? sa : 0.f, wa);
            w[u + 1] = f2(qb > 0.f ? sb : 0.f, wb);
        }
        gather();
        entries();
        if (t > 0) {
            turn_wait<kTeam>(part);
            const float2 ux = sh.sum[0][lane], uy = sh.sum[1][lane], uz = sh.sum[2][lane];
            small = min(small, sh.small[lane]);
            sx = f2(ux.x, ux.y), sy = f2(uy.x, uy.y), sz = f2(uz.x, uz.y);
        }
#pragma unroll
        for (int u = 0; u < kTurn; ++u) {
            sx = fma2(w[u], dx[u], sx);
            sy = fma2(w[u], dy[u], sy);
            sz = fma2(w[u], dz[u], sz);
        }
        if (t + 1 < turns) {
            sh.sum[0][lane] = unpack(sx);
            sh.sum[1][lane] = unpack(sy);
            sh.sum[2][lane] = unpack(sz);
            sh.small[lane] = small;
            turn_pass<kTeam>(next_part);
        }
    }
    const float2 ux = unpack(sx), uy = unpack(sy), uz = unpack(sz);
    a = PairAcc{ux.x, uy.x, uz.x, ux.y, uy.y, uz.y};
    return listed && small >= __float_as_uint(kFastR2Min) - 1u && h >= kFastHMin && h <= kFastHMax;
}

}  // namespace sf
