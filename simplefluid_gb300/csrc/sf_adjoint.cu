// sf_adjoint.cu — hand-written adjoint of the SPH sub-step and of the CIC
// histogram loss (sm_103a).
//
// The neighbour structure of each step is held fixed (piecewise constant):
// the backward pass re-runs each segment forward from a checkpoint, recording
// per step the sorted state, density/pressure, the neighbour lists and the
// force sums (AP, AV), then walks the steps in reverse.  One step's adjoint is
// three gather passes over the recorded neighbours, so every accumulation is
// per particle, deterministic and free of atomics on particle data:
//   P1  integration (symplectic Euler, box clamp with restitution) and the
//       acceleration's own inputs: a = (cp AP + cv AV) inv + g;
//   P2  force pair terms in both orientations of every pair (spiky pressure,
//       symmetrised weights, viscosity), then rho_bar from 1/rho and the EOS;
//   P4  poly6 density terms onto positions; adjoints written back by particle.
// Adjoint vectors between steps live in caller-index space (index = original
// particle id), so the per-step re-sort needs no explicit adjoint permutation.
// Scalar gradients (viscosity, stiffness) are reduced per block in double,
// then summed in block order by one block: bit-reproducible.
//
// The CPU oracle (oracle/sph_oracle.cpp, adjoint_step) performs the same
// operations in the same order.
#include "sf_device.cuh"

namespace sf {
namespace {

constexpr int kAdjBlock = 128, kAdjForceBlock = 64;
constexpr int kAdjBatch = 4;  // neighbours P4 gathers at a time

__device__ __forceinline__ float dot3f(float ax, float ay, float az, float bx, float by, float bz) {
    return fmaf(az, bz, fmaf(ay, by, ax * bx));
}

// P1: per sorted particle.  Outputs the 32-byte record abrec = apb = cp tb
// beside avb = cv tb in each axis, then (inv_bar, cv_bar); and xdir/vdir = the
// integration's direct adjoints.
__global__ void __launch_bounds__(kAdjBlock)
    k_adj_integrate(const float4* __restrict__ pos, const float4* __restrict__ vel, const float2* __restrict__ pr,
                    const float4* __restrict__ sums, uint32_t n, SimConst c, const float4* __restrict__ Xb,
                    const float4* __restrict__ Vb, float4* __restrict__ abrec, float4* __restrict__ xdir,
                    float4* __restrict__ vdir) {
    grid_dependency_wait();
    allow_dependents();
    const uint32_t i = blockIdx.x * kAdjBlock + threadIdx.x;
    if (i >= n) return;
    const float4 x4 = pos[i], v4 = vel[i];
    const uint32_t id = __float_as_uint(x4.w);
    const float inv = pr[i].y;
    const float4 AP = sums[2 * (size_t)i], AV = sums[2 * (size_t)i + 1];
    const float4 xb4 = Xb[id], vb4 = Vb[id];
    const float xs[3] = {x4.x, x4.y, x4.z}, vs[3] = {v4.x, v4.y, v4.z};
    const float aps[3] = {AP.x, AP.y, AP.z}, avs[3] = {AV.x, AV.y, AV.z};
    const float xbs[3] = {xb4.x, xb4.y, xb4.z}, vbs[3] = {vb4.x, vb4.y, vb4.z};
    float t[3], tb[3], ab[3], xd[3], vd[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        t[a] = fmaf(c.cp, aps[a], c.cv * avs[a]);
        const float acc = fmaf(t[a], inv, c.g[a]);
        const float vpre = fmaf(c.dt, acc, vs[a]);
        const float xpre = fmaf(c.dt, vpre, xs[a]);
        const bool lo = xpre < c.lo[a], hi = xpre > c.hi[a];
        const bool pass = !lo && !hi;
        const float sv = ((lo && vpre < 0.f) || (hi && vpre > 0.f)) ? -c.e : 1.f;
        const float xbpre = pass ? xbs[a] : 0.f;
        const float vbpre = fmaf(sv, vbs[a], c.dt * xbpre);
        xd[a] = xbpre;
        vd[a] = vbpre;
        ab[a] = c.dt * vbpre;
        tb[a] = ab[a] * inv;
    }
    const float invb = dot3f(ab[0], ab[1], ab[2], t[0], t[1], t[2]);
    const float cvb = dot3f(tb[0], tb[1], tb[2], avs[0], avs[1], avs[2]);
    st8(abrec + 2 * (size_t)i, make_float4(c.cp * tb[0], c.cv * tb[0], c.cp * tb[1], c.cv * tb[1]),
        make_float4(c.cp * tb[2], c.cv * tb[2], invb, cvb));
    xdir[i] = make_float4(xd[0], xd[1], xd[2], 0.f);
    vdir[i] = make_float4(vd[0], vd[1], vd[2], 0.f);
}

// dp/drho and dp/dk of the equation of state (0 where the clamp is active).
__device__ __forceinline__ void eos_derivs(const SimConst& c, float rho, float& dpdrho, float& dpdk) {
    float ppre, dr, dk;
    if (c.eos == SF_EOS_TAIT) {
        const float x = rho * c.inv_rho0;
        const float x2 = x * x;
        const float x4 = x2 * x2;
        const float x6 = x4 * x2;
        const float x7 = x6 * x;
        ppre = c.k * (x7 - 1.f);
        dr = (7.f * c.k) * (x6 * c.inv_rho0);
        dk = x7 - 1.f;
    } else {
        ppre = c.k * (rho - c.rho0);
        dr = c.k;
        dk = rho - c.rho0;
    }
    const bool act = c.attractive || ppre > 0.f;
    dpdrho = act ? dr : 0.f;
    dpdk = act ? dk : 0.f;
}

// The pair sums of P2 for particle k: x_bar and v_bar of the force terms in
// both orientations, p_bar and inv_bar.
struct AdjSums {
    float xb[3] = {0.f, 0.f, 0.f}, vb[3] = {0.f, 0.f, 0.f}, pb = 0.f, inv = 0.f;
};
// What P2 knows of a particle: (x, vx) .. (z, vz), (p, 1/rho), and P1's
// (apb, avb) of the axes, (inv_bar, cv_bar).
struct AdjRec {
    PairRec s, a;
};
__device__ __forceinline__ void ld_adj(const float4* __restrict__ pv, const float4* __restrict__ ab, uint32_t j,
                                       AdjRec& r) {
    ld_rec<true>(pv + 2 * (size_t)j, r.s);
    ld_rec<true>(ab + 2 * (size_t)j, r.a);
}

// Terms of neighbour j (not k itself), with the compiler's root and divisions.
__device__ __forceinline__ void adj_pair(float h, const AdjRec& k, const AdjRec& j, AdjSums& o) {
    const float2 ek[3] = {unpack(k.s.x), unpack(k.s.y), unpack(k.s.z)}, ck[3] = {unpack(k.a.x), unpack(k.a.y), unpack(k.a.z)};
    const float2 ej[3] = {unpack(j.s.x), unpack(j.s.y), unpack(j.s.z)}, cj[3] = {unpack(j.a.x), unpack(j.a.y), unpack(j.a.z)};
    const float pk = unpack(k.s.pw).x, invk = unpack(k.s.pw).y, pj = unpack(j.s.pw).x, invj = unpack(j.s.pw).y;
    const float d0 = ek[0].x - ej[0].x, d1 = ek[1].x - ej[1].x, d2 = ek[2].x - ej[2].x;
    const float r2 = fmaf(d2, d2, fmaf(d1, d1, d0 * d0));
    const float r = sqrtf(r2);
    const float hr = h - r;
    const float dv0 = ej[0].y - ek[0].y, dv1 = ej[1].y - ek[1].y, dv2 = ej[2].y - ek[2].y;
    const float ps = pk + pj;
    // orientation A: k is i, j the neighbour
    const float wkj = hr * invj;
#pragma unroll
    for (int q = 0; q < 3; ++q) o.vb[q] = fmaf(-wkj, ck[q].y, o.vb[q]);
    float wb = dot3f(ck[0].y, ck[1].y, ck[2].y, dv0, dv1, dv2);
    float rb = 0.f;
    // orientation B: j is i, k the neighbour
    const float wjk = hr * invk;
#pragma unroll
    for (int q = 0; q < 3; ++q) o.vb[q] = fmaf(wjk, cj[q].y, o.vb[q]);
    float wb2 = -dot3f(cj[0].y, cj[1].y, cj[2].y, dv0, dv1, dv2);
    float rb2 = 0.f;
    if (r > 0.f) {
        const float q = hr / r;
        const float S = (ps * wkj) * q;
        const float Sb = dot3f(ck[0].x, ck[1].x, ck[2].x, d0, d1, d2);
#pragma unroll
        for (int x = 0; x < 3; ++x) o.xb[x] = fmaf(S, ck[x].x, o.xb[x]);
        o.pb = fmaf(Sb, wkj * q, o.pb);
        wb = fmaf(Sb, ps * q, wb);
        const float qb = Sb * (ps * wkj);
        rb = -((qb * h) / r2);
        const float S2 = (ps * wjk) * q;
        const float Sb2 = -dot3f(cj[0].x, cj[1].x, cj[2].x, d0, d1, d2);
#pragma unroll
        for (int x = 0; x < 3; ++x) o.xb[x] = fmaf(-S2, cj[x].x, o.xb[x]);
        o.pb = fmaf(Sb2, wjk * q, o.pb);
        wb2 = fmaf(Sb2, ps * q, wb2);
        const float qb2 = Sb2 * (ps * wjk);
        rb2 = -((qb2 * h) / r2);
    }
    rb = fmaf(-wb, invj, rb);
    o.inv = fmaf(wb2, hr, o.inv);
    rb2 = fmaf(-wb2, invk, rb2);
    if (r > 0.f) {
        const float g = (rb + rb2) / r;
        o.xb[0] = fmaf(g, d0, o.xb[0]);
        o.xb[1] = fmaf(g, d1, o.xb[1]);
        o.xb[2] = fmaf(g, d2, o.xb[2]);
    }
}

// The same of two neighbours a and b at once (`va`, `vb` clear: none, its
// terms are zeros), a's added before b's, without the compiler's root and
// divisions (see root_recip; the range is kFastR2Min to kAdjHMax^2, the numerators
// are zero or at least kAdjTiny): the packed halves are the position and the
// velocity side of one neighbour in the differences, dot products and sums,
// and the two neighbours in between.  Signs differ from adj_pair's where that
// saves an operation; every rounding is the same.
constexpr float kAdjTiny = 7.8886091e-31f;  // 2^-100: quotients of smaller numerators go to adj_pair
constexpr float kAdjHMax = 1024.f;
struct AdjPairSums {
    F2 x, y, z;              // (x_bar, v_bar)
    float pb = 0.f, inv = 0.f;
    float nearest = 1.f;     // smallest r^2 so far
    uint32_t tiny = ~0u;     // smallest 2 bits(|numerator|) - 1 so far (numerators that are zero pass)
};
__device__ __forceinline__ void adj_pair2(float h, const F2 k[3], float pk, F2 invk, const PairRec& ck, const AdjRec& a,
                                          const AdjRec& b, bool va, bool vb, AdjPairSums& o) {
    const F2 flip = f2(-1.f, 1.f);
    // (xk - xj, vj - vk); k holds (xk, -vk)
    const F2 ax = fma2(a.s.x, flip, k[0]), ay = fma2(a.s.y, flip, k[1]), az = fma2(a.s.z, flip, k[2]);
    const F2 bx = fma2(b.s.x, flip, k[0]), by = fma2(b.s.y, flip, k[1]), bz = fma2(b.s.z, flip, k[2]);
    const float ra = va ? square3(ax, ay, az) : 1.f, rb = vb ? square3(bx, by, bz) : 1.f;
    o.nearest = fminf(o.nearest, fminf(ra, rb));
    const F2 n2 = f2(-ra, -rb), y0 = f2(rsqrt_approx(ra), rsqrt_approx(rb));
    const RootRecip root = root_recip(n2, y0);
    const F2 nr = root.nr, y = root.y, y2 = recip_step(n2, mul2(y0, y0));  // -r, 1 / r, 1 / r^2
    const float2 hr1 = unpack(add2(f2(h, h), nr));
    const F2 hr = f2(va ? hr1.x : 0.f, vb ? hr1.y : 0.f);  // zero weights where there is no neighbour
    const F2 q = quotient2(hr, nr, y);
    const float2 pa = unpack(a.s.pw), pb = unpack(b.s.pw);
    const F2 ps = f2(pk + pa.x, pk + pb.x), inv = f2(pa.y, pb.y);
    const F2 wkj = mul2(hr, inv), wjk = mul2(hr, invk);
    // (Sb, wb) and minus (Sb2, wb2) of each neighbour
    const float2 fa = unpack(fma2(ck.z, az, fma2(ck.y, ay, mul2(ck.x, ax))));
    const float2 fb = unpack(fma2(ck.z, bz, fma2(ck.y, by, mul2(ck.x, bx))));
    const float2 ga = unpack(fma2(a.a.z, az, fma2(a.a.y, ay, mul2(a.a.x, ax))));
    const float2 gb = unpack(fma2(b.a.z, bz, fma2(b.a.y, by, mul2(b.a.x, bx))));
    const F2 Sb = f2(fa.x, fb.x), nSb2 = f2(ga.x, gb.x);
    const F2 t1 = mul2(ps, wkj), t2 = mul2(ps, wjk), pq = mul2(ps, q);
    const F2 wb = fma2(Sb, pq, f2(fa.y, fb.y)), nwb2 = fma2(nSb2, pq, f2(ga.y, gb.y));
    const F2 hh = f2(h, h);
    const F2 n1 = mul2(mul2(Sb, t1), hh), m1 = mul2(mul2(nSb2, t2), hh);
    const F2 nrb = fma2(wb, inv, quotient2(n1, n2, y2));    // minus rb
    const F2 rb2 = fma2(nwb2, invk, quotient2(m1, n2, y2));
    const F2 gn = fma2(nrb, f2(-1.f, -1.f), rb2);           // rb + rb2
    const float2 g = unpack(quotient2(gn, nr, y));
    auto seen = [&](F2 v) {
        const float2 u = unpack(v);
        o.tiny = min(o.tiny, min(2u * __float_as_uint(u.x) - 1u, 2u * __float_as_uint(u.y) - 1u));
    };
    seen(n1);
    seen(m1);
    seen(gn);
    const float2 S = unpack(mul2(t1, q)), S2 = unpack(mul2(t2, q)), w1 = unpack(wkj), w2 = unpack(wjk);
    const float2 kq = unpack(mul2(wkj, q)), jq = unpack(mul2(wjk, q)), hru = unpack(hr), nw = unpack(nwb2);
    auto add = [&](F2 ex, F2 ey, F2 ez, const PairRec& cj, float s, float s2, float wk, float wj, float gg) {
        const F2 u = f2(s, -wk), v = f2(-s2, wj);
        auto axis = [&](F2& sum, F2 c, F2 cn, F2 e) {
            const float2 t = unpack(fma2(v, cn, fma2(u, c, sum)));
            sum = f2(fmaf(gg, unpack(e).x, t.x), t.y);
        };
        axis(o.x, ck.x, cj.x, ex);
        axis(o.y, ck.y, cj.y, ey);
        axis(o.z, ck.z, cj.z, ez);
    };
    add(ax, ay, az, a.a, S.x, S2.x, w1.x, w2.x, g.x);
    o.pb = fmaf(-ga.x, jq.x, fmaf(fa.x, kq.x, o.pb));
    o.inv = fmaf(-nw.x, hru.x, o.inv);
    add(bx, by, bz, b.a, S.y, S2.y, w1.y, w2.y, g.y);
    o.pb = fmaf(-gb.x, jq.y, fmaf(fb.x, kq.y, o.pb));
    o.inv = fmaf(-nw.y, hru.y, o.inv);
}

// P2: force pair terms of every pair in both orientations, then the density
// adjoint of the particle.  Outputs xrb = (x, y, z, rho_bar), P4's gather
// record, xf = (force x_bar, k_bar) and vf.
// A neighbour is two 32-byte records, each one 256-bit load: the step's
// gather record and P1's.
// 65,536 particles are 13.5 warps per SM, so the pass takes as long as a
// thread's chain: two neighbours share each of its steps (adj_pair2, half the
// instructions of adj_pair, none of its branches), and the next two's records
// are on their way meanwhile.  47 -> 31 us by the first, -> 24 us by the
// second (65,536 disordered particles), 84 -> 43 us at 150,000; blocks of 64
// threads spread the warps evenly (32: 26 us).
template <int kReach>
__global__ void __launch_bounds__(kAdjForceBlock)
    k_adj_forces(const float4* __restrict__ pos, const float4* __restrict__ pv, const float* __restrict__ rho,
                 const uint32_t* __restrict__ cs, const uint32_t* __restrict__ nbr, const uint32_t* __restrict__ cnt,
                 uint32_t n, SimConst c, const float4* __restrict__ ab, float4* __restrict__ xrb,
                 float4* __restrict__ xf, float4* __restrict__ vf) {
    grid_dependency_wait();
    allow_dependents();
    const uint32_t k = blockIdx.x * kAdjForceBlock + threadIdx.x;
    if (k >= n) return;
    const uint32_t m = __ldg(cnt + k);
    const uint32_t* lst = nbr + nbr_index(k, 0);  // slot s at lst[s * kNbTile]
    uint32_t ea = __ldg(lst), eb = __ldg(lst + kNbTile);
    AdjRec me;
    ld_adj(pv, ab, k, me);
    const float2 x = unpack(me.s.x), y = unpack(me.s.y), z = unpack(me.s.z), pw = unpack(me.s.pw);
    AdjSums o;
    bool summed = false;
    if (m <= (uint32_t)kNbCap) {
        const F2 mine[3] = {f2(x.x, -x.y), f2(y.x, -y.y), f2(z.x, -z.y)};
        AdjPairSums p;
        p.x = p.y = p.z = f2(0.f, 0.f);
        // The next two neighbours' records and the entries after them are on
        // their way while two are processed.  The list holds the particle
        // itself (no terms); slots past the count hold stale values, never used.
        uint32_t ja = m ? checked_index(ea, n) : k, jb = 1 < m ? checked_index(eb, n) : k;
        AdjRec a, b;
        ld_adj(pv, ab, ja, a);
        ld_adj(pv, ab, jb, b);
        lst += 2 * kNbTile;
        ea = __ldg(lst);
        eb = __ldg(lst + kNbTile);
#pragma unroll 1
        for (uint32_t s = 0; s < m; s += 2) {
            const bool va = ja != k, vb = jb != k;
            ja = s + 2 < m ? checked_index(ea, n) : k;
            jb = s + 3 < m ? checked_index(eb, n) : k;
            AdjRec na, nb;
            ld_adj(pv, ab, ja, na);
            ld_adj(pv, ab, jb, nb);
            lst += s + 4 < m ? 2 * kNbTile : 0;
            ea = __ldg(lst);
            eb = __ldg(lst + kNbTile);
            adj_pair2(c.h, mine, pw.x, f2(pw.y, pw.y), me.a, a, b, va, vb, p);
            a = na;
            b = nb;
        }
        const float2 sx = unpack(p.x), sy = unpack(p.y), sz = unpack(p.z);
        o = AdjSums{{sx.x, sy.x, sz.x}, {sx.y, sy.y, sz.y}, p.pb, p.inv};
        summed = c.h >= kFastHMin && c.h <= kAdjHMax && p.nearest >= kFastR2Min &&
                 p.tiny >= 2u * __float_as_uint(kAdjTiny) - 1u && isfinite(sx.x + sy.x + sz.x);
    }
    if (!summed) {
        o = AdjSums{};
        for_candidates_rolled<kReach>(c, cs, pos, n, x.x, y.x, z.x, [&](uint32_t j, const float4& xp) {
            if (j == k) return;
            const float dx = x.x - xp.x, dy = y.x - xp.y, dz = z.x - xp.z;
            if (!(fmaf(dz, dz, fmaf(dy, dy, dx * dx)) < c.h2)) return;
            AdjRec r;
            ld_adj(pv, ab, j, r);
            adj_pair(c.h, me, r, o);
        });
    }
    const float ib = unpack(me.a.pw).x + o.inv;
    float dpdrho, dpdk;
    eos_derivs(c, rho[k], dpdrho, dpdk);
    xrb[k] = make_float4(x.x, y.x, z.x, fmaf(o.pb, dpdrho, -((ib * pw.y) * pw.y)));
    xf[k] = make_float4(o.xb[0], o.xb[1], o.xb[2], o.pb * dpdk);
    vf[k] = make_float4(o.vb[0], o.vb[1], o.vb[2], 0.f);
}

// P4: poly6 density terms onto positions; the step's input adjoints are
// written back by particle id.
// Also reduces the step's scalar adjoints (cv_bar in the ab record's last word, k_bar in xf.w) per
// block, in thread order, into partial[blockIdx.x].
// Four neighbours in flight: 48 -> 39 registers and, with P1 and P2 chained,
// 40 steps' forward and adjoint 5.36 -> 5.28 ms at 65,536 particles.  This
// pass is launched plainly: chained, its shared memory arrives on the SMs
// beside P2's last blocks and costs 7.5 us a step.
template <int kReach>
__global__ void __launch_bounds__(kAdjBlock)
    k_adj_density(const float4* __restrict__ pos, const uint32_t* __restrict__ cs, const uint32_t* __restrict__ nbr,
                  const uint32_t* __restrict__ cnt, uint32_t n, SimConst c, float m6cd, const float4* __restrict__ xrb,
                  const float4* __restrict__ xdir, const float4* __restrict__ vdir, const float4* __restrict__ xf,
                  const float4* __restrict__ vf, const float4* __restrict__ ab, float4* __restrict__ Xb,
                  float4* __restrict__ Vb, double2* __restrict__ partial) {
    __shared__ double s0[kAdjBlock], s1[kAdjBlock];
    allow_dependents();
    const uint32_t k = blockIdx.x * kAdjBlock + threadIdx.x;
    s0[threadIdx.x] = k < n ? (double)ab[2 * (size_t)k + 1].w : 0.0;
    s1[threadIdx.x] = k < n ? (double)xf[k].w : 0.0;
    __syncthreads();
    for (int o = kAdjBlock / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) {
            s0[threadIdx.x] += s0[threadIdx.x + o];
            s1[threadIdx.x] += s1[threadIdx.x + o];
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = make_double2(s0[0], s1[0]);
    if (k >= n) return;
    const uint32_t m = __ldg(cnt + k);
    const uint32_t* lst = nbr + nbr_index(k, 0);  // slot s at lst[s * kNbTile]
    uint32_t e[kAdjBatch];
#pragma unroll
    for (int u = 0; u < kAdjBatch; ++u) e[u] = __ldg(lst + u * kNbTile);
    const float4 xk = pos[k];
    const float rbk = xrb[k].w;
    float x0 = 0.f, x1 = 0.f, x2 = 0.f;
    auto add = [&](const float4& xj, bool other) {  // xj: position and rho_bar in one load
        const float d0 = xk.x - xj.x, d1 = xk.y - xj.y, d2 = xk.z - xj.z;
        const float r2 = fmaf(d2, d2, fmaf(d1, d1, d0 * d0));
        const float q = c.h2 - r2;
        const float sc = other ? (rbk + xj.w) * (q * q) : 0.f;
        x0 = fmaf(sc, d0, x0);
        x1 = fmaf(sc, d1, x1);
        x2 = fmaf(sc, d2, x2);
    };
    if (m <= (uint32_t)kNbCap) {
        // kAdjBatch neighbours are gathered while the next entries are loaded.
        // The list holds the particle itself, which has no term and stands in
        // past the end; slots past the count hold stale values, never used.
#pragma unroll 1
        for (uint32_t s = 0; s < m; s += kAdjBatch) {
            float4 xj[kAdjBatch];
            bool other[kAdjBatch];
#pragma unroll
            for (int u = 0; u < kAdjBatch; ++u) {
                const uint32_t j = s + u < m ? checked_index(e[u], n) : k;
                other[u] = j != k;
                xj[u] = ldg4(xrb + j);
            }
            if (s + kAdjBatch < m) lst += kAdjBatch * kNbTile;
#pragma unroll
            for (int u = 0; u < kAdjBatch; ++u) e[u] = __ldg(lst + u * kNbTile);
#pragma unroll
            for (int u = 0; u < kAdjBatch; ++u) add(xj[u], other[u]);
        }
    } else {
        for_candidates_rolled<kReach>(c, cs, pos, n, xk.x, xk.y, xk.z, [&](uint32_t j, const float4& xp) {
            if (j == k) return;
            const float dx = xk.x - xp.x, dy = xk.y - xp.y, dz = xk.z - xp.z;
            if (fmaf(dz, dz, fmaf(dy, dy, dx * dx)) < c.h2) add(ldg4(xrb + j), true);
        });
    }
    const uint32_t id = __float_as_uint(xk.w);
    const float4 xd = xdir[k], xfk = xf[k], vd = vdir[k], vfk = vf[k];
    Xb[id] = make_float4(fmaf(m6cd, x0, xd.x + xfk.x), fmaf(m6cd, x1, xd.y + xfk.y), fmaf(m6cd, x2, xd.z + xfk.z), 0.f);
    Vb[id] = make_float4(vd.x + vfk.x, vd.y + vfk.y, vd.z + vfk.z, 0.f);
}

// Adds the block partials of `nsteps` steps to acc[0..1].  Eight steps at a
// time, one warp per step: lane l sums blocks l, l + 32, ... in order and a
// fixed shuffle tree combines the lanes; thread 0 then adds the step sums
// last step first (the order the adjoint visits them).  Deterministic.
constexpr int kAccThreads = 256;

__global__ void __launch_bounds__(kAccThreads)
    k_accumulate_scalars(const double2* __restrict__ partial, uint32_t nsteps, uint32_t nblocks,
                         double* __restrict__ acc) {
    constexpr int kWarps = kAccThreads / 32;
    __shared__ double s0[kWarps], s1[kWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double a = 0.0, b = 0.0;
    if (threadIdx.x == 0) {
        a = acc[0];
        b = acc[1];
    }
    for (int64_t hi = (int64_t)nsteps; hi > 0; hi -= kWarps) {
        const int64_t st = hi - 1 - warp;  // the same in every lane of the warp
        double x = 0.0, y = 0.0;
        if (st >= 0) {
            for (uint32_t t = lane; t < nblocks; t += 32) {
                const double2 v = partial[(size_t)st * nblocks + t];
                x += v.x;
                y += v.y;
            }
            for (int o = 16; o > 0; o >>= 1) {
                x += __shfl_down_sync(0xffffffffu, x, o);
                y += __shfl_down_sync(0xffffffffu, y, o);
            }
        }
        if (lane == 0) {
            s0[warp] = x;
            s1[warp] = y;
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            for (int w = 0; w < kWarps && hi - 1 - w >= 0; ++w) {  // steps hi-1, hi-2, ...
                a += s0[w];
                b += s1[w];
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        acc[0] = a;
        acc[1] = b;
    }
}

constexpr int kRedBlock = 256;

// ------------------------------------------------------------------ loss
// CIC (cloud-in-cell) histogram on res^3 cell-centred bins over the box,
// normalised by the particle count.  Deposits are 2^-32 fixed point in 64-bit
// integer atomics, so the histogram does not depend on the order of arrival.
__device__ __forceinline__ void cic(const SimConst& c, const float ext_inv[3], float x, float y, float z, int i0[3],
                                    float w0[3], float w1[3]) {
    const float p3[3] = {x, y, z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float u = (p3[a] - c.bmin[a]) * ext_inv[a] - 0.5f;
        const float fl = floorf(u);
        const float f = u - fl;
        i0[a] = (int)fl;
        w0[a] = 1.f - f;
        w1[a] = f;
    }
}

struct HistDims {
    float inv[3];  // res / extent per axis
    int res;
};

__global__ void k_hist_deposit(const float4* __restrict__ pos, uint32_t n, SimConst c, HistDims hd,
                               unsigned long long* __restrict__ hist) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 x = pos[i];
    int i0[3];
    float w0[3], w1[3];
    cic(c, hd.inv, x.x, x.y, x.z, i0, w0, w1);
    const int R = hd.res;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int ix = i0[0] + (q & 1), iy = i0[1] + ((q >> 1) & 1), iz = i0[2] + ((q >> 2) & 1);
        if (ix < 0 || iy < 0 || iz < 0 || ix >= R || iy >= R || iz >= R) continue;
        const float w = ((q & 1) ? w1[0] : w0[0]) * ((q & 2) ? w1[1] : w0[1]) * ((q & 4) ? w1[2] : w0[2]);
        if (!(w > 0.f)) continue;
        atomicAdd(hist + ((size_t)iz * R + iy) * R + ix, (unsigned long long)llrint((double)w * 4294967296.0));
    }
}

// e[c] = 2 (H_c - T_c) / n and per-block partial sums of (H_c - T_c)^2.
__global__ void __launch_bounds__(kRedBlock)
    k_hist_error(const unsigned long long* __restrict__ hist, const float* __restrict__ target, uint32_t ncells,
                 uint32_t n, float* __restrict__ e2, double* __restrict__ partial) {
    __shared__ double s[kRedBlock];
    const uint32_t cidx = blockIdx.x * kRedBlock + threadIdx.x;
    double sq = 0.0;
    if (cidx < ncells) {
        const double H = (double)hist[cidx] * (1.0 / 4294967296.0) / (double)n;
        const double e = H - (double)target[cidx];
        e2[cidx] = (float)(2.0 * e / (double)n);
        sq = e * e;
    }
    s[threadIdx.x] = sq;
    __syncthreads();
    for (int o = kRedBlock / 2; o > 0; o >>= 1) {
        if ((int)threadIdx.x < o) s[threadIdx.x] += s[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.x] = s[0];
}

// dL/dx of each particle, written by particle id.
__global__ void k_hist_grad(const float4* __restrict__ pos, uint32_t n, SimConst c, HistDims hd,
                            const float* __restrict__ e2, float4* __restrict__ Xb) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 x = pos[i];
    int i0[3];
    float w0[3], w1[3];
    cic(c, hd.inv, x.x, x.y, x.z, i0, w0, w1);
    const int R = hd.res;
    float g0 = 0.f, g1 = 0.f, g2 = 0.f;
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int ix = i0[0] + (q & 1), iy = i0[1] + ((q >> 1) & 1), iz = i0[2] + ((q >> 2) & 1);
        if (ix < 0 || iy < 0 || iz < 0 || ix >= R || iy >= R || iz >= R) continue;
        const float e = e2[((size_t)iz * R + iy) * R + ix];
        const float wx = (q & 1) ? w1[0] : w0[0], wy = (q & 2) ? w1[1] : w0[1], wz = (q & 4) ? w1[2] : w0[2];
        const float sx = (q & 1) ? hd.inv[0] : -hd.inv[0], sy = (q & 2) ? hd.inv[1] : -hd.inv[1],
                    sz = (q & 4) ? hd.inv[2] : -hd.inv[2];
        g0 += e * (sx * (wy * wz));
        g1 += e * (sy * (wx * wz));
        g2 += e * (sz * (wx * wy));
    }
    Xb[__float_as_uint(x.w)] = make_float4(g0, g1, g2, 0.f);
}

}  // namespace

SF_INDEX_CHECK_ACCESSOR(index_check_failures_adjoint)

// ------------------------------------------------------------------ launchers
const char* const kAdjointPassNames[kAdjointPasses] = {"adj_integrate", "adj_forces", "adj_density"};

void launch_adjoint_pass(uint32_t pass, const AdjointStep& st, const SimConst& c, AdjointWork& w, double2* partial,
                         cudaStream_t s) {
    const uint32_t n = st.n;
    if (!n) return;
    const unsigned g = grid_for(n, kAdjBlock);
    if (pass == 0) {
        launch_chained(k_adj_integrate, g, kAdjBlock, s, st.pos, st.vel, st.pr, st.sums, n, c, w.Xb, w.Vb, w.ab, w.xdir,
                       w.vdir);
        return;
    }
    const float m6cd = (float)(-6.0 * (double)c.cd);
    with_reach(c.reach, [&](auto R) {
        constexpr int K = decltype(R)::value;
        if (pass == 1)
            launch_chained(k_adj_forces<K>, grid_for(n, kAdjForceBlock), kAdjForceBlock, s, st.pos, st.pv, st.rho,
                           st.cs, st.nbr, st.cnt, n, c, w.ab, w.xrb, w.xf, w.vf);
        else if (pass == 2)
            k_adj_density<K><<<g, kAdjBlock, 0, s>>>(st.pos, st.cs, st.nbr, st.cnt, n, c, m6cd, w.xrb, w.xdir, w.vdir,
                                                     w.xf, w.vf, w.ab, w.Xb, w.Vb, partial);
    });
}

void launch_adjoint_step(const AdjointStep& st, const SimConst& c, AdjointWork& w, double2* partial,
                         cudaStream_t s) {
    for (uint32_t p = 0; p < kAdjointPasses; ++p) launch_adjoint_pass(p, st, c, w, partial, s);
}

uint32_t adjoint_partial_count(uint32_t n) { return grid_for(n, kAdjBlock); }

void launch_adjoint_accumulate(const double2* partial, uint32_t nsteps, uint32_t n, double* scalars, cudaStream_t s) {
    k_accumulate_scalars<<<1, kAccThreads, 0, s>>>(partial, nsteps, adjoint_partial_count(n), scalars);
}

void launch_histogram_loss(const float4* pos, uint32_t n, const SimConst& c, const float box_ext[3], uint32_t res,
                           const float* target, unsigned long long* hist, float* e2, double* partial, float4* Xb,
                           cudaStream_t s) {
    HistDims hd;
    hd.res = (int)res;
    for (int a = 0; a < 3; ++a) hd.inv[a] = (float)((double)res / (double)box_ext[a]);
    const uint32_t ncells = res * res * res;
    cudaMemsetAsync(hist, 0, (size_t)ncells * sizeof(unsigned long long), s);
    if (n) k_hist_deposit<<<grid_for(n, kBlock), kBlock, 0, s>>>(pos, n, c, hd, hist);
    k_hist_error<<<grid_for(ncells, kRedBlock), kRedBlock, 0, s>>>(hist, target, ncells, n ? n : 1, e2, partial);
    if (n && Xb) k_hist_grad<<<grid_for(n, kBlock), kBlock, 0, s>>>(pos, n, c, hd, e2, Xb);
}

uint32_t histogram_partial_count(uint32_t res) { return grid_for(res * res * res, kRedBlock); }

}  // namespace sf
