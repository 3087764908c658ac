// e4c_fused_ws64.cuh -- the fused stage of the FP64 form for tiles 32 cells
// wide (i) and TJ rows (j), marching in k over a chunk of planes.
//
// The CTA has TJ cell warps (warp = tile row, lane = cell) and two edge warps,
// as the FP32-flux form's kernel (e4c_fused_ws.cuh): the edge warps keep a
// four-slot ring of halo planes in shared memory (cp.async, three planes
// ahead), reconstruct the halo cells around the tile and compute the faces on
// its east and north edges; each cell thread reconstructs its own cell once
// per direction and computes its west, south and top faces.
//
// What bounds it: FP64 instruction issue and the latency of its dependency
// chains (the reference's rounding allows no fused multiply-adds outside the
// quotients), not HBM.
// So the split is chosen for operations and for warps in flight:
//   * per-cell reconstruction: one set of differences, limiter values and MUSCL
//     values per cell and direction (the per-face form computes the
//     differences of a cell for each of its faces);
//   * i-direction values and face fluxes pass between lanes (shuffles), only
//     the j-direction ones through shared memory;
//   * one barrier per plane: what crosses rows is double-buffered, the
//     j-direction values of a plane are made one plane ahead, and the edge
//     warps' loads follow a plan made once per work item, so no warp waits for
//     a phase of its own (with two barriers and the loads decided position by
//     position a third of the stall cycles were barrier waits);
//   * the halo planes come by cp.async, the conserved state is prefetched into
//     L2 by the edge warps and loaded before the barrier.
// 16 warps at 128 registers: fewer registers spill, more of them cost warps
// (20 warps at 96 registers measured 6.7 ms/step where 16 took 5.8).
// Measured on the 256^3 block, HLLC, per step: 7.53 ms for the per-face kernel
// with the 32x8 tile and 32-plane chunks, 6.57 with its best tile (32x16; both
// before the batched quotients, 6.47 with them); 5.99 here with 32x8, 5.57 with
// 32x14, 5.46 with that and 40-plane chunks.  128^3, 32x14 (ncu): 31 % of the
// instructions are FP64, 0.47 issued per cycle and scheduler, stalls led by the
// FP64 chains (2.2 cycles per instruction issued) and the barrier (1.2).
//
// The arithmetic is that of the per-face kernel (e4c_fused.cuh), operation for
// operation, so results are the same bits.  On a uniform grid the left state of
// a face depends on its left cell and that cell's two neighbours alone:
// interp_l2r2_scalar (onedinterp.d:136-162) with equal lengths gives the cell's
// value at its high face as q + (s a0) (b two + a len) and at its low face as
// q - (s a0) (b len + a two), with a, b the scaled differences, s the van
// Albada value, a0 = 0.5 len / (len + 2 len + len), two = 2 len + len.
#pragma once

#include "e4c_fused_ws.cuh"

namespace e4c {
namespace ws64 {

using ws::NE;
using ws::NEW;
using ws::PI;
using ws::TI;

// resident warps per SM the launch bounds aim at
#ifndef E4C_WS64_WARPS
#define E4C_WS64_WARPS 16
#endif

template <int TJ>
struct Lay {
    static_assert(PI * (TJ + 4) <= 16 * NE, "tile too tall for the edge threads' fixups");
    static constexpr int PLANE = PI * (TJ + 4);   // one field of one plane
    static constexpr int NR = (TJ + 1) * TI;      // rows -1..TJ-1, or j-faces 0..TJ
    static constexpr int NL = TJ * TI;            // the tile's cells
    // (two slots by plane parity for what one plane's threads read while others
    // already write the next plane's)
    static constexpr int o_hj = 20 * PLANE;       // ring: 4 slots x 5 fields
    static constexpr int o_fj = o_hj + 2 * 5 * NR;    // after [2][5] j-direction high values
    static constexpr int o_a = o_fj + 2 * 5 * NR;     // [2][5] j-face fluxes
    static constexpr int o_fb = o_a + 2 * NR;         // [2] sound speeds, rows -1..TJ-1
    static constexpr int o_hw = o_fb + 5 * NL;        // [5] fluxes of the cells' bottom faces
    static constexpr int o_aw = o_hw + 2 * 5 * TJ;    // [2][5] i-direction high values of column -1
    static constexpr int o_fe = o_aw + 2 * TJ;        // [2] sound speeds there
    static constexpr int o_plan = o_fe + 2 * 5 * TJ;  // [2][5] fluxes of the tile's east faces
    static constexpr int words = o_plan + (PLANE + 1) / 2;   // plan_tile's table (ints)
    static constexpr size_t bytes = sizeof(double) * size_t(words);
    static constexpr int threads = 32 * (TJ + NEW);
    // CTAs per SM: as many as the shared memory holds (228 KB per SM, 1 KB
    // reserved per CTA)
    static constexpr int fit = int((228 * 1024) / (bytes + 1024));
    static constexpr int want = E4C_WS64_WARPS / (TJ + NEW) > 0 ? E4C_WS64_WARPS / (TJ + NEW) : 1;
    static constexpr int min_blocks = fit < want ? fit : want;
    static_assert(fit >= 1, "tile too tall for the shared memory");
};

// l2r2_prepare (onedinterp.d:118-133) for equal lengths
struct Weights {
    double tw, a0, two, len;
};

// The MUSCL values of N scalars at a cell's high and low faces from the cell
// (q0) and its neighbours below and above (qm, qp) along one direction.
template <int N>
__device__ __forceinline__ void muscl_cell(const Weights& w, bool lim, const double* qm,
                                           const double* q0, const double* qp, double* hi,
                                           double* lo) {
    double a[N], b[N], s[N];
#pragma unroll
    for (int f = 0; f < N; ++f) {
        a[f] = (q0[f] - qm[f]) * w.tw;
        b[f] = (qp[f] - q0[f]) * w.tw;
        s[f] = 1.0;
    }
    if (lim) {
        double nu[N], de[N];
#pragma unroll
        for (int f = 0; f < N; ++f) {
            const double ab = a[f] * b[f];
            nu[f] = ab + fabs(ab) + 1.0e-12;
            de[f] = a[f] * a[f] + b[f] * b[f] + 1.0e-12;
        }
        fdiv_va<N>(nu, de, s);
    }
#pragma unroll
    for (int f = 0; f < N; ++f) {
        const double sa = s[f] * w.a0;
        hi[f] = q0[f] + sa * (b[f] * w.two + a[f] * w.len);
        lo[f] = q0[f] - sa * (b[f] * w.len + a[f] * w.two);
    }
}

// A face from its two cells' values (order rho, vx, vy, vz, u, global frame):
// hL the left cell's high value, cL the left cell, aL its sound speed; lR, cR,
// aR on the right.  The operations of face_flux (e4c_fused.cuh).
template <int FLUX, int DIR>
__device__ __forceinline__ void face_cells(const double* hL, const double* cL, double aL,
                                           const double* lR, const double* cR, double aR,
                                           const FluxOpts& o, int shock, double* F) {
    Prim<double, 1> Lf, Rt;
    double l[5], r[5];
#pragma unroll
    for (int f = 0; f < 5; ++f) {
        l[f] = hL[f];
        r[f] = lR[f];
        if (o.order2 && o.clip) {
            l[f] = clip_to_limits(l[f], cL[f], cR[f]);
            r[f] = clip_to_limits(r[f], cL[f], cR[f]);
        }
    }
    if (o.order2) {
        // a failed thermo update falls back on the cell (onedinterp.d:1039-1068)
        if (l[4] <= 0.0 || l[0] <= 0.0) {
#pragma unroll
            for (int f = 0; f < 5; ++f) l[f] = cL[f];
        }
        if (r[4] <= 0.0 || r[0] <= 0.0) {
#pragma unroll
            for (int f = 0; f < 5; ++f) r[f] = cR[f];
        }
    }
    Lf.rho = l[0]; Lf.vel = {l[1], l[2], l[3]}; Lf.u = l[4]; Lf.a = aL;
    Rt.rho = r[0]; Rt.vel = {r[1], r[2], r[3]}; Rt.u = r[4]; Rt.a = aR;
    Lf.massf[0] = Rt.massf[0] = 1.0;
    Lf.p = Lf.rho * o.gas.Rgas * (Lf.u * o.gas.Cvinv);
    Rt.p = Rt.rho * o.gas.Rgas * (Rt.u * o.gas.Cvinv);
    axis_to_local<DIR>(Lf.vel);
    axis_to_local<DIR>(Rt.vel);
    if (FLUX == 1) {
        hllc<double, 1, 0>(Lf, Rt, F);
    } else if (FLUX == 2) {
        hanel<double, 1, 0>(Lf, Rt, F);
    } else if (FLUX == 3) {
        // adaptive_hanel_ausmdv (fluxcalc.d:824-838)
        bool use_hanel = false;
        if (shock) {
            const double sound = 0.5 * (Lf.a + Rt.a);
            const double shear_y = fabs(Lf.vel.y - Rt.vel.y) / sound;
            const double shear_z = fabs(Lf.vel.z - Rt.vel.z) / sound;
            use_hanel = fmax(shear_y, shear_z) <= o.shear_tol;
        }
        if (use_hanel) hanel<double, 1, 0>(Lf, Rt, F);
        else ausmdv<double, 1, 0>(Lf, Rt, F);
    } else {
        ausmdv<double, 1, 0>(Lf, Rt, F);
    }
    V3<double> m{F[1], F[2], F[3]};
    axis_to_global<DIR>(m);
    F[1] = m.x; F[2] = m.y; F[3] = m.z;
}

__device__ __forceinline__ double sound_speed(double u, const GasConsts& g) {
    return sqrt(g.gamma * g.Rgas * (u * g.Cvinv));
}

// The sound speed of a cell whose value is not that of its u: while the
// uploaded sound speed is in use, and beyond an inflow face.  (gi, gj, gk) is
// an interior cell or lies beyond exactly one face; elsewhere the value is
// never used.  Out of line: only the first stage after an upload and the
// cells beyond a boundary come here.
static __device__ __noinline__ double special_sound_speed(const FusedDesc* __restrict__ descs,
                                                          const FusedDesc& d, int stage,
                                                          int use_a0, int gi, int gj, int gk,
                                                          double a_of_u) {
    const bool oi = gi < 0 || gi >= d.ni;
    const bool oj = gj < 0 || gj >= d.nj;
    const bool ok = gk < 0 || gk >= d.nk;
    if (int(oi) + int(oj) + int(ok) > 1) return a_of_u;
    int which = -1, layer = 0;
    if (oi) {
        if (gi < 0) { which = WEST; layer = -gi - 1; }
        else { which = EAST; layer = gi - d.ni; }
    } else if (oj) {
        if (gj < 0) { which = SOUTH; layer = -gj - 1; }
        else { which = NORTH; layer = gj - d.nj; }
    } else if (ok) {
        if (gk < 0) { which = BOTTOM; layer = -gk - 1; }
        else { which = TOP; layer = gk - d.nk; }
    }
    if (layer > 1) return a_of_u;
    const int type = which >= 0 ? d.bc[which] : -1;
    if (type == 1) return d.inflow[5];
    if (type == 3) {
        const FusedDesc& o = descs[d.ex[which]];
        if (!(stage == 1 && *o.use_a0)) return a_of_u;
        switch (which) {
            case WEST: gi = o.ni - 1 - layer; break;
            case EAST: gi = layer; break;
            case SOUTH: gj = o.nj - 1 - layer; break;
            case NORTH: gj = layer; break;
            case BOTTOM: gk = o.nk - 1 - layer; break;
            default: gk = layer; break;
        }
        return o.A0[(size_t(gk) * o.nj + gj) * o.ni + gi];
    }
    if (!use_a0) return a_of_u;
    if (which >= 0) {
        const int s = (type == 2) ? 0 : layer;
        switch (which) {
            case WEST: gi = s; break;
            case EAST: gi = d.ni - 1 - s; break;
            case SOUTH: gj = s; break;
            case NORTH: gj = d.nj - 1 - s; break;
            case BOTTOM: gk = s; break;
            default: gk = d.nk - 1 - s; break;
        }
    }
    return d.A0[(size_t(gk) * d.nj + gj) * d.ni + gi];
}

// Shock flag of the cell (gi, gj, gk), interior or the first one beyond a
// face (k_fused_shock has written the stage's flags).
__device__ __forceinline__ int flag_of(const FusedDesc* __restrict__ descs, const FusedDesc& d,
                                       int stage, int gi, int gj, int gk) {
    const int out = int(gi < 0 || gi >= d.ni) + int(gj < 0 || gj >= d.nj) +
                    int(gk < 0 || gk >= d.nk);
    if (out > 1) return 0;
    if (out == 1) {
        if (gi < -1 || gi > d.ni || gj < -1 || gj > d.nj || gk < -1 || gk > d.nk) return 0;
        return ghost_shock(descs, d, stage, gi, gj, gk);
    }
    return d.S[stage == 1 ? 0 : 1][(size_t(gk) * d.nj + gj) * d.ni + gi];
}

__device__ __forceinline__ void prefetch_l2(const double* p) {
    asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

template <int FLUX, int TJ>
__global__ void __launch_bounds__(Lay<TJ>::threads, Lay<TJ>::min_blocks)
k_fused_stage_ws64(const FusedDesc* __restrict__ descs, int nblocks, long long nitems, int kc,
                   SimDev* sim, GasConsts gas, FluxOpts o, int stage,
                   const int* __restrict__ order) {
    using L = Lay<TJ>;
    constexpr int NPOS = L::PLANE;
    constexpr unsigned FULL = 0xffffffffu;
    // one decision per CTA (another CTA may set the status while this one
    // starts): every thread leaves, or none
    __shared__ int s_stop;
    pdl_wait();
    if (threadIdx.x == 0) s_stop = (sim->status != 0 || sim->finished) ? 1 : 0;
    __syncthreads();
    if (s_stop) return;
    if (blockIdx.x == 0 && threadIdx.x == 0) sim->item_next[stage == 1 ? 1 : 0] = 0u;
    __shared__ unsigned int s_item;
    __shared__ Weights s_w[3];
    __shared__ double s_volinv, s_area[3];   // of the current work item's block
    __shared__ ws::PlanSrc<double> s_src[5];
    extern __shared__ __align__(16) double sm64[];
    double* ring = sm64;
    double* Hj = sm64 + L::o_hj;
    double* Fj = sm64 + L::o_fj;
    double* As = sm64 + L::o_a;
    double* Fb = sm64 + L::o_fb;
    double* Hw = sm64 + L::o_hw;
    double* Aw = sm64 + L::o_aw;
    double* Fe = sm64 + L::o_fe;
    int* plan = reinterpret_cast<int*>(sm64 + L::o_plan);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const bool edge = warp >= TJ;
    const int et = threadIdx.x - 32 * TJ;   // edge thread index (edge warps)
    const int tj = warp <= TJ ? warp : -1;  // this warp's row of the tile
    const double dt = sim->dt_global;
    const bool lim = o.limiter != 0;
    constexpr bool ADAPT = (FLUX == 3);
    // isfinite(a) of a cell that passes the temperature tests depends on the
    // gas constants alone
    const double gR = gas.gamma * gas.Rgas;
    const bool a_ok = gR >= 0.0 && isfinite(gR * 50000.0);
    int bad = 0;
    auto slot_of = [&](int kk) { return ring + ((kk + 8) & 3) * (5 * NPOS); };
    // Positions the boundary conditions never fill (the block's corners, beyond
    // the second ghost layer of a partial tile) are read by lanes whose results
    // are not used.  They start as a cell of the first block: with zeros there
    // the density, pressure and sound speed of such a lane are out of the
    // batched quotients' range, and its whole warp goes through the plain
    // divisions as well (flux_ieee), every plane.  AUSMDV, 125x122x151 (29 of
    // 32 lanes in the last tile): 2.96 ms/step with zeros, 1.13 with a cell (the
    // per-face kernel's 32x8 tile: 1.74); over 24 layouts of partial tiles the
    // step is 0.57 of that with zeros (Hanel 0.75, adaptive 0.69, HLLC, whose
    // supersonic faces need no quotient, 1.00).  A gas at rest in its place made
    // HLLC take its subsonic side for those lanes (1.03).
    double first[5];
    {
        const double* c = static_cast<const double*>(stage == 1 ? descs[0].WA : descs[0].WB);
        const size_t n = size_t(descs[0].ni) * descs[0].nj * descs[0].nk;
#pragma unroll
        for (int f = 0; f < 5; ++f) first[f] = c[f * n];
    }
    for (int e = threadIdx.x; e < L::words - L::o_hj; e += blockDim.x) Hj[e] = 0.0;
    for (int e = threadIdx.x; e < NPOS; e += blockDim.x) {
#pragma unroll
        for (int q = 0; q < 20; ++q) ring[q * NPOS + e] = first[q % 5];
    }

    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) s_item = atomicAdd(&sim->item_next[stage == 1 ? 0 : 1], 1u);
        __syncthreads();
        if (s_item >= (unsigned long long)nitems) break;
        const long long item = order[s_item];
        const int b = find_block(descs, nblocks, item);
        const FusedDesc& d = descs[b];
        long long local = item - d.item0;
        const int kch = int(local % d.kchunks);
        local /= d.kchunks;
        const int tile_i = int(local % d.tiles_i), tile_j = int(local / d.tiles_i);
        const int i0 = tile_i * TI, j0 = tile_j * TJ;
        const int k0 = kch * kc, k1 = min(k0 + kc, d.nk);
        const size_t nc = size_t(d.ni) * d.nj * d.nk;
        if (threadIdx.x < 3) {
            // l2r2_prepare and the block's constants, read after a barrier
            L2R2<double> w;
            const double len = d.len[threadIdx.x];
            w.prepare(len, len, len, len);
            s_w[threadIdx.x] = Weights{w.tw_R0L0, w.aL0, w.two_L0_L1, len};
            s_area[threadIdx.x] = d.area[threadIdx.x];
            if (threadIdx.x == 0) s_volinv = 1.0 / d.vol;
        }
        const double* __restrict__ Win = static_cast<const double*>(stage == 1 ? d.WA : d.WB);
        if (threadIdx.x == 0) ws::plan_sources<double>(descs, stage, d, Win, s_src);
        __syncthreads();
        double* __restrict__ Wout = static_cast<double*>(stage == 1 ? d.WB : d.WA);
        const int use_a0 = (stage == 1) ? *d.use_a0 : 0;
        // a cell's sound speed: that of its u, except as special_sound_speed says
        auto cell_a = [&](double u, int gi, int gj, int gk) {
            const double a = sound_speed(u, gas);
            const bool inside = gi >= 0 && gi < d.ni && gj >= 0 && gj < d.nj && gk >= 0 && gk < d.nk;
            if (inside && !use_a0) return a;
            return special_sound_speed(descs, d, stage, use_a0, gi, gj, gk, a);
        };

        // prologue: planes k0-2 .. k0
        unsigned plan_fix = 0u, fx_next = 0u;
        if (edge) {
            plan_fix = ws::plan_tile<TJ>(descs, d, plan, ring, i0, j0, et);
            unsigned fx[3];
#pragma unroll
            for (int q = 0; q < 3; ++q)
                fx[q] = ws::queue_planned<TJ>(descs, stage, d, Win, slot_of(k0 - 2 + q), i0, j0,
                                              k0 - 2 + q, et, plan, s_src, plan_fix);
            ws::cp_async_wait_all();
#pragma unroll
            for (int q = 0; q < 3; ++q) ws::fixup_plane<TJ>(slot_of(k0 - 2 + q), fx[q], et);
        }
        __syncthreads();
        const int i = i0 + lane, j = j0 + tj;
        const int coff = (tj + 2) * PI + (lane + 2);   // own cell in the ring
        const bool row = !edge && j < d.nj;            // all three faces, and the update
        const bool face_row = tj >= 0 && j <= d.nj;    // the south face
        double hK[5];       // high value (k-direction) of the own cell at the current plane
        double lJ[5];       // low value (j-direction) of the own cell at the current plane
        double aK = 0.0;    // its sound speed
        int s_cur = 0;      // its shock flag

        // Planes k0-2 and k0-1 only start the k direction (their cells' high
        // values and the flux through the bottom of plane k0).
        for (int k = k0 - 2; k < k1; ++k) {
            const int par = k & 1;
            const double* sk = slot_of(k);
            const bool live = k >= k0;
            // plane k+3 into the slot plane k-1 has left
            const bool load = edge && k + 3 <= k1 + 1;
            if (load)
                fx_next = ws::queue_planned<TJ>(descs, stage, d, Win, slot_of(k + 3), i0, j0, k + 3,
                                                et, plan, s_src, plan_fix);
            if (live && face_row) {
                // south face: cells j-1 and j
                double hL[5], cL[5], cR[5], F[5];
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    hL[f] = Hj[(par * 5 + f) * L::NR + tj * TI + lane];
                    cL[f] = sk[f * NPOS + coff - PI];
                    cR[f] = sk[f * NPOS + coff];
                }
                int sh = 0;
                if (ADAPT) {
                    const int own = row ? s_cur : flag_of(descs, d, stage, i, j, k);
                    sh = own | flag_of(descs, d, stage, i, j - 1, k);
                }
                face_cells<FLUX, 1>(hL, cL, As[par * L::NR + tj * TI + lane], lJ, cR, aK, o, sh, F);
#pragma unroll
                for (int f = 0; f < 5; ++f) Fj[(par * 5 + f) * L::NR + tj * TI + lane] = F[f];
            }
            double Fw[5], Ftop[5];
            if (row) {
                if (live) {
                    // west face: cells i-1 and i
                    double qm[5], q0[5], qp[5], h[5], l[5];
#pragma unroll
                    for (int f = 0; f < 5; ++f) {
                        const double* q = sk + f * NPOS + coff;
                        qm[f] = q[-1]; q0[f] = q[0]; qp[f] = q[1];
                    }
                    if (o.order2) muscl_cell<5>(s_w[0], lim, qm, q0, qp, h, l);
                    else {
#pragma unroll
                        for (int f = 0; f < 5; ++f) h[f] = l[f] = q0[f];
                    }
#pragma unroll
                    for (int f = 0; f < 5; ++f) {
                        h[f] = __shfl_up_sync(FULL, h[f], 1);
                        if (lane == 0) h[f] = Hw[(par * 5 + f) * TJ + tj];
                    }
                    double aL = __shfl_up_sync(FULL, aK, 1);
                    if (lane == 0) aL = Aw[par * TJ + tj];
                    int sh = 0;
                    if (ADAPT) {
                        const int left = __shfl_up_sync(FULL, s_cur, 1);
                        sh = s_cur | (lane == 0 ? flag_of(descs, d, stage, i - 1, j, k) : left);
                    }
                    face_cells<FLUX, 0>(h, qm, aL, l, q0, aK, o, sh, Fw);
                }
                {   // top face: cells k and k+1
                    const double* s1 = slot_of(k + 1);
                    const double* s2 = slot_of(k + 2);
                    double q0[5], c1[5], c2[5], hN[5], lo1[5];
#pragma unroll
                    for (int f = 0; f < 5; ++f) {
                        q0[f] = sk[f * NPOS + coff];
                        c1[f] = s1[f * NPOS + coff];
                        c2[f] = s2[f * NPOS + coff];
                    }
                    if (o.order2) muscl_cell<5>(s_w[2], lim, q0, c1, c2, hN, lo1);
                    else {
#pragma unroll
                        for (int f = 0; f < 5; ++f) hN[f] = lo1[f] = c1[f];
                    }
                    const double aN = cell_a(c1[4], i, j, k + 1);
                    int sh = 0, s_next = 0;
                    if (ADAPT) {
                        s_next = flag_of(descs, d, stage, i, j, k + 1);
                        sh = s_cur | s_next;
                    }
                    if (k > k0 - 2) face_cells<FLUX, 2>(hK, q0, aK, lo1, c1, aN, o, sh, Ftop);
#pragma unroll
                    for (int f = 0; f < 5; ++f) hK[f] = hN[f];
                    aK = aN;
                    s_cur = s_next;
                }
            } else if (live && warp > TJ && lane < TJ) {
                // the faces on the tile's east edge, both cells reconstructed here
                const int off = (lane + 2) * PI + (TI + 1);
                double qm[5], q0[5], q1[5], q2[5], hL[5], lR[5], unused[5], F[5];
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    const double* q = sk + f * NPOS + off;
                    qm[f] = q[-1]; q0[f] = q[0]; q1[f] = q[1]; q2[f] = q[2];
                }
                if (o.order2) {
                    muscl_cell<5>(s_w[0], lim, qm, q0, q1, hL, unused);
                    muscl_cell<5>(s_w[0], lim, q0, q1, q2, unused, lR);
                } else {
#pragma unroll
                    for (int f = 0; f < 5; ++f) { hL[f] = q0[f]; lR[f] = q1[f]; }
                }
                const double aR = cell_a(q1[4], i0 + TI, j0 + lane, k);
                const int sh = ADAPT ? (flag_of(descs, d, stage, i0 + TI - 1, j0 + lane, k) |
                                        flag_of(descs, d, stage, i0 + TI, j0 + lane, k))
                                     : 0;
                face_cells<FLUX, 0>(hL, q0, As[par * L::NR + (lane + 1) * TI + TI - 1], lR, q1, aR, o,
                                    sh, F);
#pragma unroll
                for (int f = 0; f < 5; ++f) Fe[(par * 5 + f) * TJ + lane] = F[f];
            }
            // the next plane's j-direction values, and those of column -1
            const double* s1 = slot_of(k + 1);
            const int nxt = par ^ 1;
            if (k + 1 >= k0 && k + 1 < k1) {
                if (j <= d.nj) {
                    double qm[5], q0[5], qp[5], h[5];
#pragma unroll
                    for (int f = 0; f < 5; ++f) {
                        const double* q = s1 + f * NPOS + coff;
                        qm[f] = q[-PI]; q0[f] = q[0]; qp[f] = q[PI];
                    }
                    if (o.order2) muscl_cell<5>(s_w[1], lim, qm, q0, qp, h, lJ);
                    else {
#pragma unroll
                        for (int f = 0; f < 5; ++f) h[f] = lJ[f] = q0[f];
                    }
                    if (!row) aK = cell_a(q0[4], i, j, k + 1);
                    if (tj < TJ) {
#pragma unroll
                        for (int f = 0; f < 5; ++f)
                            Hj[(nxt * 5 + f) * L::NR + (tj + 1) * TI + lane] = h[f];
                        As[nxt * L::NR + (tj + 1) * TI + lane] = aK;
                    }
                }
                if (warp > TJ && lane < TJ) {
                    const int off = (lane + 2) * PI + 1;
                    double qm[5], q0[5], qp[5], h[5], unused[5];
#pragma unroll
                    for (int f = 0; f < 5; ++f) {
                        const double* q = s1 + f * NPOS + off;
                        qm[f] = q[-1]; q0[f] = q[0]; qp[f] = q[1];
                    }
                    if (o.order2) muscl_cell<5>(s_w[0], lim, qm, q0, qp, h, unused);
                    else {
#pragma unroll
                        for (int f = 0; f < 5; ++f) h[f] = q0[f];
                    }
#pragma unroll
                    for (int f = 0; f < 5; ++f) Hw[(nxt * 5 + f) * TJ + lane] = h[f];
                    Aw[nxt * TJ + lane] = cell_a(q0[4], i0 - 1, j0 + lane, k + 1);
                }
            }
            if (edge) {
                // the next plane's conserved state on its way into L2
                if (k + 1 >= k0 && k + 1 < k1) {
                    for (int t = et; t < TJ * 10; t += NE) {
                        const int f = t / (2 * TJ), r = t % (2 * TJ);
                        const int pj = j0 + (r >> 1), pi = i0 + (r & 1) * 16;
                        if (pj < d.nj && pi < d.ni) {
                            const size_t c = (size_t(k + 1) * d.nj + pj) * d.ni + pi + f * nc;
                            prefetch_l2(d.U0 + c);
                            if (stage == 2) prefetch_l2(d.dUdt0 + c);
                        }
                    }
                }
                // plane k+3 must be in place before the next plane's faces
                if (load) {
                    ws::cp_async_wait_all();
                    ws::fixup_plane<TJ>(slot_of(k + 3), fx_next, et);
                }
            }
            // the cell's conserved state, on its way while the warp waits
            const size_t c = (size_t(k) * d.nj + j) * d.ni + i;
            const bool update = row && live && i < d.ni;
            double U[5], D[5];
            if (update) {
#pragma unroll
                for (int v = 0; v < 5; ++v) U[v] = d.U0[v * nc + c];
                if (stage == 2) {
#pragma unroll
                    for (int v = 0; v < 5; ++v) D[v] = d.dUdt0[v * nc + c];
                }
            }
            __syncthreads();
            // ---- update and decode (cell warps) -----------------------------------
            if (row && live) {
                double Fx[5];   // east faces: the next lane's west faces
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    Fx[f] = __shfl_down_sync(FULL, Fw[f], 1);
                    if (lane == 31) Fx[f] = Fe[(par * 5 + f) * TJ + tj];
                }
                if (update) {
                    // time_derivatives: faces north, east, south, west, top, bottom
                    const double aN = s_area[1], aE = s_area[0], aT = s_area[2];
                    const double vol_inv = s_volinv;
                    double Un[5];
#pragma unroll
                    for (int v = 0; v < 5; ++v) {
                        const double* fj = Fj + (par * 5 + v) * L::NR + tj * TI + lane;
                        double s = 0.0;
                        s -= fj[TI] * (1.0 * aN);
                        s -= Fx[v] * (1.0 * aE);
                        s -= fj[0] * (-1.0 * aN);
                        s -= Fw[v] * (-1.0 * aE);
                        s -= Ftop[v] * (1.0 * aT);
                        s -= Fb[v * L::NL + tj * TI + lane] * (-1.0 * aT);
                        const double rate = vol_inv * s;
                        if (stage == 1) {
                            d.dUdt0[v * nc + c] = rate;
                            Un[v] = U[v] + dt * 1.0 * rate;
                        } else {
                            Un[v] = U[v] + dt * (0.5 * D[v] + 0.5 * rate);
                        }
                    }
                    // decode_conserved (fvcell.d:563-732), ideal gas
                    bool ok = a_ok;
                    double rho = Un[0], vx = 0.0, vy = 0.0, vz = 0.0, u = 0.0, p = 0.0, T = 0.0;
                    if (!(Un[0] > 0.0)) {
                        if (atomicCAS(&sim->status, 0, -5) == 0) sim->status_step = sim->step;
                        ok = false;
                    } else {
                        const double dinv = fdiv(1.0, rho);
                        vx = Un[1] * dinv; vy = Un[2] * dinv; vz = Un[3] * dinv;
                        u = Un[4] * dinv;
                        const double ke = 0.5 * (vx * vx + vy * vy + vz * vz);
                        u -= ke;
                        if (!ideal_rhou<double>(gas, rho, u, p, T)) {
                            T = 200.0;
                            p = rho * gas.Rgas * T;
                            u = gas.Cv * T;
                            Un[0] = rho;
                            Un[1] = rho * vx; Un[2] = rho * vy; Un[3] = rho * vz;
                            const double ke2 = 0.5 * (vx * vx + vy * vy + vz * vz);
                            Un[4] = rho * (u + ke2);
                        }
                    }
                    Wout[0 * nc + c] = rho;
                    Wout[1 * nc + c] = vx; Wout[2 * nc + c] = vy; Wout[3 * nc + c] = vz;
                    Wout[4 * nc + c] = u;
                    if (stage == 2) {
#pragma unroll
                        for (int v = 0; v < 5; ++v) d.U0[v * nc + c] = Un[v];
                    }
                    // FlowState.check_data (flowstate.d:345-388); the sound speed
                    // is finite for every T that passes (a_ok)
                    if (!isfinite(rho) || rho < 0.0) ok = false;
                    if (!isfinite(T) || T < 1.01) ok = false;
                    if (!isfinite(p)) ok = false;
                    if (fabs(vx) > 30000.0 || fabs(vy) > 30000.0 || fabs(vz) > 30000.0) ok = false;
                    if (T > 50000.0) ok = false;
                    if (!ok) ++bad;
                }
            }
            if (row) {
#pragma unroll
                for (int v = 0; v < 5; ++v) Fb[v * L::NL + tj * TI + lane] = Ftop[v];
            }
            // one barrier per plane: what is read after it (the j-face and east
            // fluxes, the own bottom flux) is rewritten two planes on, or by its
            // own reader
        }
    }
    if (stage == 2 && blockIdx.x == 0 && threadIdx.x == 0) {
        // from now on the sound speed comes from the decoded state
        for (int b = 0; b < nblocks; ++b) *descs[b].use_a0 = 0;
    }
    if (bad) atomicAdd(&sim->bad_acc, bad);
}

// Shock points of every fused block before a stage of the adaptive flux
// (detect_shock_points, fluidblock.d:415-431, with PJ_ShockDetector,
// shockdetectors.d:20-59): a face flags compression when
// (uR - uL) / min(aL, aR) < tol with u the velocity along the face normal (an
// axis); a cell is a shock point if any of its six faces does.  A pass of its
// own: it reads the state once (memory bound), where detecting inside the
// stage costs every tile its ring of neighbours' flags, a barrier and
// registers.  One block per blockIdx.y.
__global__ void k_fused_shock(const FusedDesc* __restrict__ descs, const SimDev* sim,
                              GasConsts gas, double tol, int stage) {
    pdl_wait();
    if (sim->status != 0 || sim->finished) return;
    const FusedDesc& d = descs[blockIdx.y];
    const double* W = static_cast<const double*>(stage == 1 ? d.WA : d.WB);
    const size_t nc = size_t(d.ni) * d.nj * d.nk;
    const int use_a0 = (stage == 1) ? *d.use_a0 : 0;
    unsigned char* S = d.S[stage == 1 ? 0 : 1];
    for (size_t c = blockIdx.x * size_t(blockDim.x) + threadIdx.x; c < nc;
         c += size_t(gridDim.x) * blockDim.x) {
        const int x[3] = {int(c % d.ni), int((c / d.ni) % d.nj), int(c / (size_t(d.ni) * d.nj))};
        const int n[3] = {d.ni, d.nj, d.nk};
        const size_t step[3] = {1, size_t(d.ni), size_t(d.ni) * d.nj};
        const int lo[3] = {WEST, SOUTH, BOTTOM}, hi[3] = {EAST, NORTH, TOP};
        const double u0 = W[4 * nc + c];
        const double a0 = use_a0 ? d.A0[c] : sound_speed(u0, gas);
        int flag = 0;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            const double v0 = W[(1 + q) * nc + c];
#pragma unroll
            for (int side = 0; side < 2; ++side) {
                const bool at_face = side == 0 ? x[q] == 0 : x[q] == n[q] - 1;
                double v, a;
                if (!at_face) {
                    const size_t m = side == 0 ? c - step[q] : c + step[q];
                    v = W[(1 + q) * nc + m];
                    a = use_a0 ? d.A0[m] : sound_speed(W[4 * nc + m], gas);
                } else {
                    // the first ghost cell of this face
                    const int which = side == 0 ? lo[q] : hi[q];
                    const int type = d.bc[which];
                    if (type == 1) {
                        v = d.inflow[1 + q];
                        a = d.inflow[5];
                    } else if (type == 3) {
                        const FusedDesc& p = descs[d.ex[which]];
                        int y[3] = {x[0], x[1], x[2]};
                        const int pn[3] = {p.ni, p.nj, p.nk};
                        y[q] = side == 0 ? pn[q] - 1 : 0;
                        const size_t pc = (size_t(y[2]) * p.nj + y[1]) * p.ni + y[0];
                        const size_t pnc = size_t(p.ni) * p.nj * p.nk;
                        const double* PW = static_cast<const double*>(stage == 1 ? p.WA : p.WB);
                        v = PW[(1 + q) * pnc + pc];
                        a = (stage == 1 && *p.use_a0) ? p.A0[pc] : sound_speed(PW[4 * pnc + pc], gas);
                    } else {
                        v = (type == 0) ? -v0 : v0;   // mirrored, or extrapolated
                        a = a0;
                    }
                }
                const double aL = side == 0 ? a : a0, aR = side == 0 ? a0 : a;
                const double a_min = (aL < aR) ? aL : aR;
                const double du = side == 0 ? v0 - v : v - v0;
                if (quotient_below(du, a_min, tol)) flag = 1;
            }
        }
        S[c] = (unsigned char)flag;
    }
}

}  // namespace ws64
}  // namespace e4c
