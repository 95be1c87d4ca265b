// The FP64 gather of the cooperative reverse step (included by adjoint_kernels.cuh): a thread per cell,
// or for a flow over few tiles four lanes per cell, one per side.
//
// As the FP32 one (adjoint_staged.cuh) it works on a tile and its halo in shared memory, with the global
// path's arithmetic and order of sums (adj_gather_phase, adjoint_impl.cuh), so results are identical.
// A face took 9 divisions and 2 square roots one after another; here the velocities and wave speeds
// are those the coefficient phase of the replayed step kept (staged_impl.cuh) and the remaining
// quotients are formed branch-free (quot.cuh) where the staged states allow it.  The terms of a cell's
// faces on four lanes meet by shuffles and every lane of the cell adds them in face order.
#pragma once

namespace da {
namespace adj {
namespace {

using fwd::kSlots;

struct GatherBuf64 {
    uint4 nl[kTileCells];                            // the tile's cells' neighbour slots (8 x int16)
    double vx[kSlots], vy[kSlots];                   // velocities of wet cells
    double wave[kSlots];                             // their wave speeds
    double b[4][kSlots];                             // slope coefficients B per side
    double a[3][kTileCells];                         // A of the tile's cells
    double gb[kTileCells], gi[kTileCells];           // running d J / d phi_bed, phi_int of the tile's cells
    double h[kSlots], hu[kSlots], hv[kSlots];        // U^n
    double lh[kSlots], lhu[kSlots], lhv[kSlots];     // lambda^{n+1}
    double sx[kSlots], sy[kSlots];                   // cell sizes
    uint8_t mask[kSlots], bf[kSlots], mat[kSlots];   // recorded branch byte (0 outside this recording), flags, material
};

struct GatherSmem64 {
    GatherBuf64 g;
    int hoff[kTileCells];  // halo range of each listed unit of the round
    int hcnt[kTileCells];
};

__device__ __forceinline__ void gather_slot64(GatherBuf64 &g, int s, int e, const MeshArgs &m, const StateRef<double> &U,
                                              const StateRef<double> &L, const AdjArgs &aa, const double *kept) {
    using fwd::cp_async;
    cp_async<8>(&g.h[s], U.h + e);
    cp_async<8>(&g.hu[s], U.hu + e);
    cp_async<8>(&g.hv[s], U.hv + e);
    cp_async<8>(&g.lh[s], L.h + e);
    cp_async<8>(&g.lhu[s], L.hu + e);
    cp_async<8>(&g.lhv[s], L.hv + e);
    cp_async<8>(&g.vx[s], kept + (size_t)2 * m.n + e);
    cp_async<8>(&g.vy[s], kept + (size_t)3 * m.n + e);
    cp_async<8>(&g.wave[s], kept + (size_t)4 * m.n + e);
    cp_async<8>(&g.sx[s], m.dx + e);
    cp_async<8>(&g.sy[s], m.dy + e);
#pragma unroll
    for (int q = 0; q < 4; ++q) cp_async<8>(&g.b[q][s], aa.B + (size_t)q * m.n + e);
}

// Tile t and its halo into g; returns with every value in shared memory and every thread past the
// copy.  True: every staged state and dt allow quot.cuh's quotients.  Thread c copies cell c of the tile
// and halo cell c.
__device__ __forceinline__ bool gather_stage64(GatherBuf64 &g, int t, int hoff, int hc, const fwd::HaloArgs &ha,
                                               const MeshArgs &m, const StateRef<double> &U, const StateRef<double> &L,
                                               const AdjArgs &aa, int rec_id, double dt) {
    static_assert(kHaloMax <= kTileCells, "one halo cell per thread");
    const int c = threadIdx.x;
    const int i = t * kTileCells + c;
    const bool own = i < m.n;
    const int e = c < hc ? ha.idx[hoff + c] : -1;
    const double *kept = (const double *)ha.kept;
    uint8_t mk = 0, bf = 0, mat = 0, hmk = 0, hbf = 0, hmat = 0;
    if (own) {
        gather_bytes(mk, bf, mat, i, m, aa, rec_id);
        gather_slot64(g, c, i, m, U, L, aa, kept);
        fwd::cp_async<16>(&g.nl[c], ha.nloc + (size_t)i * 8);
#pragma unroll
        for (int q = 0; q < 3; ++q) fwd::cp_async<8>(&g.a[q][c], aa.A + (size_t)q * m.n + i);
        fwd::cp_async<8>(&g.gb[c], aa.gbed + i);
        fwd::cp_async<8>(&g.gi[c], aa.gint + i);
    }
    if (e >= 0) {
        gather_bytes(hmk, hbf, hmat, e, m, aa, rec_id);
        gather_slot64(g, kTileCells + c, e, m, U, L, aa, kept);
    }
    fwd::cp_async_commit();
    // the byte fields, their loads in flight with the copies
    g.mask[c] = mk;
    g.bf[c] = bf;
    g.mat[c] = mat;
    if (e >= 0) {
        g.mask[kTileCells + c] = hmk;
        g.bf[kTileCells + c] = hbf;
        g.mat[kTileCells + c] = hmat;
    }
    fwd::cp_async_wait_all();
    const auto odd = [&](int s) {
        return !(quot::ordinary(g.h[s]) && quot::ordinary(g.hu[s]) && quot::ordinary(g.hv[s]));
    };
    return !__syncthreads_or(!ha.fast || !quot::ordinary(dt) || (own && odd(c)) || (e >= 0 && odd(kTileCells + c)));
}

template <bool FAST>
struct QuotPolicy {
    static __device__ __forceinline__ double div(double a, double b) { return fwd::Divisor<double, FAST>(b)(a); }
};

// A side of a face from the staged values (make_side).
__device__ __forceinline__ void gather_side64(const GatherBuf64 &g, const MatConsts &mc, int d, int e, uint8_t mk,
                                              Side<double> &s) {
    const double h = g.h[e];
    const bool wet = h >= DA_TINY;
    s.h = h;
    s.hu = g.hu[e];
    s.hv = g.hv[e];
    s.gz = 0.0;  // not read by the derivatives
    s.k = wet ? kact_of<double>(mc, g.mat[e], mk & 3) : 0.0;
    s.vel = wet ? (d == 0 ? g.vx[e] : g.vy[e]) : 0.0;
    s.a = wet ? g.wave[e] : 0.0;
    Hfv<double> &o = s.f;
    o.u[0] = wet ? s.h : 0.0;
    o.u[1] = wet ? s.hu : 0.0;
    o.u[2] = wet ? s.hv : 0.0;
    const double p = 0.5 * s.a * s.a * o.u[0];
    const double fu = o.u[1] * s.vel, fv = o.u[2] * s.vel;
    o.f[0] = d == 0 ? o.u[1] : o.u[2];
    o.f[1] = d == 0 ? fu + p : fu;
    o.f[2] = d == 0 ? fv : fv + p;
    o.s[0] = s.vel - s.a;
    o.s[1] = s.vel;
    o.s[2] = s.vel + s.a;
}

// The terms face (s, qq) of cell c adds to lambda_j (gather_face, adjoint_staged.cuh); a term the face
// does not have is left as it is.
template <bool FAST>
__device__ __forceinline__ void gather_face64(const GatherBuf64 &g, const MatConsts &mc, int c, int s, int qq,
                                              uint8_t bf, uint8_t mj, double h_j, const double lj[3], double dt,
                                              double &tb, double tg[3], double &tk) {
    const int d = s & 1;
    const bool plus = s < 2;
    const int sl = reinterpret_cast<const int16_t *>(&g.nl[c])[s + 4 * qq];
    const uint8_t bk = g.bf[sl];
    const double h_k = g.h[sl];
    if (h_k > DA_TINY) {
        // slope coefficient of neighbour k for j (k's side s^2 faces j)
        double bk_s = g.b[s ^ 2][sl];
        if (bk & (0x10 << (s ^ 2))) bk_s *= 0.5;
        tb = bk_s;
    }
    if (!(h_k >= DA_TINY || h_j >= DA_TINY)) return;
    const auto weight = [&](int cell, uint8_t f, int sd) {
        if (side_outflow<double>(f, sd)) return 0.0;
        double w = QuotPolicy<FAST>::div(sd < 2 ? -dt : dt, d == 0 ? g.sx[cell] : g.sy[cell]);
        if (f & (0x10 << sd)) w = 0.5 * w;
        return w;
    };
    const double wj = weight(c, bf, s), wk = weight(sl, bk, s ^ 2);
    if (wj == 0.0 && wk == 0.0) return;
    const uint8_t mk = g.mask[sl];
    const double lk[3] = {(mk & 4) ? 0.0 : g.lh[sl], g.lhu[sl], g.lhv[sl]};
    const double mu[3] = {wj * lj[0] + wk * lk[0], wj * lj[1] + wk * lk[1], wj * lj[2] + wk * lk[2]};
    if (mu[0] == 0.0 && mu[1] == 0.0 && mu[2] == 0.0) return;
    // the edge's left and right sides: j then k on a plus side, k then j on a minus side
    const int eL = plus ? c : sl, eR = plus ? sl : c;
    const uint8_t mL = plus ? mj : mk, mR = plus ? mk : mj;
    Side<double> sL, sR;
    gather_side64(g, mc, d, eL, mL, sL);
    gather_side64(g, mc, d, eR, mR, sR);
    double gL[3], gR[3], gkL, gkR;
    riemann_adj<double, QuotPolicy<FAST>>(d, sL, sR, mu, gL, gR, gkL, gkR);
    tg[0] = plus ? gL[0] : gR[0];
    tg[1] = plus ? gL[1] : gR[1];
    tg[2] = plus ? gL[2] : gR[2];
    tk = plus ? gkL : gkR;
}

// adj_gather_phase with every listed tile staged (see adj_gather_phase_staged for the listing).
// quarter: a block per listed quarter tile, which spreads a flow over few tiles over four times as many
// blocks and a cell's faces over four lanes; else a block per tile, a thread per cell.  An absent term
// is -0.0, the exact additive identity.
template <bool BATCH>
__device__ __forceinline__ void adj_gather_phase64(const MeshArgs &m, const fwd::HaloArgs &ha, const StateRef<double> &U,
                                                   const StateRef<double> &Lnext, const StateOut<double> &Lout,
                                                   const MatConsts &mc0, const AdjArgs &aa, int rec_id, double dt0,
                                                   int *list, const InstArgs &ia, GatherSmem64 &S, bool quarter, const fwd::FirstTiles<double> &first) {
    const GatherBuf64 &g = S.g;
    const int lane = threadIdx.x & 31, s = lane & 3;
    const int nunits = quarter ? 4 * aa.ntiles : aa.ntiles;
    for (int round = 0; sched_more(round, nunits); ++round) {
        const int uq = quarter ? fwd::staged_quarter<double, BATCH>(ha, round, first, aa.ntiles)
                               : fwd::staged_tile<double, BATCH>(ha, round, first, aa.ntiles);
        const int tq = quarter ? uq >> 2 : uq;
        bool need = false;
        if (uq < nunits) {
            const int ep = aa.tile_epoch[tq];
            if (quarter) {
                // the quarter's two segments
                const size_t o = (size_t)tq * 8 + 2 * (uq & 3);
                const unsigned sa = *reinterpret_cast<const uint16_t *>(aa.seg_act + o);
                const unsigned lc = *reinterpret_cast<const uint16_t *>(aa.lam_clean + o);
                need = (ep == rec_id && sa != 0u) || lc != 0x0101u;
            } else {
                const unsigned long long sa = seg_flags8(aa.seg_act, tq), lc = seg_flags8(aa.lam_clean, tq);
                need = (ep == rec_id && sa != 0ull) || lc != 0x0101010101010101ull;
            }
        }
        int ho, hc;
        fwd::halo_range(ha, uq < nunits ? tq : aa.ntiles, aa.ntiles, ho, hc);
        const int cnt = compact_tiles(need, uq, list, ho, hc, S.hoff, S.hcnt);
        for (int q = 0; q < cnt; ++q) {
            const int u = list[q];
            const int t = quarter ? u >> 2 : u;
            const int inst = BATCH ? ia.tile_inst[t] : 0;
            const MatConsts &mc = BATCH ? ia.mcs[inst] : mc0;
            const double dt = BATCH ? ia.dt[inst] : dt0;
            const bool fast = gather_stage64(S.g, t, S.hoff[q], S.hcnt[q], ha, m, U, Lnext, aa, rec_id, dt);
            // a recorded tile's segment activity is the OR of its cells' active bits
            if (threadIdx.x < (quarter ? 2 : 8)) {
                const int seg = t * 8 + (quarter ? 2 * (u & 3) : 0) + (int)threadIdx.x;
                aa.lam_clean[seg] = aa.tile_epoch[t] == rec_id && aa.seg_act[seg] ? 0 : 1;
            }
            const int c = quarter ? (u & 3) * 64 + ((int)threadIdx.x >> 2) : (int)threadIdx.x;
            const int j = t * kTileCells + c;
            const uint8_t mj = g.mask[c];  // 0 for cells past n
            const bool act = (mj & 8) != 0;
            const uint8_t bf = g.bf[c];
            const double h_j = g.h[c];
            const double lj[3] = {(mj & 4) ? 0.0 : g.lh[c], g.lhu[c], g.lhv[c]};
            double out[3] = {lj[0], lj[1], lj[2]}, dJ_dkj = 0.0;
            if (h_j > DA_TINY) {
                out[0] += g.a[0][c];
                out[1] += g.a[1][c];
                out[2] += g.a[2][c];
            }
            // the lane's faces (side, neighbour): its own side's two, or all eight of the cell in turn
            double tb[2], tg[2][3], tk[2];
            const bool any_two = __any_sync(0xffffffffu, act && (bf & 0xF0));
            const int sides = quarter ? 1 : 4;
#pragma unroll 1
            for (int k = 0; k < sides; ++k) {
                const int sd = quarter ? s : k;
#pragma unroll
                for (int qq = 0; qq < 2; ++qq) {
                    tb[qq] = tg[qq][0] = tg[qq][1] = tg[qq][2] = tk[qq] = -0.0;
                    if (qq && !any_two) continue;
                    if (!act || (bf & (1 << sd)) || (qq && !(bf & (0x10 << sd)))) continue;
                    if (fast)
                        gather_face64<true>(g, mc, c, sd, qq, bf, mj, h_j, lj, dt, tb[qq], tg[qq], tk[qq]);
                    else
                        gather_face64<false>(g, mc, c, sd, qq, bf, mj, h_j, lj, dt, tb[qq], tg[qq], tk[qq]);
                }
                // the terms in face order: this lane's, or those of the cell's four lanes
#pragma unroll 1
                for (int f = 0; f < (quarter ? 4 : 1); ++f) {
                    const int src = quarter ? (lane & ~3) + f : lane;
#pragma unroll
                    for (int qq = 0; qq < 2; ++qq) {
                        if (qq && !any_two) continue;
                        out[0] += __shfl_sync(0xffffffffu, tb[qq], src);
                        out[0] += __shfl_sync(0xffffffffu, tg[qq][0], src);
                        out[1] += __shfl_sync(0xffffffffu, tg[qq][1], src);
                        out[2] += __shfl_sync(0xffffffffu, tg[qq][2], src);
                        dJ_dkj += __shfl_sync(0xffffffffu, tk[qq], src);
                    }
                }
            }
            if (j < m.n) {
                // not active in the forward step: its update was the identity, and no neighbour is wet.  A
                // quarter's four lanes share the cell's stores out.
                const auto mine = [&](int k) { return !quarter || s == k; };
                if (mine(0)) Lout.h[j] = act ? out[0] : g.lh[c];
                if (mine(1)) Lout.hu[j] = act ? out[1] : g.lhu[c];
                if (mine(2)) Lout.hv[j] = act ? out[2] : g.lhv[c];
                if (mine(3) && act && dJ_dkj != 0.0) {
                    const InstTables it = inst_tables<BATCH>(aa, ia, inst);
                    const int mat = g.mat[c];
                    aa.gbed[j] = g.gb[c] + dJ_dkj * dk_of(it.dk_dbed, mat, mj & 3);
                    aa.gint[j] = g.gi[c] + dJ_dkj * dk_of(it.dk_dint, mat, mj & 3);
                }
            }
            __syncthreads();  // every thread is done with the tile before the next one is copied
        }
    }
}

}  // namespace
}  // namespace adj
}  // namespace da
