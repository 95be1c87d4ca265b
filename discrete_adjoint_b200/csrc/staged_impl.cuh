// Staged coefficient and update phases of the cooperative step kernels (included by
// forward_impl.cuh).
//
// A block works through its listed tiles one after another.  The values a tile's cells read at
// their neighbours (depth, momenta, k act/pass, g_z and the centres or sizes) are copied, for the
// tile's 256 cells and its halo (the outside cells they name as neighbours, at most kHaloMax),
// into a shared-memory buffer by asynchronous copies (cp.async) one tile ahead: while the block
// computes tile q, the copies of tile q + 1 and the halo list of tile q + 2 are in flight.  The
// per-cell arithmetic is the global path's (the same helpers through StagedView), so results are
// identical; only where the operands come from changes.  Each cell's neighbour entries come from
// the host-built table of tile-local slots (one 16-byte load per cell).
//
// What both phases need of a wet cell and of its wet neighbours is formed once per cell, in the
// coefficient phase: the velocities hu / h and hv / h and the flux's wave speed sqrt(k h g_z) go to
// global memory, are staged with the tile, and replace k act/pass and g_z there, so the four side
// fluxes of a cell take no division and no square root besides the HLL quotients; the four friction
// signs (a byte) and the two depth slopes are all that the sources take from the slopes.
// FP64 quotients that share a divisor are formed branch-free (quot.cuh) as long as every staged state is ordinary
// there (tested as the copies land, folded into the tile's barrier); a tile with any other value, and
// a mesh or material outside the range, takes the division operator.  The results are the
// reference's bits either way (FP32: the unstaged phases' bits).  A recording step also keeps the depth
// slopes' derivatives for the source adjoint (kept_deriv).  Bound: not memory (740k wet cells: a third of HBM's rate) but the
// instructions and the latency of one warp's FP64 chain.  46 divisions and 6 square roots per cell and
// step became 13 divisors and 2 square roots: 2894 -> 2060 instructions per warp and step, 125 -> 95 us
// per step on 740k wet cells (2 x 296 blocks), 14.0 -> 10.7 us on a flow of 18 tiles.  Three blocks
// per SM with one buffer each (80 registers) took 100 us.  FP32 (approximate quotients): 1650 -> 1380
// instructions, 137 -> 133 us on 2.1M wet cells (2 x 296 blocks), a flow on 262k cells 15.4 -> 13.9 us per
// step and 26.2 -> 25.0 us per reverse step.
//
// Activity: a cell is updated when it or a face neighbour is wet.  The global path marks every
// neighbour of a wet cell in the active bitmask with atomics; here the update phase recomputes
// that set from the staged depths of the tile and its halo, and the coefficient phase only marks
// neighbours in other tiles (and each warp's own wet cells), which the tile listing needs.
#pragma once

#include "quot.cuh"

namespace da {
namespace fwd {
namespace {

constexpr int kSlots = kTileCells + kHaloMax;  // slot s < 256: cell 256 t + s; 256 + k: halo cell k

template <class R>
struct StageBuf {
    // the tile's own cells
    uint4 nl[kTileCells];                      // neighbour slots (8 x int16)
    uint8_t bf[kTileCells], mat[kTileCells];   // boundary flags, material
    R sz[2][kTileCells];                       // dx, dy (FP32: in the update phase)
    R src[6][kTileCells];                      // update phase: g_x, g_y, the gravity derivatives, curvatures
    // every slot
    R h[kSlots], hu[kSlots], hv[kSlots];
    R c0[kSlots];  // coefficient phase: x centre (FP32: dx); update phase: hu / h of wet cells
    R c1[kSlots];  // y centre (FP32: dy); hv / h
    R a[kSlots];   // wave speed of wet cells (update phase)
    // the tile's own cells
    R k[kTileCells];   // k act/pass (update phase)
    R gz[kTileCells];  // g_z
};

template <class R>
struct StageSmem {
    StageBuf<R> buf[2];
    int hidx[3][kHaloMax];  // halo cells of three tiles in flight
    int hoff[kTileCells];   // halo range of each listed tile of the round
    int hcnt[kTileCells];
};

template <class R>
constexpr size_t stage_smem_bytes() {
    return sizeof(StageSmem<R>);
}

struct HaloArgs {
    const int32_t *off;   // [ntiles + 1]
    const int32_t *idx;   // halo cells, tile after tile
    const int16_t *nloc;  // [n][8] tile-local neighbour slots
    // written by the coefficient phase for each wet cell and read by the same step's update phase:
    void *kept;           // [5][n]: d h / dx, d h / dy, hu / h, hv / h, sqrt(k h g_z)
    uint8_t *fsign;       // [n]: the four friction signs of the sources, two bits each (sign + 1)
    double *deriv;        // [4][n]: when recording, the derivatives of d h / dx and d h / dy by the neighbours'
                          // depths (kept_deriv): the adjoint's array B, whose entry of a wet cell the update
                          // phase writes after it has read this one (no memory of their own: 32 B a cell)
    int fast;             // FP64: the mesh and the materials allow quot.cuh's quotients
    const int *order;     // [ntiles] the order of the tiles (tile_order.cu), null: plain
};

inline HaloArgs halo_args(const da_ctx *ctx) {
    const bool kact = ctx->ninst > 0 ? ctx->inst_ordinary : kact_ordinary(ctx->mc);
    return HaloArgs{ctx->mesh.halo_off, ctx->mesh.halo_idx, ctx->mesh.nloc,
                    ctx->slopes,        ctx->fsign,         ctx->adjB,
                    ctx->mesh.ordinary && kact ? 1 : 0,     ctx->tile_ordered ? ctx->tile_order : nullptr};
}

// The place of side q's kept derivative of cell i: the first bytes of B's own entry.
template <class R>
__device__ __forceinline__ R *kept_deriv(double *deriv, int q, int n, int i) {
    return reinterpret_cast<R *>(deriv + (size_t)q * n + i);
}

// Which kernels take the tiles in the order of tile_order.cu: those of an ensemble, whose members' flows fall
// on the same blocks (24 members, 310 wet of 6212 tiles: step 37 -> 31 us, reverse step 92 -> 64 us), and the
// FP32 ones (13 wet of 1024 tiles: 13.7 -> 12.0 and 24.9 -> 20.7 us).  The FP64 kernels of a single flow have
// no register left for it: there it cost every step 0.3 us of 11, more than it gives a compact flow.
template <class R, bool BATCH>
constexpr bool kOrdered = BATCH || sizeof(R) == 4;

// The tile at entry q of the list (q itself past its end).
__device__ __forceinline__ int ordered_tile(const HaloArgs &ha, int q, int ntiles) {
    return ha.order != nullptr && q < ntiles ? ha.order[q] : q;
}

// A thread's tile of round 0 (and in FP32 that of its first quarter tile) is the same in every phase of a
// launch and waits in shared memory: read from memory it cost each phase 0.2 us, and so did a register, which
// spilled.  It is loaded before a launch's restore and stored after it; waited for at its start it cost 3 us.
template <class R>
struct FirstTiles {
    uint16_t tile[kTileCells], quarter[sizeof(R) == 4 ? kTileCells : 1];  // an ordered list has at most 2^16 tiles
};
template <class R, bool BATCH>
struct FirstLoad {
    int tile = 0, quarter = 0;
    __device__ __forceinline__ FirstLoad(const HaloArgs &ha, int ntiles) {
        if constexpr (kOrdered<R, BATCH>) tile = ordered_tile(ha, sched_tile(0), ntiles);
        if constexpr (sizeof(R) == 4) quarter = ordered_tile(ha, sched_tile(0) >> 2, ntiles);
    }
    __device__ __forceinline__ void store(const HaloArgs &ha, FirstTiles<R> &first) const {
        if constexpr (kOrdered<R, BATCH>) {
            if (ha.order == nullptr) return;
            first.tile[threadIdx.x] = uint16_t(min(tile, 0xffff));
            if constexpr (sizeof(R) == 4) first.quarter[threadIdx.x] = uint16_t(min(quarter, 0xffff));
        }
    }
};

// The thread's tile of a round, and its unit 4 t + quarter of a gather by quarter tiles.
template <class R, bool BATCH>
__device__ __forceinline__ int staged_tile(const HaloArgs &ha, int round, const FirstTiles<R> &first, int ntiles) {
    const int q = sched_tile(round);
    if constexpr (kOrdered<R, BATCH>) {
        if (ha.order != nullptr) return round == 0 ? first.tile[threadIdx.x] : ordered_tile(ha, q, ntiles);
    }
    return q;
}
template <class R, bool BATCH>
__device__ __forceinline__ int staged_quarter(const HaloArgs &ha, int round, const FirstTiles<R> &first, int ntiles) {
    const int q = sched_tile(round);
    if constexpr (sizeof(R) == 4) {
        if (ha.order != nullptr)
            return 4 * (round == 0 ? first.quarter[threadIdx.x] : ordered_tile(ha, q >> 2, ntiles)) + (q & 3);
    } else if constexpr (BATCH) {
        if (ha.order != nullptr) return 4 * ordered_tile(ha, q >> 2, ntiles) + (q & 3);
    }
    return q;
}

// The staged phases run when the parameters ask for them, the mesh's halo tables exist and the
// slopes are kept (the staged update of the forward step reads them instead of staging the centres).
inline bool staged_ok(const da_ctx *ctx) {
    return ctx->p.tile_staging >= 1 && ctx->mesh.nloc != nullptr && ctx->slopes != nullptr;
}

// cp.async of BYTES (4 or 8) from global to shared memory; completes at the group's wait.
template <int BYTES>
__device__ __forceinline__ void cp_async(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(s), "l"(gmem), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <class R>
struct StagedView {
    const StageBuf<R> &b;
    int nl[8];  // the cell's neighbour slots
    __device__ __forceinline__ int nb(int s, int) const { return nl[s]; }
    __device__ __forceinline__ R h(int e) const { return b.h[e]; }
    __device__ __forceinline__ R hu(int e) const { return b.hu[e]; }
    __device__ __forceinline__ R hv(int e) const { return b.hv[e]; }
    __device__ __forceinline__ double coord(int dir, int e) const { return double(dir == 0 ? b.c0[e] : b.c1[e]); }
    __device__ __forceinline__ float size(int dir, int e) const { return float(dir == 0 ? b.c0[e] : b.c1[e]); }
};

// The eight neighbour slots of cell i (one 16-byte load).
__device__ __forceinline__ void load_slots(const int16_t *nloc, int i, int nl[8]) {
    const uint4 w = *reinterpret_cast<const uint4 *>(nloc + (size_t)i * 8);
    const unsigned u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        nl[2 * q] = int(int16_t(u[q] & 0xffffu));
        nl[2 * q + 1] = int(int16_t(u[q] >> 16));
    }
}

// Copies of one slot's values.  UPD: also what the update phase reads at neighbours (the velocities and
// the wave speed, at the cell itself k act/pass and g_z).  The coefficient phase reads the centres (FP32:
// the sizes) instead.
template <class R, bool UPD>
__device__ __forceinline__ void stage_slot(StageBuf<R> &b, int s, int e, bool own, const MeshArgs &m,
                                           const StateRef<R> &U, const R *kact, const HaloArgs &ha) {
    constexpr int B = sizeof(R);
    cp_async<B>(&b.h[s], U.h + e);
    cp_async<B>(&b.hu[s], U.hu + e);
    cp_async<B>(&b.hv[s], U.hv + e);
    if (own) cp_async<B>(&b.gz[s], (sizeof(R) == 8 ? (const R *)m.g : (const R *)m.fg) + (size_t)2 * m.n + e);
    if (UPD) {
        const R *kept = (const R *)ha.kept;
        if (own) cp_async<B>(&b.k[s], kact + e);
        cp_async<B>(&b.c0[s], kept + (size_t)2 * m.n + e);
        cp_async<B>(&b.c1[s], kept + (size_t)3 * m.n + e);
        cp_async<B>(&b.a[s], kept + (size_t)4 * m.n + e);
    } else {
        cp_async<B>(&b.c0[s], sizeof(R) == 8 ? (const R *)m.x + e : (const R *)m.fdx + e);
        cp_async<B>(&b.c1[s], sizeof(R) == 8 ? (const R *)m.y + e : (const R *)m.fdy + e);
    }
}

// What only the tile's own cells need: neighbour slots, sizes, source coefficients (UPD),
// and the tile's flag and material bytes in 16-byte pieces (the byte arrays are padded to tiles).
template <class R, bool UPD>
__device__ __forceinline__ void stage_own(StageBuf<R> &b, int t, const MeshArgs &m, const int16_t *nloc) {
    constexpr int B = sizeof(R);
    const int c = threadIdx.x;
    const int i = t * kTileCells + c;
    if (i < m.n) {
        cp_async<16>(&b.nl[c], nloc + (size_t)i * 8);
        if (sizeof(R) == 8 || UPD) {
            cp_async<B>(&b.sz[0][c], sizeof(R) == 8 ? (const R *)m.dx + i : (const R *)m.fdx + i);
            cp_async<B>(&b.sz[1][c], sizeof(R) == 8 ? (const R *)m.dy + i : (const R *)m.fdy + i);
        }
        if (UPD) {
            const R *g = sizeof(R) == 8 ? (const R *)m.g : (const R *)m.fg;
            const R *dg = sizeof(R) == 8 ? (const R *)m.dg : (const R *)m.fdg;
            const R *cv = sizeof(R) == 8 ? (const R *)m.curv : (const R *)m.fcurv;
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                cp_async<B>(&b.src[q][c], g + (size_t)q * m.n + i);
                cp_async<B>(&b.src[2 + q][c], dg + (size_t)q * m.n + i);
                cp_async<B>(&b.src[4 + q][c], cv + (size_t)q * m.n + i);
            }
        }
    }
    if (c < kTileCells / 16)
        cp_async<16>(&b.bf[16 * c], m.bflag + (size_t)t * kTileCells + 16 * c);
    else if (c < kTileCells / 8)
        cp_async<16>(&b.mat[16 * (c - kTileCells / 16)], m.mat + (size_t)t * kTileCells + 16 * (c - kTileCells / 16));
}

// The staged source coefficients of own cell c.
template <class R>
__device__ __forceinline__ CellSrc<R> staged_src(const StageBuf<R> &b, int c) {
    CellSrc<R> s;
#pragma unroll
    for (int q = 0; q < 2; ++q) {
        s.g[q] = b.src[q][c];
        s.dg[q] = b.src[2 + q][c];
        s.cv[q] = b.src[4 + q][c];
    }
    s.mat = b.mat[c];
    return s;
}

// The eight neighbour slots of own cell c from the staged table.
template <class R>
__device__ __forceinline__ void staged_slots(const StageBuf<R> &b, int c, int nl[8]) {
    const uint4 w = b.nl[c];
    const unsigned u[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        nl[2 * q] = int(int16_t(u[q] & 0xffffu));
        nl[2 * q + 1] = int(int16_t(u[q] >> 16));
    }
}

// Tile t's own cells and its halo (halo list already in shared memory) into buffer b.
template <class R, bool UPD>
__device__ __forceinline__ void stage_tile(StageBuf<R> &b, int t, const int *hidx, int hcnt, const MeshArgs &m,
                                           const StateRef<R> &U, const R *kact, const HaloArgs &ha) {
    const int i = t * kTileCells + (int)threadIdx.x;
    if (i < m.n) stage_slot<R, UPD>(b, threadIdx.x, i, true, m, U, kact, ha);
    stage_own<R, UPD>(b, t, m, ha.nloc);
    for (int k = threadIdx.x; k < hcnt; k += kTileCells)
        stage_slot<R, UPD>(b, kTileCells + k, hidx[k], false, m, U, kact, ha);
}

// Whether a state this thread staged (its own cell of tile t, its halo cells) is outside the range
// of quot.cuh; after the thread's copies have landed.
__device__ __forceinline__ bool staged_odd(const StageBuf<double> &b, int t, int hcnt, int n) {
    auto odd = [&](int s) { return !(quot::ordinary(b.h[s]) && quot::ordinary(b.hu[s]) && quot::ordinary(b.hv[s])); };
    const int c = (int)threadIdx.x;
    bool r = t * kTileCells + c < n && odd(c);
    for (int k = c; k < hcnt; k += kTileCells) r = r || odd(kTileCells + k);
    return r;
}

__device__ __forceinline__ void stage_halo_list(int *dst, const int32_t *src, int cnt) {
    for (int k = threadIdx.x; k < cnt; k += kTileCells) cp_async<4>(dst + k, src + k);
}

// The halo range of tile tq (or nothing past the last tile), loaded beside its flags by the scan
// and kept with the tile by compact_tiles.
__device__ __forceinline__ void halo_range(const HaloArgs &ha, int tq, int ntiles, int &off, int &cnt) {
    off = 0;
    cnt = 0;
    if (tq < ntiles) {
        off = ha.off[tq];
        cnt = ha.off[tq + 1] - off;
    }
}

// The listed tiles of a round, pipelined: fn(t, buffer, halo list, fast) computes tile t from shared
// memory (fast: FP64 quotients by quot.cuh).  Needs blockDim.x == kTileCells; every thread of the
// block calls it with the same cnt; S.hoff / S.hcnt hold the listed tiles' halo ranges
// (compact_tiles).  The first tile's halo cells are read by the threads that copy them; later
// tiles' lists arrive two tiles ahead.
template <class R, bool UPD, class F>
__device__ __forceinline__ void staged_tiles(const MeshArgs &m, const HaloArgs &ha, const StateRef<R> &U,
                                             const R *kact, int cnt, const int *list, StageSmem<R> &S, F &&fn) {
    {
        const int t0 = list[0], hc = S.hcnt[0];
        const int32_t *src = ha.idx + S.hoff[0];
        const int i = t0 * kTileCells + (int)threadIdx.x;
        if (i < m.n) stage_slot<R, UPD>(S.buf[0], threadIdx.x, i, true, m, U, kact, ha);
        stage_own<R, UPD>(S.buf[0], t0, m, ha.nloc);
        for (int k = threadIdx.x; k < hc; k += kTileCells) {
            const int e = src[k];
            S.hidx[0][k] = e;
            stage_slot<R, UPD>(S.buf[0], kTileCells + k, e, false, m, U, kact, ha);
        }
    }
    if (cnt > 1) stage_halo_list(S.hidx[1], ha.idx + S.hoff[1], S.hcnt[1]);
    cp_async_commit();
    for (int q = 0; q < cnt; ++q) {
        // tile q's values and tile q + 1's halo list have landed; every thread is past tile q - 1
        cp_async_wait_all();
        bool fast = false;
        if constexpr (sizeof(R) == 8)
            fast = !__syncthreads_or(!ha.fast || staged_odd(S.buf[q & 1], list[q], S.hcnt[q], m.n));
        else
            __syncthreads();
        if (q + 1 < cnt) {
            stage_tile<R, UPD>(S.buf[(q + 1) & 1], list[q + 1], S.hidx[(q + 1) % 3], S.hcnt[q + 1], m, U, kact, ha);
            if (q + 2 < cnt) stage_halo_list(S.hidx[(q + 2) % 3], ha.idx + S.hoff[q + 2], S.hcnt[q + 2]);
        }
        cp_async_commit();
        fn(list[q], S.buf[q & 1], S.hidx[q % 3], fast);
    }
    __syncthreads();
}

// ------------------------------------------------------------------------------- FP64 arithmetic
// The cold path's division, out of line (the kernels stay small).
__device__ __noinline__ double div_operator(double a, double b) { return a / b; }

// A divisor and its quotients.  FP64: FAST by quot.cuh, else the operator; FP32: its inverse.
template <class R, bool FAST>
struct Divisor {
    quot::Recip r;
    __device__ __forceinline__ explicit Divisor(double b) {
        if constexpr (FAST)
            r = quot::recip(b);
        else
            r.b = b;
    }
    __device__ __forceinline__ double operator()(double a) const {
        if constexpr (FAST)
            return quot::div(a, r);
        else
            return div_operator(a, r.b);
    }
};
template <bool FAST>
struct Divisor<float, FAST> {
    float y;
    __device__ __forceinline__ explicit Divisor(float b) : y(1.0f / b) {}
    __device__ __forceinline__ float operator()(float a) const { return a * y; }
};

// cell_slopes (fv_device.cuh, FP64) with one divisor per centre distance.  DERIV: also the derivatives
// of the depth slopes by the depth across each side, q[s] (h_slope_deriv, fv_device.cuh: the
// slope's derivative by dp or dm over the centre distance).
template <bool FAST, bool DERIV>
__device__ __forceinline__ void staged_slopes64(const StagedView<double> &v, int i, uint8_t bf, double gamma,
                                                const double ui[3], double out[6], double q[4]) {
    if (bf & 0x0F) {
#pragma unroll
        for (int j = 0; j < 6; ++j) out[j] = 0.0;
        if (DERIV) q[0] = q[1] = q[2] = q[3] = 0.0;
        return;
    }
#pragma unroll
    for (int dir = 0; dir < 2; ++dir) {
        const int ep = v.nb(dir, i), em = v.nb(dir + 2, i);
        const bool two_p = bf & (0x10 << dir), two_m = bf & (0x10 << (dir + 2));
        const double ci = v.coord(dir, i);
        const double dxp = v.coord(dir, ep) - ci, dxm = ci - v.coord(dir, em);
        const Divisor<double, FAST> dvp(dxp), dvm(dxm), dvs(dxm + dxp);
        const double up[3] = {v.h(ep), v.hu(ep), v.hv(ep)}, um[3] = {v.h(em), v.hu(em), v.hv(em)};
        double dp[3], dm[3];
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            dp[j] = dvp(up[j] - ui[j]);
            dm[j] = dvm(ui[j] - um[j]);
        }
        if (two_p) {
            const int e = v.nb(dir + 4, i);
            const double u2[3] = {v.h(e), v.hu(e), v.hv(e)};
#pragma unroll
            for (int j = 0; j < 3; ++j) dp[j] = .5 * (dp[j] + dvp(u2[j] - ui[j]));
        }
        if (two_m) {
            const int e = v.nb(dir + 6, i);
            const double u2[3] = {v.h(e), v.hu(e), v.hv(e)};
#pragma unroll
            for (int j = 0; j < 3; ++j) dm[j] = .5 * (dm[j] + dvm(ui[j] - u2[j]));
        }
#pragma unroll
        for (int j = 0; j < 3; ++j) {
            const double dc = dvs(dp[j] * dxm + dm[j] * dxp);
            double mn = gamma * dabs(dp[j]);
            const double b = gamma * dabs(dm[j]), c = dabs(dc);
            int sel = 0;
            if (mn > b) { mn = b; sel = 1; }
            if (mn > c) { mn = c; sel = 2; }
            const double fac = .5 * (c_sgn(dp[j]) + c_sgn(dm[j]));
            out[j + 3 * dir] = fac * mn;
            if (DERIV && j == 0) {
                const auto sgnf = [](double x) { return x > 0.0 ? 1.0 : (x < 0.0 ? -1.0 : 0.0); };
                const double gc = dvs(fac * sgnf(dc));
                const double gp = sel == 0 ? fac * gamma * sgnf(dp[0]) : (sel == 1 ? 0.0 : gc * dxm);
                const double gm = sel == 1 ? fac * gamma * sgnf(dm[0]) : (sel == 0 ? 0.0 : gc * dxp);
                q[dir] = dvp(gp);
                q[dir + 2] = dvm(gm);
            }
        }
    }
}

// What the coefficient phase forms of a wet cell.
template <class R>
struct StagedCoef {
    R s[6];        // limited slopes
    R vx, vy, a;   // hu / h, hv / h, sqrt(k h g_z)
    R k, ev;       // k act/pass, largest wave speed
    uint8_t code;  // branch of k act/pass
    uint8_t sgn;   // friction signs, two bits each
    R q[4];        // recording: derivatives of the depth slopes by the neighbours' depths
};

// The four friction signs (-1, 0 or 1) in two bits each.
__device__ __forceinline__ uint8_t pack_signs(int s0, int s1, int s2, int s3) {
    return uint8_t((s0 + 1) | (s1 + 1) << 2 | (s2 + 1) << 4 | (s3 + 1) << 6);
}

// A cell with h > GEOFLOW_TINY: get_slopes, gmfggetcoef, eigen, and the velocities, wave speed and
// friction signs that the corrector forms from the same values (update_cell).
template <bool FAST, bool DERIV>
__device__ __forceinline__ void staged_coef64(const StagedView<double> &v, int c, uint8_t bf, int mat, double gz,
                                              const MatConsts &mc, double ft, const double ui[3],
                                              StagedCoef<double> &o) {
    staged_slopes64<FAST, DERIV>(v, c, bf, mc.gamma, ui, o.s, o.q);
    const double *s = o.s;
    const double h = ui[0], hu = ui[1], hv = ui[2];
    const Divisor<double, FAST> dh(h), dhh(h * h);
    o.vx = dh(hu);
    o.vy = dh(hv);
    const double vel = dh(s[1]) - dhh(hu * s[0]) + dh(s[5]) - dhh(hv * s[3]);
    const int sg = fsgn(vel, DA_TINY);
    o.k = mc.kact_sgn[mat][sg + 1];
    o.code = uint8_t(sg + 2);
    if (dabs(o.vx) < DA_TINY && dabs(o.vy) < DA_TINY) {
        o.k = mc.kact_rest;
        o.code = 0;
    }
    const double cc = sqrt(o.k * gz * h);
    o.a = sqrt(o.k * h * gz);
    const double evx = dabs(o.vx) + cc, evy = dabs(o.vy) + cc;
    o.ev = evx > evy ? evx : evy;
    const double h_inv = dh(1.0);
    const int s0 = int(tiny_sgn(h_inv * (s[4] - o.vx * s[3]), ft)), s2 = int(tiny_sgn(o.vx, ft));
    const int s1 = int(tiny_sgn(h_inv * (s[2] - o.vy * s[0]), ft)), s3 = int(tiny_sgn(o.vy, ft));
    o.sgn = pack_signs(s0, s1, s2, s3);
}

// The same in FP32, from the helpers of the unstaged phases (their operations, hence their bits).
template <bool DERIV>
__device__ __forceinline__ void staged_coef32(const StagedView<float> &v, int c, uint8_t bf, int mat, float gz,
                                              const MatConsts &mc, float ft, const float ui[3], StagedCoef<float> &o) {
    cell_slopes<float>(v, c, bf, float(mc.gamma), ui, o.s);
    const float *s = o.s;
    const float h = ui[0];
    o.k = cell_kact<float>(mc, mat, h, ui[1], ui[2], s, &o.code);
    o.vx = ui[1] / h;
    o.vy = ui[2] / h;
    const float cc = sqrt(o.k * gz * h);
    o.a = sqrt(o.k * h * gz);
    const float evx = dabs(o.vx) + cc, evy = dabs(o.vy) + cc;
    o.ev = evx > evy ? evx : evy;
    const float h_inv = 1.0f / h, vel0 = ui[1] * h_inv, vel1 = ui[2] * h_inv;
    const int s0 = int(tiny_sgn(h_inv * (s[4] - vel0 * s[3]), ft)), s2 = int(tiny_sgn(vel0, ft));
    const int s1 = int(tiny_sgn(h_inv * (s[2] - vel1 * s[0]), ft)), s3 = int(tiny_sgn(vel1, ft));
    o.sgn = pack_signs(s0, s1, s2, s3);
    if (DERIV) {
        o.q[0] = o.q[1] = o.q[2] = o.q[3] = 0.0f;
        if (!(bf & 0x0F)) slope_quotients<float>(v, c, bf, float(mc.gamma), h, o.q);
    }
}

// A side of a Riemann problem from the staged values (dirflux): zero for a dry cell.
template <class R>
struct StagedSide {
    R u[3], f[3], s0, s1, s2;
};

template <class R, int DIR>
__device__ __forceinline__ StagedSide<R> staged_side(const StageBuf<R> &b, int e) {
    StagedSide<R> o;
    const R h = b.h[e];
    const bool wet = !(h < R(DA_TINY));
    o.u[0] = wet ? h : R(0);
    o.u[1] = wet ? b.hu[e] : R(0);
    o.u[2] = wet ? b.hv[e] : R(0);
    const R vel = wet ? (DIR == 0 ? b.c0[e] : b.c1[e]) : R(0), a = wet ? b.a[e] : R(0);
    if (DIR == 0) {
        o.f[0] = o.u[1];
        o.f[1] = o.u[1] * vel + R(0.5) * a * a * o.u[0];
        o.f[2] = o.u[2] * vel;
    } else {
        o.f[0] = o.u[2];
        o.f[1] = o.u[1] * vel;
        o.f[2] = o.u[2] * vel + R(0.5) * a * a * o.u[0];
    }
    o.s0 = vel - a;
    o.s1 = vel;
    o.s2 = vel + a;
    return o;
}

// riemann (fv_device.cuh) with one divisor for the three components.  Two dry sides give zero speeds,
// hence the left flux, which is zero.
template <class R, bool FAST>
__device__ __forceinline__ void staged_riemann(const StagedSide<R> &l, const StagedSide<R> &r, R F[3]) {
    const bool ld = l.u[0] == R(0), rd = r.u[0] == R(0);
    const R a0 = R(2.0) * r.s0 - r.s1, a2 = R(2.0) * r.s2 - r.s1;
    const R b0 = R(2.0) * l.s0 - l.s1, b2 = R(2.0) * l.s2 - l.s1;
    const R lo = ld ? a0 : (rd ? b0 : rmin(l.s0, r.s0));
    const R hi = ld ? a2 : (rd ? b2 : rmax(l.s2, r.s2));
    const R sl = rmin(R(0), lo), sr = rmax(R(0), hi);
    if (sl >= R(0)) {
        F[0] = l.f[0]; F[1] = l.f[1]; F[2] = l.f[2];
    } else if (sr <= R(0)) {
        F[0] = r.f[0]; F[1] = r.f[1]; F[2] = r.f[2];
    } else {
        const Divisor<R, FAST> den(sr - sl);
#pragma unroll
        for (int v = 0; v < 3; ++v) F[v] = den(sr * l.f[v] - sl * r.f[v] + sl * sr * (r.u[v] - l.u[v]));
    }
}

// F(+side) - F(-side) in direction DIR of cell c (flux_div).
template <class R, bool FAST, int DIR>
__device__ __forceinline__ void staged_div(const StagedView<R> &v, int c, uint8_t bf, R div[3]) {
    if (bf & ((1 << DIR) | (1 << (DIR + 2)))) {
        div[0] = div[1] = div[2] = R(0);
        return;
    }
    const StagedSide<R> self = staged_side<R, DIR>(v.b, c);
    R Fm[3], Fp[3];
    staged_riemann<R, FAST>(staged_side<R, DIR>(v.b, v.nl[DIR + 2]), self, Fm);
    staged_riemann<R, FAST>(self, staged_side<R, DIR>(v.b, v.nl[DIR]), Fp);
    if (bf & (0x10 << (DIR + 2))) {
        R F2[3];
        staged_riemann<R, FAST>(staged_side<R, DIR>(v.b, v.nl[DIR + 6]), self, F2);
#pragma unroll
        for (int q = 0; q < 3; ++q) Fm[q] = R(0.5) * (Fm[q] + F2[q]);
    }
    if (bf & (0x10 << DIR)) {
        R F2[3];
        staged_riemann<R, FAST>(self, staged_side<R, DIR>(v.b, v.nl[DIR + 4]), F2);
#pragma unroll
        for (int q = 0; q < 3; ++q) Fp[q] = R(0.5) * (Fp[q] + F2[q]);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) div[q] = Fp[q] - Fm[q];
}

// What the update phase loads of a cell ahead of the fluxes.
template <class R>
struct Kept {
    R sx, sy;  // depth slopes
    uint8_t sgn;
};

// update_cell (forward_impl.cuh) of an active cell from the staged and kept values.
template <class R, bool FAST, class Hook>
__device__ __forceinline__ bool staged_update(const StagedView<R> &v, int c, uint8_t bf, const CellSrc<R> &cs,
                                              const MatConsts &mc, R dt, const R prev[3], R dxc, R dyc, R st[3],
                                              const Kept<R> &kp, const Hook &hook) {
    R dx3[3], dy3[3];
    staged_div<R, FAST, 0>(v, c, bf, dx3);
    staged_div<R, FAST, 1>(v, c, bf, dy3);
    R dtdx, dtdy;
    if constexpr (sizeof(R) == 8) {
        dtdx = dt / dxc;
        dtdy = dyc == dxc ? dtdx : dt / dyc;
    } else {
        dtdx = dt * (1.0f / dxc);
        dtdy = dt * (1.0f / dyc);
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) st[q] = prev[q] - dtdx * dx3[q] - dtdy * dy3[q];
    const bool clamped = st[0] < R(0);
    if (clamped) st[0] = R(0);
    if (prev[0] > R(DA_TINY)) {
        R vel0, vel1;
        if constexpr (sizeof(R) == 8) {
            vel0 = v.b.c0[c];
            vel1 = v.b.c1[c];
        } else {  // the sources' velocities are products with 1 / h
            const float h_inv = 1.0f / prev[0];
            vel0 = prev[1] * h_inv;
            vel1 = prev[2] * h_inv;
        }
        auto sg = [&](int q) { return R(int((kp.sgn >> (2 * q)) & 3) - 1); };
        const R sg0 = sg(0), sg1 = sg(1), sg2 = sg(2), sg3 = sg(3);
        hook(SrcFwd<R>{{kp.sx, R(0), R(0), kp.sy, R(0), R(0)}, vel0, vel1, R(0), sg0, sg1, sg2, sg3}, clamped);
        const R ki = v.b.k[c], gz = v.b.gz[c];
        const R sin_int = R(mc.sin_int), tan_bed = R(mc.tan_bed[cs.mat]);
        R s1 = cs.g[0] * prev[0];
        R s2 = sg0 * prev[0] * ki * slope_term(gz, kp.sy, cs.dg[1], prev[0]) * sin_int;
        R s3 = sg2 * rmax(gz * prev[0] + vel0 * prev[1] * cs.cv[0], R(0)) * tan_bed;
        st[1] += dt * (s1 - s2 - s3);
        s1 = cs.g[1] * prev[0];
        s2 = sg1 * prev[0] * ki * slope_term(gz, kp.sx, cs.dg[0], prev[0]) * sin_int;
        s3 = sg3 * rmax(gz * prev[0] + vel1 * prev[2] * cs.cv[1], R(0)) * tan_bed;
        st[2] += dt * (s1 - s2 - s3);
    }
    return clamped;
}

// Coefficient phase (see coef_phase) with the tile and its halo staged.
template <class R, bool RECORD, bool BATCH = false>
__device__ __forceinline__ void coef_phase_staged(const MeshArgs &m, const HaloArgs &ha, const StateRef<R> &U,
                                                  R *kact, unsigned *active, const uint8_t *seg_wet, int ntiles,
                                                  int cull, const MatConsts &mc0, DevScalars *sc, uint8_t *mask,
                                                  int *list, unsigned long long &my_min, unsigned long long &my_max,
                                                  const InstArgs &ia, StageSmem<R> &S, R ft, const FirstTiles<R> &first) {
    for (int round = 0; sched_more(round, ntiles); ++round) {
        const int tq = staged_tile<R, BATCH>(ha, round, first, ntiles);
        const bool need = tq < ntiles && (!cull || seg_flags(seg_wet, tq) != 0ull);
        int ho, hc;
        halo_range(ha, tq, ntiles, ho, hc);
        const int cnt = compact_tiles(need, tq, list, ho, hc, S.hoff, S.hcnt);
        if (cnt == 0) continue;
        staged_tiles<R, false>(m, ha, U, kact, cnt, list, S, [&](int t, const StageBuf<R> &b, const int *hidx, bool fast) {
            const int inst = BATCH ? ia.tile_inst[t] : 0;
            const MatConsts &mc = BATCH ? ia.mcs[inst] : mc0;
            const int c = threadIdx.x;
            const int i = t * kTileCells + c;
            bool wet = false;
            if (i < m.n) {
                const R h = b.h[c];
                if (!(h == h)) raise_err(sc, DA_ERR_NAN);
                wet = h >= R(DA_TINY);
                uint8_t code = 0;
                if (wet) {
                    const uint8_t bf = b.bf[c];
                    const int mat = b.mat[c];
                    R dxm, dym;
                    if constexpr (sizeof(R) == 8) {
                        dxm = b.sz[0][c];
                        dym = b.sz[1][c];
                    } else {
                        dxm = b.c0[c];
                        dym = b.c1[c];
                    }
                    StagedView<R> v{b};
                    staged_slots(b, c, v.nl);
                    // neighbours in other tiles: mark them for the tile listing of the update
#pragma unroll
                    for (int s = 0; s < 4; ++s) {
                        if (bf & (1 << s)) continue;
                        const int ne = (bf & (0x10 << s)) ? 2 : 1;
                        for (int q = 0; q < ne; ++q) {
                            const int sl = v.nl[s + 4 * q];
                            if (sl >= kTileCells) {
                                const int e = hidx[sl - kTileCells];
                                atomicOr(&active[e >> 5], 1u << (e & 31));
                            }
                        }
                    }
                    const R ui[3] = {h, b.hu[c], b.hv[c]};
                    const R gz = b.gz[c];
                    R *kept = (R *)ha.kept;
                    if (!(h > R(DA_TINY))) {  // h == GEOFLOW_TINY: dry for get_coef_and_eigen, wet for the fluxes
                        const R k = R(mc.kact_rest);
                        kact[i] = k;
                        kept[(size_t)2 * m.n + i] = ui[1] / h;
                        kept[(size_t)3 * m.n + i] = ui[2] / h;
                        kept[(size_t)4 * m.n + i] = sqrt(k * h * gz);
                    } else {
                        StagedCoef<R> o;
                        if constexpr (sizeof(R) == 8) {
                            if (fast)
                                staged_coef64<true, RECORD>(v, c, bf, mat, gz, mc, ft, ui, o);
                            else
                                staged_coef64<false, RECORD>(v, c, bf, mat, gz, mc, ft, ui, o);
                        } else {
                            staged_coef32<RECORD>(v, c, bf, mat, gz, mc, ft, ui, o);
                        }
                        code = o.code;
                        kact[i] = o.k;
                        kept[i] = o.s[0];
                        kept[(size_t)m.n + i] = o.s[3];
                        kept[(size_t)2 * m.n + i] = o.vx;
                        kept[(size_t)3 * m.n + i] = o.vy;
                        kept[(size_t)4 * m.n + i] = o.a;
                        ha.fsign[i] = o.sgn;
                        if (RECORD)
#pragma unroll
                            for (int q = 0; q < 4; ++q) *kept_deriv<R>(ha.deriv, q, m.n, i) = o.q[q];
                        const R ev = o.ev;
                        if (ev > R(1000000000.)) raise_err(sc, DA_ERR_EIGEN);
                        const unsigned long long rb = __double_as_longlong(double((dxm > dym ? dym : dxm) / ev));
                        const unsigned long long hb = __double_as_longlong(double(h));
                        my_min = rb < my_min ? rb : my_min;
                        my_max = hb > my_max ? hb : my_max;
                    }
                }
                if (RECORD) mask[i] = code;
            }
            const unsigned self = __ballot_sync(0xffffffffu, wet);
            if (self && (threadIdx.x & 31) == 0) atomicOr(&active[i >> 5], self);
            if (BATCH) {
                push_minmax(my_min, my_max, ia.acc_min + inst, ia.acc_max + inst);
                my_min = 0x7FF0000000000000ull;
                my_max = 0ull;
            }
        });
    }
}

// No per-cell epilogue.
struct NoEpilogue {
    struct Pre {};
    __device__ __forceinline__ Pre pre(int, bool) const { return Pre{}; }
    template <class... A>
    __device__ __forceinline__ void operator()(A &&...) const {}
};

// Update phase (see update_phase) with the tile and its halo staged.  A listed tile's cells
// recompute their activity from the staged depths; the segment flags follow it.
// epi(t, i, v, c, prev, bf, code, gz, cs, pre, f) runs for every wet cell i of a listed tile t inside
// its update, where the corrector has formed the source terms' slopes, velocities and friction
// signs f (the reverse step's source adjoint, which needs exactly these), with the staged view v
// of the cell (slot c), its U^n, boundary flags, recorded branch byte, g_z and source coefficients,
// and what epi.pre(i, wet) loaded before the update (so that those loads overlap it).
// STATE false: a reverse step whose new state nobody reads -- the state, the segments' volumes and their
// wet, clean and dirty flags are left alone, and only active tiles are listed.
template <class R, bool RECORD, bool BATCH = false, bool STATE = true, class Epi = NoEpilogue>
__device__ __forceinline__ void update_phase_staged(const MeshArgs &m, const HaloArgs &ha, const StateRef<R> &U,
                                                    const StateOut<R> &O, const R *kact, unsigned *active,
                                                    uint8_t *seg_clean, uint8_t *seg_wet, double *seg_vol,
                                                    uint8_t *seg_dirty, int ntiles, int cull, const MatConsts &mc0,
                                                    DevScalars *sc, R dt0, R ft, uint8_t *mask, int *tile_epoch,
                                                    uint8_t *seg_act, int rec_id, int *list, const InstArgs &ia,
                                                    StageSmem<R> &S, const FirstTiles<R> &first, const Epi &epi = Epi{}) {
    const int lane = threadIdx.x & 31;
    for (int round = 0; sched_more(round, ntiles); ++round) {
        const int tq = staged_tile<R, BATCH>(ha, round, first, ntiles);
        bool need = false;
        if (tq < ntiles) {
            // the clean flags and the bitmask words of the tile, loaded together
            const unsigned long long cf = STATE ? seg_flags(seg_clean, tq) : kAllSegs;
            const uint4 *w4 = reinterpret_cast<const uint4 *>(active + (size_t)tq * (kTileCells / 32));
            const uint4 a = w4[0], b = w4[1];
            need = !cull || cf != kAllSegs || (a.x | a.y | a.z | a.w | b.x | b.y | b.z | b.w) != 0u;
        }
        int ho, hc;
        halo_range(ha, tq, ntiles, ho, hc);
        const int cnt = compact_tiles(need, tq, list, ho, hc, S.hoff, S.hcnt);
        if (cnt == 0) continue;
        if (RECORD && threadIdx.x == 0) atomicAdd(&sc->listed, (unsigned)cnt);
        staged_tiles<R, true>(m, ha, U, kact, cnt, list, S, [&](int t, const StageBuf<R> &b, const int *, bool fast) {
            const int inst = BATCH ? ia.tile_inst[t] : 0;
            const MatConsts &mc = BATCH ? ia.mcs[inst] : mc0;
            const R dt = BATCH ? R(ia.dt[inst]) : dt0;
            const int c = threadIdx.x;
            const int i = t * kTileCells + c;
            const int seg = i >> 5;
            const unsigned word = active[seg];  // marks to clear (padded: bits of cells >= n never set)
            double vol = 0.0;
            bool wet_after = false, act = false;
            if (i < m.n) {
                const R prev[3] = {b.h[c], b.hu[c], b.hv[c]};
                // what this step's coefficient phase left for a wet cell, loaded ahead of the fluxes
                const bool wet = prev[0] > R(DA_TINY);
                const R *kept = (const R *)ha.kept;
                Kept<R> kp{};
                if (wet) {
                    kp.sx = kept[i];
                    kp.sy = kept[(size_t)m.n + i];
                    kp.sgn = ha.fsign[i];
                }
                const auto pre = epi.pre(i, wet);
                const uint8_t bf = b.bf[c];
                StagedView<R> v{b};
                staged_slots(b, c, v.nl);
                act = prev[0] >= R(DA_TINY);
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    if (bf & (1 << s)) continue;
                    act |= b.h[v.nl[s]] >= R(DA_TINY);
                    if (bf & (0x10 << s)) act |= b.h[v.nl[s + 4]] >= R(DA_TINY);
                }
                const R dxc = b.sz[0][c], dyc = b.sz[1][c];
                R st[3] = {prev[0], prev[1], prev[2]};
                bool clamped = false;
                const CellSrc<R> cs = staged_src(b, c);
                // the k act/pass code the coefficient phase recorded
                const uint8_t kcode = RECORD && prev[0] >= R(DA_TINY) ? uint8_t(mask[i] & 3) : uint8_t(0);
                // a wet cell is active: its branch byte as recorded below
                const auto hook = [&](const SrcFwd<R> &f, bool cl) {
                    epi(t, i, v, c, prev, bf, uint8_t(kcode | 8 | (cl ? 4 : 0)), b.gz[c], cs, pre, f);
                };
                if (act) {
                    if constexpr (sizeof(R) == 8) {
                        if (fast)
                            clamped = staged_update<R, true>(v, c, bf, cs, mc, dt, prev, dxc, dyc, st, kp, hook);
                        else
                            clamped = staged_update<R, false>(v, c, bf, cs, mc, dt, prev, dxc, dyc, st, kp, hook);
                    } else {
                        clamped = staged_update<R, true>(v, c, bf, cs, mc, dt, prev, dxc, dyc, st, kp, hook);
                    }
                }
                const uint8_t code = RECORD ? uint8_t(kcode | (act ? 8 : 0) | (clamped ? 4 : 0)) : 0;
                if (RECORD) mask[i] = code;
                if (!isfinite(st[0]) || !isfinite(st[1]) || !isfinite(st[2])) raise_err(sc, DA_ERR_NAN);
                if (STATE) {
                    O.h[i] = st[0];
                    O.hu[i] = st[1];
                    O.hv[i] = st[2];
                }
                vol = double(dxc) * double(dyc) * double(st[0]);
                wet_after = st[0] >= R(DA_TINY);
            }
            const unsigned wet_bits = __ballot_sync(0xffffffffu, wet_after);
            const unsigned act_bits = __ballot_sync(0xffffffffu, act);
            if (STATE) vol = warp_sum(vol);
            if (lane == 0) {
                if (word) active[seg] = 0u;
                if (STATE) {
                    if (act_bits) seg_dirty[seg] = 1;  // changed since the base checkpoint
                    seg_vol[seg] = vol;
                    seg_clean[seg] = act_bits ? 0 : 1;
                    seg_wet[seg] = wet_bits ? 1 : 0;
                }
                if (RECORD) seg_act[seg] = act_bits ? 1 : 0;
            }
            if (RECORD && threadIdx.x == 0) tile_epoch[t] = rec_id;
        });
    }
}

}  // namespace
}  // namespace fwd
}  // namespace da
