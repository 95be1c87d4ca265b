// Launchers of the adjoint kernels for one precision (included by adjoint_fp64.cu / _fp32.cu).
#pragma once
#include <algorithm>

#include "adjoint_impl.cuh"
#include "forward_impl.cuh"
#include "adjoint_staged.cuh"
#include "adjoint_staged64.cuh"

namespace da {
namespace adj {
namespace {

template <class R>
AdjArgs adj_args(da_ctx *ctx, const double *sec2, double cos_int) {
    AdjArgs a;
    a.mask = ctx->mask;
    a.tile_epoch = ctx->tile_epoch;
    a.seg_act = ctx->seg_act;
    a.lam_clean = ctx->lam_clean;
    a.rec_id = ctx->rec_id;
    a.ntiles = ctx->ntiles;
    a.A = ctx->adjA;
    a.B = ctx->adjB;
    a.gbed = ctx->gbed;
    a.gint = ctx->gint;
    a.dk_dbed = ctx->dk_tab;
    a.dk_dint = ctx->dk_tab + DA_MAX_MATERIALS * 3;
    for (int m = 0; m < DA_MAX_MATERIALS; ++m) a.sec2_bed[m] = sec2[m];
    a.cos_int = cos_int;
    return a;
}

template <class R>
int step_t(da_ctx *ctx, int lam_in, int lam_out, const double *sec2, double cos_int) {
    // the forward step of U^n has just been replayed: U^n is in buffer 1 - cur, its codes in mask
    const MeshArgs m = mesh_args(ctx);
    const int un = 1 - ctx->cur;
    StateRef<R> U{(const R *)ctx->U[un][0], (const R *)ctx->U[un][1], (const R *)ctx->U[un][2]};
    StateRef<R> Ln{(const R *)ctx->lam[lam_in][0], (const R *)ctx->lam[lam_in][1], (const R *)ctx->lam[lam_in][2]};
    StateOut<R> Lo{(R *)ctx->lam[lam_out][0], (R *)ctx->lam[lam_out][1], (R *)ctx->lam[lam_out][2]};
    const AdjArgs aa = adj_args<R>(ctx, sec2, cos_int);
    const int grid = ctx->grid;
    const R floor = R(ctx->mc.sign_floor);
    trace_begin(ctx, TR_ADJ_SRC);
    k_adj_src<R><<<grid, kBlock, 0, ctx->stream>>>(m, U, Ln, ctx->mc, aa, ctx->dsc, floor);
    trace_end(ctx);
    trace_begin(ctx, TR_ADJ_GATHER);
    k_adj_gather<R><<<grid, kBlock, 0, ctx->stream>>>(m, U, Ln, Lo, ctx->mc, aa, ctx->dsc);
    trace_end(ctx);
    return cuda_check(ctx, cudaGetLastError(), "adjoint step launch");
}

template <class R>
int reduce_t(da_ctx *ctx, int lam0, int n_piles) {
    const MeshArgs m = mesh_args(ctx);
    StateRef<R> L{(const R *)ctx->lam[lam0][0], (const R *)ctx->lam[lam0][1], (const R *)ctx->lam[lam0][2]};
    const int nout = ctx->p.n_materials + 1 + n_piles;
    trace_begin(ctx, TR_ADJ_REDUCE);
    k_adj_reduce<R><<<dim3(kReduceParts, nout), kBlock, 0, ctx->stream>>>(m, L, ctx->gbed, ctx->gint, ctx->dh0,
                                                                           ctx->p.n_materials, n_piles, ctx->red_part);
    k_adj_reduce_final<<<nout, kReduceParts, 0, ctx->stream>>>(ctx->red_part, ctx->red_out);
    trace_end(ctx);
    return cuda_check(ctx, cudaGetLastError(), "adjoint reduce launch");
}

// Ensemble gradients: (n_mat + 2) outputs per member into red_out, n_mat the largest material
// count of the members.
template <class R>
int reduce_inst_t(da_ctx *ctx, int lam0) {
    const MeshArgs m = mesh_args(ctx);
    StateRef<R> L{(const R *)ctx->lam[lam0][0], (const R *)ctx->lam[lam0][1], (const R *)ctx->lam[lam0][2]};
    trace_begin(ctx, TR_ADJ_REDUCE);
    const int nout = ctx->inst_mat + 2, n = ctx->ninst * nout;
    // a launch takes at most 65535 members across
    for (int k0 = 0; k0 < ctx->ninst; k0 += 65535) {
        const int nk = ctx->ninst - k0 < 65535 ? ctx->ninst - k0 : 65535;
        k_adj_reduce_inst<R><<<dim3(kInstParts, nk, nout), kBlock, 0, ctx->stream>>>(
            m, L, ctx->gbed, ctx->gint, ctx->dh0, ctx->inst_mat, ctx->ia.seg0 + k0,
            ctx->red_part + (size_t)k0 * nout * kInstParts);
    }
    k_adj_reduce_inst_final<<<(n * 32 + kBlock - 1) / kBlock, kBlock, 0, ctx->stream>>>(ctx->red_part, n, ctx->red_out);
    trace_end(ctx);
    return cuda_check(ctx, cudaGetLastError(), "ensemble reduce launch");
}

// The gather shares its work out by quarter tiles when four times the tiles the recording update
// listed fit in the grid (a flow over few tiles), else by tiles; every block reads the same count
// after the barrier that ends the update.
// split: 0 by that rule, 1 tiles, 2 quarters (da_params.tile_staging 1, 2, 3).
__device__ __forceinline__ bool gather_quarters(const DevScalars *sc, int split) {
    if (split) return split == 2;
    return 4ull * __ldcg(&sc->listed) <= gridDim.x;
}

// The gather of a staged launch in its precision.
template <class R, bool BATCH>
__device__ __forceinline__ void gather_staged(const MeshArgs &m, const fwd::HaloArgs &ha, const StateRef<R> &U,
                                              const StateRef<R> &Ln, const StateOut<R> &Lo, const MatConsts &mc,
                                              const AdjArgs &aa, int rec_id, double dt, int *list, const InstArgs &ia,
                                              void *smem, bool quarter, const fwd::FirstTiles<R> &first) {
    if constexpr (sizeof(R) == 8)
        adj_gather_phase64<BATCH>(m, ha, U, Ln, Lo, mc, aa, rec_id, dt, list, ia, *(GatherSmem64 *)smem, quarter, first);
    else
        adj_gather_phase_staged<R, BATCH>(m, ha, U, Ln, Lo, mc, aa, rec_id, R(dt), list, ia, *(GatherSmem<R> *)smem, quarter, first);
}
template <class R>
constexpr size_t gather_staged_bytes() {
    if constexpr (sizeof(R) == 8)
        return sizeof(GatherSmem64);
    else
        return gather_smem_bytes<R>();
}

// ------------------------------------------------------------------------ k_youturn
// One whole reverse step in one cooperative launch: the forward step of U^n replayed with its
// branch codes recorded (coefficient phase, barrier, dt, update phase), a barrier, the source
// adjoint, a barrier and the gather, i.e. the four launches of the separate path with grid
// barriers instead of kernel boundaries.  U^n stays in buffer cur; U^{n+1} goes to cur ^ 1.
// SEED (the last step of the horizon): lambda^N is seeded from the U^N just produced before the
// adjoint phases, with each segment's part of J.  BATCH: every member with its own constants and
// dt (the members' dt pass between two barriers).  Block 0 writes the step's scalars at the end,
// as the separate kernels do.  pre (mode NONE when unused): a checkpoint restore before the step,
// followed by a barrier.  STAGED: the replayed forward phases stage tiles and halos in shared
// memory (staged_impl.cuh).
template <class R, bool BATCH, bool SEED, int OCC, bool STAGED>
__global__ void __launch_bounds__(kBlock, OCC) k_youturn(MeshArgs m, fwd::StatePair<R> S, int cur, R *kact, unsigned *active,
                                                    uint8_t *seg_clean, uint8_t *seg_wet, double *seg_vol,
                                                    uint8_t *seg_dirty, int ntiles, int cull, MatConsts mc,
                                                    TimeConsts tc, DevScalars *sc, uint8_t *mask, int *tile_epoch,
                                                    uint8_t *seg_act, int rec_id, StateRef<R> Ln, StateOut<R> Lseed,
                                                    StateOut<R> Lo, AdjArgs aa, InstArgs ia, Box box, double *seg_J,
                                                    snap::SnapArgs<R> pre, fwd::HaloArgs ha, int gsplit) {
    __shared__ int list[kBlock];
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    fwd::StageSmem<R> &stg = *reinterpret_cast<fwd::StageSmem<R> *>(dyn_smem);
    __shared__ fwd::FirstTiles<R> first;
    const fwd::FirstLoad<R, BATCH> fl(ha, STAGED ? ntiles : 0);
    // the recording update counts its listed tiles from zero (the adds follow a barrier)
    if (blockIdx.x == 0 && threadIdx.x == 0) sc->listed = 0u;
    if (pre.mode != snap::NONE) {
        snap::snap_segments<R>(pre);
        snap::snap_scalars<R>(pre);
        if (STAGED) fl.store(ha, first);
        if (!fwd::grid_sync(sc)) return;
    } else if (STAGED) {
        fl.store(ha, first);
    }
    const double time = __ldcg(&sc->time);
    const long long iter = __ldcg(&sc->iter);
    const StateRef<R> U{S.h[cur], S.hu[cur], S.hv[cur]};
    const StateOut<R> O{S.h[cur ^ 1], S.hu[cur ^ 1], S.hv[cur ^ 1]};
    unsigned long long my_min = 0x7FF0000000000000ull, my_max = 0ull;
    if (STAGED)
        fwd::coef_phase_staged<R, true, BATCH>(m, ha, U, kact, active, seg_wet, ntiles, cull, mc, sc, mask, list, my_min,
                                               my_max, ia, stg, fwd::sign_threshold<R>(iter, tc, mc), first);
    else
        fwd::coef_phase<R, true, BATCH>(m, U, kact, active, seg_wet, ntiles, cull, mc, sc, mask, list, my_min, my_max,
                                        ia);
    if (!BATCH) fwd::push_minmax(my_min, my_max, &sc->acc_min_dxe, &sc->acc_hmax);
    if (!fwd::grid_sync(sc)) return;
    double dt = 0.0, ft, min_dxe = 0.0, hmax = 0.0;
    if (BATCH) {
        ft = iter < tc.frict_tiny_iters ? tc.frict_tiny_early : tc.frict_tiny_late;
        fwd::inst_dt_pass(ia, iter, tc, sc);
        if (!fwd::grid_sync(sc)) return;
    } else {
        min_dxe = __longlong_as_double(__ldcg(&sc->acc_min_dxe));
        hmax = __longlong_as_double(__ldcg(&sc->acc_hmax));
        fwd::step_dt(min_dxe, hmax, time, iter, tc, dt, ft);
        if (blockIdx.x == 0 && threadIdx.x == 0 && !isfinite(dt)) raise_err(sc, DA_ERR_NAN);
    }
    const R ftr = R(ft) > R(mc.sign_floor) ? R(ft) : R(mc.sign_floor);
    if (STAGED && !SEED) {
        // the source adjoint of each wet cell right after its update, from the tile and halo
        // staged for it (its own branches and lambda^{n+1}, U^n around it: nothing another cell
        // writes in this phase), so the reverse step needs no source phase of its own
        const SrcEpilogue<R, BATCH> src{m, Ln, mc, aa, ia, R(dt)};
        fwd::update_phase_staged<R, true, BATCH>(m, ha, U, O, kact, active, seg_clean, seg_wet, seg_vol, seg_dirty,
                                                 ntiles, cull, mc, sc, R(dt), ftr, mask, tile_epoch, seg_act, rec_id,
                                                 list, ia, stg, first, src);
        if (!fwd::grid_sync(sc)) return;
        gather_staged<R, BATCH>(m, ha, U, Ln, Lo, mc, aa, rec_id, dt, list, ia, dyn_smem, gather_quarters(sc, gsplit), first);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            sc->iter = iter + 1;
            sc->frict_tiny = ft;
            if (!BATCH) {
                sc->time = time + dt;
                sc->dt = dt;
                sc->min_dxe = min_dxe;
                sc->hmax = hmax;
                sc->acc_min_dxe = fwd::kMinDxeStart;
                sc->acc_hmax = 0ull;
            }
        }
        fwd::grid_exit(sc);
        return;
    }
    if (STAGED)
        fwd::update_phase_staged<R, true, BATCH>(m, ha, U, O, kact, active, seg_clean, seg_wet, seg_vol, seg_dirty,
                                                 ntiles, cull, mc, sc, R(dt), ftr, mask, tile_epoch, seg_act, rec_id,
                                                 list, ia, stg, first);
    else
        fwd::update_phase<R, true, BATCH>(m, U, O, kact, active, seg_clean, seg_wet, seg_vol, seg_dirty, ntiles, cull,
                                          mc, sc, R(dt), ftr, mask, tile_epoch, seg_act, rec_id, list, ia);
    if (!fwd::grid_sync(sc)) return;
    if (SEED) {
        seed_phase<R, BATCH>(m, StateRef<R>{O.h, O.hu, O.hv}, Lseed, box, seg_J, ntiles * (kBlock / 32), ia);
        if (!fwd::grid_sync(sc)) return;
    }
    adj_src_phase<R, BATCH>(m, U, Ln, mc, aa, R(dt), ftr, list, ia);
    if (!fwd::grid_sync(sc)) return;
    if (STAGED)
        gather_staged<R, BATCH>(m, ha, U, Ln, Lo, mc, aa, rec_id, dt, list, ia, dyn_smem, gather_quarters(sc, gsplit), first);
    else
        adj_gather_phase<R, BATCH>(m, U, Ln, Lo, mc, aa, R(dt), list, ia);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        sc->iter = iter + 1;
        sc->frict_tiny = ft;
        if (!BATCH) {
            sc->time = time + dt;
            sc->dt = dt;
            sc->min_dxe = min_dxe;
            sc->hmax = hmax;
            sc->acc_min_dxe = fwd::kMinDxeStart;
            sc->acc_hmax = 0ull;
        }
    }
    fwd::grid_exit(sc);
}

// Blocks of a reverse step's launch, cap of them co-resident.
// FP64: every co-resident block, at most four per tile, whatever the forward steps' tuned grid:
// the gather spreads a sparse flow's quarter tiles over them, which outweighs the dearer
// barriers (the forward phases split no tile and keep the tuned grid; in FP32 the shorter
// gather gains less than the barriers cost).  FP32: the tuned grid, but never below one block
// per SM (a forward grid of half the SMs leaves the reverse step short of memory parallelism).
// Results do not depend on it.
template <class R>
int reverse_grid(const da_ctx *ctx, int cap) {
    int want = ctx->grid;
    const int per_sm1 = ctx->sm_count > 0 ? ctx->sm_count : 148;
    if (want < per_sm1) want = per_sm1 < ctx->ntiles ? per_sm1 : ctx->ntiles;
    if (sizeof(R) == 8 && want < 4 * ctx->ntiles) want = 4 * ctx->ntiles;
    return want < cap ? want : cap;
}

// --------------------------------------------------------------------- k_reverse_run
// Consecutive reverse steps, each from a checkpoint of its own state, in one cooperative launch (most
// of a binomial schedule: after a chain of forward steps has stored its checkpoints they are taken
// back one after another).  Per step three phases and barriers -- coefficients, update with the source
// adjoint, gather -- where a launch per step has a fourth for the restore and a kernel boundary: the
// next step's checkpoint goes into the state buffer that this step does not read, while its gather
// runs, and the replayed steps write no state.  A step's chain of phases is latency (a flow of 18 tiles:
// restore 2, coefficients 5, update 7, gather 6, each barrier 1.2, the launch 4 us), so what counts is
// how many there are.  Against a launch per step: 200 steps of 37k cells with 16 checkpoints (runs of
// 5 steps) 10.1 -> 9.6 ms, 512 steps of 1M cells with 32 (runs of 16) 28.3 -> 26.4 ms, 48 steps of 262k
// cells in FP32 3.31 -> 3.14 ms, 24 steps of 191k wet cells 4.03 -> 3.88 ms.
//
// The two state buffers are tracked on their own: dirty[b] the segments of buffer b that may differ
// from the base checkpoint, wet[b] those with a wet cell (of the base where they do not differ).  The
// live dirty flags cover both buffers at every moment, as the restore that follows every run expects:
// also the one after a run that a barrier timeout has cut short.
constexpr int kRunMax = 32;  // steps of a launch

template <class R>
struct RunArgs {
    int n;                         // steps
    unsigned char *slot[kRunMax];  // their checkpoints (slot[0] null: the live state in buffer cur)
    size_t array_bytes;            // a slot's layout: three state arrays, the dirty flags, the scalars
    size_t scalars_at;
    const R *base[3];              // the base checkpoint
    uint8_t *dirty[2], *wet[2];    // [nseg]
    int nseg;
};

// Checkpoint k of the run into state buffer b (snap_segments' division of the work).
template <class R>
__device__ __forceinline__ void run_restore(const RunArgs<R> &ra, int k, int b, const fwd::StatePair<R> &S, int n,
                                            uint8_t *seg_dirty) {
    const int lane = threadIdx.x & 31;
    const int W = (gridDim.x * blockDim.x) >> 5;
    const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const unsigned char *slot = ra.slot[k];
    const bool is_base = (const R *)slot == ra.base[0];  // whose cells all hold the base
    const uint8_t *snap_dirty = slot + 3 * ra.array_bytes;
    uint8_t *dirty = b ? ra.dirty[1] : ra.dirty[0], *wet = b ? ra.wet[1] : ra.wet[0];
    R *dst[3] = {b ? S.h[1] : S.h[0], b ? S.hu[1] : S.hu[0], b ? S.hv[1] : S.hv[0]};
    for (int s0 = 0; s0 < ra.nseg; s0 += 32 * W) {
        const int s = s0 + lane * W + w;
        bool flag = false, work = false;
        if (s < ra.nseg) {
            flag = !is_base && snap_dirty[s] != 0;
            work = flag || dirty[s];
            if (work) dirty[s] = flag;
            if (flag) seg_dirty[s] = 1;
        }
        unsigned bits = __ballot_sync(0xffffffffu, work);
        const unsigned from = __ballot_sync(0xffffffffu, flag);
        while (bits) {
            const int q = __ffs(bits) - 1;
            bits &= bits - 1;
            const int seg = s0 + q * W + w, i = seg * 32 + lane;
            R h = R(0);
            if (i < n) {
#pragma unroll
                for (int v = 0; v < 3; ++v) {
                    const R x = (from >> q) & 1u ? ((const R *)(slot + v * ra.array_bytes))[i] : ra.base[v][i];
                    dst[v][i] = x;
                    if (v == 0) h = x;
                }
            }
            const bool any = __any_sync(0xffffffffu, h >= R(DA_TINY));
            if (lane == 0) wet[seg] = any;
        }
    }
}

template <class R, int OCC>
__global__ void __launch_bounds__(kBlock, OCC) k_reverse_run(MeshArgs m, fwd::StatePair<R> S, int cur, R *kact,
                                                             unsigned *active, uint8_t *seg_wet, uint8_t *seg_dirty,
                                                             int ntiles, int cull, MatConsts mc, TimeConsts tc,
                                                             DevScalars *sc, uint8_t *mask, int *tile_epoch,
                                                             uint8_t *seg_act, int rec_id0, fwd::StatePair<R> L,
                                                             int lam_in, AdjArgs aa, RunArgs<R> ra, fwd::HaloArgs ha,
                                                             int gsplit) {
    __shared__ int list[kBlock];
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    fwd::StageSmem<R> &stg = *reinterpret_cast<fwd::StageSmem<R> *>(dyn_smem);
    const int t0 = blockIdx.x * blockDim.x + threadIdx.x, nt = gridDim.x * blockDim.x;
    __shared__ fwd::FirstTiles<R> first;
    const fwd::FirstLoad<R, false> fl(ha, ntiles);
    for (int s = t0; s < ra.nseg; s += nt) {
        const uint8_t d = seg_dirty[s], w = seg_wet[s];
        ra.dirty[0][s] = ra.dirty[1][s] = d;
        ra.wet[0][s] = ra.wet[1][s] = w;
    }
    // the first step's state: live (its wet flags too), or its checkpoint after a barrier
    if (ra.slot[0]) {
        if (!fwd::grid_sync(sc)) return;
        run_restore<R>(ra, 0, cur, S, m.n, seg_dirty);
        fl.store(ha, first);
        if (!fwd::grid_sync(sc)) return;
    } else {
        fl.store(ha, first);
    }
    for (int k = 0; k < ra.n; ++k) {
        const int p = (cur + k) & 1, rec_id = rec_id0 + k;
        const DevScalars *from = ra.slot[k] ? (const DevScalars *)(ra.slot[k] + ra.scalars_at) : sc;
        const double time = __ldcg(&from->time);
        const long long iter = __ldcg(&from->iter);
        const R ftr = fwd::sign_threshold<R>(iter, tc, mc);
        const StateRef<R> U{S.h[p], S.hu[p], S.hv[p]};
        const int li = (lam_in + k) & 1;
        const StateRef<R> Ln{L.h[li], L.hu[li], L.hv[li]};
        const StateOut<R> Lo{L.h[li ^ 1], L.hu[li ^ 1], L.hv[li ^ 1]};
        unsigned long long *acc_min = k & 1 ? &sc->acc_alt_min_dxe : &sc->acc_min_dxe;
        unsigned long long *acc_max = k & 1 ? &sc->acc_alt_hmax : &sc->acc_hmax;
        // the recording update counts its listed tiles from zero (the adds follow a barrier)
        if (blockIdx.x == 0 && threadIdx.x == 0) sc->listed = 0u;
        unsigned long long my_min = 0x7FF0000000000000ull, my_max = 0ull;
        fwd::coef_phase_staged<R, true>(m, ha, U, kact, active, ra.slot[k] ? ra.wet[p] : seg_wet, ntiles, cull, mc, sc,
                                        mask, list, my_min, my_max, InstArgs{}, stg, ftr, first);
        fwd::push_minmax(my_min, my_max, acc_min, acc_max);
        if (!fwd::grid_sync(sc)) return;
        const double min_dxe = __longlong_as_double(__ldcg(acc_min)), hmax = __longlong_as_double(__ldcg(acc_max));
        double dt, ft;
        fwd::step_dt(min_dxe, hmax, time, iter, tc, dt, ft);
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            if (!isfinite(dt)) raise_err(sc, DA_ERR_NAN);
            // the other pair was read by every block before the last step's second barrier
            *(k & 1 ? &sc->acc_min_dxe : &sc->acc_alt_min_dxe) = fwd::kMinDxeStart;
            *(k & 1 ? &sc->acc_hmax : &sc->acc_alt_hmax) = 0ull;
        }
        const SrcEpilogue<R, false> src{m, Ln, mc, aa, InstArgs{}, R(dt)};
        fwd::update_phase_staged<R, true, false, false>(m, ha, U, StateOut<R>{}, kact, active, nullptr, nullptr, nullptr,
                                                        nullptr, ntiles, cull, mc, sc, R(dt), ftr, mask, tile_epoch,
                                                        seg_act, rec_id, list, InstArgs{}, stg, first, src);
        if (!fwd::grid_sync(sc)) return;
        gather_staged<R, false>(m, ha, U, Ln, Lo, mc, aa, rec_id, dt, list, InstArgs{}, dyn_smem,
                                gather_quarters(sc, gsplit), first);
        if (k + 1 < ra.n) {
            run_restore<R>(ra, k + 1, p ^ 1, S, m.n, seg_dirty);
            if (!fwd::grid_sync(sc)) return;
        } else if (blockIdx.x == 0 && threadIdx.x == 0) {
            // the last step's scalars, as a launch of its own leaves them
            sc->iter = iter + 1;
            sc->frict_tiny = ft;
            sc->time = time + dt;
            sc->dt = dt;
            sc->min_dxe = min_dxe;
            sc->hmax = hmax;
            sc->acc_min_dxe = sc->acc_alt_min_dxe = fwd::kMinDxeStart;
            sc->acc_hmax = sc->acc_alt_hmax = 0ull;
        }
    }
    fwd::grid_exit(sc);
}

// The steps of slots[0..n) (slots[0] may be null: the live state), lambda from buffer lam_in; afterwards
// it is in lam_in ^ (n & 1) and the state is to be restored.
template <class R>
int reverse_run_t(da_ctx *ctx, int lam_in, const double *sec2, double cos_int, void *const *slots, int n) {
    if (n < 1 || n > kRunMax || ctx->ninst > 0 || !fwd::staged_ok(ctx))
        return set_error(ctx, DA_ERR_INVALID, "reverse run: not for this context");
    const int pi = sizeof(R) == 8, occ3 = ctx->p.blocks_per_sm == 3;
    const void *kern = occ3 ? (const void *)k_reverse_run<R, 3> : (const void *)k_reverse_run<R, 2>;
    const size_t smem = std::max(fwd::stage_smem_bytes<R>(), gather_staged_bytes<R>());
    int &cap = ctx->coop_cap_run[pi + 2 * occ3];
    if (cap <= 0) {
        int st = cuda_check(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                            "shared memory attribute");
        int per_sm = 0;
        if (!st)
            st = cuda_check(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBlock, smem), "occupancy");
        if (st) return st;
        cap = per_sm * (ctx->sm_count > 0 ? ctx->sm_count : 1);
    }
    if (cap <= 0) return set_error(ctx, DA_ERR_UNSUPPORTED, "reverse-run kernel cannot be resident");
    const int grid = reverse_grid<R>(ctx, cap);
    const int rec_id0 = ctx->rec_id + 1;
    ctx->rec_id += n;
    MeshArgs m = mesh_args(ctx);
    fwd::StatePair<R> S, L;
    for (int b = 0; b < 2; ++b) {
        S.h[b] = (R *)ctx->U[b][0];
        S.hu[b] = (R *)ctx->U[b][1];
        S.hv[b] = (R *)ctx->U[b][2];
        L.h[b] = (R *)ctx->lam[b][0];
        L.hu[b] = (R *)ctx->lam[b][1];
        L.hv[b] = (R *)ctx->lam[b][2];
    }
    const snap::SnapArgs<R> sa = snap::snap_args<R>(ctx, ctx->snaps[0], false, ctx->cur);
    RunArgs<R> ra{};
    ra.n = n;
    for (int k = 0; k < n; ++k) ra.slot[k] = (unsigned char *)slots[k];
    ra.array_bytes = (size_t)((unsigned char *)sa.snap[1] - (unsigned char *)sa.snap[0]);
    ra.scalars_at = (size_t)((unsigned char *)sa.snap_sc - (unsigned char *)ctx->snaps[0]);
    for (int v = 0; v < 3; ++v) ra.base[v] = sa.base[v];
    ra.nseg = ctx->nseg;
    for (int b = 0; b < 2; ++b) {
        ra.dirty[b] = ctx->run_flags + (size_t)(2 * b) * ctx->nseg;
        ra.wet[b] = ctx->run_flags + (size_t)(2 * b + 1) * ctx->nseg;
    }
    int cur = ctx->cur, ntiles = ctx->ntiles, cull = ctx->p.tile_culling, rid = rec_id0, li = lam_in;
    R *kact = (R *)ctx->kact;
    unsigned *active = ctx->active;
    uint8_t *seg_wet = ctx->seg_wet, *seg_dirty = ctx->seg_dirty, *mask = ctx->mask, *seg_act = ctx->seg_act;
    int *tile_epoch = ctx->tile_epoch;
    MatConsts mc = ctx->mc;
    TimeConsts tc = ctx->tc;
    DevScalars *sc = ctx->dsc;
    AdjArgs aa = adj_args<R>(ctx, sec2, cos_int);
    fwd::HaloArgs ha = fwd::halo_args(ctx);
    int gsplit = ctx->p.tile_staging >= 2 ? ctx->p.tile_staging - 1 : 0;
    void *args[] = {&m,    &S,          &cur,     &kact, &active, &seg_wet, &seg_dirty, &ntiles, &cull, &mc, &tc,
                    &sc,   &mask,       &tile_epoch, &seg_act, &rid, &L, &li, &aa, &ra, &ha, &gsplit};
    trace_begin(ctx, TR_YOUTURN);
    const cudaError_t e = cudaLaunchCooperativeKernel(kern, grid, kBlock, args, smem, ctx->stream);
    trace_end(ctx, n);
    return cuda_check(ctx, e, "reverse-run launch");
}

// The k_youturn instantiation for the launch's flags.
template <class R>
const void *youturn_kernel(bool batch, bool seed, bool occ3, bool staged) {
#define DA_YT(B, S, O, G) (const void *)k_youturn<R, B, S, O, G>
#define DA_YT_OCC(B, S, G) (occ3 ? DA_YT(B, S, 3, G) : DA_YT(B, S, 2, G))
#define DA_YT_SEED(B, G) (seed ? DA_YT_OCC(B, true, G) : DA_YT_OCC(B, false, G))
#define DA_YT_BATCH(G) (batch ? DA_YT_SEED(true, G) : DA_YT_SEED(false, G))
    return staged ? DA_YT_BATCH(true) : DA_YT_BATCH(false);
#undef DA_YT_BATCH
#undef DA_YT_SEED
#undef DA_YT_OCC
#undef DA_YT
}

// The live state is U^n in buffer cur; afterwards U^{n+1} is (cur flips) and lambda^n is in
// lam_out.  seed: lambda^N goes into lam_in first (from U^{n+1} = U^N) with J's segment parts.
// pre_slot (or null): a checkpoint slot restored first, in the same launch (the live state is then
// the restored one).
template <class R>
int youturn_t(da_ctx *ctx, int lam_in, int lam_out, const double *sec2, double cos_int, bool seed,
              const double *box4, void *pre_slot) {
    const int pi = sizeof(R) == 8;
    const bool batch = ctx->ninst > 0;
    const int occ3 = ctx->p.blocks_per_sm == 3;
    const bool staged = fwd::staged_ok(ctx);
    const void *kern = youturn_kernel<R>(batch, seed, occ3, staged);
    // the staged phases and the staged gather use the same dynamic shared memory in turn
    const size_t smem = staged ? std::max(fwd::stage_smem_bytes<R>(), gather_staged_bytes<R>()) : 0;
    int &cap_ref = ctx->coop_cap_yt[pi + 2 * batch + 4 * seed + 8 * occ3 + 16 * staged];
    if (cap_ref <= 0) {
        int st = DA_OK;
        if (staged)
            st = cuda_check(ctx, cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem),
                            "shared memory attribute");
        int per_sm = 0;
        if (!st)
            st = cuda_check(ctx, cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBlock, smem),
                            "occupancy");
        if (st) return st;
        cap_ref = per_sm * (ctx->sm_count > 0 ? ctx->sm_count : 1);
    }
    const int cap = cap_ref;
    if (cap <= 0) return set_error(ctx, DA_ERR_UNSUPPORTED, "reverse-step kernel cannot be resident");
    const int grid = reverse_grid<R>(ctx, cap);
    ++ctx->rec_id;
    MeshArgs m = mesh_args(ctx);
    fwd::StatePair<R> S;
    for (int b = 0; b < 2; ++b) {
        S.h[b] = (R *)ctx->U[b][0];
        S.hu[b] = (R *)ctx->U[b][1];
        S.hv[b] = (R *)ctx->U[b][2];
    }
    int cur = ctx->cur, ntiles = ctx->ntiles, cull = ctx->p.tile_culling, rec_id = ctx->rec_id;
    R *kact = (R *)ctx->kact;
    unsigned *active = ctx->active;
    uint8_t *seg_clean = ctx->seg_clean, *seg_wet = ctx->seg_wet, *mask = ctx->mask, *seg_act = ctx->seg_act;
    int *tile_epoch = ctx->tile_epoch;
    double *seg_vol = ctx->seg_vol, *seg_J = ctx->seg_J;
    uint8_t *seg_dirty = ctx->seg_dirty;
    MatConsts mc = ctx->mc;
    TimeConsts tc = ctx->tc;
    DevScalars *sc = ctx->dsc;
    StateRef<R> Ln{(const R *)ctx->lam[lam_in][0], (const R *)ctx->lam[lam_in][1], (const R *)ctx->lam[lam_in][2]};
    StateOut<R> Ls{(R *)ctx->lam[lam_in][0], (R *)ctx->lam[lam_in][1], (R *)ctx->lam[lam_in][2]};
    StateOut<R> Lo{(R *)ctx->lam[lam_out][0], (R *)ctx->lam[lam_out][1], (R *)ctx->lam[lam_out][2]};
    AdjArgs aa = adj_args<R>(ctx, sec2, cos_int);
    InstArgs ia = ctx->ia;
    Box box{};
    if (box4)
        for (int q = 0; q < 4; ++q) box.v[q] = box4[q];
    if (seed) {
        // lambda^N is written everywhere: the two adjoint buffers differ on every segment
        int st = cuda_check(ctx, cudaMemsetAsync(ctx->lam_clean, 0, ctx->nseg, ctx->stream), "memset");
        if (st) return st;
    }
    snap::SnapArgs<R> pre = pre_slot ? snap::snap_args<R>(ctx, pre_slot, false, cur) : snap::no_snap<R>();
    fwd::HaloArgs ha = fwd::halo_args(ctx);
    int gsplit = ctx->p.tile_staging >= 2 ? ctx->p.tile_staging - 1 : 0;
    void *args[] = {&m,      &S,    &cur, &kact, &active, &seg_clean, &seg_wet,    &seg_vol, &seg_dirty,
                    &ntiles, &cull, &mc,  &tc,   &sc,     &mask,      &tile_epoch, &seg_act, &rec_id,
                    &Ln,     &Ls,   &Lo,  &aa,   &ia,     &box,       &seg_J,      &pre,     &ha,      &gsplit};
    trace_begin(ctx, TR_YOUTURN);
    const cudaError_t e = cudaLaunchCooperativeKernel(kern, grid, kBlock, args, smem, ctx->stream);
    trace_end(ctx);
    if (e != cudaSuccess) return cuda_check(ctx, e, "reverse-step launch");
    ctx->cur = cur ^ 1;
    return DA_OK;
}

// Per-member J (or the single J) from the segments' parts, fixed order; one block per member.
template <class R>
int functional_t(da_ctx *ctx, double *out) {
    const int nm = ctx->ninst > 0 ? ctx->ninst : 1;
    trace_begin(ctx, TR_ADJ_SEED);
    k_inst_sum<<<nm, kBlock, 0, ctx->stream>>>(ctx->seg_J, ctx->ninst > 0 ? ctx->ia.seg0 : nullptr, ctx->nseg, out);
    trace_end(ctx);
    return cuda_check(ctx, cudaGetLastError(), "functional launch");
}

}  // namespace
}  // namespace adj
}  // namespace da
