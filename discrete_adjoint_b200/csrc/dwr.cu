// Dual-weighted-residual error indicator on the device (error_compute.C:24-119 with the refined
// grid of uniform_refine.C and the reconstruction of bilinear_interp.C).
//
// The context keeps a second context for the error grid (the coarse mesh refined once).  One
// indicator step n -> n+1 from the live state U^n:
//   1. the coarse step U^n -> U^{n+1} (its dt), the state put back afterwards;
//   2. k_dwr_interp: on every fine cell the reconstructed U~^n (written as the error grid's state),
//      U~^{n+1} and lambda~ from the coarse fields through the fixed (cell, weight) pairs;
//   3. one step of the error grid from U~^n with the coarse dt (frozen-dt replay of the device's own
//      value, same iteration);
//   4. k_dwr_residual: r = step(U~^n) - U~^{n+1}; per fine cell |r . (lambda - lambda~)| summed
//      over the three fields (el_error) and r . lambda (correction), lambda the parent's adjoint; per
//      coarse cell the sum over its four children (fixed order), and the totals as compensated FP64
//      sums in a fixed order.
// The error grid's context works on the coarse context's stream and nothing is read on the host, so
// the reverse sweep's indicator steps queue up behind its kernels (three launches a step; with a
// host round trip for dt, iteration and totals, a dt array allocated and freed and the sums' 256 parts
// added by one thread, a step of 10k coarse cells took 210 us).
// An error that the error grid's step raises (a barrier wait that ran out, a state that is not finite, a
// wave speed above the bound) is carried into the coarse scalars, where the end of the sweep or step reads
// it; the next indicator step starts without it.
#include <cuda_runtime.h>

#include <cmath>
#include <cstring>
#include <vector>

#include "da_internal.h"

namespace da {
namespace {

constexpr int kBlock = 256;
constexpr int kParts = 256;

template <class R>
struct Fields {
    const R *h, *hu, *hv;
    __device__ R get(int v, int i) const { return v == 0 ? h[i] : (v == 1 ? hu[i] : hv[i]); }
};

template <class R>
__global__ void __launch_bounds__(kBlock) k_dwr_interp(int nf, const int32_t *__restrict__ idx,
                                                       const double *__restrict__ w, Fields<R> un, Fields<R> unext,
                                                       Fields<R> lam, R *fh, R *fhu, R *fhv,
                                                       double *__restrict__ ut_next, double *__restrict__ lamt,
                                                       uint8_t *__restrict__ seg_clean, uint8_t *__restrict__ seg_wet,
                                                       unsigned *__restrict__ active, int nseg,
                                                       const DevScalars *__restrict__ coarse,
                                                       DevScalars *__restrict__ fine) {
    // the error grid's state is new everywhere, its time that of the step's beginning; nothing of a
    // step that did not end is left (no kernel of the error grid runs beside this one)
    for (int s = blockIdx.x * blockDim.x + threadIdx.x; s < nseg; s += gridDim.x * blockDim.x) {
        seg_clean[s] = 0;
        seg_wet[s] = 1;
        active[s] = 0u;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        fine->time = coarse->time - coarse->dt;  // enters the step only through clipping, which the replay skips
        fine->iter = coarse->iter - 1;
        fine->err = 0;
        fine->bar = 0ull;
        fine->bar_exit = 0ull;
    }
    for (int f = blockIdx.x * blockDim.x + threadIdx.x; f < nf; f += gridDim.x * blockDim.x) {
        double a[3] = {0, 0, 0}, b[3] = {0, 0, 0}, c[3] = {0, 0, 0};
        for (int q = 0; q < 4; ++q) {
            const int k = idx[(size_t)q * nf + f];
            if (k < 0) continue;
            const double wq = w[(size_t)q * nf + f];
            for (int v = 0; v < 3; ++v) {
                a[v] += wq * double(un.get(v, k));
                b[v] += wq * double(unext.get(v, k));
                c[v] += wq * double(lam.get(v, k));
            }
        }
        fh[f] = R(a[0]);
        fhu[f] = R(a[1]);
        fhv[f] = R(a[2]);
        for (int v = 0; v < 3; ++v) {
            ut_next[(size_t)v * nf + f] = b[v];
            lamt[(size_t)v * nf + f] = c[v];
        }
    }
}

// Neumaier's compensated addition: (s, c) += x.
__device__ __forceinline__ void neumaier(double &s, double &c, double x) {
    const double t = s + x;
    if (fabs(s) >= fabs(x))
        c += (s - t) + x;
    else
        c += (x - t) + s;
    s = t;
}

// (s, c) += (s2, c2), both compensated sums: the rounding error of s + s2 goes to the compensation.
__device__ __forceinline__ void add_sums(double &s, double &c, double s2, double c2) {
    neumaier(s, c, s2);
    c += c2;
}
__device__ __forceinline__ void warp_sums(double &s, double &c) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double s2 = __shfl_down_sync(0xffffffffu, s, o), c2 = __shfl_down_sync(0xffffffffu, c, o);
        add_sums(s, c, s2, c2);
    }
}
// Thread 0: the sum over the block's threads, warps in order.
__device__ __forceinline__ void block_sums(double &s, double &c, double (*red)[2]) {
    warp_sums(s, c);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        red[threadIdx.x >> 5][0] = s;
        red[threadIdx.x >> 5][1] = c;
    }
    __syncthreads();
    if (threadIdx.x == 0)
        for (int w = 1; w < kBlock / 32; ++w) add_sums(s, c, red[w][0], red[w][1]);
}

// One thread per coarse cell: its children's residuals and estimates in child order.  Block b takes a
// fixed contiguous range of coarse cells; the last block adds the parts and writes the totals to
// out[0..1].  acc (or null): the estimate per coarse cell is added there too.
template <class R>
__global__ void __launch_bounds__(kBlock) k_dwr_residual(int n, int nf, const int32_t *__restrict__ children, Fields<R> uf,
                                                         const double *__restrict__ ut_next,
                                                         const double *__restrict__ lamt, Fields<R> lam,
                                                         double *__restrict__ err, double *__restrict__ cell,
                                                         double *__restrict__ acc, double *parts, unsigned *done,
                                                         double *__restrict__ out, const DevScalars *__restrict__ fine,
                                                         DevScalars *__restrict__ coarse) {
    __shared__ double red[kBlock / 32][2];
    __shared__ bool last;
    const int per = (n + kParts - 1) / kParts;
    const int i0 = blockIdx.x * per, i1 = min(n, i0 + per);
    double es = 0, ec = 0, cs = 0, cc = 0;
    for (int i = i0 + threadIdx.x; i < i1; i += kBlock) {
        const double l[3] = {double(lam.h[i]), double(lam.hu[i]), double(lam.hv[i])};
        double sum = 0.0;
        for (int q = 0; q < 4; ++q) {
            const int f = children[(size_t)q * n + i];
            if (f < 0) continue;
            double e = 0.0, c = 0.0;
            for (int v = 0; v < 3; ++v) {
                const double r = double(uf.get(v, f)) - ut_next[(size_t)v * nf + f];
                e += fabs(r * (l[v] - lamt[(size_t)v * nf + f]));
                c += r * l[v];
            }
            err[f] = e;
            sum += e;
            neumaier(es, ec, e);
            neumaier(cs, cc, c);
        }
        cell[i] = sum;
        if (acc) acc[i] += sum;
    }
    block_sums(es, ec, red);
    block_sums(cs, cc, red);
    double *p = parts + (size_t)4 * blockIdx.x;
    if (threadIdx.x == 0) {
        p[0] = es;
        p[1] = ec;
        p[2] = cs;
        p[3] = cc;
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    static_assert(kParts == kBlock, "one thread per part");
    p = parts + (size_t)4 * threadIdx.x;
    es = __ldcg(p);
    ec = __ldcg(p + 1);
    cs = __ldcg(p + 2);
    cc = __ldcg(p + 3);
    block_sums(es, ec, red);
    block_sums(cs, cc, red);
    if (threadIdx.x == 0) {
        out[0] = es + ec;
        out[1] = cs + cc;
        *done = 0u;
        if (fine->err != 0 && coarse->dwr_err == 0) coarse->dwr_err = fine->err;
    }
}

template <class R>
Fields<R> fields(void *const U[3]) {
    return Fields<R>{(const R *)U[0], (const R *)U[1], (const R *)U[2]};
}

template <class R>
int run_t(da_ctx *ctx, DwrState &d, int un, int unext, int lam, double *acc, double *out) {
    da_ctx *fc = d.fine;
    const int nf = fc->mesh.n, grid = (ctx->sm_count > 0 ? ctx->sm_count : 148) * 8;
    fc->cur = 0;  // every indicator step uses the same buffers
    k_dwr_interp<R><<<grid, kBlock, 0, ctx->stream>>>(nf, d.interp, d.weight, fields<R>(ctx->U[un]),
                                                      fields<R>(ctx->U[unext]), fields<R>(ctx->lam[lam]),
                                                      (R *)fc->U[0][0], (R *)fc->U[0][1], (R *)fc->U[0][2], d.ut_next,
                                                      d.lamt, fc->seg_clean, fc->seg_wet, fc->active, fc->nseg, ctx->dsc,
                                                      fc->dsc);
    int st = cuda_check(ctx, cudaGetLastError(), "dwr interpolation");
    fc->have_state = true;
    // one step of the error grid from U~^n with the coarse dt, read where the coarse step left it
    fc->tc.dt_replay = &ctx->dsc->dt;
    fc->tc.n_replay = kReplayOne;
    if (!st) {
        st = launch_single_step(fc);
        if (st) set_error(ctx, st, std::string("dwr step of the error grid: ") + da_last_error(fc));
    }
    if (!st) {
        k_dwr_residual<R><<<kParts, kBlock, 0, ctx->stream>>>(ctx->mesh.n, nf, d.children, fields<R>(fc->U[fc->cur]),
                                                              d.ut_next, d.lamt, fields<R>(ctx->lam[lam]), d.err, d.cell,
                                                              acc, d.parts, d.done, out, fc->dsc, ctx->dsc);
        st = cuda_check(ctx, cudaGetLastError(), "dwr residual");
    }
    return st;
}

// The context's scalars in stream order (its stream does not synchronise with the legacy stream).
int read_scalars(da_ctx *ctx) {
    int st = cuda_check(ctx, cudaMemcpyAsync(ctx->hsc, ctx->dsc, sizeof(DevScalars), cudaMemcpyDeviceToHost, ctx->stream),
                        "scalars");
    return st ? st : cuda_check(ctx, cudaStreamSynchronize(ctx->stream), "sync");
}

void free_dwr(da_ctx *ctx) {
    DwrState &d = ctx->dwr;
    if (d.fine) {
        if (ctx->stream) cudaStreamSynchronize(ctx->stream);
        if (d.fine_stream) d.fine->stream = d.fine_stream;  // its own again
        da_destroy(d.fine);
        ctx->sweeps[1].drop();  // it holds launches on the error grid
    }
    if (d.mem) cudaFree(d.mem);
    if (d.acc) cudaFree(d.acc);
    if (d.step_sums) cudaFree(d.step_sums);
    d = DwrState{};
}

}  // namespace

void dwr_release(da_ctx *ctx) { free_dwr(ctx); }

int dwr_indicator(da_ctx *ctx, int un, int unext, int lam, double *acc, double *out) {
    return ctx->p.precision == DA_PREC_FP64 ? run_t<double>(ctx, ctx->dwr, un, unext, lam, acc, out)
                                            : run_t<float>(ctx, ctx->dwr, un, unext, lam, acc, out);
}

int dwr_clear_error(da_ctx *ctx) {
    if (ctx->hsc->dwr_err == 0) return DA_OK;
    return cuda_check(ctx, cudaMemsetAsync(&ctx->dsc->dwr_err, 0, sizeof(int), ctx->stream), "memset");
}

int dwr_error(da_ctx *ctx, const char *where) {
    const int code = ctx->hsc->dwr_err;
    return code ? set_error(ctx, code, std::string(where) + ": the error grid's step: " + da_strerror(code)) : DA_OK;
}

int dwr_accumulators(da_ctx *ctx, int nsteps) {
    DwrState &d = ctx->dwr;
    int st = DA_OK;
    if (!d.acc) st = cuda_check(ctx, cudaMalloc((void **)&d.acc, sizeof(double) * (size_t)ctx->mesh.n), "cudaMalloc(dwr cells)");
    if (!st && d.step_cap < nsteps) {
        if (d.step_sums) cudaFree(d.step_sums);
        d.step_sums = nullptr;
        d.step_cap = 0;
        st = cuda_check(ctx, cudaMalloc((void **)&d.step_sums, sizeof(double) * 2 * (size_t)nsteps), "cudaMalloc(dwr sums)");
        if (!st) d.step_cap = nsteps;
    }
    return st;
}

}  // namespace da

using namespace da;

extern "C" {

int da_dwr_setup(da_ctx *ctx, const da_mesh_soa *fine, const int32_t *parent, const int32_t *interp,
                 const double *weight) {
    if (!ctx || !fine || !parent || !interp || !weight) return DA_ERR_INVALID;
    if (ctx->mesh.n <= 0) return set_error(ctx, DA_ERR_NO_MESH, "da_dwr_setup: no mesh");
    if (ctx->ninst > 0) return set_error(ctx, DA_ERR_INVALID, "da_dwr_setup: ensemble context");
    const int n = ctx->mesh.n, nf = fine->n_cells;
    if (nf <= 0) return set_error(ctx, DA_ERR_INVALID, "da_dwr_setup: empty error grid");
    // host checks: every index in range, every coarse cell with at most four children
    std::vector<int32_t> children((size_t)4 * n, -1);
    std::vector<int> count(n, 0);
    for (int f = 0; f < nf; ++f) {
        const int p = parent[f];
        if (p < 0 || p >= n || count[p] >= 4) return set_error(ctx, DA_ERR_INVALID, "da_dwr_setup: parent map");
        children[(size_t)count[p]++ * n + p] = f;
        for (int q = 0; q < 4; ++q) {
            const int k = interp[(size_t)q * nf + f];
            if (k < -1 || k >= n) return set_error(ctx, DA_ERR_INVALID, "da_dwr_setup: interpolant index");
        }
    }
    cudaSetDevice(ctx->device);
    free_dwr(ctx);
    DwrState &d = ctx->dwr;
    int err = 0;
    d.fine = da_create(&ctx->p, &err);
    if (!d.fine) return set_error(ctx, err, "da_dwr_setup: error-grid context");
    int st = da_upload_mesh(d.fine, fine, 0);
    if (st) {
        set_error(ctx, st, std::string("da_dwr_setup: ") + da_last_error(d.fine));
        free_dwr(ctx);
        return st;
    }
    // the error grid's launches go out on the coarse context's stream, in order with its own
    cudaStreamSynchronize(d.fine->stream);
    d.fine_stream = d.fine->stream;
    d.fine->stream = ctx->stream;
    // device tables: children, interpolants, weights, work arrays
    size_t off = 0;
    auto take = [&](size_t bytes) { const size_t o = off; off = (off + bytes + 255) & ~size_t(255); return o; };
    const size_t o_ch = take(4 * (size_t)4 * n), o_idx = take(4 * (size_t)4 * nf),
                 o_w = take(8 * (size_t)4 * nf), o_ut = take(8 * (size_t)3 * nf), o_lt = take(8 * (size_t)3 * nf),
                 o_err = take(8 * (size_t)nf), o_cell = take(8 * (size_t)n),
                 o_parts = take(8 * (size_t)4 * kParts), o_sums = take(8 * 2), o_done = take(sizeof(unsigned));
    st = cuda_check(ctx, cudaMalloc(&d.mem, off), "cudaMalloc(dwr)");
    if (st) {
        free_dwr(ctx);
        return st;
    }
    unsigned char *b = (unsigned char *)d.mem;
    d.children = (int32_t *)(b + o_ch);
    d.interp = (int32_t *)(b + o_idx);
    d.weight = (double *)(b + o_w);
    d.ut_next = (double *)(b + o_ut);
    d.lamt = (double *)(b + o_lt);
    d.err = (double *)(b + o_err);
    d.cell = (double *)(b + o_cell);
    d.parts = (double *)(b + o_parts);
    d.sums = (double *)(b + o_sums);
    d.done = (unsigned *)(b + o_done);
    d.nf = nf;
    st = cuda_check(ctx, cudaMemsetAsync(d.done, 0, sizeof(unsigned), ctx->stream), "memset");
    if (!st) st = copy_h2d(ctx, d.children, children.data(), 4 * (size_t)4 * n, "copy");
    if (!st) st = copy_h2d(ctx, d.interp, interp, 4 * (size_t)4 * nf, "copy");
    if (!st) st = copy_h2d(ctx, d.weight, weight, 8 * (size_t)4 * nf, "copy");
    if (st) free_dwr(ctx);
    return st;
}

int da_dwr_step(da_ctx *ctx, const double *lambda_next, double *el_error, double *cell_error, double *sums) {
    if (!ctx || !lambda_next) return DA_ERR_INVALID;
    if (!ctx->dwr.fine) return set_error(ctx, DA_ERR_INVALID, "da_dwr_step: no error grid (da_dwr_setup)");
    if (!ctx->have_state) return set_error(ctx, DA_ERR_INVALID, "da_dwr_step: no state");
    cudaSetDevice(ctx->device);
    const size_t n = (size_t)ctx->mesh.n;
    int st = adj_alloc_for_dwr(ctx);
    for (int v = 0; v < 3 && !st; ++v) st = upload_real(ctx, ctx->lam[0][v], lambda_next + v * n);
    // the coarse step n -> n+1 from a base checkpoint, put back afterwards
    if (!st) st = launch_snapshot(ctx, ctx->snaps[0], true);
    if (!st) st = read_scalars(ctx);
    if (!st) st = dwr_clear_error(ctx);
    if (!st) st = launch_single_step(ctx);
    if (!st) st = read_scalars(ctx);
    if (!st) st = device_error(ctx, "da_dwr_step: the coarse step");
    if (!st) st = dwr_indicator(ctx, 1 - ctx->cur, ctx->cur, 0, nullptr, ctx->dwr.sums);
    if (!st) st = launch_snapshot(ctx, ctx->snaps[0], false);
    if (!st) st = read_scalars(ctx);
    if (!st) st = dwr_error(ctx, "da_dwr_step");
    const int nf = ctx->dwr.nf;
    if (!st && el_error) st = copy_d2h(ctx, el_error, ctx->dwr.err, 8 * (size_t)nf, "copy");
    if (!st && cell_error) st = copy_d2h(ctx, cell_error, ctx->dwr.cell, 8 * n, "copy");
    if (!st && sums) st = copy_d2h(ctx, sums, ctx->dwr.sums, 16, "copy");
    return st;
}

}  // extern "C"
