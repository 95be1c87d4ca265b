// Flow statistics of the current state (calc_stats, src/geoflow/stats.C:31-360) and the
// discharge through planes (DISCHARGE::update, src/header/properties.h:964-1133), on the device.
//
// One launch, one pass over the cells: block b of kParts sums a fixed contiguous range of cells
// (thread-strided, then a shuffle tree per warp, then the warps in order), the last block to finish
// adds the parts (a warp per value): FP64 sums in a fixed order (the reference sums in hash-table
// order, so the two agree to rounding).  The pass is a latency chain at ordinary sizes, not
// bandwidth; summing the block's 256 values by one thread, and the 256 parts by one thread of a
// second launch, took most of it.
#include <cuda_runtime.h>

#include <cmath>
#include <vector>

#include "da_internal.h"
#include "fv_device.cuh"

namespace da {
namespace {

using namespace fv;

constexpr int kBlock = 256;
constexpr int kParts = 256;
constexpr int kSums = 14;   // xC yC rC area v_ave vx_ave vy_ave slope_ave energy slopevol testvol xVar yVar u_ave
constexpr int kMax = 3;     // max_height v_max u_max
constexpr int kMin = 4;     // xmin, -xmax, ymin, -ymax (over h >= hxyminmax)
constexpr int kPoint = kSums + kMax + kMin;  // test point: squared distance, reach
constexpr int kPlane0 = kPoint + 2;          // discharge per plane
constexpr int kPartLen = kPlane0 + DA_MAX_PLANES;
constexpr int kResPlane0 = 24;               // the result: 23 statistics, then the planes
constexpr int kResLen = kResPlane0 + DA_MAX_PLANES;

enum SlotOp { kAdd, kTakeMax, kTakeMin };
__device__ __forceinline__ int slot_op(int q) {
    return q < kSums ? kAdd : (q < kSums + kMax ? kTakeMax : (q < kPoint ? kTakeMin : kAdd));
}
__device__ __forceinline__ double combine(int op, double a, double b) {
    return op == kAdd ? a + b : (op == kTakeMax ? (b > a ? b : a) : (b < a ? b : a));
}
// the nearer test-point candidate (a tie takes the higher reach)
__device__ __forceinline__ void take_point(double &d, double &r, double d2, double r2) {
    if (d2 < d || (d2 == d && r2 > r)) {
        d = d2;
        r = r2;
    }
}
template <int OP>
__device__ __forceinline__ double warp_pick(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = combine(OP, v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ void warp_point(double &d, double &r) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double d2 = __shfl_xor_sync(0xffffffffu, d, o), r2 = __shfl_xor_sync(0xffffffffu, r, o);
        take_point(d, r, d2, r2);
    }
}

struct StatArgs {
    double min_height, hxyminmax, heightifreach, tx, ty;
    int n_planes;
    double planes[DA_MAX_PLANES][10];  // DISCHARGE::init's precomputed rows (properties.h:925-959)
};

// DISCHARGE::update for one cell and one plane (properties.h:965-1133): the plane segment clipped
// to the cell, the flux (hu dy - hv dx) through it.  nodes: 4 corners (SW, SE, NE, NW), 4 edge
// midpoints (S, E, N, W), centre.
__device__ double plane_flux(const double nodes[9][2], double hu, double hv, const double *pl) {
    double nearest[2], ip[2][2];
    double dxn[4], dyn[4];
    const double half = (fabs(nodes[6][0] - nodes[4][0]) + fabs(nodes[6][1] - nodes[4][1]) +
                         fabs(nodes[7][0] - nodes[5][0]) + fabs(nodes[7][1] - nodes[5][1])) *
                        0.25;
    const double half2 = half * half;
    const double err = half / 524288.0;
    for (int c1 = 0; c1 < 4; ++c1) {
        const int c2 = (c1 + 1) % 4;
        dxn[c1] = nodes[c2][0] - nodes[c1][0];
        dyn[c1] = nodes[c2][1] - nodes[c1][1];
    }
    double s1 = nodes[8][1] * pl[5] + nodes[8][0] * pl[4];
    nearest[0] = (-pl[5] * pl[7] + pl[4] * s1) / pl[6];
    nearest[1] = (+pl[4] * pl[7] + pl[5] * s1) / pl[6];
    const double d2 = (nodes[8][0] - nearest[0]) * (nodes[8][0] - nearest[0]) +
                      (nodes[8][1] - nearest[1]) * (nodes[8][1] - nearest[1]);
    if (!(d2 < half2 * pl[8])) return 0.0;
    int ni = 0;
    for (int c1 = 0; c1 < 4; ++c1) {
        s1 = nodes[c1][1] * dxn[c1] - nodes[c1][0] * dyn[c1];
        const double s2 = dxn[c1] * pl[5] - dyn[c1] * pl[4];
        if ((s2 < 0) || (s2 > 0)) {
            ip[ni][0] = (pl[4] * s1 - dxn[c1] * pl[7]) / s2;
            ip[ni][1] = (pl[5] * s1 - dyn[c1] * pl[7]) / s2;
            if (((ip[ni][0] < pl[0] - err) && (pl[0] < pl[1])) || ((ip[ni][0] > pl[0] + err) && (pl[0] > pl[1])) ||
                ((ip[ni][1] < pl[2] - err) && (pl[2] < pl[3])) || ((ip[ni][1] > pl[2] + err) && (pl[2] > pl[3]))) {
                ip[ni][0] = pl[0];
                ip[ni][1] = pl[2];
            } else if (((ip[ni][0] < pl[1] - err) && (pl[1] < pl[0])) ||
                       ((ip[ni][0] > pl[1] + err) && (pl[1] > pl[0])) ||
                       ((ip[ni][1] < pl[3] - err) && (pl[3] < pl[2])) ||
                       ((ip[ni][1] > pl[3] + err) && (pl[3] > pl[2]))) {
                ip[ni][0] = pl[1];
                ip[ni][1] = pl[3];
            }
            if (((((ip[ni][0] - ip[0][0]) * (ip[ni][0] - ip[0][0]) + (ip[ni][1] - ip[0][1]) * (ip[ni][1] - ip[0][1])) >
                  (half / 512.0)) ||
                 (ni == 0)) &&
                (s2 != 0.0))
                ++ni;
            if (ni == 2) {
                if ((ip[1][0] - ip[0][0]) * (pl[1] - pl[0]) + (ip[1][1] - ip[0][1]) * (pl[3] - pl[2]) < 0.0) {
                    double t = ip[0][0];
                    ip[0][0] = ip[1][0];
                    ip[1][0] = t;
                    t = ip[0][1];
                    ip[0][1] = ip[1][1];
                    ip[1][1] = t;
                }
                break;
            }
        }
    }
    if (ni == 1) {
        const double e1 = (nodes[8][0] - pl[0]) * (nodes[8][0] - pl[0]) + (nodes[8][1] - pl[2]) * (nodes[8][1] - pl[2]);
        const double e2 = (nodes[8][0] - pl[1]) * (nodes[8][0] - pl[1]) + (nodes[8][1] - pl[3]) * (nodes[8][1] - pl[3]);
        if (e1 <= e2) {
            ip[1][0] = pl[0];
            ip[1][1] = pl[2];
        } else {
            ip[1][0] = pl[1];
            ip[1][1] = pl[3];
        }
        ni = 2;
    }
    if (ni != 2) return 0.0;
    return hu * (ip[1][1] - ip[0][1]) - hv * (ip[1][0] - ip[0][0]);
}

template <class R>
__global__ void __launch_bounds__(kBlock) k_stats(MeshArgs m, StateRef<R> U, StatArgs a, double vslump, double *parts,
                                                  unsigned *done, double *res) {
    // the owned cells (a subdomain's ghosts are another subdomain's)
    const int per = (m.n_owned + kParts - 1) / kParts;
    const int i0 = blockIdx.x * per, i1 = min(m.n_owned, i0 + per);
    double s[kSums] = {}, mx[kMax] = {}, mn[kMin], dis[DA_MAX_PLANES] = {};
    for (int q = 0; q < kMin; ++q) mn[q] = HUGE_VAL;
    double tdist = 1073741824.0, treach = 0.0;  // stats.C:58
    for (int i = i0 + threadIdx.x; i < i1; i += kBlock) {
        const double h = double(U.h[i]), hu = double(U.hu[i]), hv = double(U.hv[i]);
        const double x = m.x[i], y = m.y[i], dx = m.dx ? m.dx[i] : double(m.fdx[i]), dy = m.dy ? m.dy[i] : double(m.fdy[i]);
        if (a.n_planes > 0 && (hu != 0.0 || hv != 0.0)) {  // no momentum, no flux through a plane
            double nodes[9][2] = {{x - 0.5 * dx, y - 0.5 * dy}, {x + 0.5 * dx, y - 0.5 * dy}, {x + 0.5 * dx, y + 0.5 * dy},
                                  {x - 0.5 * dx, y + 0.5 * dy}, {x, y - 0.5 * dy},             {x + 0.5 * dx, y},
                                  {x, y + 0.5 * dy},             {x - 0.5 * dx, y},             {x, y}};
            for (int p = 0; p < a.n_planes; ++p) dis[p] += plane_flux(nodes, hu, hv, a.planes[p]);
        }
        if (!(h > a.min_height)) continue;
        mx[0] = h > mx[0] ? h : mx[0];
        if (h >= a.hxyminmax) {
            mn[0] = x < mn[0] ? x : mn[0];
            mn[1] = -x < mn[1] ? -x : mn[1];
            mn[2] = y < mn[2] ? y : mn[2];
            mn[3] = -y < mn[3] ? -y : mn[3];
        }
        const double d2 = (x - a.tx) * (x - a.tx) + (y - a.ty) * (y - a.ty);
        if (d2 < tdist) {
            tdist = d2;
            treach = h >= a.heightifreach ? 1.0 : 0.0;
        }
        const double dA = dx * dy, dV = h * dA;
        s[3] += dA;
        s[10] += dV;
        s[0] += x * dV;
        s[1] += y * dV;
        s[11] += x * x * dV;
        s[12] += y * y * dV;
        s[2] += sqrt((x - 1.2) * (x - 1.2) + (y - 0.3) * (y - 0.3)) * dV;  // xCen, yCen of stats.C:68-69
        const double sp = sqrt(hu * hu + hv * hv) * dA;
        s[4] += sp;
        s[13] += sp;
        double v0 = 0, v1 = 0;
        if (h > DA_TINY) {  // Element::eval_velocity at the centre
            v0 = hu / h;
            v1 = hv / h;
        }
        const double vm = sqrt(v0 * v0 + v1 * v1);
        mx[1] = vm > mx[1] ? vm : mx[1];
        mx[2] = vm > mx[2] ? vm : mx[2];
        s[5] += hu * dA;
        s[6] += hv * dA;
        s[8] += .5 * (9.8 * h * h + h * (v0 * v0 + v1 * v1)) * dA;
        if (vm > DA_TINY) {
            // terrain slope from the gravity vector: (dz/dx, dz/dy) = -(g_x, g_y) / g_z
            const double gz = m.g ? m.g[(size_t)2 * m.n + i] : double(m.fg[(size_t)2 * m.n + i]);
            const double gx = m.g ? m.g[i] : double(m.fg[i]);
            const double gy = m.g ? m.g[(size_t)m.n + i] : double(m.fg[(size_t)m.n + i]);
            const double xs = -gx / gz, ys = -gy / gz;
            s[7] += -(hu * xs + hv * ys) * dA / vm;
            s[9] += dV;
        }
    }
    // The block's values: each warp by shuffles, then the warps' values in order.  parts[slot][block].
    __shared__ double sh[kPartLen + 1][kBlock / 32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < kSums; ++q) {
        const double v = warp_sum(s[q]);
        if (lane == 0) sh[q][warp] = v;
    }
#pragma unroll
    for (int q = 0; q < kMax; ++q) {
        const double v = warp_pick<kTakeMax>(mx[q]);
        if (lane == 0) sh[kSums + q][warp] = v;
    }
#pragma unroll
    for (int q = 0; q < kMin; ++q) {
        const double v = warp_pick<kTakeMin>(mn[q]);
        if (lane == 0) sh[kSums + kMax + q][warp] = v;
    }
    warp_point(tdist, treach);
    if (lane == 0) {
        sh[kPoint][warp] = tdist;
        sh[kPoint + 1][warp] = treach;
    }
    for (int p = 0; p < a.n_planes; ++p) {
        const double v = warp_sum(dis[p]);
        if (lane == 0) sh[kPlane0 + p][warp] = v;
    }
    __syncthreads();
    const int nslot = kPlane0 + a.n_planes;
    for (int q = threadIdx.x; q < nslot; q += kBlock) {
        if (q == kPoint + 1) continue;  // with its distance
        double v = sh[q][0], r = q == kPoint ? sh[q + 1][0] : 0.0;
        for (int w = 1; w < kBlock / 32; ++w) {
            if (q == kPoint)
                take_point(v, r, sh[q][w], sh[q + 1][w]);
            else
                v = combine(slot_op(q), v, sh[q][w]);
        }
        parts[(size_t)q * kParts + blockIdx.x] = v;
        if (q == kPoint) parts[(size_t)(q + 1) * kParts + blockIdx.x] = r;
    }
    // the last block to finish adds the blocks' parts (a warp per slot: lane l takes parts l, l + 32,
    // ... in order, then a shuffle tree) and forms the statistics
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int q = warp; q < nslot; q += kBlock / 32) {
        if (q == kPoint + 1) continue;
        const double *pq = parts + (size_t)q * kParts;
        double v = __ldcg(pq + lane), r = q == kPoint ? __ldcg(pq + kParts + lane) : 0.0;
        for (int b = lane + 32; b < kParts; b += 32) {
            if (q == kPoint)
                take_point(v, r, __ldcg(pq + b), __ldcg(pq + kParts + b));
            else
                v = combine(slot_op(q), v, __ldcg(pq + b));
        }
        const int op = slot_op(q);
        if (q == kPoint)
            warp_point(v, r);
        else if (op == kTakeMax)
            v = warp_pick<kTakeMax>(v);
        else if (op == kTakeMin)
            v = warp_pick<kTakeMin>(v);
        else
            v = warp_sum(v);
        if (lane == 0) {
            sh[q][0] = v;
            if (q == kPoint) sh[q + 1][0] = r;
        }
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    *done = 0u;
    auto S = [&](int q) { return sh[q][0]; };
    // stats.C:271-302 with LENGTH_SCALE = HEIGHT_SCALE = velocity scale = 1
    const double tv = S(10);
    res[0] = S(0) / tv;                      // xcen
    res[1] = S(1) / tv;                      // ycen
    res[2] = S(11) / tv - res[0] * res[0];   // xvar
    res[3] = S(12) / tv - res[1] * res[1];   // yvar
    res[4] = S(2) / tv;                      // rmean
    res[5] = S(3);                           // area
    res[6] = S(4) / tv;                      // vmean
    res[7] = S(13) / tv;                     // umean
    res[8] = S(5) / tv;                      // vxmean
    res[9] = S(6) / tv;                      // vymean
    res[10] = S(9) > 0 ? S(7) / S(9) : 0.0;  // slopemean
    res[11] = tv;                            // statvolume
    res[12] = 3.0 * sqrt(res[2] + res[3]);   // piler
    for (int q = 0; q < kMax; ++q) res[13 + q] = S(kSums + q);  // hmax vmax umax
    res[16] = vslump != 0 ? res[6] / vslump : 0.0;              // vstar
    for (int q = 0; q < kMin; ++q) res[17 + q] = q & 1 ? -S(kSums + kMax + q) : S(kSums + kMax + q);
    res[21] = S(kPoint + 1);
    res[22] = S(8);  // the energy sum stats.C reduces in its "adjoint" slot
    for (int p = 0; p < a.n_planes; ++p) res[kResPlane0 + p] = S(kPlane0 + p);
}

template <class R>
int stats_t(da_ctx *ctx, const StatArgs &a, double vslump) {
    const MeshArgs m = mesh_args(ctx);
    const int c = ctx->cur;
    StateRef<R> U{(const R *)ctx->U[c][0], (const R *)ctx->U[c][1], (const R *)ctx->U[c][2]};
    double *parts = ctx->stats_mem, *res = parts + (size_t)kParts * kPartLen;
    k_stats<R><<<kParts, kBlock, 0, ctx->stream>>>(m, U, a, vslump, parts, (unsigned *)(res + kResLen), res);
    return cuda_check(ctx, cudaGetLastError(), "stats launch");
}

// The partial sums, the result and the block counter, kept with the context; the result's pinned copy.
int stats_alloc(da_ctx *ctx) {
    if (ctx->stats_mem) return DA_OK;
    const size_t words = (size_t)kParts * kPartLen + kResLen + 1;
    int st = DA_OK;
    if (!ctx->stats_host)
        st = cuda_check(ctx, cudaMallocHost((void **)&ctx->stats_host, sizeof(double) * kResLen), "cudaMallocHost(stats)");
    double *dev = nullptr;
    if (!st) st = cuda_check(ctx, cudaMalloc((void **)&dev, sizeof(double) * words), "cudaMalloc(stats)");
    if (!st) st = cuda_check(ctx, cudaMemsetAsync(dev, 0, sizeof(double) * words, ctx->stream), "memset");
    if (!st)
        ctx->stats_mem = dev;
    else if (dev)
        cudaFree(dev);
    return st;
}

// OutLine::update (properties.h:726-790) for every cell: the maximum depth so far over the grid
// cells its footprint covers (bit patterns of non-negative doubles order like the values, so an
// integer atomicMax is exact).
template <class R>
__global__ void __launch_bounds__(kBlock) k_outline(MeshArgs m, StateRef<R> U, OutlineGrid g) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < m.n_owned; i += gridDim.x * blockDim.x) {
        const double height = double(U.h[i]);
        if (!(height > 0.0)) continue;  // the map starts at zero
        const double x = m.x[i], y = m.y[i], dx = m.dx ? m.dx[i] : double(m.fdx[i]), dy = m.dy ? m.dy[i] : double(m.fdy[i]);
        const double xstart = x - 0.5 * dx, xstop = x + 0.5 * dx, ystart = y - 0.5 * dy, ystop = y + 0.5 * dy;
        int ixstart = (int)((xstart - g.x0) / g.dx + 0.5), ixstop = (int)((xstop - g.x0) / g.dx + 0.5);
        int iystart = (int)((ystart - g.y0) / g.dy + 0.5), iystop = (int)((ystop - g.y0) / g.dy + 0.5);
        if (ixstart < 0) ixstart = 0;
        if (ixstop == ixstart) {
            ixstart = (int)((xstart - g.x0) / g.dx);
            ixstop = ixstart + 1;
        }
        if (ixstop > g.nx) ixstop = g.nx;
        if (iystart < 0) iystart = 0;
        if (iystop == iystart) {
            iystart = (int)((ystart - g.y0) / g.dy);
            iystop = iystart + 1;
        }
        if (iystop > g.ny) iystop = g.ny;
        const unsigned long long hb = __double_as_longlong(height);
        for (int iy = iystart; iy < iystop; ++iy)
            for (int ix = ixstart; ix < ixstop; ++ix)
                if (ix >= 0 && iy >= 0) atomicMax(g.map + (size_t)iy * g.nx + ix, hb);
    }
}

}  // namespace
}  // namespace da

using namespace da;

extern "C" {

int da_outline_init(da_ctx *ctx, const double dxy[2], const double xrange[2], const double yrange[2]) {
    if (!ctx || !dxy || !xrange || !yrange || !(dxy[0] > 0) || !(dxy[1] > 0) || !(xrange[1] > xrange[0]) ||
        !(yrange[1] > yrange[0]))
        return DA_ERR_INVALID;
    cudaSetDevice(ctx->device);
    OutlineGrid &g = ctx->outline;
    if (g.map) cudaFree(g.map);
    g = OutlineGrid{};
    // OutLine::init2 (properties.h:702-724)
    g.dx = dxy[0];
    g.dy = dxy[1];
    g.x0 = xrange[0];
    g.y0 = yrange[0];
    g.nx = (int)((xrange[1] - xrange[0]) / g.dx + 0.5);
    g.ny = (int)((yrange[1] - yrange[0]) / g.dy + 0.5);
    if (g.nx <= 0 || g.ny <= 0 || (long long)g.nx * g.ny > (1ll << 28))
        return set_error(ctx, DA_ERR_INVALID, "da_outline_init: grid size");
    int st = cuda_check(ctx, cudaMalloc((void **)&g.map, sizeof(unsigned long long) * (size_t)g.nx * g.ny), "cudaMalloc");
    if (!st) st = cuda_check(ctx, cudaMemsetAsync(g.map, 0, sizeof(unsigned long long) * (size_t)g.nx * g.ny, ctx->stream),
                             "memset");
    return st;
}

int da_outline_update(da_ctx *ctx) {
    if (!ctx) return DA_ERR_INVALID;
    if (!ctx->outline.map) return set_error(ctx, DA_ERR_INVALID, "da_outline_update: no grid (da_outline_init)");
    if (!ctx->have_state) return set_error(ctx, DA_ERR_INVALID, "da_outline_update: no state");
    if (ctx->ninst > 0) return set_error(ctx, DA_ERR_INVALID, "da_outline_update: ensemble context");
    cudaSetDevice(ctx->device);
    const MeshArgs m = mesh_args(ctx);
    const int c = ctx->cur, grid = (ctx->sm_count > 0 ? ctx->sm_count : 148) * 4;
    if (ctx->p.precision == DA_PREC_FP64) {
        StateRef<double> U{(const double *)ctx->U[c][0], (const double *)ctx->U[c][1], (const double *)ctx->U[c][2]};
        k_outline<double><<<grid, kBlock, 0, ctx->stream>>>(m, U, ctx->outline);
    } else {
        StateRef<float> U{(const float *)ctx->U[c][0], (const float *)ctx->U[c][1], (const float *)ctx->U[c][2]};
        k_outline<float><<<grid, kBlock, 0, ctx->stream>>>(m, U, ctx->outline);
    }
    return cuda_check(ctx, cudaGetLastError(), "outline launch");
}

int da_outline_read(da_ctx *ctx, int32_t *nx, int32_t *ny, double *map) {
    if (!ctx) return DA_ERR_INVALID;
    const OutlineGrid &g = ctx->outline;
    if (!g.map) return set_error(ctx, DA_ERR_INVALID, "da_outline_read: no grid (da_outline_init)");
    if (nx) *nx = g.nx;
    if (ny) *ny = g.ny;
    if (!map) return DA_OK;
    cudaSetDevice(ctx->device);
    int st = cuda_check(ctx, cudaMemcpyAsync(map, g.map, sizeof(double) * (size_t)g.nx * g.ny, cudaMemcpyDeviceToHost,
                                             ctx->stream), "copy");
    return st ? st : cuda_check(ctx, cudaStreamSynchronize(ctx->stream), "sync");
}

int da_compute_stats(da_ctx *ctx, const da_stats_props *props, double d_time, da_stats *out, double *discharge) {
    if (!ctx || !props || !out || props->n_planes < 0 || props->n_planes > DA_MAX_PLANES ||
        (props->n_planes > 0 && (!props->planes || !discharge)))
        return DA_ERR_INVALID;
    if (ctx->mesh.n <= 0) return set_error(ctx, DA_ERR_NO_MESH, "da_compute_stats: no mesh");
    if (!ctx->have_state) return set_error(ctx, DA_ERR_INVALID, "da_compute_stats: no state");
    if (ctx->ninst > 0) return set_error(ctx, DA_ERR_INVALID, "da_compute_stats: ensemble context");
    cudaSetDevice(ctx->device);
    StatArgs a{};
    a.min_height = props->min_height >= 0 ? props->min_height : ctx->p.epsilon / 10000.0;  // datread.C:210
    a.hxyminmax = props->hxyminmax >= 0 ? props->hxyminmax : 10.0 * a.min_height;     // datread.C:315-316
    a.heightifreach = props->heightifreach;
    a.tx = props->xyifreach[0];
    a.ty = props->xyifreach[1];
    a.n_planes = props->n_planes;
    for (int k = 0; k < props->n_planes; ++k) {
        // DISCHARGE::init (properties.h:925-959)
        double *pl = a.planes[k];
        const double *in = props->planes + 4 * k;
        pl[0] = in[0];
        pl[1] = in[1];
        pl[2] = in[2];
        pl[3] = in[3];
        pl[4] = pl[1] - pl[0];
        pl[5] = pl[3] - pl[2];
        pl[6] = pl[4] * pl[4] + pl[5] * pl[5];
        pl[7] = pl[3] * pl[4] - pl[1] * pl[5];
        pl[8] = ((std::fabs(pl[4]) + std::fabs(pl[5])) * (std::fabs(pl[4]) + std::fabs(pl[5]))) / pl[6];
        pl[9] = 0.0;
        if (!(pl[6] > 0)) return set_error(ctx, DA_ERR_INVALID, "da_compute_stats: degenerate discharge plane");
    }
    int st = stats_alloc(ctx);
    if (!st) st = ctx->p.precision == DA_PREC_FP64 ? stats_t<double>(ctx, a, props->vslump)
                                                   : stats_t<float>(ctx, a, props->vslump);
    const double *res = ctx->stats_host;
    if (!st) st = copy_d2h(ctx, ctx->stats_host, ctx->stats_mem + (size_t)kParts * kPartLen, sizeof(double) * kResLen, "copy");
    if (st) return st;
    for (int p = 0; p < props->n_planes; ++p) discharge[p] = std::fma(d_time, res[kResPlane0 + p], discharge[p]);
    out->xcen = res[0];
    out->ycen = res[1];
    out->xvar = res[2];
    out->yvar = res[3];
    out->rmean = res[4];
    out->area = res[5];
    out->vmean = res[6];
    out->umean = res[7];
    out->vxmean = res[8];
    out->vymean = res[9];
    out->slopemean = res[10];
    out->statvolume = res[11];
    out->piler = res[12];
    out->hmax = res[13];
    out->vmax = res[14];
    out->umax = res[15];
    out->vstar = res[16];
    for (int q = 0; q < 4; ++q) out->xyminmax[q] = res[17 + q];
    out->testpoint_reach = res[21] > 0.5 ? 1 : 0;
    out->pad = 0;
    out->energy = res[22];
    return DA_OK;
}

}  // extern "C"
