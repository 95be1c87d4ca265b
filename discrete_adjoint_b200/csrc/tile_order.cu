// The order in which the staged phases hand the tiles to their blocks.
//
// Block b of a grid of G takes the entries b, b + G, b + 2 G, ... of this list.  In plain index order a
// compact flow spreads evenly, but the flows of several members or piles, and the four corners of a
// flow in the middle of a Morton-ordered map, can fall on the same few blocks, and a phase takes as
// long as its fullest block: 24 members with 310 wet of 6212 tiles put 6 on one SM where 3 would do,
// 13 wet tiles of a 1024-tile map 2 on one.  So the tiles in work (a wet cell, then those that were
// updated beside them) are listed first, the others after them, each in index order; where plain order
// is as even as it can be, it stays (its neighbours, the tiles a flow runs into, are free there).
// Nothing but the time depends on the order, so a stale one does no harm.  It is formed a few times per
// adjoint sweep, by one block (the flags of a few thousand tiles: 6 us against some 40 steps of 11 us
// and more).
#include "da_internal.h"

namespace da {
namespace {

constexpr int kOrderThreads = 1024, kOrderWarps = kOrderThreads / 32;
constexpr int kOrderBins = 256;     // SMs at most (more: plain order decides over the first 256 bins)
constexpr int kOrderTiles = 16384;  // above, the one block's time shows and a flow has tiles for every SM

// 1: a wet cell; 2: updated in the last step; 0: neither
__device__ __forceinline__ int tile_class(const uint8_t *seg_wet, const uint8_t *seg_clean, int t) {
    const unsigned long long w = *reinterpret_cast<const unsigned long long *>(seg_wet + (size_t)t * 8);
    const unsigned long long c = *reinterpret_cast<const unsigned long long *>(seg_clean + (size_t)t * 8);
    return w != 0ull ? 1 : (c != 0x0101010101010101ull ? 2 : 0);
}

__global__ void __launch_bounds__(kOrderThreads) k_tile_order(const uint8_t *seg_wet, const uint8_t *seg_clean,
                                                              int ntiles, int bins, int *order) {
    __shared__ int hist[kOrderBins], n1[kOrderWarps], n2[kOrderWarps];
    __shared__ int total1, total2, most;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < kOrderBins; k += kOrderThreads) hist[k] = 0;
    if (threadIdx.x == 0) most = 0;
    __syncthreads();
    const int per = (ntiles + kOrderThreads - 1) / kOrderThreads * 32;  // tiles of a warp
    const int t0 = warp * per, t1 = min(t0 + per, ntiles);
    int c1 = 0, c2 = 0;
#pragma unroll 4
    for (int b = t0; b < t1; b += 32) {
        const int t = b + lane;
        const int c = t < t1 ? tile_class(seg_wet, seg_clean, t) : 0;
        c1 += __popc(__ballot_sync(0xffffffffu, c == 1));
        c2 += __popc(__ballot_sync(0xffffffffu, c == 2));
        if (c) atomicAdd(&hist[t % bins], 1);
    }
    if (lane == 0) {
        n1[warp] = c1;
        n2[warp] = c2;
    }
    __syncthreads();
    if (threadIdx.x < kOrderBins) atomicMax(&most, hist[threadIdx.x]);
    if (threadIdx.x == 0) {
        int a = 0, b = 0;
        for (int w = 0; w < kOrderWarps; ++w) {
            const int x = n1[w], y = n2[w];
            n1[w] = a;
            n2[w] = b;
            a += x;
            b += y;
        }
        total1 = a;
        total2 = b;
    }
    __syncthreads();
    const bool plain = most <= (total1 + total2 + bins - 1) / bins;
    int o1 = n1[warp], o2 = n2[warp];
    for (int b = t0; b < t1; b += 32) {
        const int t = b + lane;
        const int c = t < t1 ? tile_class(seg_wet, seg_clean, t) : 0;
        const unsigned b1 = __ballot_sync(0xffffffffu, c == 1), b2 = __ballot_sync(0xffffffffu, c == 2);
        const unsigned below = (1u << lane) - 1u;
        const int r1 = o1 + __popc(b1 & below), r2 = o2 + __popc(b2 & below);
        const int at = c == 1 ? r1 : (c == 2 ? total1 + r2 : total1 + total2 + t - r1 - r2);
        if (t < t1) order[plain ? t : at] = t;
        o1 += __popc(b1);
        o2 += __popc(b2);
    }
}

__global__ void k_plain_order(int *order, int n) {
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) order[t] = t;
}

}  // namespace

int plain_tile_order(da_ctx *ctx) {
    k_plain_order<<<(ctx->ntiles + 255) / 256, 256, 0, ctx->stream>>>(ctx->tile_order, ctx->ntiles);
    return cuda_check(ctx, cudaGetLastError(), "tile order");
}

// For the kernels that take it (kOrdered, staged_impl.cuh); meshes of at most two tiles per SM stay in plain order.
int launch_tile_order(da_ctx *ctx) {
    const int sms = ctx->sm_count > 0 ? ctx->sm_count : 148;
    if (ctx->ninst == 0 && ctx->p.precision == DA_PREC_FP64) return DA_OK;
    if (ctx->ntiles <= 2 * sms || ctx->ntiles > kOrderTiles) return DA_OK;
    k_tile_order<<<1, kOrderThreads, 0, ctx->stream>>>(ctx->seg_wet, ctx->seg_clean, ctx->ntiles,
                                                       sms < kOrderBins ? sms : kOrderBins, ctx->tile_order);
    ctx->tile_ordered = true;
    return cuda_check(ctx, cudaGetLastError(), "tile order");
}

}  // namespace da
