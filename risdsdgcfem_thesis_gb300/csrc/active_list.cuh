// active_list.cuh -- work lists of a batch launch: the tiles and node chunks
// of a set of meshes, in mesh order.
//
//  * CG lists (mixed path): meshes whose CG loop is running. The last block
//    of a node pass rebuilds them when the set has changed; the tile product
//    and the node pass walk them instead of every tile and chunk of the
//    batch, so an iteration costs what its running meshes cost.
//  * start lists: meshes that start a step in this launch (active mask 1),
//    walked by the start-of-step kernels;
//  * launch lists: meshes that take part in this launch (mask 1 or 2),
//    walked by integration and energies.
// The start and launch lists are built by the launch's first kernel (one
// block).
#pragma once
#include "batch.cuh"

namespace femgb {

// Exclusive block scan of one value per thread (blockDim.x <= 1024, a
// multiple of 32); returns this thread's offset, *total the block's sum.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* sh, uint32_t* total)
{
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    __syncthreads();
    if (lane == 31) sh[wid] = x;
    __syncthreads();
    if (wid == 0) {
        uint32_t w = lane < nw ? sh[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < nw) sh[lane] = w;  // inclusive warp totals
    }
    __syncthreads();
    const uint32_t before = wid ? sh[wid - 1] : 0u;
    *total = sh[nw - 1];
    __syncthreads();
    return before + x - v;
}

// Tiles and chunks of the meshes m with pred(m), in mesh order, into
// tiles[] / chunks[] and their counts into count2[0..1]. Called by every
// thread of one block: a thread per mesh finds where the mesh's entries go and
// writes them, or, when some mesh of its warp has more than kListOwn, the warp
// does, mesh by mesh (a 27,000-tet mesh's 107 tiles one after the other: 92 us
// for the two lists of 192 such meshes, 25 us by warps; 24 meshes of 5 tiles:
// 6 us against 16 by warps).
constexpr uint32_t kListOwn = 16;
template <typename S, typename P>
__device__ void build_mesh_lists(const BatchView<S>& b, P pred, uint32_t* tiles, uint32_t* chunks,
                                 uint32_t* count2)
{
    __shared__ uint32_t sh[32];
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t done_t = 0, done_c = 0;
    for (uint32_t base = 0; base < b.M; base += blockDim.x) {
        const uint32_t m = base + threadIdx.x;
        uint32_t t0 = 0, nt = 0, c0 = 0, nc = 0;
        if (m < b.M) {
            const MeshConsts& c = b.mc[m];
            const bool in = pred(m);
            t0 = c.tile0;
            c0 = c.chunk0;
            nt = in ? c.ntiles : 0u;
            nc = in ? c.nchunks : 0u;
        }
        uint32_t tot_t, tot_c;
        const uint32_t pt = done_t + block_excl_scan(nt, sh, &tot_t);
        const uint32_t pc = done_c + block_excl_scan(nc, sh, &tot_c);
        if (__all_sync(0xffffffffu, nt <= kListOwn && nc <= kListOwn)) {
            for (uint32_t k = 0; k < nt; k++) tiles[pt + k] = t0 + k;
            for (uint32_t k = 0; k < nc; k++) chunks[pc + k] = c0 + k;
            nt = nc = 0;
        }
        for (unsigned left = __ballot_sync(0xffffffffu, nt | nc); left; left &= left - 1) {
            const int l = __ffs(left) - 1;
            const uint32_t wt0 = __shfl_sync(0xffffffffu, t0, l), wnt = __shfl_sync(0xffffffffu, nt, l);
            const uint32_t wc0 = __shfl_sync(0xffffffffu, c0, l), wnc = __shfl_sync(0xffffffffu, nc, l);
            const uint32_t wpt = __shfl_sync(0xffffffffu, pt, l), wpc = __shfl_sync(0xffffffffu, pc, l);
            for (uint32_t k = lane; k < wnt; k += 32) tiles[wpt + k] = wt0 + k;
            for (uint32_t k = lane; k < wnc; k += 32) chunks[wpc + k] = wc0 + k;
        }
        done_t += tot_t;
        done_c += tot_c;
    }
    if (threadIdx.x == 0) {
        count2[0] = done_t;
        count2[1] = done_c;
    }
    __syncthreads();
}

// The CG work lists: meshes whose loop is running. Called by every thread
// of one block, after every other block of the grid has finished its writes
// to the meshes' done flags.
template <typename S>
__device__ void build_active_lists(const BatchView<S>& b)
{
    build_mesh_lists(
        b, [&](uint32_t m) { return ((volatile const StepScalars*)(b.st + m))->done == 0u; }, b.act_tiles,
        b.act_chunks, b.act_count);
    if (threadIdx.x == 0) *b.list_dirty = 0u;
}

// The tiles of the meshes whose next iteration recomputes the residual in
// FP64 (walked by the FP64 product of y). Same calling rule as above.
template <typename S>
__device__ void build_refresh_lists(const BatchView<S>& b)
{
    build_mesh_lists(
        b,
        [&](uint32_t m) {
            volatile const StepScalars* sp = b.st + m;
            return sp->done == 0u && sp->refresh_next != 0u;
        },
        b.refresh_tiles, b.refresh_chunks, b.list_count + 4);
}

// list_count[4] when every running mesh refreshes: the refresh product walks
// the CG list itself (no copy; its per-tile test skips the meshes that have
// left their loop).
constexpr uint32_t kRefreshUsesCgList = 0xffffffffu;

// The refresh work list of the next iteration; `all` = every running mesh
// refreshes (then the CG list serves and nothing is copied: in a batch whose
// meshes started together that is every periodic refresh, while exit
// confirmations and staggered starts give short lists). Same calling rule
// as above.
template <typename S>
__device__ void set_refresh_lists(const BatchView<S>& b, bool all)
{
    if (all && b.act_tiles) {
        if (threadIdx.x == 0) b.list_count[4] = kRefreshUsesCgList;
        __syncthreads();
    } else {
        build_refresh_lists(b);
    }
}

// Entry i of a work list, or i itself when the launch has no list.
__device__ __forceinline__ uint32_t list_entry(const uint32_t* list, uint32_t i) { return list ? list[i] : i; }

}  // namespace femgb
