// rows_build.cu -- kernels of rows_build.h: the assembled stiffness's pattern and
// the resident solve's layout, made from the mesh's tables on the device.
//
// Pattern: a warp per node, its entries in shared memory; an entry looks at all
// of the row's (73 on grid meshes), so the row needs no sort. Layout: a block of
// threads per block of rows, its rim a bit per node of the mesh in shared
// memory.
#include "bounds.cuh"
#include "fem_device.cuh"
#include "rows_build.h"

namespace femgb {

namespace {

constexpr uint32_t kPatternWarps = 4;

struct RowWarp {
    uint32_t *e, *before, lane, n, beg, entries;
};
__device__ __forceinline__ bool row_warp(const MeshView<double>& m, uint32_t most, uint32_t* smem, RowWarp& w)
{
    w.lane = threadIdx.x & 31u;
    w.n = blockIdx.x * kPatternWarps + (threadIdx.x >> 5);
    if (w.n >= m.N) return false;
    w.e = smem + 2 * most * (threadIdx.x >> 5);
    w.before = w.e + most;
    w.beg = m.csr_ptr[w.n];
    w.entries = 3 * (m.csr_ptr[w.n + 1] - w.beg) + 1;
    row_entries(w.n, w.beg, w.entries, reinterpret_cast<const uint32_t*>(m.tets), m.csr_idx, w.e, w.lane, 32u);
    for (uint32_t i = w.lane; i < w.entries; i += 32) w.e[i] = bounds_idx(w.e[i], m.N, kSiteBsrEntry);
    __syncwarp();
    return true;
}

__global__ void __launch_bounds__(32 * kPatternWarps) k_row_lengths(MeshView<double> m, uint32_t most, uint32_t* used)
{
    extern __shared__ uint32_t row_smem[];
    RowWarp w;
    if (!row_warp(m, most, row_smem, w)) return;
    const uint32_t k = __reduce_add_sync(0xffffffffu, row_columns(w.e, w.entries, w.before, w.lane, 32u));
    if (w.lane == 0) used[w.n] = k;
}

// row[n]: the groups of four ahead of row n (one block).
__global__ void __launch_bounds__(1024) k_row_starts(uint32_t N, const uint32_t* __restrict__ used, uint32_t* row)
{
    __shared__ uint32_t sh[32];
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    uint32_t done = 0;
    for (uint32_t a = 0; a < N; a += 4096) {  // four nodes per thread
        uint32_t v[4], sum = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t n = a + 4 * t + k;
            v[k] = n < N ? (used[n] + 3) / 4 : 0u;
            sum += v[k];
        }
        uint32_t up = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, up, o);
            if (lane >= (uint32_t)o) up += x;
        }
        if (lane == 31) sh[warp] = up;
        __syncthreads();
        uint32_t w = sh[lane];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t x = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= (uint32_t)o) w += x;
        }
        const uint32_t before = warp ? __shfl_sync(0xffffffffu, w, warp - 1) : 0u, all = __shfl_sync(0xffffffffu, w, 31);
        uint32_t at = done + before + up - sum;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t n = a + 4 * t + k;
            if (n < N) row[n] = at;
            at += v[k];
        }
        done += all;
        __syncthreads();
    }
    if (t == 0) row[N] = done;
}

__global__ void __launch_bounds__(32 * kPatternWarps)
    k_row_write(MeshView<double> m, uint32_t most, const uint32_t* __restrict__ used, const uint32_t* __restrict__ row,
                uint32_t* col, uint32_t* cptr, uint32_t* contrib)
{
    extern __shared__ uint32_t row_smem[];
    RowWarp w;
    if (blockIdx.x == 0 && threadIdx.x == 0) cptr[4 * (size_t)row[m.N]] = 12 * m.T;
    if (!row_warp(m, most, row_smem, w)) return;
    (void)row_columns(w.e, w.entries, w.before, w.lane, 32u);
    __syncwarp();
    row_write(w.e, w.before, w.entries, w.beg, used[w.n], 4 * row[w.n], m.csr_idx, col, cptr, contrib, w.lane, 32u);
}

__device__ __forceinline__ LayoutSpan layout_count(const LayoutShape& s, const LayoutRows& m, LayoutWork& w)
{
    const LayoutSpan b = layout_span(s, blockIdx.x);
    layout_begin(b, m, w, threadIdx.x, kLayoutThreads);
    __syncthreads();
    layout_rim(b, m, w, threadIdx.x, kLayoutThreads);
    __syncthreads();
    layout_parts(s, b, w, threadIdx.x, kLayoutThreads);
    __syncthreads();
    layout_sum(w, threadIdx.x, kLayoutThreads);
    __syncthreads();
    return b;
}

__global__ void __launch_bounds__(kLayoutThreads) k_layout_count(LayoutShape s, LayoutRows m, CgRowsCount* count)
{
    __shared__ LayoutWork w;
    (void)layout_count(s, m, w);
    if (threadIdx.x == 0) count[blockIdx.x] = CgRowsCount{w.units, w.halo};
}

__global__ void __launch_bounds__(kLayoutThreads) k_layout_write(LayoutShape s, LayoutRows m, LayoutOut o)
{
    __shared__ LayoutWork w;
    const LayoutSpan b = layout_count(s, m, w);
    layout_ahead(b, w, threadIdx.x, kLayoutThreads);
    __syncthreads();
    layout_write(s, b, blockIdx.x, m, w, o, threadIdx.x, kLayoutThreads);
}

__global__ void __launch_bounds__(kLayoutThreads) k_layout_owners(LayoutShape s, LayoutOut o)
{
    layout_owners(s, blockIdx.x, o, threadIdx.x, kLayoutThreads);
}

uint32_t pattern_grid(uint32_t N) { return (N + kPatternWarps - 1) / kPatternWarps; }
size_t pattern_smem(uint32_t most) { return 2 * sizeof(uint32_t) * kPatternWarps * (size_t)most; }

}  // namespace

FEMGB_BOUNDS_ACCESSOR(bounds_read_rows_build)

static_assert(2 * sizeof(uint32_t) * kPatternWarps * kRowEntries <= 48 * 1024 && sizeof(LayoutWork) <= 48 * 1024,
              "shared memory of a launch without the opt-in");

void launch_row_lengths(const MeshView<double>& m, uint32_t most, uint32_t* used, uint32_t* row, cudaStream_t s)
{
    k_row_lengths<<<pattern_grid(m.N), 32 * kPatternWarps, pattern_smem(most), s>>>(m, most, used);
    k_row_starts<<<1, 1024, 0, s>>>(m.N, used, row);
    launch_counter() += 2;
}

void launch_row_write(const MeshView<double>& m, uint32_t most, const uint32_t* used, const uint32_t* row, uint32_t* col,
                      uint32_t* cptr, uint32_t* contrib, cudaStream_t s)
{
    k_row_write<<<pattern_grid(m.N), 32 * kPatternWarps, pattern_smem(most), s>>>(m, most, used, row, col, cptr, contrib);
    launch_counter()++;
}

void launch_layout_count(const LayoutShape& s, uint32_t blocks, const LayoutRows& m, CgRowsCount* count, cudaStream_t st)
{
    k_layout_count<<<blocks, kLayoutThreads, 0, st>>>(s, m, count);
    launch_counter()++;
}

void launch_layout_write(const LayoutShape& s, uint32_t blocks, const LayoutRows& m, const LayoutOut& o, cudaStream_t st)
{
    k_layout_write<<<blocks, kLayoutThreads, 0, st>>>(s, m, o);
    k_layout_owners<<<blocks, kLayoutThreads, 0, st>>>(s, o);
    launch_counter() += 2;
}

}  // namespace femgb
