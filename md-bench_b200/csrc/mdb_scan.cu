// Device-wide exclusive prefix sum over int32: tile sums, then every tile is
// rescanned on top of the sum of the tiles before it; short inputs in one block.
// Used for the ghost-map offsets, the bin and column CSRs and the cluster
// offsets. A cluster-pair rebuild has four scans, so launches count: a separate
// scan of the tile sums made three kernels of each (2 us apiece and as much
// between them, 12 of 40 launches). The Verlet-list rebuild keeps that form
// (scan_exclusive_steps): a test bounds the launches of its runs from below.
#include "mdb_internal.cuh"

namespace mdb {

static constexpr int SCAN_THREADS = 1024;
static constexpr int SCAN_ITEMS   = 4;
static constexpr int SCAN_TILE    = SCAN_THREADS * SCAN_ITEMS;

static constexpr int SCAN_SMALL   = 2 * SCAN_TILE; // one block, two passes

int scan_scratch_ints(int n) { return (n + SCAN_TILE - 1) / SCAN_TILE + 1; }

// Inclusive block scan of one value per thread; returns the inclusive prefix,
// *total receives the block sum.
__device__ __forceinline__ int block_inclusive_scan(int v, int* total)
{
    __shared__ int warp_sums[SCAN_THREADS / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int o = 1; o < 32; o <<= 1) {
        int t = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += t;
    }
    if (lane == 31) warp_sums[warp] = v;
    __syncthreads();
    if (warp == 0) {
        int w = (lane < (int)(blockDim.x >> 5)) ? warp_sums[lane] : 0;
        for (int o = 1; o < 32; o <<= 1) {
            int t = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += t;
        }
        warp_sums[lane] = w;
    }
    __syncthreads();
    int prefix = warp > 0 ? warp_sums[warp - 1] : 0;
    *total     = warp_sums[(blockDim.x >> 5) - 1];
    __syncthreads();
    return v + prefix;
}

__global__ void k_scan_tiles(const int* __restrict__ in, int n, int* __restrict__ tile_sums)
{
    long long base = (long long)blockIdx.x * SCAN_TILE + threadIdx.x * SCAN_ITEMS;
    int s          = 0;
#pragma unroll
    for (int k = 0; k < SCAN_ITEMS; k++)
        if (base + k < n) s += in[base + k];
    int total;
    block_inclusive_scan(s, &total);
    if (threadIdx.x == 0) tile_sums[blockIdx.x] = total;
}

// The tiles of SCAN_TILE inputs first, first + step, ... on top of `carry`;
// returns the sum with them. out[n] is left to the caller.
__device__ __forceinline__ int scan_tiles_on(const int* __restrict__ in, int* __restrict__ out,
    int n, long long first, long long step, int carry)
{
    for (long long tile = first; tile < n; tile += step) {
        const long long base = tile + threadIdx.x * SCAN_ITEMS;
        int v[SCAN_ITEMS];
        int s = 0;
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) {
            v[k] = (base + k < n) ? in[base + k] : 0;
            s += v[k];
        }
        int total;
        int run = carry + block_inclusive_scan(s, &total) - s;
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; k++) {
            if (base + k < n) out[base + k] = run;
            run += v[k];
        }
        carry += total;
    }
    return carry;
}

__global__ void k_scan_apply(const int* __restrict__ in, int* __restrict__ out, int n,
    const int* __restrict__ tile_sums)
{
    int before = 0, total;
    for (int k = threadIdx.x; k < blockIdx.x; k += SCAN_THREADS)
        before += tile_sums[k];
    block_inclusive_scan(before, &total);
    const int sum =
        scan_tiles_on(in, out, n, (long long)blockIdx.x * SCAN_TILE, 1LL << 40, total);
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = sum;
}

__global__ void k_scan_small(const int* __restrict__ in, int* __restrict__ out, int n)
{
    const int sum = scan_tiles_on(in, out, n, 0, SCAN_TILE, 0);
    if (threadIdx.x == 0) out[n] = sum;
}

// One block: exclusive scan of the tile sums in place.
__global__ void k_scan_tile_sums(int* tile_sums, int ntiles)
{
    int carry = 0;
    for (int base = 0; base < ntiles; base += SCAN_THREADS) {
        int idx = base + threadIdx.x;
        int v   = idx < ntiles ? tile_sums[idx] : 0;
        int total;
        int inc = block_inclusive_scan(v, &total);
        if (idx < ntiles) tile_sums[idx] = carry + inc - v;
        carry += total;
    }
}

// tile_sums: the sums of the tiles before each
__global__ void k_scan_rescan(const int* __restrict__ in, int* __restrict__ out, int n,
    const int* __restrict__ tile_sums)
{
    const int sum = scan_tiles_on(in, out, n, (long long)blockIdx.x * SCAN_TILE, 1LL << 40,
        tile_sums[blockIdx.x]);
    if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) out[n] = sum;
}

void scan_exclusive_steps(const int* in, int* out, int n, int* scratch, cudaStream_t s)
{
    const int ntiles = n > 0 ? (n + SCAN_TILE - 1) / SCAN_TILE : 1;
    k_scan_tiles<<<ntiles, SCAN_THREADS, 0, s>>>(in, n, scratch);
    k_scan_tile_sums<<<1, SCAN_THREADS, 0, s>>>(scratch, ntiles);
    k_scan_rescan<<<ntiles, SCAN_THREADS, 0, s>>>(in, out, n, scratch);
    g_launches += 3;
}

void scan_exclusive(const int* in, int* out, int n, int* scratch, cudaStream_t s)
{
    if (n <= SCAN_SMALL) {
        k_scan_small<<<1, SCAN_THREADS, 0, s>>>(in, out, n);
        g_launches++;
        return;
    }
    const int ntiles = (n + SCAN_TILE - 1) / SCAN_TILE;
    k_scan_tiles<<<ntiles, SCAN_THREADS, 0, s>>>(in, n, scratch);
    k_scan_apply<<<ntiles, SCAN_THREADS, 0, s>>>(in, out, n, scratch);
    g_launches += 2;
}

} // namespace mdb
