// Routing of many tokens to their experts: choice and weights, slots grouped by expert, the table of token
// tiles the expert products walk, and the copy of the rows into their slots.  (Up to DENSE_GEMV_ROWS tokens,
// DENSE_FEW_ROWS in float32, need none of this: the matrix-vector products choose for themselves.)
#include "decoder.cuh"

namespace rb {

// One warp per row: choices, weights, and how many rows each expert gets.
__global__ void __launch_bounds__(256) route_choose_kernel(const __grid_constant__ Routing r, int rows) {
    __shared__ int hist[EXPERTS_MAX];
    for (int e = threadIdx.x; e < r.experts; e += blockDim.x) hist[e] = 0;
    pdl_wait();
    pdl_trigger();
    __syncthreads();
    const int lane = threadIdx.x & 31, per = blockDim.x >> 5;
    for (int row = blockIdx.x * per + (threadIdx.x >> 5); row < rows; row += gridDim.x * per) {
        int sel;
        float w;
        route_row(r, row, lane, sel, w);
        if (lane < r.top) {
            r.chosen[(size_t)row * r.top + lane] = sel;
            r.weight[(size_t)row * r.top + lane] = w;
            atomicAdd(&hist[sel], 1);
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < r.experts; e += blockDim.x)
        if (hist[e]) atomicAdd(&r.counts[e], hist[e]);
}

// One CTA of EXPERTS_MAX threads: first slot of every expert, the tile table; counts are zeroed for the next call.
__global__ void __launch_bounds__(EXPERTS_MAX) route_table_kernel(const __grid_constant__ Routing r, int pairs) {
    __shared__ int2 warp_sums[32];
    pdl_wait();
    pdl_trigger();
    const int e = threadIdx.x, lane = e & 31, warp = e >> 5;
    const int n = e < r.experts ? min(max(r.counts[e], 0), pairs) : 0, tiles = (n + r.tile_rows - 1) / r.tile_rows;
    int2 s = make_int2(n, tiles);  // inclusive sums
    auto scan = [&]() {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int a = __shfl_up_sync(0xffffffffu, s.x, o), b = __shfl_up_sync(0xffffffffu, s.y, o);
            if (lane >= o) {
                s.x += a;
                s.y += b;
            }
        }
    };
    scan();
    if (lane == 31) warp_sums[warp] = s;
    __syncthreads();
    const int2 own = s;
    if (warp == 0) {
        s = warp_sums[lane];
        scan();
        warp_sums[lane] = s;
    }
    __syncthreads();
    int first = own.x - n, tile = own.y - tiles;
    if (warp > 0) {
        first += warp_sums[warp - 1].x;
        tile += warp_sums[warp - 1].y;
    }
    if (e < r.experts) {
        r.cursor[e] = first;
        r.counts[e] = 0;
        for (int t = 0; t < tiles && tile + t < r.max_tiles && first + t * r.tile_rows < pairs; ++t) {
            int* out = r.table + 1 + 3 * (tile + t);
            out[0] = e;
            out[1] = first + t * r.tile_rows;
            out[2] = min(min(r.tile_rows, n - t * r.tile_rows), pairs - out[1]);
        }
    }
    if (e == 0) r.table[0] = min(warp_sums[31].y, r.max_tiles);
}

// One warp per row: takes the next slot of each of its experts and copies the row there, read once.
__global__ void __launch_bounds__(256) route_scatter_kernel(const __grid_constant__ Routing r, int rows, const uint4* x, int pieces, uint4* permuted) {
    pdl_wait();
    pdl_trigger();
    const int lane = threadIdx.x & 31, per = blockDim.x >> 5, pairs = rows * r.top;
    constexpr int U = 4;  // pieces per lane requested together
    for (int row = blockIdx.x * per + (threadIdx.x >> 5); row < rows; row += gridDim.x * per) {
        const uint4* src = x + (size_t)row * pieces;
        uint4 v[U];
        auto fetch = [&](int c0) {
#pragma unroll
            for (int u = 0; u < U; ++u)
                if (c0 + 32 * u + lane < pieces) v[u] = __ldcg(src + c0 + 32 * u + lane);
        };
        fetch(0);
        int slot = 0;
        if (lane < r.top) {
            slot = min(max(atomicAdd(&r.cursor[r.chosen[(size_t)row * r.top + lane]], 1), 0), pairs - 1);
            r.slot_of[(size_t)row * r.top + lane] = slot;
        }
        for (int c0 = 0; c0 < pieces; c0 += 32 * U) {
            if (c0) fetch(c0);
            for (int k = 0; k < r.top; ++k) {
                uint4* dst = permuted + (size_t)__shfl_sync(0xffffffffu, slot, k) * pieces;
#pragma unroll
                for (int u = 0; u < U; ++u)
                    if (c0 + 32 * u + lane < pieces) dst[c0 + 32 * u + lane] = v[u];
            }
        }
    }
}

// Up to 32 rows: all of it in one launch.  Every CTA makes the choices and the slots for itself (a row is a bit of its experts' masks, so
// that a token's slot is a count of bits and nobody has to take turns), the first one writes them down, and each copies its
// share of the rows.  8 rows, 64 experts, 6 of them: 11.7 us of a step in three launches, 5.5 here.
constexpr int ROUTE_ROWS = 32, ROUTE_TH = 256, ROUTE_EACH = EXPERTS_MAX / ROUTE_TH;
__global__ void __launch_bounds__(ROUTE_TH) route_few_kernel(const __grid_constant__ Routing r, int rows, const uint4* x, int pieces, uint4* permuted) {
    __shared__ unsigned mask[EXPERTS_MAX];
    __shared__ int first_of[EXPERTS_MAX], chosen[ROUTE_ROWS * EXPERT_TOP_MAX];
    __shared__ int2 warp_sums[ROUTE_TH / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, pairs = rows * r.top;
    for (int e = threadIdx.x; e < EXPERTS_MAX; e += ROUTE_TH) mask[e] = 0u;
    pdl_wait();
    pdl_trigger();
    __syncthreads();
    for (int row = warp; row < rows; row += ROUTE_TH / 32) {
        int sel;
        float w;
        route_row(r, row, lane, sel, w);
        if (lane < r.top) {
            chosen[row * r.top + lane] = sel;
            atomicOr(&mask[sel], 1u << row);
            if (blockIdx.x == 0) {
                r.chosen[row * r.top + lane] = sel;
                r.weight[row * r.top + lane] = w;
            }
        }
    }
    __syncthreads();
    // first slot and first tile of every expert: a thread's experts one after the other, then sums over the threads before it
    const int e0 = ROUTE_EACH * threadIdx.x;
    int2 own = make_int2(0, 0);
#pragma unroll
    for (int i = 0; i < ROUTE_EACH; ++i) {
        const int n = __popc(mask[e0 + i]);
        own.x += n;
        own.y += (n + r.tile_rows - 1) / r.tile_rows;
    }
    int2 sum = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, sum.x, o), b = __shfl_up_sync(0xffffffffu, sum.y, o);
        if (lane >= o) {
            sum.x += a;
            sum.y += b;
        }
    }
    if (lane == 31) warp_sums[warp] = sum;
    __syncthreads();
    int first = sum.x - own.x, tile = sum.y - own.y;
    for (int w = 0; w < warp; ++w) {
        first += warp_sums[w].x;
        tile += warp_sums[w].y;
    }
#pragma unroll
    for (int i = 0; i < ROUTE_EACH; ++i) {
        const int e = e0 + i, n = __popc(mask[e]), tiles = (n + r.tile_rows - 1) / r.tile_rows;
        first_of[e] = first;
        for (int t = 0; blockIdx.x == 0 && t < tiles && tile + t < r.max_tiles; ++t) {
            int* out = r.table + 1 + 3 * (tile + t);
            out[0] = e;
            out[1] = first + t * r.tile_rows;
            out[2] = min(r.tile_rows, n - t * r.tile_rows);
        }
        first += n;
        tile += tiles;
    }
    if (blockIdx.x == 0 && threadIdx.x == ROUTE_TH - 1) r.table[0] = min(tile, r.max_tiles);
    __syncthreads();
    for (int p = blockIdx.x; p < pairs; p += gridDim.x) {
        const int row = p / r.top, e = chosen[p], slot = first_of[e] + __popc(mask[e] & ((1u << row) - 1u));
        if (threadIdx.x == 0) r.slot_of[p] = slot;
        for (int c = threadIdx.x; c < pieces; c += ROUTE_TH) permuted[(size_t)slot * pieces + c] = __ldcg(x + (size_t)row * pieces + c);
    }
}

int launch_route(const Routing& r, int rows, const void* x, size_t row_bytes, void* permuted, cudaStream_t st) {
    RB_REQUIRE(r.logits && r.slot_of && r.weight && r.chosen && r.counts && r.cursor && r.table && x && permuted && rows > 0);
    RB_REQUIRE(r.experts >= 1 && r.experts <= EXPERTS_MAX && r.top >= 1 && r.top <= r.experts && r.top <= EXPERT_TOP_MAX);
    RB_REQUIRE(row_bytes % 16 == 0 && (long long)rows * r.top < 0x7fffffffLL);
    const int pairs = rows * r.top, most = 148 * 8;
    RB_REQUIRE(r.max_tiles >= route_tiles(pairs, r.experts, r.tile_rows));
    if (rows <= ROUTE_ROWS)
        return launch_chained(route_few_kernel, dim3(pairs < 148 ? pairs : 148), dim3(ROUTE_TH), 0, st, 1, r, rows,
                              static_cast<const uint4*>(x), (int)(row_bytes / 16), static_cast<uint4*>(permuted));
    int rc = launch_chained(route_choose_kernel, dim3((rows + 7) / 8 < most ? (rows + 7) / 8 : most), dim3(256), 0, st, 1, r, rows);
    if (!rc) rc = launch_chained(route_table_kernel, dim3(1), dim3(EXPERTS_MAX), 0, st, 1, r, pairs);
    if (!rc)
        rc = launch_chained(route_scatter_kernel, dim3((rows + 7) / 8 < most ? (rows + 7) / 8 : most), dim3(256), 0, st, 1, r, rows,
                            static_cast<const uint4*>(x), (int)(row_bytes / 16), static_cast<uint4*>(permuted));
    return rc;
}

}  // namespace rb
