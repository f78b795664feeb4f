// grid.cu -- uniform-grid neighbour search: cell keys, stable sort by (cell,
// id), cell-ordered reindexing with cell ranges, neighbour lists. The sort is a
// counting sort over the cells, or, where the grid is too sparse for the
// particles, an LSD radix sort of the keys (api.cu, counting_pays).
//
// Replaces the reference's bucket grid (64 atomically filled slots per cell,
// src/Utils/Neighborhood/UniformGrid/UniformGridKernel.cu:30-55) and its
// 27-cell neighbour walk writing 200-slot lists (UniformGridKernel.cu:58-95).
// What stays identical, bit for bit:
//   * the cell index i = floor((x - Min)/sizeCell) in FP64 from the float
//     corner and cell edge (UniformGridKernel.cu:46-49), linearised as
//     i + j*nx + k*nx*ny (:50);
//   * the neighbour test length(x_i - x_j) <= h, self included (:81-82):
//     decided in FP32 (the sign of |d|^2 - h^2, collected per row of cells)
//     and, within a band about h, re-evaluated in FP64 with separately rounded
//     operations in the reference's order.
// What differs by design: particles are sorted stably by (cell, id), so the
// neighbour order is deterministic; particles outside the grid are clamped
// into the border cells (the reference writes out of bounds there); lists
// are bounded (overflow raises a flag, never a trap).
#include <algorithm>

#include "psb_internal.cuh"

namespace psb {

namespace {

__device__ __forceinline__ int cell_coord(float x, float corner, float cell, int dim, int& clamped) {
    const double t = floor(__ddiv_rn(__dsub_rn((double)x, (double)corner), (double)cell));
    if (!(t >= 0.0)) { clamped = 1; return 0; }          // also NaN
    if (t >= (double)dim) { clamped = 1; return dim - 1; }
    return (int)t;
}

// Clears the start entry of every cell the previous sort occupied.
__global__ void k_reset_cells(int n, const uint32_t* __restrict__ sorted_keys, uint32_t* __restrict__ cell_start) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= n) return;
    const uint32_t k = sorted_keys[s];
    if (s == 0 || sorted_keys[s - 1] != k) cell_start[k] = kEmpty;
}

// Cell of the particle in slot s; c is set where it was clamped.
template <bool BATCH>
__device__ __forceinline__ uint32_t cell_key(const Params& P, int s, float4 p, int& c) {
    const Grid g = BATCH ? P.scenes[P.slot_scene[s]].g : P.g;
    const uint32_t base = BATCH ? P.scenes[P.slot_scene[s]].cell_base : 0u;
    const int i = cell_coord(p.x, g.gx, g.cell, g.nx, c);
    const int j = cell_coord(p.y, g.gy, g.cell, g.ny, c);
    const int k = cell_coord(p.z, g.gz, g.cell, g.nz, c);
    return base + (uint32_t)i + (uint32_t)j * (uint32_t)g.nx + (uint32_t)k * (uint32_t)g.nx * (uint32_t)g.ny;
}

__device__ __forceinline__ void count_clamped(int c, int* __restrict__ clamped) {
    const unsigned ballot = __ballot_sync(__activemask(), c);
    if (ballot && (threadIdx.x & 31) == __ffs(ballot) - 1) atomicAdd(clamped, __popc(ballot));
}

// Cell key of every particle, written at its id so that a stable sort of
// the id-ordered keys yields (cell, id) order. A batch gives each scene its
// own grid and a block of keys after the previous scene's, so the sort keeps
// every scene in its own contiguous slot range, in the order it has alone.
template <bool BATCH>
__global__ void k_cell_keys(Params P, const float4* __restrict__ pos, const int* __restrict__ ids,
                            uint32_t* __restrict__ keys_by_id, uint32_t* __restrict__ slot_by_id,
                            int* __restrict__ clamped) {
    after_previous();
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= P.n) return;
    int c = 0;
    const uint32_t key = cell_key<BATCH>(P, s, pos[s], c);
    const int id = ids[s];
    keys_by_id[id] = key;
    slot_by_id[id] = (uint32_t)s;
    count_clamped(c, clamped);
}

// ---- LSD radix sort, 8-bit digits, three kernels per pass ----------------
constexpr int kItems = 8;                      // keys per thread per tile
constexpr int kTile = kBlock * kItems;         // 2048 keys per block

__global__ void k_radix_hist(int n, int shift, int nblocks, const uint32_t* __restrict__ keys,
                             uint32_t* __restrict__ hist) {
    after_previous();
    __shared__ uint32_t h[256];
    h[threadIdx.x] = 0;
    __syncthreads();
    const int base = blockIdx.x * kTile;
#pragma unroll
    for (int r = 0; r < kItems; ++r) {
        const int i = base + r * kBlock + threadIdx.x;
        if (i < n) atomicAdd(&h[(keys[i] >> shift) & 255u], 1u);
    }
    __syncthreads();
    hist[threadIdx.x * nblocks + blockIdx.x] = h[threadIdx.x];
}

// Block-wide exclusive scan of one value per thread (blockDim == 256).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* s_warp, uint32_t& total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    if (warp == 0) {
        uint32_t w = lane < kBlock / 32 ? s_warp[lane] : 0u;
#pragma unroll
        for (int o = 1; o < kBlock / 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        if (lane < kBlock / 32) s_warp[lane] = w;
    }
    __syncthreads();
    total = s_warp[kBlock / 32 - 1];
    const uint32_t before = warp ? s_warp[warp - 1] : 0u;
    __syncthreads();
    return before + x - v;
}

// Per-digit exclusive scan of the tiles' counts: block d scans hist[d][0..nb)
// in place and writes the digit's total.
__global__ void __launch_bounds__(kBlock) k_radix_scan(int nb, uint32_t* __restrict__ hist,
                                                       uint32_t* __restrict__ totals) {
    after_previous();
    __shared__ uint32_t s_warp[kBlock / 32];
    uint32_t* h = hist + (size_t)blockIdx.x * nb;
    uint32_t carry = 0;
    for (int base = 0; base < nb; base += kBlock) {
        const int i = base + threadIdx.x;
        const uint32_t v = i < nb ? h[i] : 0u;
        uint32_t tot;
        const uint32_t ex = block_exclusive_scan(v, s_warp, tot);
        if (i < nb) h[i] = carry + ex;
        carry += tot;
    }
    if (threadIdx.x == 0) totals[blockIdx.x] = carry;
}

// Stable scatter. Tile items are ranked round by round (round r covers 256
// consecutive keys); inside a round, lanes holding the same digit are found
// with __match_any_sync and ranked by lane, warps by warp index.
__global__ void __launch_bounds__(kBlock) k_radix_scatter(int n, int shift, int nblocks,
                                                          const uint32_t* __restrict__ keys_in,
                                                          const uint32_t* __restrict__ vals_in,
                                                          uint32_t* __restrict__ keys_out,
                                                          uint32_t* __restrict__ vals_out,
                                                          const uint32_t* __restrict__ offsets,
                                                          const uint32_t* __restrict__ totals) {
    after_previous();
    __shared__ uint32_t s_off[256];
    __shared__ uint32_t s_wc[kBlock / 32][256];
    __shared__ uint32_t s_warp[kBlock / 32];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t all;
    const uint32_t digit_base = block_exclusive_scan(totals[tid], s_warp, all);
    s_off[tid] = digit_base + offsets[tid * nblocks + blockIdx.x];
#pragma unroll
    for (int w = 0; w < kBlock / 32; ++w) s_wc[w][tid] = 0;
    __syncthreads();
    const int base = blockIdx.x * kTile;
    for (int r = 0; r < kItems; ++r) {
        const int i = base + r * kBlock + tid;
        const bool valid = i < n;
        const uint32_t key = valid ? keys_in[i] : 0u;
        const uint32_t val = valid ? vals_in[i] : 0u;
        const uint32_t d = valid ? ((key >> shift) & 255u) : 256u;
        const unsigned peers = __match_any_sync(0xffffffffu, d);
        const int wrank = __popc(peers & ((1u << lane) - 1u));
        if (valid && lane == __ffs(peers) - 1) s_wc[warp][d] = __popc(peers);
        __syncthreads();
        if (valid) {
            uint32_t dst = s_off[d] + (uint32_t)wrank;
            for (int w = 0; w < warp; ++w) dst += s_wc[w][d];
            keys_out[dst] = key;
            vals_out[dst] = val;
        }
        __syncthreads();
        uint32_t tot = 0;
#pragma unroll
        for (int w = 0; w < kBlock / 32; ++w) { tot += s_wc[w][tid]; s_wc[w][tid] = 0; }
        s_off[tid] += tot;
        __syncthreads();
    }
}

// Lists slot t (position x) in P.wall_list when it lies near a box face, and
// writes the warp's flag word; every thread of the block calls it. One atomic
// add per block that has such a particle (one per warp queued at the count's
// address: 40 us of the positions' reorder at 1M, 14 without); the list's
// order is left open.
template <bool BATCH>
__device__ __forceinline__ void list_near_walls(const Params& P, int t, float4 x) {
    if (!P.wall_list || P.n < kWallListMin) return;
    bool near = false;
    if (t < P.n) {
        const float reach = kWallReach * P.hf;
        float lo_x = P.bx0, lo_y = P.by0, lo_z = P.bz0, hi_x = P.bx1, hi_y = P.by1, hi_z = P.bz1;
        if (BATCH) {
            const SceneGeom* G = P.scenes + P.slot_scene[t];
            lo_x = G->bx0; lo_y = G->by0; lo_z = G->bz0; hi_x = G->bx1; hi_y = G->by1; hi_z = G->bz1;
        }
        near = x.x - lo_x < reach || hi_x - x.x < reach || x.y - lo_y < reach || hi_y - x.y < reach ||
               x.z - lo_z < reach || hi_z - x.z < reach;
    }
    const unsigned word = __ballot_sync(0xffffffffu, near);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ int s_count[kBlock / 32], s_base;
    if (lane == 0) {
        if (t < P.n) P.wall_bits[t >> 5] = word;
        s_count[warp] = __popc(word);
    }
    __syncthreads();
    int before = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kBlock / 32; ++w) {
        if (w < warp) before += s_count[w];
        total += s_count[w];
    }
    if (total == 0) return;
    if (threadIdx.x == 0) s_base = atomicAdd(P.wall_count, total);
    __syncthreads();
    if (near) P.wall_list[s_base + before + __popc(word & ((1u << lane) - 1u))] = t;
}

// ---- sort of up to kSmallSort pairs in one block -----------------------------
// Below this size the passes above are launches: 8 kernels of 2-5 us each for
// 5,000 pairs, 45 us with the gaps. One block keeps the pairs in registers
// and shared memory through every pass (same 8-bit digits, same stable order)
// and touches global memory once each way. Warp w owns items 256 w .. 256 w +
// 255, a row of 32 per turn: a row's equal digits are found with
// __match_any_sync and ranked by lane behind the warp's count so far; the
// (digit, warp) counts are then scanned and each pair moves to its place.
constexpr int kSmallSort = 8192, kSmallThreads = 1024, kSmallItems = kSmallSort / kSmallThreads;
struct SmallSortSmem {
    uint32_t key[kSmallSort], val[kSmallSort];
    uint16_t count[256][kSmallThreads / 32];      // per digit and warp, then exclusive offsets
    uint32_t warp_sum[kSmallThreads / 32];
};

__global__ void __launch_bounds__(kSmallThreads) k_small_sort(int n, int bits, const uint32_t* keys_in,
                                                              const uint32_t* vals_in, uint32_t* keys_out,
                                                              uint32_t* vals_out) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    SmallSortSmem& S = *reinterpret_cast<SmallSortSmem*>(smem_raw);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    uint32_t key[kSmallItems], val[kSmallItems], rank[kSmallItems];
    const int first = warp * 32 * kSmallItems + lane;
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
        const int i = first + r * 32;
        key[r] = i < n ? keys_in[i] : 0u;
        val[r] = i < n ? vals_in[i] : 0u;
    }
    for (int shift = 0; shift < bits; shift += 8) {
        for (int i = tid; i < 256 * (kSmallThreads / 32) / 2; i += kSmallThreads) ((uint32_t*)S.count)[i] = 0u;
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSmallItems; ++r) {
            if (first - lane + r * 32 >= n) break;               // warp-uniform
            const bool valid = first + r * 32 < n;
            const uint32_t d = (key[r] >> shift) & 255u;
            const unsigned peers = __match_any_sync(0xffffffffu, valid ? d : 256u);
            uint32_t before = 0u;
            if (valid) before = S.count[d][warp];
            __syncwarp();
            rank[r] = before + __popc(peers & ((1u << lane) - 1u));
            if (valid && lane == __ffs(peers) - 1) S.count[d][warp] = (uint16_t)(before + __popc(peers));
            __syncwarp();
        }
        __syncthreads();
        // exclusive scan over (digit, warp), eight entries a thread
        uint16_t* c = &S.count[0][0] + tid * 8;
        uint32_t v[8], tot = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) { v[k] = tot; tot += c[k]; }
        uint32_t x = tot;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) S.warp_sum[warp] = x;
        __syncthreads();
        if (warp == 0) {
            const uint32_t w = S.warp_sum[lane];
            uint32_t y = w;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t z = __shfl_up_sync(0xffffffffu, y, o);
                if (lane >= o) y += z;
            }
            S.warp_sum[lane] = y - w;
        }
        __syncthreads();
        const uint32_t base = S.warp_sum[warp] + x - tot;
#pragma unroll
        for (int k = 0; k < 8; ++k) c[k] = (uint16_t)(base + v[k]);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSmallItems; ++r) {
            if (first + r * 32 < n) {
                const uint32_t dst = S.count[(key[r] >> shift) & 255u][warp] + rank[r];
                S.key[dst] = key[r];
                S.val[dst] = val[r];
            }
        }
        __syncthreads();
#pragma unroll
        for (int r = 0; r < kSmallItems; ++r) {
            const int i = first + r * 32;
            if (i < n) { key[r] = S.key[i]; val[r] = S.val[i]; }
        }
    }
#pragma unroll
    for (int r = 0; r < kSmallItems; ++r) {
        const int i = first + r * 32;
        if (i < n) { keys_out[i] = key[r]; vals_out[i] = val[r]; }
    }
}

// ---- counting sort by cell ------------------------------------------------------
// A step's particles are sorted over cells whose number is known, so one
// counting pass replaces the radix passes: count the cells' particles, scan
// the counts over the grid, place each particle in its cell's range, then
// order every cell's few particles by id (the arrival order is the atomics').
// The result is the radix sort's, (cell, id) order, and the scanned counts
// are the cell ranges of every cell, empty ones included: cell c holds slots
// [cell_start[c], cell_start[c + 1]).
constexpr int kScanCells = 8192;      // cells per block of the scan, 32 per thread

// Keys by slot, and each particle's arrival rank in its cell; one atomic per
// distinct cell and per distinct scan tile of a warp (slots are nearly in
// cell order from the previous step, so a warp holds a few of each).
template <bool BATCH>
__global__ void __launch_bounds__(kBlock) k_cell_count(Params P, const float4* __restrict__ pos,
                                                       uint32_t* __restrict__ keys, uint32_t* __restrict__ ranks,
                                                       uint32_t* __restrict__ cell_count,
                                                       uint32_t* __restrict__ tile_sum, int* __restrict__ clamped) {
    after_previous();
    const int s = blockIdx.x * kBlock + threadIdx.x, lane = threadIdx.x & 31;
    const bool valid = s < P.n;
    int c = 0;
    const uint32_t key = valid ? cell_key<BATCH>(P, s, pos[s], c) : kEmpty;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int leader = __ffs(peers) - 1;
    uint32_t before = 0u;
    if (valid && lane == leader) before = atomicAdd(&cell_count[key], (uint32_t)__popc(peers));
    before = __shfl_sync(0xffffffffu, before, leader);
    const unsigned tile = valid ? key / kScanCells : kEmpty;
    const unsigned mates = __match_any_sync(0xffffffffu, tile);
    if (!valid) return;
    if (lane == __ffs(mates) - 1) atomicAdd(&tile_sum[tile], (uint32_t)__popc(mates));
    keys[s] = key;
    ranks[s] = before + (uint32_t)__popc(peers & ((1u << lane) - 1u));
    count_clamped(c, clamped);
}

// Exclusive scan of the counts of one tile of cells, behind the particles of
// the tiles before it; leaves the counts at zero for the next step. A tile
// without particles (most of a dam break's box) only writes. Cells are scanned
// in rows of 1,024, four to a thread: all rows' counts are loaded at once, each
// warp scans its part of every row, and the 64 (row, warp) totals are scanned
// by one warp -- two barriers; a block scan per row, one after another, took
// 12 us for the five tiles of a 38,000-cell grid.
__global__ void __launch_bounds__(kBlock) k_cell_scan(uint32_t* __restrict__ cell_count,
                                                      const uint32_t* __restrict__ tile_sum,
                                                      uint32_t* __restrict__ cell_start, int* __restrict__ flags) {
    after_previous();
    // the build's words: cleared here, not by a memset before the count pass,
    // which cannot be placed early (16 DEM steps 597 -> 493 us without it and
    // the error history's); the count pass has left its clamped count in flags[6]
    if (blockIdx.x == 0 && threadIdx.x < 8) {
        const int clamped = flags[6];
        __syncwarp(0xffu);
        flags[threadIdx.x] = threadIdx.x == 4 ? clamped : 0;
    }
    constexpr int kRowsPerTile = kScanCells / (kBlock * 4), kWarps = kBlock / 32;
    static_assert(kRowsPerTile * kWarps == 64, "one warp scans the (row, warp) totals, two each");
    __shared__ uint32_t s_warp[kWarps], s_total[kRowsPerTile * kWarps];
    const int tile = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t first = (size_t)tile * kScanCells + tid * 4;
    const uint32_t here = tile_sum[tile];
    uint4 v[kRowsPerTile];
    if (here) {
#pragma unroll
        for (int r = 0; r < kRowsPerTile; ++r) v[r] = *reinterpret_cast<const uint4*>(cell_count + first + r * kBlock * 4);
    }
    uint32_t mine = 0, before;
    for (int i = tid; i < tile; i += kBlock) mine += tile_sum[i];
    mine = __reduce_add_sync(0xffffffffu, mine);
    if (lane == 0) s_warp[warp] = mine;
    uint32_t e[kRowsPerTile];       // exclusive within the warp's part of the row
    if (here) {
#pragma unroll
        for (int r = 0; r < kRowsPerTile; ++r) {
            const uint32_t t = v[r].x + v[r].y + v[r].z + v[r].w;
            uint32_t x = t;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            e[r] = x - t;
            if (lane == 31) s_total[r * kWarps + warp] = x;
        }
    }
    __syncthreads();
    before = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) before += s_warp[w];
    if (here && warp == 0) {
        const uint32_t a = s_total[2 * lane], b = s_total[2 * lane + 1];
        uint32_t x = a + b;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        s_total[2 * lane] = x - a - b;
        s_total[2 * lane + 1] = x - b;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRowsPerTile; ++r) {
        uint4 start = make_uint4(before, before, before, before);
        if (here) {
            start.x += s_total[r * kWarps + warp] + e[r];
            start.y = start.x + v[r].x;
            start.z = start.y + v[r].y;
            start.w = start.z + v[r].z;
            *reinterpret_cast<uint4*>(cell_count + first + r * kBlock * 4) = make_uint4(0u, 0u, 0u, 0u);
        }
        *reinterpret_cast<uint4*>(cell_start + first + r * kBlock * 4) = start;
    }
    if (tid == 0 && tile == (int)gridDim.x - 1) cell_start[(size_t)(tile + 1) * kScanCells] = before + here;
}

// Each particle's (id, slot) into its cell's range, in arrival order; clears
// the tile sums for the next step.
__global__ void __launch_bounds__(kBlock) k_cell_place(int n, int ntiles, const uint32_t* __restrict__ keys,
                                                       const uint32_t* __restrict__ ranks, const int* __restrict__ ids,
                                                       const uint32_t* __restrict__ cell_start,
                                                       uint2* __restrict__ placed, uint32_t* __restrict__ tile_sum) {
    after_previous();
    const int s = blockIdx.x * kBlock + threadIdx.x;
    if (s < ntiles) tile_sum[s] = 0u;
    if (s >= n) return;
    placed[cell_start[keys[s]] + ranks[s]] = make_uint2((uint32_t)ids[s], (uint32_t)s);
}

// Orders every cell's particles by id: a particle's place is the number of
// smaller ids in its cell.
__global__ void __launch_bounds__(kBlock) k_cell_rank(int n, const uint32_t* __restrict__ keys,
                                                      const uint2* __restrict__ placed,
                                                      const uint32_t* __restrict__ cell_start,
                                                      uint32_t* __restrict__ keys_out, uint32_t* __restrict__ vals_out) {
    after_previous();
    const int p = blockIdx.x * kBlock + threadIdx.x;
    if (p >= n) return;
    const uint2 me = placed[p];
    const uint32_t key = keys[me.y];
    const uint32_t lo = cell_start[key], hi = cell_start[key + 1];
    uint32_t t = lo;
    for (uint32_t q = lo; q < hi; ++q) t += placed[q].x < me.x ? 1u : 0u;
    keys_out[t] = key;
    vals_out[t] = me.y;
}

// A set of the particle state's arrays.
struct State {
    float4 *pos, *vel, *vap;
    float2* rp;
    int* ids;
};

// The particle of slot s, at x, into sorted slot t.
__device__ __forceinline__ void move_particle(const Params& P, uint32_t s, uint32_t t, float4 x,
                                              const float4* __restrict__ vel, const float4* __restrict__ vap,
                                              const float2* __restrict__ rp, int id, const State& out) {
    const float4 v = vel[s];
    out.pos[t] = x;
    out.vel[t] = v;
    P.cx[t] = x.x;
    P.cy[t] = x.y;
    P.x0.z[t] = x.z;
    if (P.x0.xy) {
        P.x0.xy[t] = make_float2(x.x, x.y);
        P.v0.xy[t] = make_float2(v.x, v.y);
        P.v0.z[t] = v.z;
    }
    out.vap[t] = vap[s];
    out.rp[t] = rp[s];
    out.ids[t] = id;
}

// k_cell_rank and the reorder in one launch: each particle finds its place
// and moves its state there, reads coalesced, writes within its cell's range.
// Below kWallListMin particles, where nothing is listed by sorted slot on the
// way and a launch counts (WCSPH frame of 8 steps at 16k 641 -> 620 us).
__global__ void __launch_bounds__(kBlock) k_rank_reorder(Params P, const uint32_t* __restrict__ keys,
                                                         const uint2* __restrict__ placed,
                                                         const uint32_t* __restrict__ cell_start,
                                                         const float4* __restrict__ pos, const float4* __restrict__ vel,
                                                         const float4* __restrict__ vap, const float2* __restrict__ rp,
                                                         const int* __restrict__ ids, uint32_t* __restrict__ keys_out,
                                                         uint32_t* __restrict__ vals_out, State out) {
    after_previous();
    const int s = blockIdx.x * kBlock + threadIdx.x;
    if (s >= P.n) return;
    const uint32_t key = keys[s];
    const int id = ids[s];
    const uint32_t lo = cell_start[key], hi = cell_start[key + 1];
    uint32_t t = lo;
    for (uint32_t q = lo; q < hi; ++q) t += placed[q].x < (uint32_t)id ? 1u : 0u;
    keys_out[t] = key;
    vals_out[t] = (uint32_t)s;
    move_particle(P, s, t, pos[s], vel, vap, rp, id, out);
}

// Gathers the particle state into sorted order and records each occupied
// cell's [start, end) slot range (cell_start null: the counting sort has).
template <bool BATCH>
__global__ void k_reorder(Params P, const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                          const float4* __restrict__ pos, const float4* __restrict__ vel,
                          const float4* __restrict__ vap, const float2* __restrict__ rp, const int* __restrict__ ids,
                          float4* __restrict__ pos2, float4* __restrict__ vel2, float4* __restrict__ vap2,
                          float2* __restrict__ rp2, int* __restrict__ ids2, uint32_t* __restrict__ cell_start,
                          uint32_t* __restrict__ cell_end) {
    after_previous();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = P.n;
    const uint32_t s = t < n ? vals[t] : 0u;
    const float4 x = t < n ? pos[s] : make_float4(0.f, 0.f, 0.f, 0.f);
    list_near_walls<BATCH>(P, t, x);
    if (t >= n) return;
    move_particle(P, s, (uint32_t)t, x, vel, vap, rp, ids[s], State{pos2, vel2, vap2, rp2, ids2});
    if (!cell_start) return;
    const uint32_t k = keys[t];
    if (t == 0 || keys[t - 1] != k) cell_start[k] = (uint32_t)t;
    if (t == n - 1 || keys[t + 1] != k) cell_end[k] = (uint32_t)t + 1u;
}

// The same in two launches, for the first step after an upload: positions,
// ids and cell ranges (all that the neighbour build reads) here, the rest
// in k_reorder_state once the upload's copies of it are in.
template <bool BATCH>
__global__ void k_reorder_pos(Params P, const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                              const float4* __restrict__ pos, const int* __restrict__ ids, float4* __restrict__ pos2,
                              int* __restrict__ ids2, uint32_t* __restrict__ cell_start,
                              uint32_t* __restrict__ cell_end) {
    after_previous();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int n = P.n;
    const uint32_t s = t < n ? vals[t] : 0u;
    const float4 x = t < n ? pos[s] : make_float4(0.f, 0.f, 0.f, 0.f);
    list_near_walls<BATCH>(P, t, x);
    if (t >= n) return;
    pos2[t] = x;
    P.cx[t] = x.x;
    P.cy[t] = x.y;
    P.x0.z[t] = x.z;
    if (P.x0.xy) {
        P.x0.xy[t] = make_float2(x.x, x.y);
    }
    ids2[t] = ids[s];
    if (!cell_start) return;
    const uint32_t k = keys[t];
    if (t == 0 || keys[t - 1] != k) cell_start[k] = (uint32_t)t;
    if (t == n - 1 || keys[t + 1] != k) cell_end[k] = (uint32_t)t + 1u;
}

// Gathers velocities, half-step velocities and (density, pressure) into
// sorted order.
__global__ void k_reorder_state(Params P, const uint32_t* __restrict__ vals, const float4* __restrict__ vel,
                                const float4* __restrict__ vap, const float2* __restrict__ rp,
                                float4* __restrict__ vel2, float4* __restrict__ vap2, float2* __restrict__ rp2) {
    after_previous();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= P.n) return;
    const uint32_t s = vals[t];
    const float4 v = vel[s];
    vel2[t] = v;
    if (P.v0.xy) {
        P.v0.xy[t] = make_float2(v.x, v.y);
        P.v0.z[t] = v.z;
    }
    vap2[t] = vap[s];
    rp2[t] = rp[s];
}

// Per-thread schedule: one thread per sorted particle. The three cells of a
// grid row are adjacent in sorted order, so each of the nine rows is one
// contiguous slot range; candidates are taken in increasing slot order and
// the list is sorted. In a batch the walk stays inside the particle's
// scene's grid.
//
// ~216 candidates are tested for ~33 kept, so the kernel is bound by the
// instructions and the L1 wavefronts of the test. It is kept to seven
// instructions a candidate: x, y and z lie in arrays of their own (the reorder
// writes them beside the position), a row is read in aligned fours -- three
// 16-byte loads for four candidates instead of four -- and two candidates
// share an instruction of the FMA chain e = |d|^2 - h^2 (f32x2). A funnel
// shift collects e's sign into the row's mask, and a second mask says which
// fours hold a candidate within rounding of the cut-off: only those are gone
// over again with the reference's FP64 test. (A block of fluid started on a
// lattice of spacing h/2 has candidates at exactly h in five of its nine rows;
// going over the whole row took 198 us at 1M such particles and 26.9 at 16k,
// the fours 184 and 23.0.) Of a NaN coordinate e is the canonical NaN, whose
// sign bit is clear: the particle is nobody's neighbour, as in a comparison. The masks of the nine rows wait in shared memory;
// the list is then written quad by quad, every lane's k-th quad in the same
// store (512 contiguous bytes a warp), where one 4-byte store per entry was a
// sector write for each of 34M entries at 1M particles.
// One candidate after another from the float4 positions, eleven instructions
// each: 184 us at 1M particles, 654 at 4M, 36 at 97k; now 151, 555 and 27.
// Loading a four ahead of the one in use: 12 registers more, 163 us at 1M.
constexpr int kRows = 9;

// Two FP32 operations of one instruction.
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 d;
    asm("add.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
    return d;
}
__device__ __forceinline__ float2 square_plus2(float2 a, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(c)));
    return d;
}

// The candidates of the row [lo, hi) among the 32 slots from w on (a multiple
// of four below hi): bit 31 - c of the result is set when slot w + c is one
// and a neighbour of the particle at pi. Reads whole fours.
__device__ __forceinline__ uint32_t row_mask(const Params& P, float4 pi, uint32_t w, uint32_t lo, uint32_t hi) {
    const float4* __restrict__ X = reinterpret_cast<const float4*>(P.cx + w);
    const float4* __restrict__ Y = reinterpret_cast<const float4*>(P.cy + w);
    const float4* __restrict__ Z = reinterpret_cast<const float4*>(P.x0.z + w);
    // h2_hi - h2 is 1e-5 h^2, some thirty times the rounding of e near h
    const float band = P.h2_hi - P.h2;
    const uint32_t first = lo > w ? lo - w : 0u, end = min(hi - w, 32u), groups = (end + 3u) >> 2;
    uint32_t mask = 0u, close = 0u;      // close: one bit per four candidates, the last four lowest
    const float2 px = make_float2(-pi.x, -pi.x), py = make_float2(-pi.y, -pi.y), pz = make_float2(-pi.z, -pi.z);
    const float2 cut = make_float2(-P.h2, -P.h2);
    auto excess = [&](float2 x, float2 y, float2 z) {
        return square_plus2(add2(z, pz), square_plus2(add2(y, py), square_plus2(add2(x, px), cut)));
    };
    for (uint32_t g = 0; g < groups; ++g) {
        const float4 x = X[g], y = Y[g], z = Z[g];
        const float2 a = excess(make_float2(x.x, x.y), make_float2(y.x, y.y), make_float2(z.x, z.y));
        const float2 b = excess(make_float2(x.z, x.w), make_float2(y.z, y.w), make_float2(z.z, z.w));
        mask = __funnelshift_l(__float_as_uint(a.x), mask, 1);
        mask = __funnelshift_l(__float_as_uint(a.y), mask, 1);
        mask = __funnelshift_l(__float_as_uint(b.x), mask, 1);
        mask = __funnelshift_l(__float_as_uint(b.y), mask, 1);
        const float near = fminf(fminf(fabsf(a.x), fabsf(a.y)), fminf(fabsf(b.x), fabsf(b.y)));
        close = __funnelshift_l(__float_as_uint(near - band), close, 1);
    }
    mask = (mask << (32u - 4u * groups)) & (kEmpty << (32u - end)) & (kEmpty >> first);
    while (close) {
        const uint32_t low = (uint32_t)__ffs((int)close) - 1u;
        close &= close - 1u;
        const uint32_t c0 = 4u * (groups - 1u - low);
        for (uint32_t c = max(c0, first); c < min(c0 + 4u, end); ++c) {
            const float4 pj = make_float4(P.cx[w + c], P.cy[w + c], P.x0.z[w + c], 0.f);
            const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
            const float e = __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmaf_rn(dx, dx, -P.h2)));
            if (!(fabsf(e) <= band)) continue;
            const uint32_t bit = 0x80000000u >> c;
            if (exact_neighbor(pi, pj, P.h2_exact)) mask |= bit;
            else mask &= ~bit;
        }
    }
    return mask;
}

template <bool BATCH, int BS>
__global__ void __launch_bounds__(BS) k_build_nbr(Params P, const uint32_t* __restrict__ keys,
                                                  const uint32_t* __restrict__ cell_start,
                                                  const uint32_t* __restrict__ cell_end, int* __restrict__ counts,
                                                  int* __restrict__ list, int* __restrict__ flags) {
    after_previous();
    __shared__ uint32_t s_first[kRows][BS], s_mask[kRows][BS];     // each thread uses its own column
    const int tid = threadIdx.x;
    const int t = blockIdx.x * BS + tid;
    const bool valid = t < P.n;       // every lane stays for the warp reductions below
    const int n = P.n;
    int cnt = 0;
    if (valid) {
        const Grid g = BATCH ? P.scenes[P.slot_scene[t]].g : P.g;
        const uint32_t base = BATCH ? P.scenes[P.slot_scene[t]].cell_base : 0u;
        const uint32_t nx = (uint32_t)g.nx, ny = (uint32_t)g.ny;
        const uint32_t key = keys[t] - base;
        const int ci = (int)(key % nx), cj = (int)((key / nx) % ny), ck = (int)(key / (nx * ny));
        const int a0 = max(ci - 1, 0), a1 = min(ci + 1, g.nx - 1);
        // the nine rows' slot ranges: independent loads, in flight together
        uint32_t longest = 0u;
#pragma unroll
        for (int r = 0; r < kRows; ++r) {
            const int j = cj + r % 3 - 1, k = ck + r / 3 - 1;
            uint32_t lo = 0u, hi = 0u;
            if (j >= 0 && j < g.ny && k >= 0 && k < g.nz) {
                const uint32_t row = base + (uint32_t)j * nx + (uint32_t)k * nx * ny;
                if (P.dense_cells) {
                    lo = cell_start[row + a0];
                    hi = cell_end[row + a1];
                } else {
                    row_range(cell_start, cell_end, row, a0, a1, lo, hi);
                }
            }
            s_first[r][tid] = lo;
            s_mask[r][tid] = hi;
            longest = max(longest, hi - (lo & ~3u));
        }
        const float4 pi = make_float4(P.cx[t], P.cy[t], P.x0.z[t], 0.f);
        if (longest <= 32u) {
            for (int r = 0; r < kRows; ++r) {
                const uint32_t lo = s_first[r][tid], hi = s_mask[r][tid], w = lo & ~3u;
                const uint32_t mask = lo < hi ? row_mask(P, pi, w, lo, hi) : 0u;
                s_first[r][tid] = w;
                s_mask[r][tid] = mask;
                cnt += __popc(mask);
            }
            // the set bits of the nine masks in order, four to a store
            const int kept = min(cnt, P.cap);
            int4* __restrict__ out = reinterpret_cast<int4*>(list) + t;
            int r = -1;
            uint32_t mask = 0u, q = 0u;
            auto next = [&] {
                while (mask == 0u) {
                    ++r;
                    mask = s_mask[r][tid];
                    q = s_first[r][tid];
                }
                const int z = __clz((int)mask);
                mask = (mask << z) << 1;
                q += (uint32_t)z;
                return (int)q++;
            };
            for (int c = 0; c < kept; c += 4, out += n) {
                int4 e = make_int4(0, 0, 0, 0);
                e.x = next();
                if (c + 1 < kept) e.y = next();
                if (c + 2 < kept) e.z = next();
                if (c + 3 < kept) e.w = next();
                *out = e;
            }
        } else {        // a row of more than 32 candidates: 32 at a time, an entry a store
            for (int r = 0; r < kRows; ++r) {
                const uint32_t lo = s_first[r][tid], hi = s_mask[r][tid];
                if (lo >= hi) continue;
                for (uint32_t w = lo & ~3u; w < hi; w += 32u) {
                    uint32_t mask = row_mask(P, pi, w, lo, hi), q = w;
                    while (mask) {
                        const int z = __clz((int)mask);
                        mask = (mask << z) << 1;
                        q += (uint32_t)z;
                        if (cnt < P.cap) list[nbr_index(cnt, n, t)] = (int)q;
                        ++q;
                        ++cnt;
                    }
                }
            }
        }
        counts[t] = cnt;
        if (cnt > P.cap) atomicOr(&flags[0], 1);
    }
    nbr_flags(cnt, flags);
}

// Warp-cooperative schedule (row tiles). The lanes of a warp whose particles
// lie in the same grid row (same scene, j and k; consecutive sorted
// particles mostly do) form a group and walk its nine neighbour rows
// together. For each row the group's slot span -- the union of its lanes'
// three-cell ranges, one contiguous run of cells -- is staged 32 candidates
// at a time in shared memory, one coalesced load per lane, and each lane
// tests the staged candidates that lie inside its own range, in slot order.
// A lane therefore accepts the same candidates in the same order as in the
// per-thread schedule; the gathers become one load per candidate per group
// instead of one per candidate per lane.
template <bool BATCH, int BS>
__global__ void __launch_bounds__(BS) k_build_nbr_tile(Params P, const float4* __restrict__ pos,
                                                       const uint32_t* __restrict__ keys,
                                                       const uint32_t* __restrict__ cell_start,
                                                       const uint32_t* __restrict__ cell_end,
                                                       int* __restrict__ counts, int* __restrict__ list,
                                                       int* __restrict__ flags) {
    after_previous();
    __shared__ float4 s_tile[BS];
    float4* tile = s_tile + (threadIdx.x & ~31u);
    const int lane = threadIdx.x & 31;
    const int t = blockIdx.x * BS + threadIdx.x;
    const bool valid = t < P.n;
    const int n = P.n;
    int cnt = 0;
    float4 pi = make_float4(0.f, 0.f, 0.f, 0.f);
    int nx = 1, ny = 1, nz = 1, ci = 0, cj = 0, ck = 0;
    uint32_t base = 0, rowkey = kEmpty;     // rowkey: the global key of cell (0, j, k) of the particle's row
    if (valid) {
        const Grid g = BATCH ? P.scenes[P.slot_scene[t]].g : P.g;
        base = BATCH ? P.scenes[P.slot_scene[t]].cell_base : 0u;
        nx = g.nx; ny = g.ny; nz = g.nz;
        pi = pos[t];
        const uint32_t key = keys[t] - base;
        ci = (int)(key % (uint32_t)nx);
        cj = (int)((key / (uint32_t)nx) % (uint32_t)ny);
        ck = (int)(key / ((uint32_t)nx * (uint32_t)ny));
        rowkey = keys[t] - (uint32_t)ci;
    }
    const int a0 = max(ci - 1, 0), a1 = min(ci + 1, nx - 1);
    unsigned todo = __ballot_sync(0xffffffffu, valid);
    while (todo) {
        const int leader = __ffs(todo) - 1;
        const uint32_t rk = __shfl_sync(0xffffffffu, rowkey, leader);
        const unsigned grp = __ballot_sync(0xffffffffu, valid && rowkey == rk);
        todo &= ~grp;
        const bool mine = (grp >> lane) & 1u;
        // the group shares scene, j, k and the grid: take them from the leader
        const int gj = __shfl_sync(0xffffffffu, cj, leader), gk = __shfl_sync(0xffffffffu, ck, leader);
        const int gnx = __shfl_sync(0xffffffffu, nx, leader), gny = __shfl_sync(0xffffffffu, ny, leader);
        const int gnz = __shfl_sync(0xffffffffu, nz, leader);
        const uint32_t gbase = __shfl_sync(0xffffffffu, base, leader);
        for (int k = max(gk - 1, 0); k <= min(gk + 1, gnz - 1); ++k) {
            for (int j = max(gj - 1, 0); j <= min(gj + 1, gny - 1); ++j) {
                const uint32_t row = gbase + (uint32_t)j * (uint32_t)gnx + (uint32_t)k * (uint32_t)gnx * (uint32_t)gny;
                uint32_t lo = kEmpty, hi = 0;
                if (mine) {
                    for (int a = a0; a <= a1; ++a) {
                        const uint32_t s = cell_start[row + a];
                        if (s != kEmpty) {
                            if (lo == kEmpty) lo = s;
                            hi = cell_end[row + a];
                        }
                    }
                }
                const uint32_t L = __reduce_min_sync(0xffffffffu, lo);
                const uint32_t H = __reduce_max_sync(0xffffffffu, hi);
                if (L == kEmpty) continue;
                for (uint32_t q0 = L; q0 < H; q0 += 32u) {
                    if (q0 + lane < H) tile[lane] = pos[q0 + lane];
                    __syncwarp();
                    if (mine && lo != kEmpty) {
                        // this lane's part of the staged chunk [q0, q0 + 32): [c0, c1)
                        const uint32_t c0 = lo > q0 ? lo - q0 : 0u;
                        const uint32_t c1 = hi > q0 ? min(hi - q0, 32u) : 0u;
                        for (uint32_t c = c0; c < c1; ++c) {
                            const float4 pj = tile[c];
                            const float dx = pi.x - pj.x, dy = pi.y - pj.y, dz = pi.z - pj.z;
                            const float d2 = dist2(dx, dy, dz);
                            bool acc;
                            if (d2 < P.h2_lo) acc = true;
                            else if (d2 > P.h2_hi) acc = false;
                            else acc = exact_neighbor(pi, pj, P.h2_exact);
                            if (acc) {
                                if (cnt < P.cap) list[nbr_index(cnt, n, t)] = (int)(q0 + c);
                                ++cnt;
                            }
                        }
                    }
                    __syncwarp();
                }
            }
        }
    }
    if (valid) {
        counts[t] = cnt;
        if (cnt > P.cap) atomicOr(&flags[0], 1);
    }
    nbr_flags(cnt, flags);
}

inline int grid_of(int n) { return (n + kBlock - 1) / kBlock; }

}  // namespace

void launch_reset_cells(cudaStream_t st, int n, const uint32_t* sorted_keys, uint32_t* cell_start) {
    if (n > 0) k_reset_cells<<<grid_of(n), kBlock, 0, st>>>(n, sorted_keys, cell_start);
}

void launch_cell_keys(cudaStream_t st, const Params& P, const float4* pos, const int* ids, uint32_t* keys_by_id,
                      uint32_t* slot_by_id, int* clamped) {
    if (P.n <= 0) return;
    if (P.scenes) k_cell_keys<true><<<grid_of(P.n), kBlock, 0, st>>>(P, pos, ids, keys_by_id, slot_by_id, clamped);
    else k_cell_keys<false><<<grid_of(P.n), kBlock, 0, st>>>(P, pos, ids, keys_by_id, slot_by_id, clamped);
}

int radix_blocks(int n) { return (n + kTile - 1) / kTile; }

bool small_sort(cudaStream_t st, int n, int bits, const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out,
                uint32_t* vals_out) {
    if (n > kSmallSort) return false;
    cudaFuncSetAttribute(k_small_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallSortSmem));
    k_small_sort<<<1, kSmallThreads, sizeof(SmallSortSmem), st>>>(n, bits, keys_in, vals_in, keys_out, vals_out);
    return true;
}

size_t cell_sort_tiles(size_t ncells) { return (ncells + kScanCells - 1) / kScanCells; }
size_t cell_sort_cells(size_t ncells) { return cell_sort_tiles(ncells) * kScanCells + 4; }

void launch_cell_count(cudaStream_t st, const Params& P, const float4* pos, uint32_t* keys, uint32_t* ranks,
                       uint32_t* cell_count, uint32_t* tile_sum, int* clamped) {
    if (P.n <= 0) return;
    auto kernel = P.scenes ? k_cell_count<true> : k_cell_count<false>;
    launch_chained(kernel, grid_of(P.n), kBlock, 0, st, P, pos, keys, ranks, cell_count, tile_sum, clamped);
}

void launch_cell_sort(cudaStream_t st, int n, size_t ncells, const int* ids, const uint32_t* keys, const uint32_t* ranks,
                      uint32_t* cell_count, uint32_t* tile_sum, uint32_t* cell_start, int* flags, uint2* placed,
                      uint32_t* keys_out, uint32_t* vals_out) {
    launch_cell_place(st, n, ncells, ids, keys, ranks, cell_count, tile_sum, cell_start, flags, placed);
    if (n > 0) launch_chained(k_cell_rank, grid_of(n), kBlock, 0, st, n, keys, placed, cell_start, keys_out, vals_out);
}

void launch_cell_place(cudaStream_t st, int n, size_t ncells, const int* ids, const uint32_t* keys,
                       const uint32_t* ranks, uint32_t* cell_count, uint32_t* tile_sum, uint32_t* cell_start,
                       int* flags, uint2* placed) {
    if (n <= 0) return;
    const int tiles = (int)cell_sort_tiles(ncells);
    launch_chained(k_cell_scan, tiles, kBlock, 0, st, cell_count, tile_sum, cell_start, flags);
    launch_chained(k_cell_place, grid_of(std::max(n, tiles)), kBlock, 0, st, n, tiles, keys, ranks, ids, cell_start,
                   placed, tile_sum);
}

void launch_rank_reorder(cudaStream_t st, const Params& P, const uint32_t* keys, const uint2* placed,
                         const uint32_t* cell_start, const float4* pos, const float4* vel, const float4* vap,
                         const float2* rp, const int* ids, uint32_t* keys_out, uint32_t* vals_out, float4* pos2,
                         float4* vel2, float4* vap2, float2* rp2, int* ids2) {
    if (P.n <= 0) return;
    launch_chained(k_rank_reorder, grid_of(P.n), kBlock, 0, st, P, keys, placed, cell_start, pos, vel, vap, rp, ids,
                   keys_out, vals_out, State{pos2, vel2, vap2, rp2, ids2});
}

int radix_sort(cudaStream_t st, int n, int bits, uint32_t* keys[2], uint32_t* vals[2], uint32_t* hist, int nblocks_cap) {
    const int nb = radix_blocks(n);
    if (nb > nblocks_cap || n <= 0) return 0;
    if (small_sort(st, n, bits, keys[0], vals[0], keys[0], vals[0])) return 0;
    int cur = 0;
    for (int shift = 0; shift < bits; shift += 8) {
        launch_chained(k_radix_hist, nb, kBlock, 0, st, n, shift, nb, keys[cur], hist);
        launch_chained(k_radix_scan, 256, kBlock, 0, st, nb, hist, hist + (size_t)256 * nb);
        launch_chained(k_radix_scatter, nb, kBlock, 0, st, n, shift, nb, keys[cur], vals[cur], keys[cur ^ 1],
                       vals[cur ^ 1], hist, hist + (size_t)256 * nb);
        cur ^= 1;
    }
    return cur;
}

void launch_reorder(cudaStream_t st, const Params& P, const uint32_t* keys, const uint32_t* vals, const float4* pos,
                    const float4* vel, const float4* vap, const float2* rp, const int* ids, float4* pos2, float4* vel2,
                    float4* vap2, float2* rp2, int* ids2, uint32_t* cell_start, uint32_t* cell_end) {
    if (P.n <= 0) return;
    auto kernel = P.scenes ? k_reorder<true> : k_reorder<false>;
    launch_chained(kernel, grid_of(P.n), kBlock, 0, st, P, keys, vals, pos, vel, vap, rp, ids, pos2, vel2, vap2, rp2,
                   ids2, cell_start, cell_end);
}

void launch_reorder_pos(cudaStream_t st, const Params& P, const uint32_t* keys, const uint32_t* vals, const float4* pos,
                        const int* ids, float4* pos2, int* ids2, uint32_t* cell_start, uint32_t* cell_end) {
    if (P.n <= 0) return;
    auto kernel = P.scenes ? k_reorder_pos<true> : k_reorder_pos<false>;
    launch_chained(kernel, grid_of(P.n), kBlock, 0, st, P, keys, vals, pos, ids, pos2, ids2, cell_start, cell_end);
}

void launch_reorder_state(cudaStream_t st, const Params& P, const uint32_t* vals, const float4* vel, const float4* vap,
                          const float2* rp, float4* vel2, float4* vap2, float2* rp2) {
    if (P.n > 0) k_reorder_state<<<grid_of(P.n), kBlock, 0, st>>>(P, vals, vel, vap, rp, vel2, vap2, rp2);
}

void launch_build_nbr(cudaStream_t st, const Params& P, const float4* pos, const uint32_t* keys,
                      const uint32_t* cell_start, const uint32_t* cell_end, int* counts, int* list, int* flags) {
    if (P.n <= 0) return;
    with_block(P.tune.nbr_block, [&](auto B) {
        constexpr int BS = decltype(B)::value;
        const unsigned g = (unsigned)((P.n + BS - 1) / BS);
        auto go = [&](auto kernel) {
            launch_chained(kernel, g, BS, 0, st, P, keys, cell_start, cell_end, counts, list, flags);
        };
        auto go_tile = [&](auto kernel) {
            launch_chained(kernel, g, BS, 0, st, P, pos, keys, cell_start, cell_end, counts, list, flags);
        };
        if (P.tune.nbr_schedule == 1) {
            if (P.scenes) go_tile(k_build_nbr_tile<true, BS>); else go_tile(k_build_nbr_tile<false, BS>);
        } else {
            if (P.scenes) go(k_build_nbr<true, BS>); else go(k_build_nbr<false, BS>);
        }
    });
}

}  // namespace psb
