// boundary.cu -- static boundary particles (config profile), after Akinci,
// Ihmsen, Akinci, Solenthaler & Teschner 2012, "Versatile rigid-fluid
// coupling for incompressible SPH".
//
// A solid is sampled by particles b. Each gets the volume-weighted mass
// psi_b = rho0 / sum_k W(x_b - x_k) over the boundary particles (their
// eq. 5), so that the sampling's density, whatever its spacing, stands for a
// full solid. A fluid particle i gains psi_b W_ib in density and the
// pressure term psi_b p_i/rho0^2 gradW_ib (the fluid's own pressure mirrored
// onto the solid); the kernels in sph.cu add both. The reference has no
// counterpart: its obstacles are analytic collision objects
// (src/Kernel/Collision/*), used here only as the box.
//
// The boundary set is sorted once into its own cell ranges over the scene's
// grid; each step, the fluid particles near its bounding box list their
// boundary neighbours (quads, like the fluid lists).
#include "psb_internal.cuh"

namespace psb {

namespace {

inline int blocks_for(int n) { return (n + kBlock - 1) / kBlock; }

__global__ void k_iota(int n, int* __restrict__ a) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) a[i] = i;
}

// Sorted slot t takes the boundary particle vals[t]; cell ranges from the
// sorted keys.
__global__ void k_bnd_gather(int nb, const uint32_t* __restrict__ keys, const uint32_t* __restrict__ vals,
                             const float4* __restrict__ raw, float4* __restrict__ sorted, int* __restrict__ ids,
                             uint32_t* __restrict__ cell_start, uint32_t* __restrict__ cell_end) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nb) return;
    const int s = (int)vals[t];
    const float4 x = raw[s];
    sorted[t] = make_float4(x.x, x.y, x.z, 0.f);
    ids[t] = s;
    const uint32_t k = keys[t];
    if (t == 0 || keys[t - 1] != k) cell_start[k] = (uint32_t)t;
    if (t == nb - 1 || keys[t + 1] != k) cell_end[k] = (uint32_t)t + 1u;
}

// psi_b / m of sorted boundary slot t, summed in FP64 over the boundary
// particles in its 27 cells that lie within h.
__global__ void k_bnd_psi(Params P, int nb, const uint32_t* __restrict__ keys, const float4* __restrict__ sorted,
                          const uint32_t* __restrict__ cell_start, const uint32_t* __restrict__ cell_end,
                          float* __restrict__ w) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nb) return;
    const int nx = P.g.nx, ny = P.g.ny, nz = P.g.nz;
    const float4 xb = sorted[t];
    const uint32_t key = keys[t];
    const int ci = (int)(key % (uint32_t)nx), cj = (int)((key / (uint32_t)nx) % (uint32_t)ny);
    const int ck = (int)(key / ((uint32_t)nx * (uint32_t)ny));
    double s = 0.0;
    for (int k = max(ck - 1, 0); k <= min(ck + 1, nz - 1); ++k)
        for (int j = max(cj - 1, 0); j <= min(cj + 1, ny - 1); ++j) {
            const uint32_t row = (uint32_t)j * (uint32_t)nx + (uint32_t)k * (uint32_t)nx * (uint32_t)ny;
            for (int a = max(ci - 1, 0); a <= min(ci + 1, nx - 1); ++a) {
                const uint32_t lo = cell_start[row + a];
                if (lo == kEmpty) continue;
                const uint32_t hi = cell_end[row + a];
                for (uint32_t q = lo; q < hi; ++q) {
                    const float4 xk = sorted[q];
                    const float dx = xb.x - xk.x, dy = xb.y - xk.y, dz = xb.z - xk.z;
                    const float qq = (dx * dx + dy * dy + dz * dz) * P.inv_h2;
                    if (qq >= 1.f) continue;
                    const double u = 1.0 - (double)qq;
                    s += u * u * u;
                }
            }
        }
    w[t] = (float)(P.rho0_d / ((double)P.k_rho * s));
}

__global__ void k_bnd_set_w(int nb, const float* __restrict__ w, float4* __restrict__ sorted) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nb) sorted[t].w = w[t];
}

// Fluid slot t's boundary neighbours, in increasing boundary slot order.
__global__ void __launch_bounds__(kBlock) k_build_bnd_nbr(Params P, const float4* __restrict__ pos,
                                                          const uint32_t* __restrict__ keys,
                                                          const uint32_t* __restrict__ bnd_start,
                                                          const uint32_t* __restrict__ bnd_end, int* __restrict__ counts,
                                                          int* __restrict__ list, int* __restrict__ flags) {
    after_previous();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= P.n) return;
    const float4 pi = pos[t];
    int cnt = 0;
    if (pi.x >= P.bnd_lo[0] && pi.x <= P.bnd_hi[0] && pi.y >= P.bnd_lo[1] && pi.y <= P.bnd_hi[1] &&
        pi.z >= P.bnd_lo[2] && pi.z <= P.bnd_hi[2]) {
        const int nx = P.g.nx, ny = P.g.ny, nz = P.g.nz, n = P.n;
        const uint32_t key = keys[t];
        const int ci = (int)(key % (uint32_t)nx), cj = (int)((key / (uint32_t)nx) % (uint32_t)ny);
        const int ck = (int)(key / ((uint32_t)nx * (uint32_t)ny));
        const int a0 = max(ci - 1, 0), a1 = min(ci + 1, nx - 1);
        for (int k = max(ck - 1, 0); k <= min(ck + 1, nz - 1); ++k)
            for (int j = max(cj - 1, 0); j <= min(cj + 1, ny - 1); ++j) {
                const uint32_t row = (uint32_t)j * (uint32_t)nx + (uint32_t)k * (uint32_t)nx * (uint32_t)ny;
                uint32_t lo = kEmpty, hi = 0;
                for (int a = a0; a <= a1; ++a) {
                    const uint32_t s = bnd_start[row + a];
                    if (s != kEmpty) {
                        if (lo == kEmpty) lo = s;
                        hi = bnd_end[row + a];
                    }
                }
                if (lo == kEmpty) continue;
                for (uint32_t q = lo; q < hi; ++q) {
                    const float4 xb = P.bnd[q];
                    const float dx = pi.x - xb.x, dy = pi.y - xb.y, dz = pi.z - xb.z;
                    if (dx * dx + dy * dy + dz * dz > P.h2_hi) continue;
                    if (cnt < P.bnd_cap) list[nbr_index(cnt, n, t)] = (int)q;
                    ++cnt;
                }
            }
    }
    counts[t] = cnt;
    if (cnt > P.bnd_cap) atomicOr(&flags[0], 1);
}

// F_b = - sum_j m a_j^b over the fluid particles j within h of the
// boundary particle at xb, a_j^b = k_grad (psi_b / m) pV_j (1-u)^2 x^_jb
// the mirrored-pressure acceleration the boundary particle gives j (sph.cu,
// boundary_pressure); the fluid's cells are walked around xb, row by row in
// slot order. Two forms of the same sum, term by term in the same order:
//   * one thread a boundary particle: ~216 candidates, one after another, a
//     chain of ~20 us whatever the number of particles up to ~30k;
//   * one warp a boundary particle: the lanes take 32 candidates of a row at
//     a time, all nine rows' loads in flight together, and queue the accepted
//     ones in slot order in shared memory; three lanes then add the queue, a
//     component each. A shorter chain, but several times the instructions.
// k_bnd_move, solids immersed in 262k fluid particles, threads against warps:
// 500 boundary particles 27 and 8.8 us, 2,000 24 and 9.3, 8,000 19.5 and
// 16.4, 16,000 19.5 and 23: warps up to kBndWarps.
constexpr int kBndWarps = 8192;

// The first cell of the walk in each direction, and the one behind the last.
struct BndCells {
    int lo[3], hi[3];
};
__device__ __forceinline__ BndCells bnd_cells(const Params& P, float4 xb) {
    BndCells c;
    const float lo[3] = {P.g.gx, P.g.gy, P.g.gz};
    const float x[3] = {xb.x, xb.y, xb.z};
    const int dims[3] = {P.g.nx, P.g.ny, P.g.nz};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const double q = floor(((double)x[a] - (double)lo[a]) / (double)P.g.cell);
        const int i = q < 0.0 ? 0 : (q >= (double)dims[a] ? dims[a] - 1 : (int)q);
        c.lo[a] = max(i - 1, 0);
        c.hi[a] = min(i + 2, dims[a]);
    }
    return c;
}

// The slots of the walk's cells of row (j, k).
__device__ __forceinline__ void bnd_row(const Params& P, const BndCells& c, int j, int k,
                                        const uint32_t* __restrict__ cell_start, const uint32_t* __restrict__ cell_end,
                                        uint32_t& lo, uint32_t& hi) {
    const uint32_t row = (uint32_t)j * (uint32_t)P.g.nx + (uint32_t)k * (uint32_t)P.g.nx * (uint32_t)P.g.ny;
    if (P.dense_cells) {
        lo = cell_start[row + c.lo[0]];
        hi = cell_end[row + c.hi[0] - 1];
    } else {
        row_range(cell_start, cell_end, row, c.lo[0], c.hi[0] - 1, lo, hi);
    }
}

// d = x_j - x_b and its weight in the sum; false if the pair has none.
__device__ __forceinline__ bool bnd_pair(const Params& P, float4 xb, float4 xj, const float& pj, float4& t) {
    const float ir0 = 1.f / (P.rho0 * P.rho0);
    const float dx = xj.x - xb.x, dy = xj.y - xb.y, dz = xj.z - xb.z;
    const float r2 = dist2(dx, dy, dz);
    if (!(r2 > 0.f) || r2 * P.inv_h2 >= 1.f) return false;
    const float rinv = rsqrtf(r2);
    const float om = __fmaf_rn(-(r2 * rinv), P.inv_h, 1.f);      // rounded alike in both forms
    t = make_float4(dx, dy, dz, pj * ir0 * om * om * rinv);
    return true;
}

__device__ float3 bnd_reaction_at(const Params& P, float4 xb, const float4* __restrict__ fluid_pos,
                                  const float2* __restrict__ fluid_rp, const uint32_t* __restrict__ cell_start,
                                  const uint32_t* __restrict__ cell_end) {
    const BndCells c = bnd_cells(P, xb);
    float3 s = make_float3(0.f, 0.f, 0.f);
    for (int k = c.lo[2]; k < c.hi[2]; ++k)
        for (int j = c.lo[1]; j < c.hi[1]; ++j) {
            uint32_t lo, hi;
            bnd_row(P, c, j, k, cell_start, cell_end, lo, hi);
            for (uint32_t q = lo; q < hi; ++q) {
                float4 t;
                if (!bnd_pair(P, xb, fluid_pos[q], fluid_rp[q].y, t)) continue;
                s.x = __fmaf_rn(t.w, t.x, s.x); s.y = __fmaf_rn(t.w, t.y, s.y); s.z = __fmaf_rn(t.w, t.z, s.z);
            }
        }
    const float k = -P.mass * P.k_grad * xb.w;
    return make_float3(k * s.x, k * s.y, k * s.z);
}

// The same by a whole warp (every lane calls it, every lane gets the sum);
// queue: kBndQueue entries of the warp's own.
constexpr int kBndQueue = 9 * 32;
__device__ float3 bnd_reaction_warp(const Params& P, float4 xb, const float4* __restrict__ fluid_pos,
                                    const float2* __restrict__ fluid_rp, const uint32_t* __restrict__ cell_start,
                                    const uint32_t* __restrict__ cell_end, float4* queue) {
    const int lane = threadIdx.x & 31;
    const BndCells c = bnd_cells(P, xb);
    // lane r < 9 finds row r's slots; a row outside the grid has none
    uint32_t lo = 0u, hi = 0u;
    {
        const int j = c.lo[1] + lane % 3, k = c.lo[2] + lane / 3;
        if (lane < 9 && j < c.hi[1] && k < c.hi[2]) bnd_row(P, c, j, k, cell_start, cell_end, lo, hi);
    }
    float4 x[9];
    float p[9];
#pragma unroll
    for (int r = 0; r < 9; ++r) {
        const uint32_t q = __shfl_sync(0xffffffffu, lo, r) + lane;
        const bool in = q < __shfl_sync(0xffffffffu, hi, r);
        x[r] = in ? fluid_pos[q] : make_float4(0.f, 0.f, 0.f, 0.f);
        p[r] = in ? fluid_rp[q].y : 0.f;
    }
    float s = 0.f;          // lanes 0, 1, 2: the sum's x, y, z
    int queued = 0;
    auto add_queue = [&] {
        __syncwarp();
        if (lane < 3) {
            const float* e = reinterpret_cast<const float*>(queue);
#pragma unroll 4
            for (int i = 0; i < queued; ++i) s = __fmaf_rn(e[4 * i + 3], e[4 * i + lane], s);
        }
        __syncwarp();
        queued = 0;
    };
#pragma unroll
    for (int r = 0; r < 9; ++r) {
        const uint32_t q0 = __shfl_sync(0xffffffffu, lo, r), q1 = __shfl_sync(0xffffffffu, hi, r);
        float4 xj = x[r];
        float pj = p[r];
        for (uint32_t q = q0 + lane; q - lane < q1; q += 32u) {
            if (q - lane != q0 && q < q1) {         // past the row's first 32: loaded here
                xj = fluid_pos[q];
                pj = fluid_rp[q].y;
            }
            float4 t;
            const bool take = q < q1 && bnd_pair(P, xb, xj, pj, t);
            const unsigned taken = __ballot_sync(0xffffffffu, take);
            if (take) queue[queued + __popc(taken & ((1u << lane) - 1u))] = t;
            queued += __popc(taken);
            if (queued > kBndQueue - 32) add_queue();
        }
    }
    add_queue();
    const float k = -P.mass * P.k_grad * xb.w;
    return make_float3(k * __shfl_sync(0xffffffffu, s, 0), k * __shfl_sync(0xffffffffu, s, 1),
                       k * __shfl_sync(0xffffffffu, s, 2));
}

// f(b, x_b, F) for the block's boundary slots b < nb, F the reaction on b.
template <bool WARP, class Fn>
__device__ __forceinline__ void for_each_reaction(const Params& P, int nb, const float4* __restrict__ fluid_pos,
                                                  const float2* __restrict__ fluid_rp,
                                                  const uint32_t* __restrict__ cell_start,
                                                  const uint32_t* __restrict__ cell_end, Fn&& f) {
    const int i = blockIdx.x * kBlock + threadIdx.x;
    if constexpr (WARP) {
        __shared__ float4 s_queue[kBlock / 32][kBndQueue];
        const int b = i >> 5;
        if (b >= nb) return;
        const float4 xb = P.bnd[b];
        const float3 F = bnd_reaction_warp(P, xb, fluid_pos, fluid_rp, cell_start, cell_end,
                                           s_queue[threadIdx.x >> 5]);
        if ((threadIdx.x & 31) == 0) f(b, xb, F);
    } else {
        if (i >= nb) return;
        const float4 xb = P.bnd[i];
        f(i, xb, bnd_reaction_at(P, xb, fluid_pos, fluid_rp, cell_start, cell_end));
    }
}

// Boundary slots' reaction at the fluid's state.
template <bool WARP>
__global__ void __launch_bounds__(kBlock) k_bnd_reaction(Params P, int nb, const float4* __restrict__ fluid_pos,
                                                         const float2* __restrict__ fluid_rp,
                                                         const uint32_t* __restrict__ cell_start,
                                                         const uint32_t* __restrict__ cell_end,
                                                         float4* __restrict__ force) {
    for_each_reaction<WARP>(P, nb, fluid_pos, fluid_rp, cell_start, cell_end, [&](int b, float4, float3 F) {
        force[b] = make_float4(F.x, F.y, F.z, 0.f);
    });
}

// Moving boundary: the reaction at the committed pressures of the current
// correction (the fluid at the step's start positions, as the config
// pressure force) and the boundary's prediction with it. The velocity and
// position updates are the DEM step's (v += (f + F) / m dt, x += v dt), so
// the spheres' next positions are the last prediction's wherever no wall
// projects them.
template <bool WARP>
__global__ void __launch_bounds__(kBlock) k_bnd_move(Params P, int nb, const float4* __restrict__ fluid_pos,
                                                     const float2* __restrict__ fluid_rp,
                                                     const uint32_t* __restrict__ cell_start,
                                                     const uint32_t* __restrict__ cell_end,
                                                     const float4* __restrict__ vel, const float4* __restrict__ fext,
                                                     float inv_mass, float4* __restrict__ pred,
                                                     float4* __restrict__ force) {
    after_previous();
    for_each_reaction<WARP>(P, nb, fluid_pos, fluid_rp, cell_start, cell_end, [&](int b, float4 xb, float3 F) {
        const float4 v0 = vel[b], f = fext[b];
        const float vx = v0.x + (f.x + F.x) * inv_mass * P.dt;
        const float vy = v0.y + (f.y + F.y) * inv_mass * P.dt;
        const float vz = v0.z + (f.z + F.z) * inv_mass * P.dt;
        pred[b] = make_float4(xb.x + vx * P.dt, xb.y + vy * P.dt, xb.z + vz * P.dt, xb.w);
        force[b] = make_float4(F.x, F.y, F.z, 0.f);
    });
}

// Threads for nb boundary particles' reactions.
inline int reaction_threads(int nb) { return nb <= kBndWarps ? nb * 32 : nb; }

__global__ void k_gather4(int nb, const int* __restrict__ ids, const float4* __restrict__ src,
                          float4* __restrict__ dst) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nb) dst[t] = src[ids[t]];
}

}  // namespace

void launch_bnd_move(cudaStream_t st, const Params& P, int nb, const float4* fluid_pos, const float2* fluid_rp,
                     const uint32_t* cell_start, const uint32_t* cell_end, const float4* vel, const float4* fext,
                     float inv_mass, float4* pred, float4* force) {
    if (nb <= 0) return;
    auto kernel = nb <= kBndWarps ? k_bnd_move<true> : k_bnd_move<false>;
    launch_chained(kernel, blocks_for(reaction_threads(nb)), kBlock, 0, st, P, nb, fluid_pos, fluid_rp, cell_start,
                   cell_end, vel, fext, inv_mass, pred, force);
}

void launch_bnd_gather4(cudaStream_t st, int nb, const int* ids, const float4* src, float4* dst) {
    if (nb > 0) k_gather4<<<blocks_for(nb), kBlock, 0, st>>>(nb, ids, src, dst);
}

void launch_bnd_reaction(cudaStream_t st, const Params& P, int nb, const float4* fluid_pos, const float2* fluid_rp,
                         const uint32_t* cell_start, const uint32_t* cell_end, float4* force) {
    if (nb <= 0) return;
    auto kernel = nb <= kBndWarps ? k_bnd_reaction<true> : k_bnd_reaction<false>;
    kernel<<<blocks_for(reaction_threads(nb)), kBlock, 0, st>>>(P, nb, fluid_pos, fluid_rp, cell_start, cell_end, force);
}

int launch_bnd_prepare(cudaStream_t st, const Params& P, int nb, const float4* raw, int* iota, uint32_t* keys[2],
                       uint32_t* vals[2], uint32_t* hist, int hist_blocks, int key_bits, float4* sorted, int* ids,
                       float* w, uint32_t* cell_start, uint32_t* cell_end, int* clamped) {
    if (nb <= 0) return 0;
    Params Q = P;
    Q.n = nb;
    Q.scenes = nullptr;
    k_iota<<<blocks_for(nb), kBlock, 0, st>>>(nb, iota);
    launch_cell_keys(st, Q, raw, iota, keys[0], vals[0], clamped);
    const int res = radix_sort(st, nb, key_bits, keys, vals, hist, hist_blocks);
    k_bnd_gather<<<blocks_for(nb), kBlock, 0, st>>>(nb, keys[res], vals[res], raw, sorted, ids, cell_start, cell_end);
    k_bnd_psi<<<blocks_for(nb), kBlock, 0, st>>>(Q, nb, keys[res], sorted, cell_start, cell_end, w);
    k_bnd_set_w<<<blocks_for(nb), kBlock, 0, st>>>(nb, w, sorted);
    return res;
}

void launch_build_bnd_nbr(cudaStream_t st, const Params& P, const float4* pos, const uint32_t* keys,
                          const uint32_t* bnd_start, const uint32_t* bnd_end, int* counts, int* list, int* flags) {
    if (P.n > 0)
        launch_chained(k_build_bnd_nbr, blocks_for(P.n), kBlock, 0, st, P, pos, keys, bnd_start, bnd_end, counts,
                       list, flags);
}

}  // namespace psb
