// psb_internal.cuh -- shared device-side types of libpsb (not part of the ABI).
//
// Data layout in HBM (all arrays in cell-sorted slot order after each step's
// sort; slot s holds particle ids[s]):
//   pos   float4  x, y, z, 0           16 B
//   vel   float4  interpolated v       16 B   (the reference's m_dVel[1])
//   vap   float4  leap-frog v+         16 B   (m_dVelInterAp)
//   rp    float2  (density, pressure)   8 B   (pressure persists across steps)
//   ids   int32   particle id           4 B
// Per-step scratch: sort keys/values (2 x 2 x 4 B), the cells' slot ranges
// (counting sort: every cell's, from the scan of the counts; radix sort: only
// occupied cells are written, and reset before the next build),
// neighbour lists (slot-major quads, see nbr_index; c < count[s]), and the
// PCISPH predictor buffers xs[2] and vs (Soa3), rpc (float2),
// fnp (float4 non-pressure force density), rho_x (float).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>
#include <utility>
#include "psb.h"

namespace psb {

constexpr uint32_t kEmpty = 0xFFFFFFFFu;
constexpr int kBlock = 256;

struct Grid {
    float gx, gy, gz;   // corner (float, as UniformGrid.Min)
    float cell;         // edge (float, as UniformGrid.sizeCell)
    int nx, ny, nz;
};

// One scene of a batch: its box and its own grid. Every other constant is
// shared by the batch's scenes and lives in Params.
struct SceneGeom {
    float bx0, by0, bz0, bx1, by1, bz1;              // faces (ghost walls, wall distance)
    float wlo_x, wlo_y, wlo_z, whi_x, whi_y, whi_z;  // projection bounds (faces -/+ particle radius)
    Grid g;                                          // the scene's grid; its cells are keys cell_base + i + j nx + k nx ny
    uint32_t cell_base;
    int first, count;                                // its particles: sorted slots [first, first + count)
};

// Launch configuration of the tunable kernels, the autotuner's choice for a
// size bucket: block sizes (128, 256 or 512; 0 = 256) and the neighbour
// build's schedule (0: each thread its own 27 cells, by sign masks; 1: the
// lanes of a warp that share a grid row walk it together, staging candidates in
// shared memory; 2: each thread's walk with the density pass at x folded in,
// single config-profile PCISPH scenes, elsewhere as 0). Every choice computes
// the same result bit for bit.
struct Tune {
    int nbr_block, nbr_schedule, density_block, init_block, pci_density_block, force_block, xsph_block;
};

// Uniform per-scene constants, FP32 in normalised form (q = r^2/h^2, u = r/h)
// so that no intermediate leaves FP32 range; derived on the host in FP64.
struct Collider;     // colliders.cuh

// A vector field split for gathers: a neighbour's vector is an 8-byte and a
// 4-byte load. The sweeps' gathers are bound by L1 wavefronts -- a warp's 32
// neighbours lie in ~10 lines of a float4 array, ~5 of the 8-byte one, ~3 of
// the 4-byte one -- so the split costs fewer of them than one 16-byte load
// (density pass at 1M particles alone: 55 against 66 us).
struct Soa3 {
    float2* xy;
    float* z;
};

struct Params {
    int n;
    int cap;            // neighbour slots per particle
    Grid g;
    double h;           // list cut-off of the exact neighbour test sqrt(d.d) <= h in FP64
                        // (reference: h; config: (1 + skin) h)
    double h2_exact;    // the largest double x with sqrt_rn(x) <= h: the same test as d.d <= h2_exact
    float h2_lo, h2_hi; // FP32 d^2 outside [h2_lo, h2_hi] is decided without the FP64 test
    float h2, inv_h, inv_h2;
    float k_rho;        // 315 m / (64 pi h^3):           rho = k_rho * sum (1-q)^3
    float k_grad;       // 45 m / (pi h^4):               a_p = k_grad * sum (pV_i+pV_j)(1-u)^2 x^
    float k_visc;       // mu m 45 / (pi h^5):            f_v = k_visc * sum (v_j-v_i)(1-u)/rho_j
    float k_surf;       // 945 m / (32 pi h^5):           normals and surface term (reference profile)
    float sigma, l;
    float k_press;      // 1 / (beta G^2), beta = 2 (m dt/rho0)^2, G = 45/(pi h^4)
    float k_delta;      // config PCISPH: prototype delta = 1/(beta (|sum gradW|^2 + sum |gradW|^2)) of a filled lattice
    float rho0;
    double rho0_d;
    float eos_k;        // REF: k (p = k (rho - rho0));  CONFIG: k rho0 / 7 (Tait, gamma 7)
    float dt;
    float gx, gy, gz;   // gravity acceleration
    float wlo_x, wlo_y, wlo_z, whi_x, whi_y, whi_z;   // box min + r, box max - r (float, as collisionBox)
    float wall_k, wall_c;
    float xsph_k;       // config PCISPH XSPH: xsph * k_rho / rho0 (0: off)
    // DEM: contact law constants (REF: k_s, c, s, a; CONFIG: k_n, c_n), the
    // distance R in k (R - d) (REF: h_A + h_B as float; CONFIG: 2r), the
    // contact range (REF: 2R; CONFIG: 2r), sphere mass and its inverse
    float dem_k, dem_c, dem_s, dem_a, dem_R, dem_range, dem_mass, dem_inv_mass;
    int dem;
    // Config-profile walls (mirror ghost particles across the box faces):
    float bx0, by0, bz0, bx1, by1, bz1;   // faces
    float hf;           // h
    int ref;            // reference profile
    int pci;            // PCISPH (else WCSPH)
    int surface;        // surface tension on
    // Batched scenes (kernels instantiated with BATCH = true read these; the
    // box and grid fields above then go unused):
    const SceneGeom* scenes;          // per scene
    const uint16_t* slot_scene;       // scene of each sorted slot (scenes occupy contiguous slot ranges)
    const uint8_t* active;            // corrector: scenes still iterating
    unsigned long long* err_scene;    // corrector: per-scene max compression error of the pass (ordered)
    int nscenes;
    Tune tune;
    // Static boundary particles (config profile; Akinci et al. 2012): sorted
    // by cell, position in .xyz and psi_b / m in .w; per fluid slot its
    // boundary neighbours within the list cut-off, stored in quads like the
    // fluid list (bnd_cap slots). bnd_count == nullptr: no boundary.
    const float4* bnd;
    const int* bnd_count;
    const int* bnd_list;
    int bnd_cap;
    float bnd_lo[3], bnd_hi[3];     // their bounding box grown by the list cut-off
    // Boundary particles that move with the corrector (two-way coupling
    // solved inside the step): their predicted positions (psi_b / m in .w),
    // which the corrector's density passes read in place of bnd; nullptr:
    // the boundary is static.
    const float4* bnd_pred;
    // DEM: an external force per sphere in particle-id order (N; nullptr:
    // none), found through the id of each sorted slot
    const float4* ext_force;
    const int* slot_ids;
    float mass;         // particle mass (FP32)
    // Collision objects applied after the integrator and the box, in order
    // (colliders.cuh); n_coll == 0: none. Single-scene contexts only.
    const Collider* coll;
    int n_coll;
    // Particles near the box faces (config-profile SPH; sph.cu): their slots
    // in any order, how many, and a flag bit per slot, all written by the
    // step's reorder. wall_list == nullptr: none. wall_blocks: the blocks of
    // a launch that take the list (set per launch).
    int* wall_list;
    int* wall_count;
    uint32_t* wall_bits;
    int wall_blocks;
    // SPH: the step's start positions and velocities in sorted order, as its
    // sweeps gather them, written by the reorder; and the two z components
    // once more beside the scalar that the pressure and set-up sums want with
    // them: (z, pressure) and (v_z, 1 / density) -- the division once a particle,
    // not once a pair. The density passes write those.
    Soa3 x0, v0;
    float *cx, *cy;     // x0's x and y once more, each alone, for the neighbour build (DEM: with x0.z, all it has of x0)
    float2* zp;
    float2* vr;
    int dense_cells;    // the cell ranges cover every cell (the counting sort's), empty ones included
};

// Distance to a face, in h, up to which the reorder lists a particle: past
// the h within which a face has ghosts, so that the corrector's predictions
// (a CFL step moves a particle well under 0.1 h) rarely bring an unlisted
// particle into range. The list is used from kWallListMin particles on, where
// a pass is no longer one chain of loads. A step (PCISPH with four
// corrections, eager) with the list against without, blocks that fill their
// box's floor: 306 / 276 us at 64,000 particles, 349 / 323 at 107,520, 365 /
// 341 at 131,072, 411 / 386 at 184,320, 438 / 442 at 230,400, 462 / 506 at
// 291,840, 671 / 760 at 522,240, 1,206 / 1,316 at 1,044,480: it pays from ~220,000
// on. Scenes that are mostly wall lose by it further up, since the
// list's blocks are sized for a quarter of the particles (four layers of
// 65,536 between two faces: 873 / 512).
constexpr float kWallReach = 1.1f;
constexpr int kWallListMin = 131072;

// Programmatic dependent launch. A kernel launched with launch_chained may be
// placed while the stream's previous kernel still runs, once all of that one's
// blocks have passed their own wait: its launch and block start-up overlap the
// previous kernel's tail instead of following it. Such a kernel begins with
// after_previous(), in every thread and before any access to memory that a
// chained kernel ever writes: it waits until the previous kernel has ended and
// its writes are visible -- so kernels still run one after another, and a
// kernel's end implies the end of all before it -- and then lets the next one
// be placed. (Letting it be placed before the wait put several kernels' blocks
// on the chip at once: a 16k particle WCSPH frame 843 us, 752 this way, 840
// without.) Launched the usual way the wait returns at once. Only an order
// between two kernels is loosened: behind a memset, a copy, a waited event or a
// loop node of a graph a chained kernel starts as any other.
__device__ __forceinline__ void after_previous() {
    cudaGridDependencySynchronize();
    cudaTriggerProgrammaticLaunchCompletion();
}

// Threads up to which a launch is chained: a launch's start-up is worth ~2 us,
// a part of the frame of 4k-290k particles (16 DEM steps 784 -> 600 us, four
// PCISPH steps of 97k 1670 -> 1580, 50 corrections of 262k 5680 -> 5370). In a
// step's graph, as large scenes run, the blocks placed early cost as much from
// ~350,000 particles on, chained against not: 503 / 504 us a step at 327,680,
// 574 / 569 at 405,504, 692 / 690 at 524,160, 804 / 798 at 633,600, 1,031 / 1,019
// at 860,160. Steps launched one by one still gain there (551 / 581, 670 / 702,
// 781 / 818, 1,008 / 1,038); the line is where graphs still lose next to nothing.
constexpr long long kChainThreads = 1 << 19;

template <class... Params_, class... Args>
inline void launch_chained(void (*kernel)(Params_...), unsigned grid, unsigned block, size_t smem, cudaStream_t st,
                           Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = (long long)grid * block <= kChainThreads;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);      // an error stays for cudaGetLastError
}

// Runs f(std::integral_constant<int, B>) with B the tuned block size.
template <class F>
inline void with_block(int bs, F&& f) {
    if (bs == 128) f(std::integral_constant<int, 128>{});
    else if (bs == 512) f(std::integral_constant<int, 512>{});
    else f(std::integral_constant<int, 256>{});
}

// Neighbour lists are stored in quads: entries 4q .. 4q+3 of sorted slot s
// are the int4 at index q * n + s, so one 16-byte load gives a thread four
// neighbours and a warp's 32 slots read 512 contiguous bytes per quad.
__host__ __device__ inline size_t nbr_index(int c, int n, int t) { return ((size_t)(c >> 2) * n + t) * 4 + (c & 3); }
inline size_t nbr_list_ints(size_t n, int cap) { return n * (size_t)((cap + 3) & ~3); }

// f(j) for the first cnt entries of slot t's list, in order. The next quad's
// load is issued behind the current quad's gathers, so a quad costs one
// latency, not two (density pass at 1M particles alone: 61 against 66 us).
// FRESH: the kernel that calls it writes the lists, each thread its own, so
// they are not loaded through the read-only path.
template <bool FRESH = false, class F>
__device__ __forceinline__ void for_each_nbr(const int* list, int n, int t, int cnt, F&& f) {
    const int4* L = reinterpret_cast<const int4*>(list) + t;
    auto load = [&] { return FRESH ? *L : __ldg(L); };
    int4 q = make_int4(0, 0, 0, 0);
    if (cnt > 0) q = load();
    int c = 0;
    for (; c + 4 <= cnt; c += 4) {
        int4 next = q;
        L += n;
        if (c + 4 < cnt) next = load();
        f(q.x); f(q.y); f(q.z); f(q.w);
        q = next;
    }
    if (c < cnt) {
        f(q.x);
        if (c + 1 < cnt) f(q.y);
        if (c + 2 < cnt) f(q.z);
    }
}

// |d|^2 of a pair in FP32 with the multiply-adds written out, so that every
// kernel that tests or weights the same pair rounds it the same way.
__device__ __forceinline__ float dist2(float dx, float dy, float dz) {
    return __fmaf_rn(dz, dz, __fmaf_rn(dy, dy, __fmul_rn(dx, dx)));
}

// The reference's test, sqrt((dx*dx + dy*dy) + dz*dz) <= h with every
// operation rounded separately in FP64 (double3.h:15-47). The correctly
// rounded square root is monotone, so the test is d2 <= h2_exact, the
// largest double whose root rounds to at most h (found on the host).
__device__ __forceinline__ bool exact_neighbor(float4 a, float4 b, double h2_exact) {
    const double dx = __dsub_rn((double)a.x, (double)b.x);
    const double dy = __dsub_rn((double)a.y, (double)b.y);
    const double dz = __dsub_rn((double)a.z, (double)b.z);
    const double d2 = __dadd_rn(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)), __dmul_rn(dz, dz));
    return d2 <= h2_exact;
}

// flags[1]: max count, flags[2..3]: total pairs (64-bit); every lane of the
// warp calls it.
__device__ __forceinline__ void nbr_flags(int cnt, int* __restrict__ flags) {
    int m = cnt;
    unsigned long long tot = (unsigned long long)cnt;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        tot += __shfl_xor_sync(0xffffffffu, tot, o);
    }
    if ((threadIdx.x & 31) == 0 && tot > 0) {
        atomicMax(&flags[1], m);
        atomicAdd((unsigned long long*)&flags[2], tot);
    }
}

// Slots of cells a0..a1 of a row where empty cells hold kEmpty (the radix
// sort's ranges): lo = hi = 0 when all are empty.
__device__ __forceinline__ void row_range(const uint32_t* __restrict__ cell_start,
                                          const uint32_t* __restrict__ cell_end, uint32_t row, int a0, int a1,
                                          uint32_t& lo, uint32_t& hi) {
    lo = kEmpty;
    hi = 0u;
    for (int a = a0; a <= a1; ++a) {
        const uint32_t s = cell_start[row + a];
        if (s == kEmpty) continue;
        if (lo == kEmpty) lo = s;
        hi = cell_end[row + a];
    }
    if (lo == kEmpty) lo = 0u;
}

// The 27-cell walk of sorted particle t of a single scene (one thread per
// particle; the build with the density folded in): the three cells of a grid
// row are adjacent in sorted order, so each of the nine rows is one contiguous
// slot range, and accept(slot, position) runs for every candidate within the
// list cut-off in increasing slot order, row by row -- the list order.
// Candidates beyond the FP32 window are out with one compare, those below it
// in; inside it the reference's FP64 test decides.
template <class F>
__device__ __forceinline__ void walk_neighbours(const Params& P, int t, float4 pi, const float4* __restrict__ pos,
                                                const uint32_t* __restrict__ keys,
                                                const uint32_t* __restrict__ cell_start,
                                                const uint32_t* __restrict__ cell_end, F&& accept) {
    const int nx = P.g.nx, ny = P.g.ny, nz = P.g.nz;
    const uint32_t key = keys[t];
    const int ci = (int)(key % (uint32_t)nx);
    const int cj = (int)((key / (uint32_t)nx) % (uint32_t)ny);
    const int ck = (int)(key / ((uint32_t)nx * (uint32_t)ny));
    // Skipping the cells whose faces lie beyond the cut-off (a bound from the
    // particle's distance to its own cell's faces) was measured: the lanes of
    // a warp prune different cells, so the warp still walks their union, and
    // the per-row bounds cost more than the skipped candidates save.
    const int a0 = max(ci - 1, 0), a1 = min(ci + 1, nx - 1);
    for (int k = max(ck - 1, 0); k <= min(ck + 1, nz - 1); ++k) {
        for (int j = max(cj - 1, 0); j <= min(cj + 1, ny - 1); ++j) {
            const uint32_t row = (uint32_t)j * (uint32_t)nx + (uint32_t)k * (uint32_t)nx * (uint32_t)ny;
            uint32_t lo = kEmpty, hi = 0;
            for (int a = a0; a <= a1; ++a) {
                const uint32_t s = cell_start[row + a];
                if (s != kEmpty) {
                    if (lo == kEmpty) lo = s;
                    hi = cell_end[row + a];
                }
            }
            if (lo == kEmpty) continue;
            for (uint32_t q = lo; q < hi; ++q) {
                const float4 pj = pos[q];
                const float d2 = dist2(pi.x - pj.x, pi.y - pj.y, pi.z - pj.z);
                if (d2 <= P.h2_hi && (d2 < P.h2_lo || exact_neighbor(pi, pj, P.h2_exact))) accept(q, pj);
            }
        }
    }
}

// ---- launchers (grid.cu) -------------------------------------------------
void launch_reset_cells(cudaStream_t st, int n, const uint32_t* sorted_keys, uint32_t* cell_start);
void launch_cell_keys(cudaStream_t st, const Params& P, const float4* pos, const int* ids, uint32_t* keys_by_id,
                      uint32_t* slot_by_id, int* clamped);
// Sorts (keys, vals) by key, stably; returns the buffer index (0 or 1) holding the result.
// hist holds 256 * radix_blocks(n) + 256 words.
int radix_sort(cudaStream_t st, int n, int bits, uint32_t* keys[2], uint32_t* vals[2], uint32_t* hist, int nblocks_cap);
int radix_blocks(int n);
// The same for n that one block holds (false: too many, nothing launched);
// the outputs may be the inputs.
bool small_sort(cudaStream_t st, int n, int bits, const uint32_t* keys_in, const uint32_t* vals_in, uint32_t* keys_out,
                uint32_t* vals_out);
// Counting sort of the particles by (cell, id) over a grid of ncells cells:
// launch_cell_count writes each slot's key and arrival rank and raises the
// counts; launch_cell_sort turns the counts into cell_start (every cell; slots
// [cell_start[c], cell_start[c + 1])), writes the sorted keys and the old slot
// of each sorted one, and leaves counts and tile sums at zero, as both must
// be before the first count; it clears the eight words at flags, keeping the
// count of clamped particles that the count pass left at flags[6] in flags[4].
// cell_count and cell_start hold cell_sort_cells(ncells) words, tile_sum
// cell_sort_tiles(ncells); placed: n.
size_t cell_sort_tiles(size_t ncells);
size_t cell_sort_cells(size_t ncells);
void launch_cell_count(cudaStream_t st, const Params& P, const float4* pos, uint32_t* keys, uint32_t* ranks,
                       uint32_t* cell_count, uint32_t* tile_sum, int* clamped);
void launch_cell_sort(cudaStream_t st, int n, size_t ncells, const int* ids, const uint32_t* keys, const uint32_t* ranks,
                      uint32_t* cell_count, uint32_t* tile_sum, uint32_t* cell_start, int* flags, uint2* placed,
                      uint32_t* keys_out, uint32_t* vals_out);
// The same up to the arrival order in placed, and then the places and the
// whole state into sorted order (scenes without a wall list).
void launch_cell_place(cudaStream_t st, int n, size_t ncells, const int* ids, const uint32_t* keys,
                       const uint32_t* ranks, uint32_t* cell_count, uint32_t* tile_sum, uint32_t* cell_start,
                       int* flags, uint2* placed);
void launch_rank_reorder(cudaStream_t st, const Params& P, const uint32_t* keys, const uint2* placed,
                         const uint32_t* cell_start, const float4* pos, const float4* vel, const float4* vap,
                         const float2* rp, const int* ids, uint32_t* keys_out, uint32_t* vals_out, float4* pos2,
                         float4* vel2, float4* vap2, float2* rp2, int* ids2);
// The whole state into sorted order, with the cell ranges; or in two
// launches: positions, ids and cell ranges (what the neighbour build reads),
// then the rest. cell_start null: the ranges are there already.
// Both also list the particles near the box faces (P.wall_list).
void launch_reorder(cudaStream_t st, const Params& P, const uint32_t* keys, const uint32_t* vals, const float4* pos,
                    const float4* vel, const float4* vap, const float2* rp, const int* ids, float4* pos2, float4* vel2,
                    float4* vap2, float2* rp2, int* ids2, uint32_t* cell_start, uint32_t* cell_end);
void launch_reorder_pos(cudaStream_t st, const Params& P, const uint32_t* keys, const uint32_t* vals, const float4* pos,
                        const int* ids, float4* pos2, int* ids2, uint32_t* cell_start, uint32_t* cell_end);
void launch_reorder_state(cudaStream_t st, const Params& P, const uint32_t* vals, const float4* vel, const float4* vap,
                          const float2* rp, float4* vel2, float4* vap2, float2* rp2);
void launch_build_nbr(cudaStream_t st, const Params& P, const float4* pos, const uint32_t* keys,
                      const uint32_t* cell_start, const uint32_t* cell_end, int* counts, int* list, int* flags);
// (sph.cu) The per-thread neighbour build of one config-profile scene with the
// density pass at x folded in: lists, counts and flags as launch_build_nbr,
// then density, pressure and features as launch_density_x.
void launch_build_density(cudaStream_t st, const Params& P, const float4* pos, const uint32_t* keys,
                          const uint32_t* cell_start, const uint32_t* cell_end, int* counts, int* list, int* flags,
                          float2* rp, float* rho_x, int zero_p, float p_scale, float* feats, int nfeat);

// ---- launchers (sph.cu) ---------------------------------------------------
// feats != nullptr: also the warm start's inputs f0 .. f(nfeat - 1), nfeat 6 or 7.
void launch_density_x(cudaStream_t st, const Params& P, const int* counts, const int* list, float2* rp, float* rho_x, int zero_p, float p_scale = 1.f,
                      float* feats = nullptr, int nfeat = 7);
void launch_wcsph_force(cudaStream_t st, const Params& P, const float4* vap, const float2* rp, const int* counts, const int* list, float4* pos_out, float4* vel_out,
                        float4* vap_out, float4* fnp);
void launch_pci_init(cudaStream_t st, const Params& P, const float4* vap, const float2* rp, const int* counts,
                     const int* list, int warm, float4* fnp, Soa3 xs, Soa3 vs);
void launch_pci_density(cudaStream_t st, const Params& P, Soa3 xs, const float2* rp, const int* counts,
                        const int* list, float2* rpc, unsigned long long* err_slot);
void launch_pci_force_predict(cudaStream_t st, const Params& P, const float4* vap, const float4* fnp, Soa3 xs,
                              const float2* rpc, const int* counts, const int* list, Soa3 xs_next, Soa3 vs, float2* rp);
void launch_pci_commit(cudaStream_t st, const Params& P, Soa3 xs, Soa3 vs, const float2* rpc,
                       int have_density_pass, float4* pos, float4* vel, float4* vap, float2* rp);
void launch_xsph(cudaStream_t st, const Params& P, Soa3 xs, Soa3 vs, const int* counts, const int* list, Soa3 vs_out);
void launch_dem_step(cudaStream_t st, const Params& P, const float4* pos, const float4* vel, const int* counts,
                     const int* list, float4* pos_out, float4* vel_out, float4* vap_out, float4* force);
// The force on each sphere (slot order) that the next step would apply
// without its external force: gravity and the contacts; nothing moves.
void launch_dem_forces(cudaStream_t st, const Params& P, const float4* pos, const float4* vel, const int* counts,
                       const int* list, float4* force);

// ---- batched scenes: the corrector loop on the device (batch.cu) ---------------
// loop: [0] pass index, [1] continue, [2, 2 + S) corrections, [2 + S, 2 + 2S) converged,
// [2 + 2S, 2 + 3S) corrections summed over steps, [2 + 3S, 2 + 4S) unconverged steps;
// host_word (if not null): set to 1 (stop) or 2 (another pass) by the decision
void launch_batch_begin(cudaStream_t st, int S, int max_it, uint8_t* active, unsigned long long* err_scene,
                        unsigned long long* err_hist, int hist_len, int* loop);
void launch_batch_decide(cudaStream_t st, int S, int min_it, int max_it, double eta, uint8_t* active,
                         unsigned long long* err_scene, unsigned long long* err_hist, int* loop,
                         cudaGraphConditionalHandle handle, int set_handle, int* host_word);
// The whole corrector loop of a config-profile scene or batch as one
// cooperative launch (begin, then {density pass, decision, pressure-force
// pass} until the decision ends it). Returns the launch's error.
cudaError_t launch_corrector_persistent(cudaStream_t st, const Params& P, const float4* vap, const float4* fnp, Soa3 xs,
                                        float2* rp, float2* rpc, const int* counts, const int* list, Soa3 vs, int S, int min_it, int max_it, double eta,
                                        uint8_t* active, unsigned long long* err_scene, unsigned long long* err_hist,
                                        int* loop);

// ---- boundary particles (boundary.cu) ------------------------------------------
// Sorts nb boundary particles by cell (stable on index), fills their cell
// ranges and writes psi_b / m to .w of sorted[]: rho0 / (k_rho sum_k (1 -
// q_bk)^3) over the boundary particles within h, self included. Returns the
// buffer (0 or 1) of keys[] that holds the sorted keys.
int launch_bnd_prepare(cudaStream_t st, const Params& P, int nb, const float4* raw, int* iota, uint32_t* keys[2],
                       uint32_t* vals[2], uint32_t* hist, int hist_blocks, int key_bits, float4* sorted, int* ids,
                       float* w, uint32_t* cell_start, uint32_t* cell_end, int* clamped);
// The force the fluid exerts on each sorted boundary particle: minus the sum
// of the mirrored-pressure forces the particle exerts on the fluid within h,
// from the fluid's positions and committed pressures (sorted slots, cell
// ranges of the last build). Written as float4 per boundary slot.
// Collision objects on the integrator's output (WCSPH and DEM; the PCISPH
// commit applies them itself). x_old: the step's start positions. vh_old
// (WCSPH): the start half-step velocities, for v = (vh_old + vap)/2; null
// (DEM): vel and vap both take the new velocity.
void launch_apply_colliders(cudaStream_t st, const Params& P, const float4* x_old, const float4* vh_old, float4* pos,
                            float4* vel, float4* vap);
// Emission (emit.cu): k particles at slots and ids n0 .. n0 + k - 1, velocity
// v, half-step velocity v (dem) or 0, density and pressure 0.
void launch_emit_list(cudaStream_t st, int n0, int k, const float* xyz, const float* v, int dem, float4* pos,
                      float4* vel, float4* vap, int* ids, float2* rp);
void launch_emit_random(cudaStream_t st, int n0, int k, int type, int count, unsigned emission,
                        unsigned long long seed, const float* params, const float* faces, const float* v, int dem,
                        float4* pos, float4* vel, float4* vap, int* ids, float2* rp);
void launch_append_ids(cudaStream_t st, int n0, int k, int* ids, float2* rp);
void launch_bnd_reaction(cudaStream_t st, const Params& P, int nb, const float4* fluid_pos, const float2* fluid_rp,
                         const uint32_t* cell_start, const uint32_t* cell_end, float4* force);
// Moving boundary (sorted slots): the reaction F_b at the pressures in
// fluid_rp (fluid at the step's start positions) into force, and the
// prediction x*_b = x_b + dt (v_b + dt (F_b + f_b) / m) into pred (.w:
// psi_b / m, from P.bnd).
void launch_bnd_move(cudaStream_t st, const Params& P, int nb, const float4* fluid_pos, const float2* fluid_rp,
                     const uint32_t* cell_start, const uint32_t* cell_end, const float4* vel, const float4* fext,
                     float inv_mass, float4* pred, float4* force);
// dst[t] = src[ids[t]] (boundary arrays from their input order to sorted slots)
void launch_bnd_gather4(cudaStream_t st, int nb, const int* ids, const float4* src, float4* dst);
// Per fluid slot: the boundary particles within the list cut-off, from a
// 27-cell walk of the boundary's cell ranges (none outside P.bnd_lo/hi);
// flags[0] is set when a slot has more than P.bnd_cap.
void launch_build_bnd_nbr(cudaStream_t st, const Params& P, const float4* pos, const uint32_t* keys,
                          const uint32_t* bnd_start, const uint32_t* bnd_end, int* counts, int* list, int* flags);

// ---- FP64 diagnostics (diag.cu) -------------------------------------------------
// terms: mass, momentum x/y/z, kinetic, potential, sum and max of |rho - rho0|/rho0
constexpr int kDiagTerms = 8;
int diag_rows(int count);
void launch_diagnostics(cudaStream_t st, int first, int count, double mass, double rho0, const float g[3],
                        const float4* pos, const float4* vel, const float2* rp, double* rows, double* out);

// ---- iso field and marching cubes (mc.cu) ----------------------------------------
constexpr int kMcMaxTri = 10;       // at most 12 active edges in loops of >= 3: 12 - 2 triangles
struct IsoParams {
    double origin[3];   // node (0, 0, 0)
    double spacing[3];  // node spacing per axis
    int dims[3];        // nodes per axis
    double level;       // iso level of the surface
    double r;           // influence radius (REF: h / scale; CONFIG: h)
    int ring;           // cells of the particle grid walked on each side of the node's cell
    double inv_r2;      // CONFIG: 1 / h^2
    double k_colour;    // CONFIG: m 315 / (64 pi h^3): c(x) = k_colour sum (1 - q)^3 / rho_j
};
void mc_build_table(uint8_t ntri[256], int8_t tri[256][kMcMaxTri * 3]);
void mc_upload_table(cudaStream_t st);
long long scan_scratch_words(long long n);
void scan_exclusive_u32(cudaStream_t st, long long n, uint32_t* data, uint32_t* scratch);
void launch_iso_field(cudaStream_t st, const IsoParams& Q, const Params& P, const float4* pos, const float2* rp,
                      const uint32_t* cell_start, const uint32_t* cell_end, double* weight, double* iso);
// Marching cubes: edge flags and cube case per node, vertices and triangles
// per block of nodes (mc_blocks of them, one trailing word for the scan's
// total); then, from the scanned block counts, the mesh. first: a word per node.
long long mc_blocks(const IsoParams& Q);
void launch_mc_classify(cudaStream_t st, const IsoParams& Q, const double* iso, uint16_t* cases, uint32_t* block_vert,
                        uint32_t* block_tri);
void launch_mc_emit(cudaStream_t st, const IsoParams& Q, const double* iso, const uint16_t* cases,
                    const uint32_t* block_vert, const uint32_t* block_tri, uint32_t* first, float* vert, int32_t* tris);
// The reference's polygonizer layout (compat): double4 nodes, per-cube vertex
// slots and counts; synchronous, reports a slot overflow on stderr.
void launch_mc_polygonize_slots(cudaStream_t st, const double* node4, int nx, int ny, int nz, double level, int* count,
                                double* vertex, int* index, int slots);

// ---- learned warm start (mlp.cu) ---------------------------------------------------
// Networks (psb.h PSB_MLP_*): arch 0 6 -> 64 -> 64 -> 1 SiLU, arch 1 7 -> 64 -> 64 -> 1 ReLU.
constexpr int kMlpParams = 4737;   // the larger network's parameters: 7x64 + 64 + 64x64 + 64 + 64 + 1
int mlp_inputs(int arch);
int mlp_params(int arch);
// The initial pressures into rp[].y and, where given, zp[].y.
void launch_mlp_infer(cudaStream_t st, int arch, int n, const float* feats, const void* wbf, float p_scale, float2* rp,
                      float2* zp);
void launch_mlp_forward(cudaStream_t st, int arch, int n, const float* X, const void* wbf, float* y);
// Training blocks per minibatch (at most) and the gradient partials they
// write: kMlpGradBlocks rows of kMlpParams + 1 floats (the caller's buffer).
constexpr int kMlpGradBlocks = 148 * 4;
constexpr size_t kMlpGradPartials = (size_t)kMlpGradBlocks * (kMlpParams + 1);
void launch_mlp_grad(cudaStream_t st, int arch, int batch, const float* X, const float* T, const void* wbf,
                     float* partial, float* grad, float* loss);
// One Adam step on a minibatch drawn from `rows` recorded rows (rows > 0);
// after_step: enqueued directly behind another one.
void launch_mlp_step(cudaStream_t st, int arch, int batch, const float* X, const float* T, uint64_t rows, uint64_t seed,
                     float* partial, float* grad, float* loss, float* w, float* m1, float* m2, void* wbf, float lr,
                     int step, bool after_step);
void launch_to_bf16(cudaStream_t st, int np, const float* w, void* wbf);
void launch_collect(cudaStream_t st, int n, int stride, int offset, uint64_t base, uint64_t cap, const float* feats,
                    const float2* rp, float p_scale, float* X, float* T);
void launch_zero_pressure(cudaStream_t st, int n, float2* rp);

// Ordered encoding of doubles for atomicMax on unsigned 64-bit words.
__host__ __device__ inline unsigned long long order_double(double v) {
    long long b;
#ifdef __CUDA_ARCH__
    b = __double_as_longlong(v);
#else
    __builtin_memcpy(&b, &v, 8);
#endif
    return b >= 0 ? (unsigned long long)b ^ 0x8000000000000000ull : ~(unsigned long long)b;
}
__host__ __device__ inline double unorder_double(unsigned long long u) {
    long long b = (u & 0x8000000000000000ull) ? (long long)(u ^ 0x8000000000000000ull) : (long long)~u;
    double v;
#ifdef __CUDA_ARCH__
    v = __longlong_as_double(b);
#else
    __builtin_memcpy(&v, &b, 8);
#endif
    return v;
}

// Start of a step's corrector, run by one block. With max_iters = 0 no pass
// runs and every scene ends unconverged with no corrections, as a single
// scene does.
__device__ inline void corrector_begin(int S, int max_it, uint8_t* active, unsigned long long* err_scene,
                                       unsigned long long* err_hist, int hist_len, int* loop) {
    for (int s = threadIdx.x; s < S; s += blockDim.x) {
        active[s] = 1;
        err_scene[s] = 0ull;
        loop[2 + s] = 0;
        loop[2 + S + s] = 0;
        if (max_it == 0) loop[2 + 3 * S + s] += 1;
    }
    for (int i = threadIdx.x; i < hist_len; i += blockDim.x) err_hist[i] = 0ull;
    if (threadIdx.x == 0) { loop[0] = 0; loop[1] = 1; }
}

// After density pass k, run by one block (every thread calls it; any is a
// shared word). A scene converges when k >= min_iters and its error is at
// most eta (the host loop's test, in FP64 on the same value). A scene that
// has not converged takes the pressure-force pass; if that pass is its
// max_iters-th, it stops after it, unconverged, with max_iters corrections.
// Returns (to every thread) whether another pass follows.
__device__ inline int corrector_decide(int S, int min_it, int max_it, double eta, uint8_t* active,
                                       unsigned long long* err_scene, unsigned long long* err_hist, int* loop,
                                       int* any) {
    if (threadIdx.x == 0) *any = 0;
    __syncthreads();
    const int k = loop[0];
    for (int s = threadIdx.x; s < S; s += blockDim.x) {
        if (!active[s]) continue;
        const unsigned long long e = err_scene[s];
        if (k < PSB_MAX_ITERS + 1) err_hist[(size_t)k * S + s] = e;
        err_scene[s] = 0ull;
        if (k >= min_it && e != 0ull && unorder_double(e) <= eta) {
            active[s] = 0;
            loop[2 + s] = k;
            loop[2 + S + s] = 1;
            loop[2 + 2 * S + s] += k;
        } else if (k + 1 >= max_it) {
            loop[2 + s] = k + 1;          // last pass; stays active for it
            loop[2 + 2 * S + s] += k + 1;
            loop[2 + 3 * S + s] += 1;
        } else {
            *any = 1;
        }
    }
    __syncthreads();
    // k + 1 < max_it <= PSB_MAX_ITERS whenever any is set: the loop ends
    const int cont = *any && k + 1 < max_it && k + 1 <= PSB_MAX_ITERS;
    __syncthreads();
    if (threadIdx.x == 0) {
        loop[0] = k + 1;
        loop[1] = cont;
    }
    return cont;
}


}  // namespace psb
