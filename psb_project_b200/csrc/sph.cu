// sph.cu -- SPH density, forces and the PCISPH predictor-corrector sweeps.
//
// One thread per cell-sorted particle, walking its neighbour list (slot-
// major, so a warp's list reads are coalesced). Sums are per-particle and
// atomic-free, in the list's fixed order; densities use Kahan-compensated
// FP32 sums. All kernel constants are pre-scaled (q = r^2/h^2, u = r/h) so
// FP32 never sees h^9.
//
// Formulas and their reference sources (paths inside the reference tree):
//   density  rho_i = m 315/(64 pi h^9) sum (h^2-r^2)^3
//            SphKernel.cu:9-27, PciSphSystem_Kernel.cu:70-85
//   pressure force density -rho_i sum m (p_i/rho_i^2 + p_j/rho_j^2) gradW,
//            gradW = -45/(pi h^6) (h-r)^2 r^     SphKernel.cu:53-61, PciSphSystem_Kernel.cu:88-114
//   viscosity sum mu (v_j-v_i) m/rho_j 45 (h-r)/(pi h^6)
//            SphKernel.cu:63-66, PciSphSystem_Kernel.cu:141-146
//   surface tension and normals (reference profile only)
//            SphKernel.cu:68-88, PciSphSystem_Kernel.cu:148-166
//   PCISPH pressure increment (rho*-rho0)/(beta(|sum gradW|^2 + sum|gradW|^2)),
//            compressed particles only     PciSphSystem_Kernel.cu:36-67
//            (config profile: Solenthaler & Pajarola's prototype factor for every
//            particle, p clamped at 0; the per-particle form diverges when
//            iterated to an eta, see the config notes in the oracle)
//   leap-frog v+ += a dt, x += v+ dt; v = (v- + v+)/2
//            SphKernel.cu:95-135
//   box walls: projection + reflection     BoxCollision_Kernel.cu:7-34
// The reference's predict/restore passes (PciSphSystem.cu:30-61) become a
// predictor that writes x*, v* to separate buffers and leaves the state
// alone; the final leap-frog is the last prediction committed.
#include <algorithm>
#include <cooperative_groups.h>

#include "psb_internal.cuh"
#include "colliders.cuh"

namespace cg = cooperative_groups;

namespace psb {

namespace {

// The sums that several kernels compute for the same pair (the corrector's
// passes in their own kernels and in the persistent one, the density at x in
// its own sweep and inside the neighbour build) round the same way in every
// kernel: wherever a product feeds a sum, the operation is written out --
// __fmaf_rn where the product is fused, __fmul_rn/__fadd_rn/__fsub_rn (never
// contracted) where it is not. Plain * and + remain only where no fused
// multiply-add can form (products of products, a sum feeding a product), so
// the results do not depend on where the compiler would fuse.
struct Kahan {
    float s = 0.f, c = 0.f;     // sum and (negated) lost low part: true sum ~ s - c
    __device__ __forceinline__ void add(float x) {
        const float y = __fsub_rn(x, c);
        const float t = __fadd_rn(s, y);
        c = __fsub_rn(__fsub_rn(t, s), y);
        s = t;
    }
    // adds a * b with the product rounded only inside the sum (one FMA)
    __device__ __forceinline__ void add_prod(float a, float b) {
        const float y = __fmaf_rn(a, b, -c);
        const float t = __fadd_rn(s, y);
        c = __fsub_rn(__fsub_rn(t, s), y);
        s = t;
    }
};

// Adds a pair's (1 - q)^3, q = r2 / h^2 < 1, as (1 - q)^2 times (1 - q).
__device__ __forceinline__ void add_poly6(Kahan& acc, float q) {
    const float w = __fsub_rn(1.f, q);
    acc.add_prod(__fmul_rn(w, w), w);
}

// 1 - r/h of a pair, from r2 and its reciprocal square root
__device__ __forceinline__ float spiky_om(const Params& P, float r2, float rinv) {
    return __fmaf_rn(-(r2 * rinv), P.inv_h, 1.f);
}

// rho - rho0 = k_rho (s - c) - rho0 with the product's low part kept by the
// FMA: the deviation, from which every pressure is computed, keeps its full
// relative precision instead of the ~6e-5 absolute step of an FP32 density.
__device__ __forceinline__ float density_deviation(const Params& P, const Kahan& a) {
    return __fsub_rn(__fmaf_rn(P.k_rho, a.s, -P.rho0), __fmul_rn(P.k_rho, a.c));
}

__device__ __forceinline__ float3 f3(float4 a) { return make_float3(a.x, a.y, a.z); }

// Element j of a split vector field (plain loads: the persistent corrector
// rewrites some of them between its passes).
__device__ __forceinline__ float4 at(const Soa3& a, int j) {
    const float2 xy = a.xy[j];
    return make_float4(xy.x, xy.y, a.z[j], 0.f);
}
// An 8-byte gather that stays one load where it is written, ahead of a pair's
// tests: of a plain load of (z, pressure) the compiler moved the pressure
// behind the tests, a second load there, and the pair waited for memory twice.
// Pressure-force pass 97 -> 88 us at 1M particles, 294 -> 264 at 4M; set-up
// sweep 146 -> 139 and 537 -> 504. (Velocities are better left to the compiler:
// gathered this way the set-up sweep took 511 us at 4M, the density pass with
// the network's inputs 132 against 124 at 1M.)
__device__ __forceinline__ float2 gather2(const float2* p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(__cvta_generic_to_global(p)));
    return v;
}
__device__ __forceinline__ void put(const Soa3& a, int t, float x, float y, float z) {
    a.xy[t] = make_float2(x, y);
    a.z[t] = z;
}

// The box faces that bound particle t (slot t): the scene's own (kernel
// parameters, read where used) or, in a batch, its scene's table entry.
template <bool BATCH> struct Faces;
template <> struct Faces<false> {
    const Params& P;
    __device__ __forceinline__ float x0() const { return P.bx0; }
    __device__ __forceinline__ float y0() const { return P.by0; }
    __device__ __forceinline__ float z0() const { return P.bz0; }
    __device__ __forceinline__ float x1() const { return P.bx1; }
    __device__ __forceinline__ float y1() const { return P.by1; }
    __device__ __forceinline__ float z1() const { return P.bz1; }
};
template <> struct Faces<true> {
    const SceneGeom* G;
    __device__ __forceinline__ float x0() const { return G->bx0; }
    __device__ __forceinline__ float y0() const { return G->by0; }
    __device__ __forceinline__ float z0() const { return G->bz0; }
    __device__ __forceinline__ float x1() const { return G->bx1; }
    __device__ __forceinline__ float y1() const { return G->by1; }
    __device__ __forceinline__ float z1() const { return G->bz1; }
};
template <bool BATCH>
__device__ __forceinline__ Faces<BATCH> faces_of(const Params& P, int t);
template <>
__device__ __forceinline__ Faces<false> faces_of<false>(const Params& P, int) { return Faces<false>{P}; }
template <>
__device__ __forceinline__ Faces<true> faces_of<true>(const Params& P, int t) {
    return Faces<true>{P.scenes + P.slot_scene[t]};
}

// Penalty walls (config profile): a = K*depth - C*v along each axis on which
// x lies outside the box (a state uploaded outside it; the projection below
// keeps stepped particles inside).
template <bool REF, bool BATCH = false>
__device__ __forceinline__ float3 wall_accel(const Params& P, int t, float4 x, float4 v) {
    float3 a = make_float3(0.f, 0.f, 0.f);
    if (REF) return a;
    const auto F = faces_of<BATCH>(P, t);
    // K * depth - C * v, depth > 0 on the outside
    auto push = [&](float depth, float vel) {
        return __fsub_rn(__fmul_rn(P.wall_k, depth), __fmul_rn(P.wall_c, vel));
    };
    if (x.x < F.x0()) a.x = __fadd_rn(a.x, push(__fsub_rn(F.x0(), x.x), v.x));
    if (x.x > F.x1()) a.x = __fadd_rn(a.x, push(-__fsub_rn(x.x, F.x1()), v.x));
    if (x.y < F.y0()) a.y = __fadd_rn(a.y, push(__fsub_rn(F.y0(), x.y), v.y));
    if (x.y > F.y1()) a.y = __fadd_rn(a.y, push(-__fsub_rn(x.y, F.y1()), v.y));
    if (x.z < F.z0()) a.z = __fadd_rn(a.z, push(__fsub_rn(F.z0(), x.z), v.z));
    if (x.z > F.z1()) a.z = __fadd_rn(a.z, push(-__fsub_rn(x.z, F.z1()), v.z));
    return a;
}

// Config-profile walls: mirror ghost particles (Libersky et al. 1993;
// Colagrossi & Landrini 2003). Every box face within h of particle i
// reflects i's neighbours (self included); for each non-empty set S of such
// faces, the ghost of j is j reflected across every face in S, provided j is
// itself within h of each. A ghost can only lie within h of i if j does, so
// the neighbour list yields all of them. Ghosts carry j's pressure continued
// hydrostatically across the faces, p_j + rho0 (-g . n) 2 d_j, so a resting
// column is held by its bottom layer as by any interior layer.
//
// The ghost walk is the longest chain of a sweep: every sweep takes at least
// as long as one corner particle's. With per-face loops over packed face
// words and every set's distance formed, that was 75-80 us at any size
// (density at x at 16,384 particles: 80 us). With the faces in registers, the
// sets unrolled and most neighbours left out by one compare per axis it is
// 20 us there, and 24 against 86 us for the density pass at 97,000.
//
// The faces near a particle at x_i, one per axis at most: inward normal
// (+1 lower, -1 upper), plane and x_i's distance inside it, clamped at 0 so
// that a particle pushed through the face still sees its ghosts on the wall
// side (unclamped, its own ghost would push it further out). An axis with no
// near face has its plane at -infinity: every distance from it is infinite,
// so no ghost across it passes the range tests below.
struct NearFaces {
    float nrm[3], plane[3], di[3];
};

__device__ __forceinline__ float comp(float4 v, int a) { return a == 0 ? v.x : (a == 1 ? v.y : v.z); }

// Fills W for x; whether any face is within h.
template <class F_>
__device__ __forceinline__ bool near_faces(const Params& P, const F_& F, float4 x, NearFaces& W) {
    const float lo[3] = {F.x0(), F.y0(), F.z0()}, hi[3] = {F.x1(), F.y1(), F.z1()};
    bool any = false;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float xa = comp(x, a);
        const bool lower = xa - lo[a] < P.hf, upper = hi[a] - xa < P.hf;
        any |= lower | upper;
        W.nrm[a] = lower || !upper ? 1.f : -1.f;
        W.plane[a] = lower ? lo[a] : (upper ? hi[a] : -INFINITY);
        W.di[a] = fmaxf(__fmul_rn(W.nrm[a], __fsub_rn(xa, W.plane[a])), 0.f);
    }
    return any;
}

// The ghosts of neighbour x_j, one per non-empty set of the near faces, in
// the order x, y, xy, z, xz, yz, xyz: add(r, dp) with r = x_i minus the
// ghost -- a reflected component is nrm (d_i + d_j) -- and dp the ghost's
// hydrostatic pressure offset (PRESSURE). A face h or more from x_j reflects
// nothing; one whose reflected component alone reaches h (with a margin over
// the rounding of the squared distance) cannot bring a ghost into range, so
// its sets are left out before their distances are formed.
template <bool PRESSURE, class F>
__device__ __forceinline__ void for_each_ghost(const Params& P, const NearFaces& W, float4 xi, float4 xj, F&& add) {
    const float n[3] = {__fsub_rn(xi.x, xj.x), __fsub_rn(xi.y, xj.y), __fsub_rn(xi.z, xj.z)};
    const float g[3] = {P.gx, P.gy, P.gz};
    const float reach = P.hf * 1.00001f;
    float r[3], dj[3], hc[3];
    bool in[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        dj[a] = fmaxf(__fmul_rn(W.nrm[a], __fsub_rn(comp(xj, a), W.plane[a])), 0.f);
        const float d = __fadd_rn(W.di[a], dj[a]);
        in[a] = !(dj[a] >= P.hf) && !(d >= reach);
        r[a] = __fmul_rn(W.nrm[a], d);
        hc[a] = PRESSURE ? __fmul_rn(__fmul_rn(P.rho0, __fmul_rn(-g[a], W.nrm[a])), 2.f) : 0.f;
    }
    if (!(in[0] || in[1] || in[2])) return;
#pragma unroll
    for (int mask = 1; mask < 8; ++mask) {
        if (((mask & 1) && !in[0]) || ((mask & 2) && !in[1]) || ((mask & 4) && !in[2])) continue;
        float dp = 0.f;
        if (PRESSURE) {
            if (mask & 1) dp = __fmaf_rn(hc[0], dj[0], dp);
            if (mask & 2) dp = __fmaf_rn(hc[1], dj[1], dp);
            if (mask & 4) dp = __fmaf_rn(hc[2], dj[2], dp);
        }
        add(make_float3(mask & 1 ? r[0] : n[0], mask & 2 ? r[1] : n[1], mask & 4 ? r[2] : n[2]), dp);
    }
}

// Density: adds (1-q)^3 of each ghost within h.
__device__ __forceinline__ void ghost_density_pair(const Params& P, const NearFaces& W, float4 xi, float4 xj,
                                                   Kahan& acc) {
    for_each_ghost<false>(P, W, xi, xj, [&](float3 r, float) {
        const float q = __fmul_rn(dist2(r.x, r.y, r.z), P.inv_h2);
        if (!(q >= 1.f)) add_poly6(acc, q);
    });
}

// Pressure: adds (pV_i + pV_ghost) (1-u)^2 x^ of each ghost within h, the
// ghost carrying p_j continued hydrostatically across its faces.
__device__ __forceinline__ void ghost_pressure_pair(const Params& P, const NearFaces& W, float4 xi, float4 xj,
                                                    float pVi, float pj, float ir0, float3& ap) {
    for_each_ghost<true>(P, W, xi, xj, [&](float3 r, float dp) {
        const float r2 = dist2(r.x, r.y, r.z);
        if (!(r2 > 0.f) || __fmul_rn(r2, P.inv_h2) >= 1.f) return;
        const float rinv = rsqrtf(r2);
        const float om = spiky_om(P, r2, rinv);
        const float sc = __fmul_rn(__fmul_rn(__fmul_rn(__fmaf_rn(__fadd_rn(pj, dp), ir0, pVi), om), om), rinv);
        ap.x = __fmaf_rn(sc, r.x, ap.x); ap.y = __fmaf_rn(sc, r.y, ap.y); ap.z = __fmaf_rn(sc, r.z, ap.z);
    });
}

// Ghost terms of particle t, in a second walk of its list that only
// particles within h of a face take (the walls are evaluated at xi). Kept
// out of the main walk: a per-neighbour wall test there slows every
// particle more than the separate walk costs the few near the faces.
template <bool BATCH = false, bool FRESH = false>
__device__ __forceinline__ void ghost_density(const Params& P, int t, float4 xi, const Soa3& x, const int* list,
                                              int cnt, Kahan& acc) {
    NearFaces W;
    if (!near_faces(P, faces_of<BATCH>(P, t), xi, W)) return;
    for_each_nbr<FRESH>(list, P.n, t, cnt, [&](const int j) { ghost_density_pair(P, W, xi, at(x, j), acc); });
}

// The neighbours at the step's start positions with the pressures of P.zp.
template <bool BATCH = false>
__device__ __forceinline__ void ghost_pressure(const Params& P, int t, float4 xi, float pVi,
                                               const int* __restrict__ list, int cnt, float3& ap) {
    NearFaces W;
    if (!near_faces(P, faces_of<BATCH>(P, t), xi, W)) return;
    const float ir0 = 1.f / __fmul_rn(P.rho0, P.rho0);
    for_each_nbr(list, P.n, t, cnt, [&](const int j) {
        const float2 xy = gather2(P.x0.xy + j), zp = gather2(P.zp + j);
        ghost_pressure_pair(P, W, xi, make_float4(xy.x, xy.y, zp.x, 0.f), pVi, zp.y, ir0, ap);
    });
}

// ---- particles near the walls -----------------------------------------------
// A particle near a face walks its list twice and sums up to seven ghosts a
// neighbour. In slot order such particles sit a few to a warp, and the warp
// waits for them with its other lanes idle. From kWallListMin particles on,
// the step's reorder therefore lists them (P.wall_list) and flags them by
// slot, and a sweep with ghost terms launches P.wall_blocks blocks over the
// list ahead of the blocks over all slots, which skip the listed ones: full
// warps of wall particles, started first. Each particle is summed by one
// thread in the same order either way, so the results are the same bits.
// Density pass / pressure-force pass (converged launches among the latter at
// 1M) with the list against without: 71 / 69 against 79 / 78 us at 1,048,576
// particles, 32 / 36 against 41 / 48 at 290,000; at 97,000, where the pass is
// one chain of loads and the list adds two, 26 / 25 against 23 / 23 us.
__device__ __forceinline__ bool in_wall_list(const Params& P, int t) {
    return P.wall_list && ((P.wall_bits[t >> 5] >> (t & 31)) & 1u);
}

// The slots of this thread in a launch of BS-thread blocks: f(slot), or f(-1)
// where it has none. Every lane of a warp makes the same calls.
template <int BS, bool GHOSTS, class F>
__device__ __forceinline__ void for_each_slot(const Params& P, F&& f) {
    if (!GHOSTS) {
        const int t = blockIdx.x * BS + threadIdx.x;
        f(t < P.n ? t : -1);
        return;
    }
    const bool wall = (int)blockIdx.x < P.wall_blocks;
    const int first = ((int)blockIdx.x - (wall ? 0 : P.wall_blocks)) * BS + threadIdx.x;
    const int end = wall ? *P.wall_count : P.n;
    int k = first;
    do {
        int t = -1;
        if (k < end) {
            if (wall) t = P.wall_list[k];
            else if (!P.wall_blocks || !in_wall_list(P, k)) t = k;
        }
        f(t);
        k += P.wall_blocks * BS;
    } while (wall && k - (int)(threadIdx.x & 31) < end);
}

// Boundary particles (config profile; boundary.cu): density psi_b W_ib, as
// (psi_b / m) (1 - q)^3 inside the k_rho-scaled sum, and the mirrored
// pressure term psi_b pV_i gradW_ib, as (psi_b / m) pV_i (1-u)^2 x^ inside
// the k_grad-scaled sum. The positions are the step's start positions of
// a static solid; x_i is the particle's current (or predicted) position.
// bx: the boundary positions the density sees (P.bnd at the step's start
// positions; in the corrector, P.bnd_pred where the boundary moves with it).
__device__ __forceinline__ void boundary_density(const Params& P, int t, float4 xi, Kahan& acc,
                                                 const float4* __restrict__ bx) {
    if (!P.bnd_count) return;
    const int cnt = min(P.bnd_count[t], P.bnd_cap);
    for_each_nbr(P.bnd_list, P.n, t, cnt, [&](const int b) {
        const float4 xb = bx[b];
        const float dx = __fsub_rn(xi.x, xb.x), dy = __fsub_rn(xi.y, xb.y), dz = __fsub_rn(xi.z, xb.z);
        const float q = __fmul_rn(dist2(dx, dy, dz), P.inv_h2);
        if (q >= 1.f) return;
        const float w = __fsub_rn(1.f, q);
        acc.add_prod(xb.w, __fmul_rn(__fmul_rn(w, w), w));
    });
}

__device__ __forceinline__ void boundary_pressure(const Params& P, int t, float4 xi, float pVi, float3& ap) {
    if (!P.bnd_count) return;
    const int cnt = min(P.bnd_count[t], P.bnd_cap);
    for_each_nbr(P.bnd_list, P.n, t, cnt, [&](const int b) {
        const float4 xb = P.bnd[b];
        const float dx = __fsub_rn(xi.x, xb.x), dy = __fsub_rn(xi.y, xb.y), dz = __fsub_rn(xi.z, xb.z);
        const float r2 = dist2(dx, dy, dz);
        if (!(r2 > 0.f) || __fmul_rn(r2, P.inv_h2) >= 1.f) return;
        const float rinv = rsqrtf(r2);
        const float om = spiky_om(P, r2, rinv);
        const float sc = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(xb.w, pVi), om), om), rinv);
        ap.x = __fmaf_rn(sc, dx, ap.x); ap.y = __fmaf_rn(sc, dy, ap.y); ap.z = __fmaf_rn(sc, dz, ap.z);
    });
}

// collisionBox (BoxCollision_Kernel.cu:7-34) with restitution 0: clamp into
// [Min+r, Max-r] (upper bounds tested first, lower bounds win), then remove
// the velocity component along the normalised sum of wall normals. PCISPH
// in both profiles: in the config profile it keeps every particle at least r
// from each face, where its own ghost still pushes back (a particle on or
// behind a face meets its ghost at distance 0, which exerts no force, and
// its density error could not be corrected). Config WCSPH keeps the penalty
// walls its scene states.
template <bool BATCH = false>
__device__ __forceinline__ void box_project(const Params& P, int t, float3& x, float3& v) {
    float wlo_x = P.wlo_x, wlo_y = P.wlo_y, wlo_z = P.wlo_z, whi_x = P.whi_x, whi_y = P.whi_y, whi_z = P.whi_z;
    if (BATCH) {
        const SceneGeom* G = P.scenes + P.slot_scene[t];
        wlo_x = G->wlo_x; wlo_y = G->wlo_y; wlo_z = G->wlo_z; whi_x = G->whi_x; whi_y = G->whi_y; whi_z = G->whi_z;
    }
    float3 pI = x, nI = make_float3(0.f, 0.f, 0.f);
    if (x.x >= whi_x) { pI.x = whi_x; nI.x = -1.f; }
    if (x.y >= whi_y) { pI.y = whi_y; nI.y = -1.f; }
    if (x.z >= whi_z) { pI.z = whi_z; nI.z = -1.f; }
    if (x.x <= wlo_x) { pI.x = wlo_x; nI.x = 1.f; }
    if (x.y <= wlo_y) { pI.y = wlo_y; nI.y = 1.f; }
    if (x.z <= wlo_z) { pI.z = wlo_z; nI.z = 1.f; }
    const float l2 = nI.x * nI.x + nI.y * nI.y + nI.z * nI.z;
    if (l2 > 0.f) {
        const float il = rsqrtf(l2);
        nI.x *= il; nI.y *= il; nI.z *= il;
        const float vd = v.x * nI.x + v.y * nI.y + v.z * nI.z;
        x = pI;
        v.x -= vd * nI.x; v.y -= vd * nI.y; v.z -= vd * nI.z;
    }
}

// ---- density at the step's start positions ---------------------------------
// WCSPH: also the equation of state (reference: p = k (rho - rho0),
// SphKernel.cu:25; config: Tait, p = k rho0/7 ((rho/rho0)^7 - 1), written as
// k rho0/7 d (1 + x + ... + x^6) with x = 1 + d to avoid cancellation).
// PCISPH: keeps the carried pressure (warm start) or zeroes it.
// NF (config PCISPH, learned warm start or data collection): the same
// neighbour walk also sums the velocity divergence and density gradient and
// writes the MLP's first NF inputs (6 or 7; feats, stride 8, the rest 0):
//   f0 neighbour count / 32
//   f1 advected density deviation (rho - dt rho div v - rho0)/rho0 * 100
//   f2 div v * dt * 100, div v = -(k_grad/rho0) sum (1-u)^2 (v_j - v_i).x^
//   f3 previous-step pressure / p_scale
//   f4 distance to the nearest box face / h, capped at 1
//   f5 k_grad |sum (1-u)^2 x^| h / rho0 (density-gradient magnitude)
//   f6 sum W_ij p_j / sum W_ij / p_scale over the list, self included: the
//      carried pressure smoothed with the poly6 weights
// The sums of the density pass at x for one particle, pair by pair in list
// order; shared by the density sweep and by the neighbour build that
// computes the density as it accepts each neighbour, so that both give the
// same bits.
template <bool REF, int NF>
struct DensityX {
    static constexpr bool FEAT = NF > 0, SMOOTH_P = NF > 6;
    Kahan acc;
    float div = 0.f, wp = 0.f, ws = 0.f;
    float3 gr = make_float3(0.f, 0.f, 0.f);
    float4 vi = make_float4(0.f, 0.f, 0.f, 0.f);

    __device__ __forceinline__ void begin(const Params& P, int t) {
        if (FEAT) vi = at(P.v0, t);
    }
    // neighbour j at xj (r2 = dist2 of xi - xj); rp[j].y is the carried
    // pressure, which the pass writes back unchanged
    __device__ __forceinline__ void pair(const Params& P, float4 xi, float4 xj, int j, const float2* __restrict__ rp) {
        // the pair's other gathers issue with its position, ahead of the tests
        const float4 vj = FEAT ? at(P.v0, j) : make_float4(0.f, 0.f, 0.f, 0.f);
        const float pj = SMOOTH_P ? rp[j].y : 0.f;
        const float dx = __fsub_rn(xi.x, xj.x), dy = __fsub_rn(xi.y, xj.y), dz = __fsub_rn(xi.z, xj.z);
        const float r2 = dist2(dx, dy, dz);
        const float q = __fmul_rn(r2, P.inv_h2);
        if (!REF && q >= 1.f) return;
        const float w = __fsub_rn(1.f, q);
        const float w2 = __fmul_rn(w, w);
        const float w3 = __fmul_rn(w2, w);
        acc.add_prod(w2, w);
        if (SMOOTH_P) {
            wp = __fmaf_rn(w3, pj, wp);
            ws = __fadd_rn(ws, w3);
        }
        if (FEAT && r2 > 0.f) {
            const float rinv = rsqrtf(r2);
            const float om = spiky_om(P, r2, rinv);
            const float s = __fmul_rn(__fmul_rn(om, om), rinv);           // (1-u)^2 / r
            gr.x = __fmaf_rn(s, dx, gr.x); gr.y = __fmaf_rn(s, dy, gr.y); gr.z = __fmaf_rn(s, dz, gr.z);
            float d = __fmul_rn(__fsub_rn(vj.x, vi.x), dx);                  // (v_j - v_i) . (x_i - x_j)
            d = __fmaf_rn(__fsub_rn(vj.y, vi.y), dy, d);
            d = __fmaf_rn(__fsub_rn(vj.z, vi.z), dz, d);
            div = __fmaf_rn(s, d, div);
        }
    }
    // wall ghosts and boundary particles (config), then density, pressure
    // (EOS, or the carried / zeroed PCISPH pressure) and the features
    // (FRESH: over lists this kernel has written)
    template <bool BATCH, bool FRESH = false>
    __device__ __forceinline__ void finish(const Params& P, int t, float4 xi, const int* list, int cnt, int count,
                                           float2* __restrict__ rp, float* __restrict__ rho_x, int zero_p,
                                           float p_scale, float* __restrict__ feats) {
        if (!REF) {
            ghost_density<BATCH, FRESH>(P, t, xi, P.x0, list, cnt, acc);
            if (!BATCH) boundary_density(P, t, xi, acc, P.bnd);
        }
        const float drho = density_deviation(P, acc);
        const float rho = __fadd_rn(P.rho0, drho);
        float p;
        if (P.pci) {
            p = zero_p ? 0.f : rp[t].y;
        } else if (REF) {
            p = P.eos_k * drho;
        } else {
            const float d = drho / P.rho0;
            const float x = 1.f + d;
            const float s = 1.f + x * (1.f + x * (1.f + x * (1.f + x * (1.f + x * (1.f + x)))));
            p = P.eos_k * d * s;
        }
        if (FEAT) {
            div = __fmul_rn(div, -P.k_grad / P.rho0);
            const auto F = faces_of<BATCH>(P, t);
            float dwall = P.hf;
            dwall = fminf(dwall, fminf(xi.x - F.x0(), F.x1() - xi.x));
            dwall = fminf(dwall, fminf(xi.y - F.y0(), F.y1() - xi.y));
            dwall = fminf(dwall, fminf(xi.z - F.z0(), F.z1() - xi.z));
            float4* f = reinterpret_cast<float4*>(feats + (size_t)t * 8);     // two 16-byte stores
            const float adv = __fsub_rn(__fsub_rn(rho, __fmul_rn(__fmul_rn(P.dt, rho), div)), P.rho0);
            const float grad = sqrtf(dist2(gr.x, gr.y, gr.z));
            f[0] = make_float4((float)count * (1.f / 32.f), __fmul_rn(adv / P.rho0, 100.f),
                               __fmul_rn(__fmul_rn(div, P.dt), 100.f),
                               rp[t].y / p_scale);     // the carried pressure, before this pass replaces it
            f[1] = make_float4(__fmul_rn(fmaxf(dwall, 0.f), P.inv_h), __fmul_rn(__fmul_rn(P.k_grad, grad), P.hf) / P.rho0,
                               SMOOTH_P && ws > 0.f ? wp / ws / p_scale : 0.f, 0.f);
        }
        rp[t] = make_float2(rho, p);
        rho_x[t] = rho;
        // what the set-up or force sweep gathers beside the xy components
        P.zp[t] = make_float2(xi.z, p);
        P.vr[t] = make_float2(FEAT ? vi.z : P.v0.z[t], 1.f / rho);
    }
};

// Resident threads per SM asked of the sweeps with ghost terms: what the
// main walk's registers allow (40 or 48 a thread), so that the ghost
// walk, which few threads take, spills rather than lowering the occupancy of
// all (density pass at 4M particles: 272 us at 40 registers, 354 at 56).
constexpr int kDensityThreads = 1536, kForceThreads = 1280;

template <bool REF, int NF, bool BATCH, int BS>
__global__ void __launch_bounds__(BS, REF ? 1 : (NF ? kForceThreads : kDensityThreads) / BS)
    k_density_x(Params P, const int* __restrict__ counts, const int* __restrict__ list, float2* __restrict__ rp,
                float* __restrict__ rho_x, int zero_p, float p_scale, float* __restrict__ feats) {
    after_previous();
    for_each_slot<BS, !REF>(P, [&](const int t) {
        if (t < 0) return;
        const float4 xi = at(P.x0, t);
        const int count = counts[t];
        const int cnt = min(count, P.cap);
        DensityX<REF, NF> D;
        D.begin(P, t);
        for_each_nbr(list, P.n, t, cnt, [&](const int j) { D.pair(P, xi, at(P.x0, j), j, rp); });
        D.template finish<BATCH>(P, t, xi, list, cnt, count, rp, rho_x, zero_p, p_scale, feats);
    });
}

// The neighbour build of one scene (config profile) with the density pass
// at x folded in: the 27-cell walk of each particle (walk_neighbours) writes
// its list and, for every neighbour it accepts, adds that pair's density and
// feature terms -- the same terms in the same order as k_density_x over the
// finished list -- so the step saves one sweep over the lists. The ghost
// and boundary terms then walk the list this thread has just written.
template <int NF, int BS>
__global__ void __launch_bounds__(BS) k_build_density(Params P, const float4* __restrict__ pos,
                                                          const uint32_t* __restrict__ keys,
                                                          const uint32_t* __restrict__ cell_start,
                                                          const uint32_t* __restrict__ cell_end,
                                                          int* __restrict__ counts, int* __restrict__ list,
                                                          int* __restrict__ flags, float2* __restrict__ rp,
                                                          float* __restrict__ rho_x, int zero_p, float p_scale,
                                                          float* __restrict__ feats) {
    after_previous();
    const int t = blockIdx.x * BS + threadIdx.x;
    const bool valid = t < P.n;     // every lane stays for the warp reductions below
    int cnt = 0;
    if (valid) {
        const float4 pi = pos[t];
        DensityX<false, NF> D;
        D.begin(P, t);
        int* wq = list + nbr_index(0, P.n, t);
        const size_t qstride = (size_t)4 * (size_t)P.n;
        walk_neighbours(P, t, pi, pos, keys, cell_start, cell_end, [&](uint32_t q, float4 pj) {
            if (cnt < P.cap) {
                wq[cnt & 3] = (int)q;
                D.pair(P, pi, pj, (int)q, rp);
            }
            ++cnt;
            if ((cnt & 3) == 0 && cnt < P.cap) wq += qstride;
        });
        counts[t] = cnt;
        if (cnt > P.cap) atomicOr(&flags[0], 1);
        D.template finish<false, true>(P, t, pi, list, min(cnt, P.cap), cnt, rp, rho_x, zero_p, p_scale, feats);
    }
    nbr_flags(cnt, flags);
}

// Viscosity (+ reference surface tension) and, when with_pressure, the
// symmetric pressure acceleration, over the list at the start positions.
struct PairSums {
    float3 ap;      // sum (pV_i + pV_j) (1-u)^2 x^_ij   (times k_grad: pressure acceleration)
    float3 fv;      // sum (v_j - v_i) (1-u) / rho_j     (times k_visc: viscosity force density)
    float3 nrm;     // sum x_ij (1-q)^2 / rho_j           (times -k_surf: surface normal)
    float fs;       // sum (1-q)(3-7q) / rho_j           (times -k_surf: surface term)
};

// Config: p/rho0^2 (the PCISPH linearisation; see k_pci_force_predict).
template <bool REF>
__device__ __forceinline__ float pressure_volume(const Params& P, float2 rp) {
    return REF ? rp.y / (rp.x * rp.x) : rp.y * (1.f / (P.rho0 * P.rho0));
}

// Adds the pair (i, j) to S; xj, inv_rj, pj: neighbour j's position, 1 / density, pressure.
template <bool REF, bool WITH_PRESSURE>
__device__ __forceinline__ void add_pair(const Params& P, PairSums& S, float4 xi, float4 vi, float pVi, float4 xj,
                                         float4 vj, float inv_rj, float pj) {
    const float ir0 = 1.f / (P.rho0 * P.rho0);
    const float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
    const float r2 = dist2(dx, dy, dz);
    if (!(r2 > 0.f)) return;
    const float q = r2 * P.inv_h2;
    if (!REF && q >= 1.f) return;
    const float rinv = rsqrtf(r2);
    const float om = 1.f - r2 * rinv * P.inv_h;
    const float sv = om * inv_rj;
    S.fv.x += (vj.x - vi.x) * sv;
    S.fv.y += (vj.y - vi.y) * sv;
    S.fv.z += (vj.z - vi.z) * sv;
    if (WITH_PRESSURE) {
        const float pVj = REF ? pj * inv_rj * inv_rj : pj * ir0;
        const float s = (pVi + pVj) * om * om * rinv;
        S.ap.x += s * dx; S.ap.y += s * dy; S.ap.z += s * dz;
    }
    if (REF) {      // surface tension and normals: reference profile only
        const float t1 = 1.f - q;
        S.fs += t1 * (3.f - 7.f * q) * inv_rj;
        const float sn = t1 * t1 * inv_rj;
        S.nrm.x += dx * sn; S.nrm.y += dy * sn; S.nrm.z += dz * sn;
    }
}

template <bool REF, bool WITH_PRESSURE, bool BATCH = false>
__device__ __forceinline__ PairSums pair_sums(const Params& P, int t, float4 xi, float4 vi, float2 rpi,
                                              const int* __restrict__ counts, const int* __restrict__ list) {
    PairSums S;
    S.ap = S.fv = S.nrm = make_float3(0.f, 0.f, 0.f);
    S.fs = 0.f;
    const float pVi = WITH_PRESSURE ? pressure_volume<REF>(P, rpi) : 0.f;
    const int cnt = min(counts[t], P.cap);
    for_each_nbr(list, P.n, t, cnt, [&](const int j) {
        // the pair's four 8-byte gathers
        const float2 xy = gather2(P.x0.xy + j), zp = gather2(P.zp + j), vxy = P.v0.xy[j], vr = P.vr[j];
        add_pair<REF, WITH_PRESSURE>(P, S, xi, vi, pVi, make_float4(xy.x, xy.y, zp.x, 0.f),
                                     make_float4(vxy.x, vxy.y, vr.x, 0.f), vr.y, zp.y);
    });
    if (WITH_PRESSURE && !REF) {
        ghost_pressure<BATCH>(P, t, xi, pVi, list, cnt, S.ap);
        if (!BATCH) boundary_pressure(P, t, xi, pVi, S.ap);
    }
    return S;
}

// Non-pressure force density f_v + f_s + rho_i g (the reference's forcesAccum
// is (0, -9.81 rho, 0) in PCISPH, PciSphSystem_Kernel.cu:168, and rho*g from
// ForceExt_Constante in WCSPH, SphSystem.cpp:307-320).
template <bool REF>
__device__ __forceinline__ float3 nonpressure_force(const Params& P, const PairSums& S, float rho) {
    float3 f = make_float3(P.k_visc * S.fv.x, P.k_visc * S.fv.y, P.k_visc * S.fv.z);
    if (REF) {
        const float3 n = make_float3(-P.k_surf * S.nrm.x, -P.k_surf * S.nrm.y, -P.k_surf * S.nrm.z);
        const float ln = sqrtf(n.x * n.x + n.y * n.y + n.z * n.z);
        if (ln >= P.l) {
            const float c = (-P.k_surf * S.fs) * (-P.sigma) / ln;
            f.x += c * n.x; f.y += c * n.y; f.z += c * n.z;
        }
    }
    f.x += rho * P.gx; f.y += rho * P.gy; f.z += rho * P.gz;
    return f;
}

// WCSPH: forces, leap-frog, walls and velocity interpolation in one sweep.
template <bool REF>
__global__ void __launch_bounds__(kBlock) k_wcsph_force(Params P, const float4* __restrict__ vap, const float2* __restrict__ rp, const int* __restrict__ counts,
                                                        const int* __restrict__ list, float4* __restrict__ pos_out,
                                                        float4* __restrict__ vel_out, float4* __restrict__ vap_out,
                                                        float4* __restrict__ fnp) {
    after_previous();
    auto integrate = [&](const int t, const float4 xi, const float2 rpi, const PairSums& S) {
        const float4 vh = vap[t];
        const float3 f = nonpressure_force<REF>(P, S, rpi.x);
        fnp[t] = make_float4(f.x, f.y, f.z, 0.f);
        const float3 aw = wall_accel<REF>(P, t, xi, vh);
        const float ir = 1.f / rpi.x;
        const float3 a = make_float3(f.x * ir + P.k_grad * S.ap.x + aw.x, f.y * ir + P.k_grad * S.ap.y + aw.y,
                                     f.z * ir + P.k_grad * S.ap.z + aw.z);
        float3 v = make_float3(vh.x + a.x * P.dt, vh.y + a.y * P.dt, vh.z + a.z * P.dt);
        float3 x = make_float3(xi.x + v.x * P.dt, xi.y + v.y * P.dt, xi.z + v.z * P.dt);
        if (REF) box_project(P, t, x, v);   // config WCSPH: penalty walls only
        pos_out[t] = make_float4(x.x, x.y, x.z, 0.f);
        vap_out[t] = make_float4(v.x, v.y, v.z, 0.f);
        vel_out[t] = make_float4((vh.x + v.x) * 0.5f, (vh.y + v.y) * 0.5f, (vh.z + v.z) * 0.5f, 0.f);
    };
    for_each_slot<kBlock, !REF>(P, [&](const int t) {
        if (t < 0) return;
        const float4 xi = at(P.x0, t), vi = at(P.v0, t);
        const float2 rpi = rp[t];
        integrate(t, xi, rpi, pair_sums<REF, true>(P, t, xi, vi, rpi, counts, list));
    });
}

// PCISPH set-up sweep: non-pressure forces at x (and, for a warm start, the
// pressure acceleration of the carried pressure), then the first prediction.
// Four 8-byte gathers a pair: bound by L1 wavefronts. With 1 / rho_j gathered
// instead of rho_j (the division was ~10 of 79 instructions a pair) it took
// 147 us at 1M particles against 166, 538 at 4M against 613; with gather2 139
// and 504.
template <bool REF, bool WARM, bool BATCH, int BS>
__global__ void __launch_bounds__(BS, REF || !WARM ? 1 : kForceThreads / BS) k_pci_init(
    Params P, const float4* __restrict__ vap, const float2* __restrict__ rp, const int* __restrict__ counts,
    const int* __restrict__ list, float4* __restrict__ fnp, Soa3 xs, Soa3 vs) {
    after_previous();
    auto predict = [&](const int t, const float4 xi, const float2 rpi, const PairSums& S) {
        const float4 vh = vap[t];
        const float3 f = nonpressure_force<REF>(P, S, rpi.x);
        fnp[t] = make_float4(f.x, f.y, f.z, 0.f);
        const float3 aw = wall_accel<REF, BATCH>(P, t, xi, vh);
        const float ir = 1.f / rpi.x;
        const float ap = WARM ? P.k_grad : 0.f;
        const float3 a = make_float3(f.x * ir + ap * S.ap.x + aw.x, f.y * ir + ap * S.ap.y + aw.y,
                                     f.z * ir + ap * S.ap.z + aw.z);
        const float3 v = make_float3(vh.x + a.x * P.dt, vh.y + a.y * P.dt, vh.z + a.z * P.dt);
        put(vs, t, v.x, v.y, v.z);
        put(xs, t, xi.x + v.x * P.dt, xi.y + v.y * P.dt, xi.z + v.z * P.dt);
    };
    for_each_slot<BS, !REF && WARM>(P, [&](const int t) {
        if (t < 0) return;
        const float4 xi = at(P.x0, t), vi = at(P.v0, t);
        const float2 rpi = rp[t];
        predict(t, xi, rpi, pair_sums<REF, WARM, BATCH>(P, t, xi, vi, rpi, counts, list));
    });
}

// PCISPH density pass at x*: rho*, the gradient sums of the pressure
// increment, the candidate pressure and the FP64 max compression error.
// The compression error (rho* - rho0)/rho0 in FP64 of sorted particle t, from
// its compensated sum; rho* and the candidate pressure into rpc[t].
template <bool REF, class F2, class F2o>
__device__ __forceinline__ double pci_density_finish(const Params& P, int t, const Kahan& acc, float3 T1, float T2,
                                                     F2 rp, F2o rpc) {
    const float drho = density_deviation(P, acc);
    const float rho = __fadd_rn(P.rho0, drho);
    float p = rp[t].y;
    if (REF) {              // per-particle factor, compressed particles only
        if (drho > 0.f && T2 > 0.f) p += P.k_press * drho / (T1.x * T1.x + T1.y * T1.y + T1.z * T1.z + T2);
    } else {                // prototype factor, every particle, p >= 0
        p = fmaxf(0.f, __fmaf_rn(P.k_delta, drho, p));
    }
    rpc[t] = make_float2(rho, p);
    if (!REF) P.zp[t] = make_float2(P.x0.z[t], p);     // as the pressure-force pass gathers it
    return (double)drho / P.rho0_d;
}

// The density pass for sorted particle t (t < P.n, its scene still iterating).
template <bool REF, bool BATCH, class F2, class F2o>
__device__ __forceinline__ double pci_density_at(const Params& P, int t, const Soa3& xs, F2 rp, const int* __restrict__ counts,
                                                 const int* __restrict__ list, F2o rpc) {
    const float4 xi = at(xs, t);
    const int cnt = min(counts[t], P.cap);
    Kahan acc;
    float3 T1 = make_float3(0.f, 0.f, 0.f);
    float T2 = 0.f;
    for_each_nbr(list, P.n, t, cnt, [&](const int j) {
        const float4 xj = at(xs, j);
        const float dx = __fsub_rn(xi.x, xj.x), dy = __fsub_rn(xi.y, xj.y), dz = __fsub_rn(xi.z, xj.z);
        const float r2 = dist2(dx, dy, dz);
        const float q = __fmul_rn(r2, P.inv_h2);
        if (!REF && q >= 1.f) return;
        add_poly6(acc, q);
        if (REF && r2 > 0.f) {
            const float rinv = rsqrtf(r2);
            const float om = 1.f - r2 * rinv * P.inv_h;
            const float g = om * om;
            const float s = g * rinv;
            T1.x += s * dx; T1.y += s * dy; T1.z += s * dz;
            T2 += g * g;
        }
    });
    if (!REF) {
        ghost_density<BATCH>(P, t, xi, xs, list, cnt, acc);
        if (!BATCH) boundary_density(P, t, xi, acc, P.bnd_pred ? P.bnd_pred : P.bnd);
    }
    return pci_density_finish<REF>(P, t, acc, T1, T2, rp, rpc);
}

// Raises *slot to err (ordered encoding; -1e300: no error). The slot only
// grows during a pass, so a value at or below what it already holds needs no
// atomic. Atomics on one sector retire one after another in L2, and a batch's
// scene words share a few sectors: its density pass took 218 us with an
// atomic from every warp (64 scenes, 2.3M particles), 171 us with the test.
__device__ __forceinline__ void raise_error(unsigned long long* slot, double err) {
    if (!(err > -1e300)) return;
    const unsigned long long e = order_double(err);
    if (e > *(volatile unsigned long long*)slot) atomicMax(slot, e);
}

// The max of the pass's errors. Batch: per scene (P.err_scene); a warp
// inside one scene reduces first, one straddling two or more reduces per
// lane; sc = the slot's scene, -1 for none. Single scene (the persistent
// corrector, once per block and pass): per block, one ordered-integer atomic
// max into err_slot; every thread of the block calls it.
template <bool BATCH, int BS>
__device__ __forceinline__ void reduce_error(const Params& P, int sc, double err, unsigned long long* err_slot,
                                             double* s_err) {
    if constexpr (BATCH) {
        const int sc0 = __shfl_sync(0xffffffffu, sc, 0);
        if (__all_sync(0xffffffffu, sc == sc0 || sc < 0)) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) err = fmax(err, __shfl_xor_sync(0xffffffffu, err, o));
            if ((threadIdx.x & 31) == 0 && sc0 >= 0) raise_error(&P.err_scene[sc0], err);
        } else if (sc >= 0) {
            raise_error(&P.err_scene[sc], err);
        }
    } else {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) err = fmax(err, __shfl_xor_sync(0xffffffffu, err, o));
        if ((threadIdx.x & 31) == 0) s_err[threadIdx.x >> 5] = err;
        __syncthreads();
        if (threadIdx.x == 0) {
            double m = s_err[0];
            for (int w = 1; w < BS / 32; ++w) m = fmax(m, s_err[w]);
            raise_error(err_slot, m);
        }
        __syncthreads();
    }
}

// PCISPH density pass at x*: rho*, the gradient sums of the pressure
// increment, the candidate pressure and the FP64 max compression error.
// Batch: scenes that have converged are left as they are, and the error is
// the max over each scene (P.err_scene).
// Single scene: the max over each warp, then one ordered-integer atomic max
// per warp (a reduction without return: the warp leaves at once). A block-
// level reduction made the block's early warps wait at its barrier for the
// slowest one, a third of the pass's stall cycles at 1M particles.
template <bool BATCH, int BS>
__device__ __forceinline__ void warp_max_error(const Params& P, int sc, double err, unsigned long long* err_slot) {
    if constexpr (BATCH) {
        reduce_error<true, BS>(P, sc, err, err_slot, nullptr);
    } else {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) err = fmax(err, __shfl_xor_sync(0xffffffffu, err, o));
        if ((threadIdx.x & 31) == 0) raise_error(err_slot, err);
    }
}

template <bool REF, bool BATCH, int BS>
__global__ void __launch_bounds__(BS, REF ? 1 : kDensityThreads / BS) k_pci_density(Params P, Soa3 xs,
                                                        const float2* __restrict__ rp, const int* __restrict__ counts,
                                                        const int* __restrict__ list, float2* __restrict__ rpc,
                                                        unsigned long long* __restrict__ err_slot) {
    after_previous();
    double worst = -1e300;
    for_each_slot<BS, !REF>(P, [&](const int t) {
        const int sc = BATCH && t >= 0 ? (int)P.slot_scene[t] : -1;
        double err = -1e300;
        if (t >= 0 && (!BATCH || P.active[sc])) err = pci_density_at<REF, BATCH>(P, t, xs, rp, counts, list, rpc);
        if (BATCH) warp_max_error<true, BS>(P, sc, err, err_slot);
        else worst = fmax(worst, err);
    });
    if (!BATCH) warp_max_error<false, BS>(P, -1, worst, err_slot);
}

// The pair (i, j) of the pressure force: (pV_i + pV_j) (1-u)^2 x^ into acc.
template <bool REF>
__device__ __forceinline__ void add_pressure_pair(const Params& P, float4 xi, float4 xj, float pVi, float2 rj, float ir0,
                                                  float3& acc) {
    const float dx = __fsub_rn(xi.x, xj.x), dy = __fsub_rn(xi.y, xj.y), dz = __fsub_rn(xi.z, xj.z);
    const float r2 = dist2(dx, dy, dz);
    if (!(r2 > 0.f)) return;
    if (!REF && __fmul_rn(r2, P.inv_h2) >= 1.f) return;
    const float rinv = rsqrtf(r2);
    const float om = spiky_om(P, r2, rinv);
    // pV_i + pV_j (config: p_j / rho0^2 fused into the sum), then products only
    const float pv = REF ? pVi + rj.y / (rj.x * rj.x) : __fmaf_rn(rj.y, ir0, pVi);
    const float s = pv * om * om * rinv;
    acc.x = __fmaf_rn(s, dx, acc.x); acc.y = __fmaf_rn(s, dy, acc.y); acc.z = __fmaf_rn(s, dz, acc.z);
}

// From the finished pressure sum of particle t: the next prediction into
// xs_next[t] and vs[t], and the candidate pressure ri committed to rp[t].
template <bool REF, bool BATCH>
__device__ __forceinline__ void pci_force_finish(const Params& P, int t, float2 ri, float3 acc,
                                                 const float4* __restrict__ vap, const float4* __restrict__ fnp,
                                                 const Soa3& xs_next, const Soa3& vs, float2* rp) {
    const float4 x0 = at(P.x0, t), vh = vap[t], f = fnp[t];
    const float3 aw = wall_accel<REF, BATCH>(P, t, x0, vh);
    const float ir = 1.f / ri.x;
    auto accel = [&](float fc, float ac, float wc) {     // f/rho + k_grad sum + wall
        return __fadd_rn(__fmaf_rn(P.k_grad, ac, __fmul_rn(fc, ir)), wc);
    };
    const float3 a = make_float3(accel(f.x, acc.x, aw.x), accel(f.y, acc.y, aw.y), accel(f.z, acc.z, aw.z));
    const float3 v = make_float3(__fmaf_rn(a.x, P.dt, vh.x), __fmaf_rn(a.y, P.dt, vh.y), __fmaf_rn(a.z, P.dt, vh.z));
    put(vs, t, v.x, v.y, v.z);
    put(xs_next, t, __fmaf_rn(v.x, P.dt, x0.x), __fmaf_rn(v.y, P.dt, x0.y), __fmaf_rn(v.z, P.dt, x0.z));
    rp[t] = ri;
}

// The pressure-force pass for sorted particle t (t < P.n, its scene still
// iterating).
template <bool REF, bool BATCH, class F2>
__device__ __forceinline__ void pci_force_at(const Params& P, int t, const float4* __restrict__ vap,
                                             const float4* __restrict__ fnp, const Soa3& xs, F2 rpc,
                                             const int* __restrict__ counts, const int* __restrict__ list,
                                             const Soa3& xs_next, const Soa3& vs, float2* rp) {
    const float4 xi = REF ? at(xs, t) : at(P.x0, t);
    const float2 ri = rpc[t];
    const float ir0 = 1.f / __fmul_rn(P.rho0, P.rho0);
    const float pVi = REF ? ri.y / __fmul_rn(ri.x, ri.x) : __fmul_rn(ri.y, ir0);
    const int cnt = min(counts[t], P.cap);
    float3 acc = make_float3(0.f, 0.f, 0.f);
    for_each_nbr(list, P.n, t, cnt, [&](const int j) {
        // the pair's gathers issue before its distance test, so a pair costs
        // one dependent load after the list, not two
        if (REF) {
            const float4 xj = at(xs, j);
            const float2 rj = rpc[j];
            add_pressure_pair<REF>(P, xi, xj, pVi, rj, ir0, acc);
        } else {
            const float2 xy = gather2(P.x0.xy + j), zp = gather2(P.zp + j);
            add_pressure_pair<REF>(P, xi, make_float4(xy.x, xy.y, zp.x, 0.f), pVi, zp, ir0, acc);
        }
    });
    if (!REF) {
        ghost_pressure<BATCH>(P, t, xi, pVi, list, cnt, acc);
        if (!BATCH) boundary_pressure(P, t, xi, pVi, acc);
    }
    pci_force_finish<REF, BATCH>(P, t, ri, acc, vap, fnp, xs_next, vs, rp);
}

// PCISPH pressure-force pass fused with the next prediction; commits the
// candidate pressure. Reference profile: at the predicted positions x*, with
// p/rho*^2 (PciSphSystem_Kernel.cu:88-114 runs on the predicted state).
// Config profile: at the step's start positions x, with p/rho0^2. That keeps
// the corrector a linear iteration in p: at x*, x* = x + dt^2 a(x*) is a
// fixed-point iteration in positions whose gain grows with p dt^2/h^2, and
// with rho* in p/rho^2 the force feeds back on the density; under a 0.64 m
// column either one makes the corrector diverge.
template <bool REF, bool BATCH, int BS>
__global__ void __launch_bounds__(BS, REF ? 1 : kForceThreads / BS) k_pci_force_predict(
    Params P, const float4* __restrict__ vap, const float4* __restrict__ fnp, Soa3 xs, const float2* __restrict__ rpc,
    const int* __restrict__ counts, const int* __restrict__ list, Soa3 xs_next, Soa3 vs, float2* __restrict__ rp) {
    after_previous();
    if (!BATCH && P.active && !P.active[0]) return;      // single scene, corrector decided on the device: converged
    for_each_slot<BS, !REF>(P, [&](const int t) {
        if (t < 0 || (BATCH && !P.active[P.slot_scene[t]])) return;     // its scene has converged
        pci_force_at<REF, BATCH>(P, t, vap, fnp, xs, rpc, counts, list, xs_next, vs, rp);
    });
}

// The whole corrector loop of a config-profile scene or batch in one
// cooperative launch: every block strides over the particles, and grid-wide
// barriers separate {density pass, decision, pressure-force pass} as kernel
// boundaries do in the graph. Block 0 takes the decision (the batch's rule,
// corrector_decide). The arrays that the passes write and the next pass
// reads (x*, the pressures, the decision's words) are read through plain
// pointers here, not the read-only path: the barrier's acquire makes other
// blocks' writes visible to ordinary loads. Same passes, same order, same
// arithmetic as the graph's loop: the results are bit-identical.
// Five resident blocks of 256 per SM (at most 48 registers, no spills),
// the occupancy of the separate pressure-force pass.
template <bool BATCH, int BS>
__global__ void __launch_bounds__(BS, 5) k_corrector_persistent(
    Params P, const float4* __restrict__ vap, const float4* __restrict__ fnp, Soa3 xs, float2* rp, float2* rpc,
    const int* __restrict__ counts, const int* __restrict__ list, Soa3 vs, unsigned long long* err_slot, int S, int min_it,
    int max_it, double eta, uint8_t* active, unsigned long long* err_scene, unsigned long long* err_hist, int* loop) {
    cg::grid_group grid = cg::this_grid();
    __shared__ double s_err[BS / 32];
    __shared__ int s_any;
    const long long stride = (long long)gridDim.x * BS;
    if (blockIdx.x == 0) corrector_begin(S, max_it, active, err_scene, err_hist, (PSB_MAX_ITERS + 1) * S, loop);
    grid.sync();
    for (int pass = 0; pass < max_it; ++pass) {
        // density pass (warp-uniform bounds: the reduction is warp-synchronous)
        double emax = -1e300;
        for (long long base = (long long)blockIdx.x * BS; base < P.n; base += stride) {
            const int t = (int)(base + threadIdx.x);
            double err = -1e300;
            const int sc = BATCH && t < P.n ? (int)P.slot_scene[t] : -1;
            const volatile uint8_t* act = active;
            if (t < P.n && (!BATCH || act[sc])) err = pci_density_at<false, BATCH>(P, t, xs, (const float2*)rp, counts, list, rpc);
            if (BATCH) reduce_error<true, BS>(P, sc, err, err_slot, s_err);
            else emax = fmax(emax, err);
        }
        if (!BATCH) reduce_error<false, BS>(P, -1, emax, err_slot, s_err);
        grid.sync();
        if (blockIdx.x == 0) corrector_decide(S, min_it, max_it, eta, active, err_scene, err_hist, loop, &s_any);
        grid.sync();
        const int cont = *(volatile int*)&loop[1];
        // pressure-force pass and the next prediction, x* in place
        for (long long base = (long long)blockIdx.x * BS; base < P.n; base += stride) {
            const int t = (int)(base + threadIdx.x);
            if (t >= P.n) continue;
            const volatile uint8_t* act = active;
            if (!act[BATCH ? (int)P.slot_scene[t] : 0]) continue;
            pci_force_at<false, BATCH>(P, t, vap, fnp, xs, (const float2*)rpc, counts, list, xs, vs, rp);
        }
        if (!cont) break;
        grid.sync();
    }
}

// Commit of the last prediction, walls, collision objects (COLL: the start
// position pos[t] is read before it is overwritten), velocity interpolation.
template <bool BATCH, bool COLL>
__global__ void __launch_bounds__(kBlock) k_pci_commit(Params P, Soa3 xs, Soa3 vs, const float2* __restrict__ rpc,
                                                       int have_density_pass, float4* __restrict__ pos,
                                                       float4* __restrict__ vel, float4* __restrict__ vap,
                                                       float2* __restrict__ rp) {
    after_previous();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= P.n) return;
    float3 x = f3(at(xs, t)), v = f3(at(vs, t));
    const float4 vh = vap[t];
    box_project<BATCH>(P, t, x, v);
    if constexpr (COLL) {
        const float4 x0 = pos[t];
        coll::V3<float> cx{x.x, x.y, x.z}, cv{v.x, v.y, v.z};
        coll::apply_colliders(P.coll, P.n_coll, P.dt, coll::V3<float>{x0.x, x0.y, x0.z}, cx, cv);
        x = make_float3(cx.x, cx.y, cx.z);
        v = make_float3(cv.x, cv.y, cv.z);
    }
    pos[t] = make_float4(x.x, x.y, x.z, 0.f);
    vap[t] = make_float4(v.x, v.y, v.z, 0.f);
    vel[t] = make_float4((vh.x + v.x) * 0.5f, (vh.y + v.y) * 0.5f, (vh.z + v.z) * 0.5f, 0.f);
    if (have_density_pass) rp[t].x = rpc[t].x;
}

// XSPH velocity smoothing (Monaghan 1989) of the committed prediction,
// config PCISPH: v_i + xsph sum_j (m/rho0) W_ij (v_j - v_i) over the list at
// x*, W the poly6 kernel (m W = k_rho (1-q)^3). Positions are not moved.
template <int BS>
__global__ void __launch_bounds__(BS) k_xsph(Params P, Soa3 xs, Soa3 vs, const int* __restrict__ counts,
                                                 const int* __restrict__ list, Soa3 vs_out) {
    after_previous();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= P.n) return;
    const float4 xi = at(xs, t), vi = at(vs, t);
    const int cnt = min(counts[t], P.cap);
    float3 dv = make_float3(0.f, 0.f, 0.f);
    for_each_nbr(list, P.n, t, cnt, [&](const int j) {
        const float4 xj = at(xs, j), vj = at(vs, j);
        const float dx = xi.x - xj.x, dy = xi.y - xj.y, dz = xi.z - xj.z;
        const float q = dist2(dx, dy, dz) * P.inv_h2;
        if (q >= 1.f) return;
        const float w = (1.f - q) * (1.f - q) * (1.f - q);
        dv.x += w * (vj.x - vi.x); dv.y += w * (vj.y - vi.y); dv.z += w * (vj.z - vi.z);
    });
    put(vs_out, t, vi.x + P.xsph_k * dv.x, vi.y + P.xsph_k * dv.y, vi.z + P.xsph_k * dv.z);
}

inline int grid_of(int n) { return (n + kBlock - 1) / kBlock; }

}  // namespace

// Kernels are specialised on the physics profile (REF), on batching
// (P.scenes set: per-scene boxes and convergence; config profile only) and
// on the tuned block size.
template <int BS>
inline unsigned blocks_of(int n) { return (unsigned)((n + BS - 1) / BS); }

// P with its wall blocks for launches of BS threads. The list's length is
// only known on the device: threads for a quarter of the particles (scenes
// of 100k to 4M list 4 to 25%), 148 x 1024 at most (blocks that find nothing
// to do cost ~2 ns each); a longer list is strided over.
template <int BS>
inline Params with_walls(const Params& P, bool ghosts = true) {
    Params Q = P;
    const bool list = ghosts && P.wall_list && P.n >= kWallListMin;
    Q.wall_blocks = list ? std::min(148 * 1024 / BS, (P.n / 4 + BS - 1) / BS) : 0;
    return Q;
}

void launch_density_x(cudaStream_t st, const Params& P, const int* counts, const int* list, float2* rp, float* rho_x,
                      int zero_p, float p_scale, float* feats, int nfeat) {
    if (P.n <= 0) return;
    with_block(P.tune.density_block, [&](auto B) {
        constexpr int BS = decltype(B)::value;
        const Params Q = with_walls<BS>(P);
        auto go = [&](auto kernel) {
            launch_chained(kernel, blocks_of<BS>(P.n) + Q.wall_blocks, BS, 0, st, Q, counts, list, rp, rho_x, zero_p,
                           p_scale, feats);
        };
        const int nf = feats ? (nfeat > 6 ? 7 : 6) : 0;
        if (P.ref) go(k_density_x<true, 0, false, BS>);
        else if (P.scenes) {
            if (nf == 7) go(k_density_x<false, 7, true, BS>);
            else if (nf == 6) go(k_density_x<false, 6, true, BS>);
            else go(k_density_x<false, 0, true, BS>);
        } else if (nf == 7) go(k_density_x<false, 7, false, BS>);
        else if (nf == 6) go(k_density_x<false, 6, false, BS>);
        else go(k_density_x<false, 0, false, BS>);
    });
}

void launch_build_density(cudaStream_t st, const Params& P, const float4* pos, const uint32_t* keys,
                          const uint32_t* cell_start, const uint32_t* cell_end, int* counts, int* list, int* flags,
                          float2* rp, float* rho_x, int zero_p, float p_scale, float* feats, int nfeat) {
    if (P.n <= 0) return;
    with_block(P.tune.nbr_block, [&](auto B) {
        constexpr int BS = decltype(B)::value;
        auto go = [&](auto kernel) {
            launch_chained(kernel, blocks_of<BS>(P.n), BS, 0, st, P, pos, keys, cell_start, cell_end, counts, list,
                           flags, rp, rho_x, zero_p, p_scale, feats);
        };
        const int nf = feats ? (nfeat > 6 ? 7 : 6) : 0;
        if (nf == 7) go(k_build_density<7, BS>);
        else if (nf == 6) go(k_build_density<6, BS>);
        else go(k_build_density<0, BS>);
    });
}

void launch_wcsph_force(cudaStream_t st, const Params& P, const float4* vap, const float2* rp, const int* counts,
                        const int* list, float4* pos_out, float4* vel_out,
                        float4* vap_out, float4* fnp) {
    if (P.n <= 0) return;
    const Params Q = with_walls<kBlock>(P);
    auto kernel = P.ref ? k_wcsph_force<true> : k_wcsph_force<false>;
    launch_chained(kernel, grid_of(P.n) + Q.wall_blocks, kBlock, 0, st, Q, vap, rp, counts, list, pos_out, vel_out,
                   vap_out, fnp);
}

void launch_pci_init(cudaStream_t st, const Params& P, const float4* vap, const float2* rp, const int* counts,
                     const int* list, int warm, float4* fnp, Soa3 xs, Soa3 vs) {
    if (P.n <= 0) return;
    with_block(P.tune.init_block, [&](auto B) {
        constexpr int BS = decltype(B)::value;
        const Params Q = with_walls<BS>(P, warm != 0);
        auto go = [&](auto kernel) {
            launch_chained(kernel, blocks_of<BS>(P.n) + Q.wall_blocks, BS, 0, st, Q, vap, rp, counts, list, fnp, xs,
                           vs);
        };
        if (P.ref) { if (warm) go(k_pci_init<true, true, false, BS>); else go(k_pci_init<true, false, false, BS>); }
        else if (P.scenes) { if (warm) go(k_pci_init<false, true, true, BS>); else go(k_pci_init<false, false, true, BS>); }
        else if (warm) go(k_pci_init<false, true, false, BS>);
        else go(k_pci_init<false, false, false, BS>);
    });
}

void launch_pci_density(cudaStream_t st, const Params& P, Soa3 xs, const float2* rp, const int* counts, const int* list,
                        float2* rpc, unsigned long long* err_slot) {
    if (P.n <= 0) return;
    with_block(P.tune.pci_density_block, [&](auto B) {
        constexpr int BS = decltype(B)::value;
        const Params Q = with_walls<BS>(P);
        auto go = [&](auto kernel) {
            launch_chained(kernel, blocks_of<BS>(P.n) + Q.wall_blocks, BS, 0, st, Q, xs, rp, counts, list, rpc,
                           err_slot);
        };
        if (P.ref) go(k_pci_density<true, false, BS>);
        else if (P.scenes) go(k_pci_density<false, true, BS>);
        else go(k_pci_density<false, false, BS>);
    });
}

cudaError_t launch_corrector_persistent(cudaStream_t st, const Params& P, const float4* vap, const float4* fnp, Soa3 xs,
                                        float2* rp, float2* rpc, const int* counts, const int* list, Soa3 vs, int S, int min_it, int max_it, double eta,
                                        uint8_t* active, unsigned long long* err_scene, unsigned long long* err_hist,
                                        int* loop) {
    constexpr int BS = 256;
    auto go = [&](auto kernel) -> cudaError_t {
        int dev = 0, sms = 0, per_sm = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, BS, 0);
        if (e != cudaSuccess) return e;
        if (per_sm < 1) return cudaErrorCooperativeLaunchTooLarge;
        // every block resident at once (the grid barrier needs it), no more
        // blocks than the particles fill
        const long long need = ((long long)P.n + BS - 1) / BS;
        const int grid = (int)std::max(1LL, std::min<long long>((long long)per_sm * sms, need));
        unsigned long long* err_slot = err_scene;
        cudaLaunchConfig_t cfg{};
        cfg.gridDim = dim3(grid);
        cfg.blockDim = dim3(BS);
        cfg.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        return cudaLaunchKernelEx(&cfg, kernel, P, vap, fnp, xs, rp, rpc, counts, list, vs, err_slot, S, min_it,
                                  max_it, eta, active, err_scene, err_hist, loop);
    };
    if (P.ref) return cudaErrorInvalidValue;
    return P.scenes ? go(k_corrector_persistent<true, BS>) : go(k_corrector_persistent<false, BS>);
}

void launch_pci_force_predict(cudaStream_t st, const Params& P, const float4* vap, const float4* fnp, Soa3 xs,
                              const float2* rpc, const int* counts, const int* list, Soa3 xs_next, Soa3 vs, float2* rp) {
    if (P.n <= 0) return;
    with_block(P.tune.force_block, [&](auto B) {
        constexpr int BS = decltype(B)::value;
        const Params Q = with_walls<BS>(P);
        auto go = [&](auto kernel) {
            launch_chained(kernel, blocks_of<BS>(P.n) + Q.wall_blocks, BS, 0, st, Q, vap, fnp, xs, rpc, counts, list,
                           xs_next, vs, rp);
        };
        if (P.ref) go(k_pci_force_predict<true, false, BS>);
        else if (P.scenes) go(k_pci_force_predict<false, true, BS>);
        else go(k_pci_force_predict<false, false, BS>);
    });
}

void launch_xsph(cudaStream_t st, const Params& P, Soa3 xs, Soa3 vs, const int* counts, const int* list, Soa3 vs_out) {
    if (P.n <= 0) return;
    with_block(P.tune.xsph_block, [&](auto B) {
        constexpr int BS = decltype(B)::value;
        k_xsph<BS><<<blocks_of<BS>(P.n), BS, 0, st>>>(P, xs, vs, counts, list, vs_out);
    });
}

void launch_pci_commit(cudaStream_t st, const Params& P, Soa3 xs, Soa3 vs, const float2* rpc,
                       int have_density_pass, float4* pos, float4* vel, float4* vap, float2* rp) {
    if (P.n <= 0) return;
    if (P.scenes)
        k_pci_commit<true, false><<<grid_of(P.n), kBlock, 0, st>>>(P, xs, vs, rpc, have_density_pass, pos, vel, vap, rp);
    else if (P.n_coll > 0)
        k_pci_commit<false, true><<<grid_of(P.n), kBlock, 0, st>>>(P, xs, vs, rpc, have_density_pass, pos, vel, vap, rp);
    else k_pci_commit<false, false><<<grid_of(P.n), kBlock, 0, st>>>(P, xs, vs, rpc, have_density_pass, pos, vel, vap, rp);
}

}  // namespace psb
