// mc.cu -- iso field on a node grid and marching-cubes surface extraction.
//
// Iso field (a thread per node or per brick of nodes, gathered over the
// particle grid's cell rings, FP64 accumulation):
//   reference profile: evaluateIso_Kernel (UniformGridKernel.cu:98-138):
//     r = h / scale, ring = floor(1/scale) cells,
//     iso(x) = sum_{|x - x_j| <= r} (1/r^6) (r^2 - d^2)^3, each term in float
//     as the reference's powf computes it;
//   config profile: the density-based colour field
//     c(x) = sum_j (m / rho_j) W_poly6(|x - x_j|, h), ring = 1 cell.
//
// Marching cubes (polygonize_MarchingCube_Kernel, MarchingCube_Kernel.cu:36-
// 160): corners and edges numbered as there, case bit c set when
// iso(corner c) <= level, vertices on the edges by linear interpolation with
// the reference's 1e-6 guards. The reference keeps 15 vertex slots per cell
// and welds vertices on the host in O(V^2) (SurfaceSPH.cpp:120-186); here
// every active grid edge owns one vertex, so the mesh is welded by
// construction. Vertices and triangles are counted per block of nodes, one scan
// over the blocks gives each block its first of both, and a second pass ranks
// inside the block again and writes them compacted.
//
// The triangle table is generated here, not copied: for each of the 256
// cases the active edges of every cube face are joined into segments (a face
// with four active edges separates its two set corners), the segments close
// into loops on the cube surface, each loop is oriented so that its normal
// points toward the set corners (iso <= level, the outside of a fluid) and
// fanned into triangles. The face rule depends only on the face's four
// corners, so neighbouring cubes agree on every shared face and the surface
// is closed wherever the field is.
#include <cuda_runtime.h>
#include <algorithm>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstdint>
#include <cstring>
#include <vector>

#include "psb_internal.cuh"

namespace psb {

namespace {

// Corner c at (x, y, z) offsets; edges as corner pairs (the reference's numbering).
#define PSB_MC_CORNERS {{0, 0, 0}, {1, 0, 0}, {1, 0, 1}, {0, 0, 1}, {0, 1, 0}, {1, 1, 0}, {1, 1, 1}, {0, 1, 1}}
#define PSB_MC_EDGES {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6}, {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}}
constexpr int kCorner[8][3] = PSB_MC_CORNERS;
constexpr int kEdge[12][2] = PSB_MC_EDGES;
constexpr int kFace[6][4] = {{0, 1, 2, 3}, {4, 5, 6, 7}, {0, 3, 7, 4}, {1, 2, 6, 5}, {0, 1, 5, 4}, {3, 2, 6, 7}};
__constant__ int c_corner[8][3] = PSB_MC_CORNERS;
__constant__ int c_edge[12][2] = PSB_MC_EDGES;

// For each edge, 5 bits: the corner offset of its lower node (x, y, z) and its axis.
constexpr uint64_t edge_pack() {
    uint64_t p = 0;
    for (int e = 0; e < 12; ++e) {
        const int* a = kCorner[kEdge[e][0]];
        const int* b = kCorner[kEdge[e][1]];
        const int* lo = a[0] + a[1] + a[2] <= b[0] + b[1] + b[2] ? a : b;
        const int* hi = lo == a ? b : a;
        const int axis = hi[0] != lo[0] ? 0 : (hi[1] != lo[1] ? 1 : 2);
        p |= (uint64_t)(lo[0] | lo[1] << 1 | lo[2] << 2 | axis << 3) << (5 * e);
    }
    return p;
}
constexpr uint64_t kEdgePack = edge_pack();

__constant__ int8_t c_tri[256][kMcMaxTri * 3];
// The same table in global memory: the lanes of a warp read different cases,
// which constant memory serves one at a time.
__device__ int8_t g_tri[256][kMcMaxTri * 3];
__constant__ uint8_t c_ntri[256];

int edge_of(int a, int b) {
    for (int e = 0; e < 12; ++e)
        if ((kEdge[e][0] == a && kEdge[e][1] == b) || (kEdge[e][0] == b && kEdge[e][1] == a)) return e;
    return -1;
}

}  // namespace

void mc_build_table(uint8_t ntri[256], int8_t tri[256][kMcMaxTri * 3]) {
    for (int cs = 0; cs < 256; ++cs) {
        ntri[cs] = 0;
        std::memset(tri[cs], -1, kMcMaxTri * 3);
        auto set = [&](int c) { return (cs >> c) & 1; };
        int link[12][2];
        int deg[12] = {0};
        auto join = [&](int e0, int e1) {
            link[e0][deg[e0]++] = e1;
            link[e1][deg[e1]++] = e0;
        };
        for (int f = 0; f < 6; ++f) {
            const int* q = kFace[f];
            int act[4], na = 0;
            for (int k = 0; k < 4; ++k) {
                const int a = q[k], b = q[(k + 1) & 3];
                if (set(a) != set(b)) act[na++] = edge_of(a, b);
            }
            if (na == 2) {
                join(act[0], act[1]);
            } else if (na == 4) {          // separate each set corner from the rest
                for (int k = 0; k < 4; ++k) {
                    if (!set(q[k])) continue;
                    join(edge_of(q[(k + 3) & 3], q[k]), edge_of(q[k], q[(k + 1) & 3]));
                }
            }
        }
        bool used[12] = {false};
        int nt = 0;
        for (int start = 0; start < 12; ++start) {
            if (deg[start] != 2 || used[start]) continue;
            int loop[12], nl = 0, prev = -1, cur = start;
            do {
                loop[nl++] = cur;
                used[cur] = true;
                const int nxt = link[cur][0] != prev ? link[cur][0] : link[cur][1];
                prev = cur;
                cur = nxt;
            } while (cur != start && nl < 12);
            // orientation: Newell normal of the edge-midpoint polygon against
            // the direction from unset to set corners across the loop's edges
            double nrm[3] = {0, 0, 0}, dir[3] = {0, 0, 0};
            double mid[12][3];
            for (int k = 0; k < nl; ++k) {
                const int a = kEdge[loop[k]][0], b = kEdge[loop[k]][1];
                for (int d = 0; d < 3; ++d) mid[k][d] = 0.5 * (kCorner[a][d] + kCorner[b][d]);
                const int s = set(a) ? a : b, u = set(a) ? b : a;
                for (int d = 0; d < 3; ++d) dir[d] += kCorner[s][d] - kCorner[u][d];
            }
            for (int k = 0; k < nl; ++k) {
                const double* p = mid[k];
                const double* r = mid[(k + 1) % nl];
                nrm[0] += (p[1] - r[1]) * (p[2] + r[2]);
                nrm[1] += (p[2] - r[2]) * (p[0] + r[0]);
                nrm[2] += (p[0] - r[0]) * (p[1] + r[1]);
            }
            const bool flip = nrm[0] * dir[0] + nrm[1] * dir[1] + nrm[2] * dir[2] < 0;
            for (int k = 1; k + 1 < nl; ++k) {
                int v0 = loop[0], v1 = loop[k], v2 = loop[k + 1];
                if (flip) { const int t = v1; v1 = v2; v2 = t; }
                tri[cs][3 * nt + 0] = (int8_t)v0;
                tri[cs][3 * nt + 1] = (int8_t)v1;
                tri[cs][3 * nt + 2] = (int8_t)v2;
                ++nt;
            }
        }
        ntri[cs] = (uint8_t)nt;
    }
}

namespace {

// ---- iso field ----------------------------------------------------------------
// k_colour / rho_j of every particle (config profile): the division once a
// particle rather than once a (node, particle) pair.
__global__ void k_iso_weight(int n, double k_colour, const float2* __restrict__ rp, double* __restrict__ w) {
    after_previous();
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < n) w[t] = k_colour / (double)rp[t].x;
}

// A thread takes a brick of E^3 nodes, a warp 4 x 2 x 4 threads, a block 1 x 2
// x 2 warps. The cells of a grid row are adjacent in slot order, so the rings
// of a thread's nodes are a few contiguous slot ranges. The sums are FP64, but
// 85% of a ring's particles lie outside the radius: those are dropped by an
// FP32 test against the nearest of the thread's nodes, with a margin over its
// own rounding (32 candidates to a mask), and only the rest, in order, see the
// FP64 distances. Config profile: a particle within the radius lies in the
// node's ring unless it was clamped into a border cell from outside the grid
// (or has a NaN coordinate), so going over the union of several rings adds
// nothing to any of them, and a candidate is loaded once for eight nodes. A
// warp with a brick whose nodes lie in different cells and whose rings reach a
// border cell adds a candidate to the nodes whose own ring holds it (OWN): the
// field at a node does not depend on the nodes it is asked for with. The field was bound
// by L1 wavefronts (93% of the data pipe with a node a thread, FP64 17%):
// 128^3 nodes over 262,144 particles took 518 us in node order with every
// candidate in FP64, 475 with the FP32 test, 412 with a warp's nodes in a
// brick, 273 with 2 x 2 x 1 nodes a thread, 247 with 2 x 2 x 2, 215 with the
// FP32 test axis by axis instead of over the eight nodes. Nodes further
// apart than half a cell share too little and take a thread each, and so do
// the nodes of grids too small to fill the chip with eighths, and the reference
// profile's, whose ring may cut the radius off. A node a thread against eight,
// spacing 0.3-0.5 / 0.15-0.4 of a cell: 48^3 nodes - / 56 against 72 us, 56^3 94 / 70
// against 100 / 84, 64^3 119 / 91 against 91 / 87, 74^3 151 / 128 against 104 / 97,
// 80^3 170 / 143 against 105 / 89: from 262,144 nodes on eight are the faster;
// the line lies above that.
constexpr long long kIsoBrickNodes = 393216;

template <bool REF, int E>
__global__ void __launch_bounds__(128) k_iso_field(IsoParams Q, Params P, const float4* __restrict__ pos,
                                                   const double* __restrict__ weight,
                                                   const uint32_t* __restrict__ cell_start,
                                                   const uint32_t* __restrict__ cell_end, double* __restrict__ iso) {
    after_previous();
    const int l = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const unsigned bx = (Q.dims[0] + 4 * E - 1) / (4 * E), by = (Q.dims[1] + 4 * E - 1) / (4 * E);
    const int ix = ((int)(blockIdx.x % bx) * 4 + (l & 3)) * E;
    const int iy = ((int)(blockIdx.x / bx % by) * 4 + (wp & 1) * 2 + (l >> 2 & 1)) * E;
    const int iz = ((int)(blockIdx.x / (bx * by)) * 8 + (wp >> 1) * 4 + (l >> 3)) * E;
    if (ix >= Q.dims[0] || iy >= Q.dims[1] || iz >= Q.dims[2]) return;
    double px[E], py[E], pz[E];
    float fx[E], fy[E], fz[E];
    int I[E], J[E], K[E];
    int lo_x = INT_MAX, hi_x = INT_MIN, lo_y = INT_MAX, hi_y = INT_MIN, lo_z = INT_MAX, hi_z = INT_MIN;
    // particle-grid cells of the nodes, as the reference computes them
    float far = 0.f;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        px[e] = Q.origin[0] + (ix + e) * Q.spacing[0];
        py[e] = Q.origin[1] + (iy + e) * Q.spacing[1];
        I[e] = (int)floor((px[e] - (double)P.g.gx) / (double)P.g.cell);
        J[e] = (int)floor((py[e] - (double)P.g.gy) / (double)P.g.cell);
        pz[e] = Q.origin[2] + (iz + e) * Q.spacing[2];
        K[e] = (int)floor((pz[e] - (double)P.g.gz) / (double)P.g.cell);
        lo_x = min(lo_x, I[e]); hi_x = max(hi_x, I[e]);
        lo_y = min(lo_y, J[e]); hi_y = max(hi_y, J[e]);
        lo_z = min(lo_z, K[e]); hi_z = max(hi_z, K[e]);
        fx[e] = (float)px[e];
        fy[e] = (float)py[e];
        fz[e] = (float)pz[e];
        far = fmaxf(far, fmaxf(fmaxf(fabsf(fx[e]), fabsf(fy[e])), fabsf(fz[e])));
    }
    const int ring = Q.ring;
    const int a0 = max(lo_x - ring, 0), a1 = min(hi_x + ring, P.g.nx - 1);
    double acc[E][E][E] = {};
    // radius of the FP32 test: a node and a particle within the ring are each
    // rounded by at most 2^-24 of their largest coordinate
    far += (float)(ring + 1) * P.g.cell;
    const float reach = (float)Q.r * 1.0001f + far * 5e-7f;
    const float r2 = -(reach * reach);
    const int k0 = max(lo_z - ring, 0), j0 = max(lo_y - ring, 0);
    const int k1 = min(hi_z + ring, P.g.nz - 1), j1 = min(hi_y + ring, P.g.ny - 1);
    // slots of cells i0..i1 of a row (none: i0 > i1)
    auto slots = [&](uint32_t row, int i0, int i1, uint32_t& lo, uint32_t& hi) {
        lo = hi = 0u;
        if (i0 > i1) return;
        if (P.dense_cells) {
            lo = cell_start[row + i0];
            hi = cell_end[row + i1];
        } else {
            row_range(cell_start, cell_end, row, i0, i1, lo, hi);
        }
    };
    auto rows = [&](auto own) {
        constexpr bool OWN = decltype(own)::value;
        for (int k = k0; k <= k1 && a0 <= a1; ++k) {
            for (int j = j0; j <= j1; ++j) {
                const uint32_t row = (uint32_t)j * P.g.nx + (uint32_t)k * P.g.nx * P.g.ny;
                uint32_t lo, hi, first[E], end[E];      // first, end: the part of the row in node e's own ring
                bool in_y[E], in_z[E];
                slots(row, a0, a1, lo, hi);
                if (OWN) {
#pragma unroll
                    for (int e = 0; e < E; ++e) {
                        in_y[e] = abs(j - J[e]) <= ring;
                        in_z[e] = abs(k - K[e]) <= ring;
                        slots(row, max(I[e] - ring, 0), min(I[e] + ring, P.g.nx - 1), first[e], end[e]);
                    }
                }
                for (; lo < hi; lo += 32u) {
                    const uint32_t m = min(hi - lo, 32u);
                    uint32_t mask = 0u;
                    for (uint32_t c = 0; c < m; c += 2) {
#pragma unroll
                        for (uint32_t u = 0; u < 2; ++u) {
                            const float4 x = pos[lo + c + u];       // padded past the last particle
                            // the nearest node's distance: the nearest on each axis, as rounding is monotonic
                            float dx = fabsf(fx[0] - x.x), dy = fabsf(fy[0] - x.y), dz = fabsf(fz[0] - x.z);
#pragma unroll
                            for (int e = 1; e < E; ++e) {
                                dx = fminf(dx, fabsf(fx[e] - x.x));
                                dy = fminf(dy, fabsf(fy[e] - x.y));
                                dz = fminf(dz, fabsf(fz[e] - x.z));
                            }
                            const float best = __fmaf_rn(dx, dx, __fmaf_rn(dy, dy, __fmaf_rn(dz, dz, r2)));
                            // a NaN position stays in, as in the FP64 test
                            const bool in = !(best >= 0.f && best < INFINITY);
                            mask = mask << 1 | (in ? 1u : 0u);
                        }
                    }
                    mask = (mask << (32u - ((m + 1u) & ~1u))) & (kEmpty << (32u - m));
                    uint32_t t = lo;
                    while (mask) {
                        const int z = __clz((int)mask);
                        mask = (mask << z) << 1;
                        t += (uint32_t)z;
                        const float4 x = pos[t];
                        if (REF) {
                            const double dx = px[0] - x.x, dy = py[0] - x.y, dz = pz[0] - x.z;
                            const double d2 = dx * dx + dy * dy + dz * dz;
                            // d = length(pos1 - pos2); (1/powf(r,6)) * powf(r*r - d*d, 3) in float
                            const double d = sqrt(d2);
                            if (d <= Q.r) {
                                const float term = (1.f / powf((float)Q.r, 6.f)) * powf((float)(Q.r * Q.r - d * d), 3.f);
                                acc[0][0][0] += (double)term;
                            }
                        } else {
                            const double wt = weight[t];
#pragma unroll
                            for (int g = 0; g < E; ++g) {
                                const double dz = pz[g] - x.z, dz2 = dz * dz;
#pragma unroll
                                for (int f = 0; f < E; ++f) {
                                    const double dy = py[f] - x.y, dy2 = dy * dy + dz2;
#pragma unroll
                                    for (int e = 0; e < E; ++e) {
                                        const double dx = px[e] - x.x;
                                        const double q = (dx * dx + dy2) * Q.inv_r2;
                                        const bool mine = !OWN || (in_z[g] && in_y[f] && t >= first[e] && t < end[e]);
                                        if (mine && !(q >= 1.0)) {
                                            const double w = 1.0 - q;
                                            acc[g][f][e] += w * w * w * wt;
                                        }
                                    }
                                }
                            }
                        }
                        ++t;
                    }
                }
            }
        }
    };
    const bool apart = lo_x != hi_x || lo_y != hi_y || lo_z != hi_z;
    const bool border = a0 == 0 || a1 == P.g.nx - 1 || j0 == 0 || j1 == P.g.ny - 1 || k0 == 0 || k1 == P.g.nz - 1;
    if (E > 1 && __any_sync(__activemask(), apart && border)) rows(std::true_type{});
    else rows(std::false_type{});
#pragma unroll
    for (int g = 0; g < E; ++g)
#pragma unroll
        for (int f = 0; f < E; ++f)
#pragma unroll
            for (int e = 0; e < E; ++e)
                if (ix + e < Q.dims[0] && iy + f < Q.dims[1] && iz + g < Q.dims[2])
                    iso[ix + e + (size_t)Q.dims[0] * (iy + f + (size_t)Q.dims[1] * (iz + g))] = acc[g][f][e];
}

// ---- marching cubes -----------------------------------------------------------
// Nodes and their coordinates fit 30 bits (psb_extract_surface's limit).
struct NodeAt {
    int x, y, z;
};
__device__ __forceinline__ NodeAt node_at(const IsoParams& Q, unsigned node) {
    const unsigned plane = node / (unsigned)Q.dims[0];
    return {(int)(node - plane * Q.dims[0]), (int)(plane % (unsigned)Q.dims[1]), (int)(plane / (unsigned)Q.dims[1])};
}

// The active edges (+x, +y, +z, bits 0-2) and the cube case (bits 8-15) of a
// node, from the corners of the cube it is the lowest node of. A node on a
// far face has no cube: case 0.
__device__ __forceinline__ unsigned node_case(const IsoParams& Q, const double* __restrict__ iso, unsigned node,
                                              const NodeAt& p) {
    const unsigned sy = Q.dims[0], sz = sy * Q.dims[1];
    const bool ix = p.x + 1 < Q.dims[0], iy = p.y + 1 < Q.dims[1], iz = p.z + 1 < Q.dims[2];
    auto in = [&](unsigned o) { return iso[o] <= Q.level; };
    const bool c0 = in(node);
    const bool cx = ix ? in(node + 1) : c0, cy = iy ? in(node + sy) : c0, cz = iz ? in(node + sz) : c0;
    unsigned r = (c0 != cx ? 1u : 0u) | (c0 != cy ? 2u : 0u) | (c0 != cz ? 4u : 0u);
    if (ix && iy && iz) {       // corners 0..7: 000 100 101 001 010 110 111 011
        unsigned cs = (c0 ? 1u : 0u) | (cx ? 2u : 0u) | (in(node + 1 + sz) ? 4u : 0u) | (cz ? 8u : 0u) |
                      (cy ? 16u : 0u) | (in(node + 1 + sy) ? 32u : 0u) | (in(node + 1 + sy + sz) ? 64u : 0u) |
                      (in(node + sy + sz) ? 128u : 0u);
        r |= cs << 8;
    }
    return r;
}

constexpr int kMcBlock = 256;

// Exclusive rank of (a, b) over the block in thread order, and the block's
// totals; both below 2^16 (at most 3 and 10 a thread).
__device__ __forceinline__ uint2 block_rank(unsigned a, unsigned b, uint2& total) {
    __shared__ unsigned s_warp[kMcBlock / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned v = a | b << 16;
    unsigned x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const unsigned y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) s_warp[warp] = x;
    __syncthreads();
    unsigned before = 0, all = 0;
#pragma unroll
    for (int w = 0; w < kMcBlock / 32; ++w) {
        if (w < warp) before += s_warp[w];
        all += s_warp[w];
    }
    total = make_uint2(all & 0xffffu, all >> 16);
    const unsigned e = before + x - v;
    return make_uint2(e & 0xffffu, e >> 16);
}

// Pass 1: every node's edge flags and cube case, and the vertices and
// triangles of each block of nodes. The offsets are scanned over the blocks
// alone (a word each for 256 nodes); pass 2 ranks inside a block again. A
// count per edge and per cube, scanned in full, was 33 MB of counters on
// 128^3 nodes: 31 us to write, 75 to scan and 85 for an emission pass with a
// thread per edge.
__global__ void __launch_bounds__(kMcBlock) k_mc_classify(IsoParams Q, const double* __restrict__ iso,
                                                          uint16_t* __restrict__ cases,
                                                          uint32_t* __restrict__ block_vert,
                                                          uint32_t* __restrict__ block_tri) {
    after_previous();
    const unsigned nn = (unsigned)Q.dims[0] * Q.dims[1] * Q.dims[2];
    const unsigned node = blockIdx.x * kMcBlock + threadIdx.x;
    unsigned nv = 0, nt = 0;
    if (node < nn) {
        const unsigned r = node_case(Q, iso, node, node_at(Q, node));
        cases[node] = (uint16_t)r;
        nv = __popc(r & 7u);
        nt = c_ntri[r >> 8];
    }
    uint2 total;
    block_rank(nv, nt, total);
    if (threadIdx.x == 0) {
        block_vert[blockIdx.x] = total.x;
        block_tri[blockIdx.x] = total.y;
        if (blockIdx.x == gridDim.x - 1) block_vert[gridDim.x] = block_tri[gridDim.x] = 0u;     // their scans' totals
    }
}

// vertexInterpolate_MarchingCube (MarchingCube_Kernel.cu:143-155)
__device__ __forceinline__ double interp(double level, double v1, double v2, double p1, double p2) {
    if (fabs(level - v1) < 0.000001) return p1;
    if (fabs(level - v2) < 0.000001) return p2;
    if (fabs(v1 - v2) < 0.000001) return p1;
    const double mu = (level - v1) / (v2 - v1);
    return p1 + mu * (p2 - p1);
}

// Pass 2: the vertices of a node's active edges, and the index of its first.
__global__ void __launch_bounds__(kMcBlock) k_mc_vertices(IsoParams Q, const double* __restrict__ iso,
                                                          const uint16_t* __restrict__ cases,
                                                          const uint32_t* __restrict__ block_vert,
                                                          uint32_t* __restrict__ first, float* __restrict__ vert) {
    after_previous();
    const unsigned nn = (unsigned)Q.dims[0] * Q.dims[1] * Q.dims[2];
    const unsigned node = blockIdx.x * kMcBlock + threadIdx.x;
    if (block_vert[blockIdx.x + 1] == block_vert[blockIdx.x]) return;       // no active edge in the block
    const unsigned edges = node < nn ? cases[node] & 7u : 0u;
    uint2 total;
    uint32_t o = block_vert[blockIdx.x] + block_rank(__popc(edges), 0u, total).x;
    if (!edges) return;
    first[node] = o;
    const NodeAt n = node_at(Q, node);
    const double p[3] = {Q.origin[0] + n.x * Q.spacing[0], Q.origin[1] + n.y * Q.spacing[1],
                         Q.origin[2] + n.z * Q.spacing[2]};
    const unsigned step[3] = {1u, (unsigned)Q.dims[0], (unsigned)Q.dims[0] * Q.dims[1]};
    const double v1 = iso[node];
#pragma unroll
    for (int axis = 0; axis < 3; ++axis) {
        if (!(edges >> axis & 1u)) continue;
        const double v2 = iso[node + step[axis]];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            const double q = d == axis ? p[d] + Q.spacing[d] : p[d];
            vert[3 * (size_t)o + d] = (float)interp(Q.level, v1, v2, p[d], q);
        }
        ++o;
    }
}

// Vertex index of cube edge e of the cube whose lowest node is `node`: the
// edge's own lower node's first vertex plus its active edges of lower axes.
__device__ __forceinline__ uint32_t edge_vertex(const IsoParams& Q, const uint16_t* __restrict__ cases,
                                                const uint32_t* __restrict__ first, unsigned node, int e) {
    const unsigned p = (unsigned)(kEdgePack >> (5 * e));
    const unsigned m = node + (p & 1u) + (p >> 1 & 1u) * Q.dims[0] + (p >> 2 & 1u) * (unsigned)Q.dims[0] * Q.dims[1];
    return first[m] + __popc(cases[m] & ((1u << (p >> 3 & 3u)) - 1u));
}

__global__ void __launch_bounds__(kMcBlock) k_mc_triangles(IsoParams Q, const uint16_t* __restrict__ cases,
                                                           const uint32_t* __restrict__ block_tri,
                                                           const uint32_t* __restrict__ first,
                                                           int32_t* __restrict__ tris) {
    after_previous();
    const unsigned nn = (unsigned)Q.dims[0] * Q.dims[1] * Q.dims[2];
    const unsigned node = blockIdx.x * kMcBlock + threadIdx.x;
    if (block_tri[blockIdx.x + 1] == block_tri[blockIdx.x]) return;
    const int cs = node < nn ? cases[node] >> 8 : 0;
    const int nt = c_ntri[cs];
    uint2 total;
    // the triangles' counts are scanned behind the vertices': less their total
    int32_t* __restrict__ out = tris + 3 * (size_t)(block_tri[blockIdx.x] - block_tri[0] + block_rank(0u, nt, total).y);
    for (int k = 0; k < 3 * nt; ++k) out[k] = (int32_t)edge_vertex(Q, cases, first, node, g_tri[cs][k]);
}

// polygonize_MarchingCube_Kernel (MarchingCube_Kernel.cu:36-139) on the
// reference's layout: nodes are double4 (x, y, z, value); every cube with a
// triangle appends its triangles' vertices, three per triangle, to its own
// `slots` vertex slots (vertex[c * slots + k], index[c * slots + k] = k) and
// counts them in count[c], which it reads first (the reference accumulates).
// Vertices are interpolated on the cube's edges in the reference's corner
// order; a cube whose slots would overflow stops and raises *overflow.
__global__ void k_mc_polygonize_slots(const double* __restrict__ node4, int nx, int ny, int nz, double level,
                                      int* __restrict__ count, double* __restrict__ vertex, int* __restrict__ index,
                                      int slots, int* __restrict__ overflow) {
    const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= (long long)nx * ny * nz) return;
    const int x = (int)(c % nx), y = (int)((c / nx) % ny), z = (int)(c / ((long long)nx * ny));
    if (x + 1 >= nx || y + 1 >= ny || z + 1 >= nz) return;
    long long corner[8];
    int cs = 0;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        corner[k] = (x + c_corner[k][0]) + (long long)(y + c_corner[k][1]) * nx +
                    (long long)(z + c_corner[k][2]) * nx * ny;
        if (node4[4 * corner[k] + 3] <= level) cs |= 1 << k;
    }
    const int nt = c_ntri[cs];
    if (nt == 0) return;
    int m = count[c];
    for (int t = 0; t < nt; ++t)
        for (int v = 0; v < 3; ++v) {
            if (m < 0 || m >= slots) { *overflow = 1; count[c] = m; return; }
            const int e = c_tri[cs][3 * t + v];
            const long long a = corner[c_edge[e][0]], b = corner[c_edge[e][1]];
            const double va = node4[4 * a + 3], vb = node4[4 * b + 3];
            double* out = vertex + 3 * ((size_t)c * slots + m);
            for (int d = 0; d < 3; ++d) out[d] = interp(level, va, vb, node4[4 * a + d], node4[4 * b + d]);
            index[(size_t)c * slots + m] = m;
            ++m;
        }
    count[c] = m;
}

// ---- exclusive scan of uint32 (three-level, 1024 items per block) ------------
constexpr int kScanThreads = 256, kScanItems = 4, kScanTile = kScanThreads * kScanItems;

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(long long n, uint32_t* __restrict__ data,
                                                             uint32_t* __restrict__ tile_sums) {
    __shared__ uint32_t s[kScanThreads];
    const long long base = (long long)blockIdx.x * kScanTile + (long long)threadIdx.x * kScanItems;
    uint32_t v[kScanItems], tot = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < n ? data[base + k] : 0u;
        tot += v[k];
    }
    s[threadIdx.x] = tot;
    __syncthreads();
    for (int off = 1; off < kScanThreads; off <<= 1) {     // Hillis-Steele over the thread totals
        const uint32_t add = threadIdx.x >= off ? s[threadIdx.x - off] : 0u;
        __syncthreads();
        s[threadIdx.x] += add;
        __syncthreads();
    }
    uint32_t run = s[threadIdx.x] - tot;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) data[base + k] = run;
        run += v[k];
    }
    if (threadIdx.x == kScanThreads - 1 && tile_sums) tile_sums[blockIdx.x] = s[threadIdx.x];
}

__global__ void k_scan_add(long long n, uint32_t* __restrict__ data, const uint32_t* __restrict__ tile_offsets) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) data[i] += tile_offsets[i / kScanTile];
}

inline unsigned blocks_for(long long n, int t) { return (unsigned)((n + t - 1) / t); }

}  // namespace

void launch_mc_polygonize_slots(cudaStream_t st, const double* node4, int nx, int ny, int nz, double level, int* count,
                                double* vertex, int* index, int slots) {
    static int* d_overflow = nullptr;
    if (!d_overflow && cudaMalloc((void**)&d_overflow, sizeof(int)) != cudaSuccess) {
        cudaGetLastError();
        d_overflow = nullptr;
    }
    int* flag = d_overflow;
    if (!flag) return;
    cudaMemsetAsync(flag, 0, sizeof(int), st);
    const long long nn = (long long)nx * ny * nz;
    k_mc_polygonize_slots<<<blocks_for(nn, 256), 256, 0, st>>>(node4, nx, ny, nz, level, count, vertex, index, slots,
                                                               flag);
    int h = 0;
    cudaMemcpyAsync(&h, flag, sizeof(int), cudaMemcpyDeviceToHost, st);
    cudaStreamSynchronize(st);
    if (h) std::fprintf(stderr, "polygonize_MarchingCube_CUDA: a cell needed more than %d vertex slots (stopped there)\n",
                        slots);
}

void mc_upload_table(cudaStream_t st) {
    static uint8_t ntri[256];
    static int8_t tri[256][kMcMaxTri * 3];
    static bool built = false;
    if (!built) {
        mc_build_table(ntri, tri);
        built = true;
    }
    cudaMemcpyToSymbolAsync(c_ntri, ntri, sizeof(ntri), 0, cudaMemcpyHostToDevice, st);
    cudaMemcpyToSymbolAsync(c_tri, tri, sizeof(tri), 0, cudaMemcpyHostToDevice, st);
    cudaMemcpyToSymbolAsync(g_tri, tri, sizeof(tri), 0, cudaMemcpyHostToDevice, st);
}

long long scan_scratch_words(long long n) {
    const long long t1 = (n + kScanTile - 1) / kScanTile;
    const long long t2 = (t1 + kScanTile - 1) / kScanTile;
    return t1 + t2 + 1;
}

void scan_exclusive_u32(cudaStream_t st, long long n, uint32_t* data, uint32_t* scratch) {
    if (n <= 0) return;
    const long long t1 = (n + kScanTile - 1) / kScanTile;
    uint32_t* s1 = scratch;
    uint32_t* s2 = scratch + t1;
    k_scan_tiles<<<(unsigned)t1, kScanThreads, 0, st>>>(n, data, s1);
    if (t1 > 1) {
        const long long t2 = (t1 + kScanTile - 1) / kScanTile;
        k_scan_tiles<<<(unsigned)t2, kScanThreads, 0, st>>>(t1, s1, s2);
        if (t2 > 1) {   // t2 <= kScanTile while n < 2^30
            k_scan_tiles<<<1, kScanThreads, 0, st>>>(t2, s2, nullptr);
            k_scan_add<<<blocks_for(t1, 256), 256, 0, st>>>(t1, s1, s2);
        }
        k_scan_add<<<blocks_for(n, 256), 256, 0, st>>>(n, data, s1);
    }
}

void launch_iso_field(cudaStream_t st, const IsoParams& Q, const Params& P, const float4* pos, const float2* rp,
                      const uint32_t* cell_start, const uint32_t* cell_end, double* weight, double* iso) {
    const long long nn = (long long)Q.dims[0] * Q.dims[1] * Q.dims[2];
    if (nn <= 0) return;
    if (!P.ref) k_iso_weight<<<blocks_for(P.n, 256), 256, 0, st>>>(P.n, Q.k_colour, rp, weight);
    const double widest = std::max(Q.spacing[0], std::max(Q.spacing[1], Q.spacing[2]));
    const int edge = !P.ref && nn >= kIsoBrickNodes && 2.0 * widest <= (double)P.g.cell ? 2 : 1;
    auto kernel = P.ref ? k_iso_field<true, 1> : edge == 2 ? k_iso_field<false, 2> : k_iso_field<false, 1>;
    const long long xy = 4 * edge, z = 8 * edge;
    const long long blocks = ((Q.dims[0] + xy - 1) / xy) * ((Q.dims[1] + xy - 1) / xy) * ((Q.dims[2] + z - 1) / z);
    launch_chained(kernel, (unsigned)blocks, 128, 0, st, Q, P, pos, weight, cell_start, cell_end, iso);
}

long long mc_blocks(const IsoParams& Q) {
    return ((long long)Q.dims[0] * Q.dims[1] * Q.dims[2] + kMcBlock - 1) / kMcBlock;
}

void launch_mc_classify(cudaStream_t st, const IsoParams& Q, const double* iso, uint16_t* cases, uint32_t* block_vert,
                        uint32_t* block_tri) {
    launch_chained(k_mc_classify, (unsigned)mc_blocks(Q), kMcBlock, 0, st, Q, iso, cases, block_vert, block_tri);
}

void launch_mc_emit(cudaStream_t st, const IsoParams& Q, const double* iso, const uint16_t* cases,
                    const uint32_t* block_vert, const uint32_t* block_tri, uint32_t* first, float* vert, int32_t* tris) {
    const unsigned blocks = (unsigned)mc_blocks(Q);
    launch_chained(k_mc_vertices, blocks, kMcBlock, 0, st, Q, iso, cases, block_vert, first, vert);
    launch_chained(k_mc_triangles, blocks, kMcBlock, 0, st, Q, cases, block_tri, first, tris);
}

}  // namespace psb
