// Coupling on an explicit (unstructured) OpenFOAM polyMesh: the reference's own algorithm on any mesh MeshInfo can
// describe (src/meshinfo.h:20-29), for cases whose mesh is graded, multi-block or polyhedral.
//
// When every cell has the same number of points (hexahedral meshes) a cell's type does not depend on the cell that the
// search came from, and the reference's breadth-first search gives the connected set, over face neighbours, of the cells
// with an inside vertex that holds the seed.  Four kernels find it, spread over the whole GPU whatever the solid count:
//   poly_plan_kernel      the blocks of 128 consecutive cells whose boxes meet each solid's bounding region;
//   poly_classify_kernel  a warp per 32 cells of those blocks: the inside test of every vertex (FP32 with a rigorous error
//                         bound, FP64 inside it), a bit per cell with an inside vertex and a list of their words; beside it a CTA
//                         per solid finds the nearest cell centre (meshSearch::findNearestCell, solidcloud.cpp:363);
//   poly_link_kernel      union-find over the face neighbours of the listed cells;
//   poly_couple_kernel    keeps the cells of the seed's set (a seed without an inside vertex: the lowest label's), computes
//                         alpha (1, or the apex / pyramid volume over the cell's faces, GeometricTools::calcCellVolume,
//                         src/geometrictools.cpp:47-116, 8 lanes a cell) and the direct forcing (solidcloud.cpp:384-417),
//                         FP64 sums per cell over the solids and per solid over its cells.
// A breadth-first search by one CTA per solid, after a scan of every cell centre, was bound by its chain of levels (dependent
// loads, eight FP64 inside tests a cell) on one SM: interact took 2.30 ms for one cylinder on 78 400 graded cells and 2.97 ms
// for 40 solids on 140 000 hexahedra; it takes 0.100 and 0.306 ms now (GB300).
// Other meshes keep the search itself, whose order decides the types:
//   poly_enum_kernel      one CTA per solid: the seed by a scan of all centres, then a level-synchronous breadth-first
//                         search with the reference's classification (CellEnumerator, src/cellenumerator.cpp:6-78): a
//                         neighbour with no inside vertex is marked visited and not followed, the others are
//                         ALL_INSIDE when every vertex of the cell being expanded is inside (the reference compares
//                         with that cell's point count), else CENTER_INSIDE / CENTER_OUTSIDE by the centre test.
// Then
//   poly_finalize_kernel  the fields from the FP64 sums: As = min(sum, 1) (checkAlpha, solidcloud.cpp:564-570), Ct of
//                         the last solid in the reference's order;
//   poly_fix_kernel       fixInternal (solidcloud.cpp:288-301) with the mesh's cell centres.
// Which points are inside is decided by the reference's FP64 operation sequence (the library is built with -fmad=false)
// wherever the FP32 bound leaves it open, and the seed by FP64 distances, so touched sets and cell types equal the FP64
// oracle's on the same mesh.  The distances that the fractions are made of take the local point from the matrix of the
// rotation (local_matrix), which differs from the reference's quaternion products in the last place (half spaces: the products).
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"
#include "poly_dev.cuh"

namespace sdfibm_dev {

__device__ inline D3 poly_point(const PolyK& m, int32_t p) {
    return D3{m.points[3 * (int64_t)p], m.points[3 * (int64_t)p + 1], m.points[3 * (int64_t)p + 2]};
}
__device__ inline D3 poly_vec(const double* a, int64_t i) { return D3{a[3 * i], a[3 * i + 1], a[3 * i + 2]}; }

// Solid::phi01 of mesh point p (shape isInside in the local frame, FP64)
__device__ inline int poly_inside_point(const ShapeK& sh, const PolyK& m, int32_t p, const D3& x, const Q4& q) {
    return inside64(sh, world2local(poly_point(m, p), x, q)) ? 1 : 0;
}
__device__ inline int poly_count_inside(const ShapeK& sh, const PolyK& m, int32_t c, const D3& x, const Q4& q) {
    int n = 0;
    for (int32_t r = m.cp_off[c]; r < m.cp_off[c + 1]; ++r) n += poly_inside_point(sh, m, m.cp[r], x, q);
    return n;
}

// block-wide minimum of (key, index) pairs, lowest index on ties; every thread receives the result
__device__ inline void block_argmin(double& key, int32_t& idx, double* sk, int32_t* si) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int o = 16; o > 0; o >>= 1) {
        const double k2 = __shfl_xor_sync(0xffffffffu, key, o);
        const int32_t i2 = __shfl_xor_sync(0xffffffffu, idx, o);
        if (k2 < key || (k2 == key && i2 < idx)) { key = k2; idx = i2; }
    }
    if (lane == 0) { sk[w] = key; si[w] = idx; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < nw; ++i)
            if (sk[i] < sk[0] || (sk[i] == sk[0] && si[i] < si[0])) { sk[0] = sk[i]; si[0] = si[i]; }
    }
    __syncthreads();
    key = sk[0];
    idx = si[0];
    __syncthreads();
}

__global__ void __launch_bounds__(256) poly_enum_kernel(PolyK m, const SolidK* __restrict__ sk,
                                                        const sdfibm_solid_state* __restrict__ st, PolyWork w) {
    __shared__ double s_key[8];
    __shared__ int32_t s_idx[8];
    __shared__ int32_t s_tail, s_over;
    const int s = blockIdx.x;
    const ShapeK& sh = sk[s].shape;
    const Q4 q = state_quat(st[s]);
    const D3 x = state_pos(st[s]);
    uint32_t* visited = w.visited + (int64_t)s * w.words;
    int32_t* queue = w.queue + (int64_t)s * w.qcap;
    int8_t* qtype = w.qtype + (int64_t)s * w.qcap;
    // seed: the cell whose centre is nearest to the solid centre, lowest label on ties
    double best = 1e300;
    int32_t seed = 0x7fffffff;
    for (int32_t c = threadIdx.x; c < m.ncells; c += blockDim.x) {
        const D3 d = poly_vec(m.Cc, c) - x;
        const double d2 = magSqr(d);
        if (d2 < best || (d2 == best && c < seed)) { best = d2; seed = c; }
    }
    block_argmin(best, seed, s_key, s_idx);
    // a seed without an inside vertex: the first cell (by label) that has one, or none
    int n_seed = 0;
    if (threadIdx.x == 0) n_seed = poly_count_inside(sh, m, seed, x, q);
    if (threadIdx.x == 0) s_idx[0] = n_seed;
    __syncthreads();
    n_seed = s_idx[0];
    __syncthreads();
    if (n_seed == 0) {
        int32_t first = 0x7fffffff;
        for (int32_t base = 0; base < m.ncells && first == 0x7fffffff; base += blockDim.x) {
            const int32_t c = base + threadIdx.x;
            int32_t mine = 0x7fffffff;
            if (c < m.ncells && poly_count_inside(sh, m, c, x, q) > 0) mine = c;
            double k = 0.0;
            block_argmin(k, mine, s_key, s_idx);
            first = mine;
        }
        seed = first;
        if (seed == 0x7fffffff) {
            if (threadIdx.x == 0) w.count[s] = 0;
            return;
        }
        if (threadIdx.x == 0) n_seed = poly_count_inside(sh, m, seed, x, q);
    }
    if (threadIdx.x == 0) {
        const int np = m.cp_off[seed + 1] - m.cp_off[seed];
        int8_t t;
        if (n_seed == np) t = 1;
        else t = inside64(sh, world2local(poly_vec(m.Cc, seed), x, q)) ? 2 : 3;
        queue[0] = seed;
        qtype[0] = t;
        atomicOr(&visited[seed >> 5], 1u << (seed & 31));
        s_tail = 1;
        s_over = 0;
    }
    __syncthreads();
    // level-synchronous breadth-first search; every level adds at least one cell or ends it (tail <= qcap)
    int32_t head = 0;
    for (;;) {
        const int32_t tail = s_tail;
        __syncthreads();
        if (head >= tail || s_over) break;
        for (int32_t e = head + threadIdx.x; e < tail; e += blockDim.x) {
            const int32_t cur = queue[e];
            const int np_cur = m.cp_off[cur + 1] - m.cp_off[cur];
            for (int32_t r = m.cc_off[cur]; r < m.cc_off[cur + 1]; ++r) {
                const int32_t nb = m.ccl[r];
                const uint32_t bit = 1u << (nb & 31);
                if (atomicOr(&visited[nb >> 5], bit) & bit) continue;
                const int n_in = poly_count_inside(sh, m, nb, x, q);
                if (n_in == 0) continue;  // ALL_OUTSIDE: visited, not followed
                int8_t t;
                if (n_in == np_cur) t = 1;
                else t = inside64(sh, world2local(poly_vec(m.Cc, nb), x, q)) ? 2 : 3;
                const int32_t pos = atomicAdd(&s_tail, 1);
                if (pos < w.qcap) {
                    queue[pos] = nb;
                    qtype[pos] = t;
                } else {
                    s_over = 1;
                }
            }
        }
        __syncthreads();
        head = tail;
    }
    if (threadIdx.x == 0) {
        if (s_over) {
            w.count[s] = 0;
            atomicCAS(w.err, 0, DERR_CAPACITY);
        } else {
            w.count[s] = s_tail;
        }
    }
}

// ---- enumeration of meshes with one point count ---------------------------------------------------------------------
// Once per context: points as FP32 pairs, the sphere of each cell, |Sf|, and the boxes of POLY_BLOCK consecutive cells.
// Radii and boxes are widened by 2^-20 of the magnitudes, far beyond their FP32 rounding.
__global__ void __launch_bounds__(256) poly_setup_kernel(PolyK m, float4* __restrict__ pt32, float4* __restrict__ cell32,
                                                         double* __restrict__ mSf, float* __restrict__ blk) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    const float W = 9.5367431640625e-7f;
    for (int64_t p = tid; p < m.npoints; p += nt) {
        const D3 x = poly_point(m, (int32_t)p);
        const float hx = (float)x.x, hy = (float)x.y, hz = (float)x.z;
        pt32[2 * p] = make_float4(hx, hy, hz, (float)(x.x - (double)hx));
        pt32[2 * p + 1] = make_float4((float)(x.y - (double)hy), (float)(x.z - (double)hz), 0.f, 0.f);
    }
    for (int64_t f = tid; f < m.nfaces; f += nt) mSf[f] = mag(poly_vec(m.Sf, f));
    const int lane = threadIdx.x & 31;
    for (int64_t b = tid >> 5; b < m.nblocks; b += nt >> 5) {  // a warp per block
        float v[12];
        for (int a = 0; a < 12; ++a) v[a] = (a / 3) & 1 ? -INFINITY : INFINITY;
        float big = 0.f;
        for (int64_t c = b * POLY_BLOCK + lane; c < min((int64_t)m.ncells, (b + 1) * POLY_BLOCK); c += 32) {
            const D3 C = poly_vec(m.Cc, c);
            const float C3[3] = {(float)C.x, (float)C.y, (float)C.z};
            float r2 = 0.f, cb = fabsf(C3[0]) + fabsf(C3[1]) + fabsf(C3[2]);
            for (int a = 0; a < 3; ++a) { v[6 + a] = fminf(v[6 + a], C3[a]); v[9 + a] = fmaxf(v[9 + a], C3[a]); }
            for (int32_t r = m.cp_off[c]; r < m.cp_off[c + 1]; ++r) {
                const D3 x = poly_point(m, m.cp[r]);
                const D3 d = x - C;
                r2 = fmaxf(r2, (float)magSqr(d));
                const float p3[3] = {(float)x.x, (float)x.y, (float)x.z};
                for (int a = 0; a < 3; ++a) {
                    v[a] = fminf(v[a], p3[a]);
                    v[3 + a] = fmaxf(v[3 + a], p3[a]);
                    cb = fmaxf(cb, fabsf(p3[a]));
                }
            }
            cell32[c] = make_float4(C3[0], C3[1], C3[2], sqrtf(r2) * (1.f + W) + W * cb);
            big = fmaxf(big, cb);
        }
        for (int o = 16; o > 0; o >>= 1) {
            for (int a = 0; a < 12; ++a) {
                const float y = __shfl_xor_sync(0xffffffffu, v[a], o);
                v[a] = (a / 3) & 1 ? fmaxf(v[a], y) : fminf(v[a], y);
            }
            big = fmaxf(big, __shfl_xor_sync(0xffffffffu, big, o));
        }
        if (lane == 0)
            for (int a = 0; a < 12; ++a) blk[12 * b + a] = v[a] + ((a / 3) & 1 ? W * big : -W * big);
    }
}

// Solid and blocks.  The bounding region of the solid's inside points is widened far beyond FP32 rounding, so a block left
// out holds no inside vertex.  Also clears what the call sums into.
__global__ void __launch_bounds__(256) poly_plan_kernel(PolyK m, const SolidK* __restrict__ sk,
                                                        const sdfibm_solid_state* __restrict__ st, PolyWork w,
                                                        double* __restrict__ ftacc) {
    __shared__ PolySolid P;
    const int s = blockIdx.x, tid = threadIdx.x;
    if (tid == 0) {
        const ShapeK& sh = sk[s].shape;
        const Q4 q = state_quat(st[s]);
        const D3 x = state_pos(st[s]);
        local_matrix(q, P.R);
        P.mn = 0.f;
        for (int r = 0; r < 9; ++r) P.M[r] = (float)P.R[r];
        for (int r = 0; r < 3; ++r)
            P.mn = fmaxf(P.mn, fabsf(P.M[3 * r]) + fabsf(P.M[3 * r + 1]) + fabsf(P.M[3 * r + 2]));
        const double xs[3] = {x.x, x.y, x.z};
        P.xabs = 0.f;
        for (int a = 0; a < 3; ++a) {
            P.xh[a] = (float)xs[a];
            P.xl[a] = (float)(xs[a] - (double)P.xh[a]);
            P.xabs += fabsf(P.xh[a]);
        }
        // local = M (p - x), M M^T = |q|^4: p - x = M^T local / |q|^4
        const float i2 = 1.f / (P.M[0] * P.M[0] + P.M[1] * P.M[1] + P.M[2] * P.M[2]), i1 = sqrtf(i2);
        const bool ell = sh.type == SDFIBM_SHAPE_ELLIPSOID;  // ignores com
        const float l[3] = {ell ? 0.f : -sh.com32[0], ell ? 0.f : -sh.com32[1], ell || sh.prism ? 0.f : -sh.com32[2]};
        float cabs = P.xabs + fabsf(l[0]) + fabsf(l[1]) + fabsf(l[2]);
        for (int a = 0; a < 3; ++a) {
            P.c[a] = P.xh[a] + (P.M[a] * l[0] + P.M[3 + a] * l[1] + P.M[6 + a] * l[2]) * i2;
            P.axis[a] = P.M[6 + a] * i1;
        }
        P.r = (float)sh.bound_r * i1 * (1.f + 1e-4f) + 1e-5f * cabs;
        P.kind = sh.type == SDFIBM_SHAPE_PLANE ? 3 : (!sh.prism ? 0 : (q.v.x == 0.0 && q.v.y == 0.0 ? 1 : 2));
        if (blockIdx.y == 0) {
            w.plan[s] = P;
            w.wcount[s] = 0;
            w.count[s] = 0;
            w.mincand[s] = 0x7fffffff;
            for (int r = 0; r < 6; ++r) ftacc[6 * s + r] = 0.0;
        }
    }
    uint32_t* bits = w.visited + (int64_t)s * w.words;
    for (int64_t i = blockIdx.y * 256 + tid; i < w.words; i += gridDim.y * 256) bits[i] = 0u;
    __syncthreads();
    const int lane = tid & 31;
    for (int b0 = blockIdx.y * 256; b0 < m.nblocks; b0 += gridDim.y * 256) {
        const int b = b0 + tid;
        bool hit = false;
        if (b < m.nblocks) {
            const float* B = m.blk + 12 * (int64_t)b;
            if (P.kind <= 1) {  // distance of the centre (of the axis, which is z) to the box
                float d2 = 0.f;
                const int na = P.kind == 0 ? 3 : 2;
                for (int a = 0; a < na; ++a) {
                    const float d = fmaxf(fmaxf(B[a] - P.c[a], P.c[a] - B[3 + a]), 0.f);
                    d2 = __fmaf_rn(d, d, d2);
                }
                hit = !(d2 > P.r * P.r * (1.f + 1e-4f));
            } else {
                float ctr[3], half[3];
                for (int a = 0; a < 3; ++a) {
                    ctr[a] = 0.5f * (B[a] + B[3 + a]);
                    half[a] = 0.5f * (B[3 + a] - B[a]);
                }
                const float mag = fabsf(ctr[0]) + fabsf(ctr[1]) + fabsf(ctr[2]) + half[0] + half[1] + half[2] + P.xabs;
                if (P.kind == 2) {  // distance of the box's bounding sphere to the axis
                    const float dx = ctr[0] - P.c[0], dy = ctr[1] - P.c[1], dz = ctr[2] - P.c[2];
                    const float t = dx * P.axis[0] + dy * P.axis[1] + dz * P.axis[2];
                    const float ex = dx - t * P.axis[0], ey = dy - t * P.axis[1], ez = dz - t * P.axis[2];
                    const float d = sqrtf(ex * ex + ey * ey + ez * ez),
                                hd = sqrtf(half[0] * half[0] + half[1] * half[1] + half[2] * half[2]);
                    hit = !(d > P.r + hd + 1e-4f * mag);
                } else {  // lowest local y of the box
                    const float* n = P.M + 3;
                    const float y = n[0] * (ctr[0] - P.xh[0]) + n[1] * (ctr[1] - P.xh[1]) + n[2] * (ctr[2] - P.xh[2]);
                    const float e = fabsf(n[0]) * half[0] + fabsf(n[1]) * half[1] + fabsf(n[2]) * half[2];
                    hit = !(y - e > 1e-4f * P.mn * mag);
                }
            }
        }
        const unsigned bal = __ballot_sync(0xffffffffu, hit);
        int base = 0;
        if (lane == 0 && bal) base = atomicAdd(w.nitems, __popc(bal));
        base = __shfl_sync(0xffffffffu, base, 0);
        if (hit) w.items[base + __popc(bal & ((1u << lane) - 1u))] = make_int2(s, b);
    }
}

// FP32 inside test of a point given as FP32 pairs relative to the solid centre; 2: undecided.  The offset p - x carries
// a rounding of 2 u per component beside the pairs' own 2^-48, the map 4 u of |M| |d|: 16 u mn |d|_1 covers both, the
// last term the FP64 reference's rounding and the pairs' (8 times to spare).
__device__ inline int poly_inside32(const ShapeK& sh, const PolySolid& P, float hx, float hy, float hz, float lx,
                                    float ly, float lz) {
    const float dx = (hx - P.xh[0]) + (lx - P.xl[0]), dy = (hy - P.xh[1]) + (ly - P.xl[1]),
                dz = (hz - P.xh[2]) + (lz - P.xl[2]);
    const float* M = P.M;
    const float px = __fmaf_rn(M[0], dx, __fmaf_rn(M[1], dy, M[2] * dz));
    const float py = __fmaf_rn(M[3], dx, __fmaf_rn(M[4], dy, M[5] * dz));
    const float pz = __fmaf_rn(M[6], dx, __fmaf_rn(M[7], dy, M[8] * dz));
    const float E = P.mn * (16.f * U32 * (fabsf(dx) + fabsf(dy) + fabsf(dz)) +
                            1e-13f * (fabsf(hx) + fabsf(hy) + fabsf(hz) + P.xabs)) + 1e-30f;
    return inside32(sh, px, py, pz, E);
}

// One CTA: the cell whose centre is nearest to the solid's (lowest label on ties).  The block whose box reaches least far
// gives an upper bound (the nearest box would not do: a block that wraps from one mesh layer to the next has a box that
// holds nearly everything and no near centre); then only the blocks whose boxes come as near as that are read.
__device__ void poly_nearest(const PolyK& m, const D3& x, int32_t* seed, double* s_key, int32_t* s_idx) {
    const float X[3] = {(float)x.x, (float)x.y, (float)x.z};
    auto box_d2 = [&](int b) {  // at most the squared distance to any centre of the block
        const float* B = m.blk + 12 * (int64_t)b + 6;
        float d2 = 0.f;
        for (int a = 0; a < 3; ++a) {
            const float g = fmaxf(B[a] - X[a], X[a] - B[3 + a]) - 4.f * U32 * (fabsf(X[a]) + fabsf(B[a]) + fabsf(B[3 + a]));
            const float d = fmaxf(g, 0.f);
            d2 = __fmaf_rn(d, d, d2);
        }
        return d2 * (1.f - 1e-6f);
    };
    auto centre_d2 = [&](int32_t c) {
        const D3 d = poly_vec(m.Cc, c) - x;
        return magSqr(d);
    };
    double key = 1e300;
    int32_t idx = 0x7fffffff;
    for (int b = threadIdx.x; b < m.nblocks; b += blockDim.x) {
        const float* B = m.blk + 12 * (int64_t)b + 6;
        float d2 = 0.f;
        for (int a = 0; a < 3; ++a) {
            const float d = fmaxf(B[3 + a] - X[a], X[a] - B[a]);
            d2 = __fmaf_rn(d, d, d2);
        }
        if ((double)d2 < key) { key = (double)d2; idx = b; }
    }
    block_argmin(key, idx, s_key, s_idx);
    double best = 1e300;
    int32_t cell = 0x7fffffff;
    const int32_t c0 = (idx == 0x7fffffff ? 0 : idx) * POLY_BLOCK + threadIdx.x;
    if (threadIdx.x < POLY_BLOCK && c0 < m.ncells) { best = centre_d2(c0); cell = c0; }
    block_argmin(best, cell, s_key, s_idx);
    const double ub = best;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int b0 = 0; b0 < m.nblocks; b0 += 32 * nw) {
        const int b = b0 + lane * nw + wid;
        unsigned bal = __ballot_sync(0xffffffffu, b < m.nblocks && !((double)box_d2(min(b, m.nblocks - 1)) > ub));
        while (bal) {
            const int bb = b0 + (__ffs(bal) - 1) * nw + wid;
            bal &= bal - 1;
            for (int32_t c = bb * POLY_BLOCK + lane; c < min(m.ncells, (bb + 1) * POLY_BLOCK); c += 32) {
                const double d2 = centre_d2(c);
                if (d2 < best || (d2 == best && c < cell)) { best = d2; cell = c; }
            }
        }
    }
    block_argmin(best, cell, s_key, s_idx);
    if (threadIdx.x == 0) *seed = cell;
}

// CTAs 0 .. S-1: the seed of each solid.  The others: a warp per 32 cells of the listed blocks.  The FP32 test decides
// nearly every vertex (an FP64 test costs about fifty instructions at 1/64 of the FP32 rate); cells whose sphere misses the
// solid's region are left out first (140 000 hexahedra, 40 solids: 283 us with FP32 alone and every block of a mesh layer
// scanned for the seed, 37 us now, latency).
__global__ void __launch_bounds__(256) poly_classify_kernel(PolyK m, const SolidK* __restrict__ sk,
                                                            const sdfibm_solid_state* __restrict__ st, PolyWork w,
                                                            int S) {
    __shared__ double s_key[8];
    __shared__ int32_t s_idx[8];
    if (blockIdx.x < S) {
        poly_nearest(m, state_pos(st[blockIdx.x]), w.seed + blockIdx.x, s_key, s_idx);
        return;
    }
    const int lane = threadIdx.x & 31;
    const int64_t nw = (int64_t)(gridDim.x - S) * 8;
    constexpr int WPB = POLY_BLOCK / 32;
    const int64_t units = (int64_t)*w.nitems * WPB;
    for (int64_t u = ((int64_t)(blockIdx.x - S) * 256 + threadIdx.x) >> 5; u < units; u += nw) {
        const int2 it = w.items[u / WPB];
        const int s = it.x;
        const int32_t word = it.y * WPB + (int32_t)(u % WPB), c = word * 32 + lane;
        if (word * 32 >= m.ncells) continue;
        const ShapeK& sh = sk[s].shape;
        const PolySolid& P = w.plan[s];
        int n_in = 0, np = 1;
        bool near = false;
        if (c < m.ncells) {  // the cell's sphere against the solid's region
            const float4 q = m.cell32[c];
            const float dx = q.x - P.c[0], dy = q.y - P.c[1], dz = q.z - P.c[2], reach = P.r + q.w;
            if (P.kind == 0) {
                near = !(dx * dx + dy * dy + dz * dz > reach * reach * (1.f + 1e-4f));
            } else if (P.kind == 3) {
                const float y = P.M[3] * (q.x - P.xh[0]) + P.M[4] * (q.y - P.xh[1]) + P.M[5] * (q.z - P.xh[2]);
                near = !(y > P.mn * (q.w + 1e-5f * (fabsf(q.x) + fabsf(q.y) + fabsf(q.z) + P.xabs)));
            } else {
                const float t = dx * P.axis[0] + dy * P.axis[1] + dz * P.axis[2];
                const float ex = dx - t * P.axis[0], ey = dy - t * P.axis[1], ez = dz - t * P.axis[2];
                near = !(sqrtf(ex * ex + ey * ey + ez * ez) > reach + 1e-5f * (fabsf(dx) + fabsf(dy) + fabsf(dz)));
            }
        }
        if (near) {
            const int32_t p0 = m.cp_off[c];
            np = m.cp_off[c + 1] - p0;
#pragma unroll 4
            for (int r = 0; r < np; ++r) {
                const int32_t p = m.cp[p0 + r];
                const float4 a = m.pt32[2 * (int64_t)p], b = m.pt32[2 * (int64_t)p + 1];
                int in = poly_inside32(sh, P, a.x, a.y, a.z, a.w, b.x, b.y);
                if (in == 2) in = poly_inside_point(sh, m, p, state_pos(st[s]), state_quat(st[s]));
                n_in += in;
            }
        }
        const bool cand = n_in > 0;
        const unsigned bal = __ballot_sync(0xffffffffu, cand);
        if (!bal) continue;
        const int64_t at = (int64_t)s * w.words;
        if (lane == 0) {
            w.visited[at + word] = bal;
            // its place in the list, and how many cells lie before it
            const unsigned long long before = atomicAdd(w.wcount + s, (1ull << 32) | (unsigned)__popc(bal));
            const int32_t pos = (int32_t)(before >> 32), cells = (int32_t)before, batch = (cells + POLY_BATCH - 1) / POLY_BATCH;
            w.wlist[at + pos] = make_int2(word, cells);
            if (batch * POLY_BATCH < cells + __popc(bal)) w.wstart[s * w.batches + batch] = pos;
            atomicMin(w.mincand + s, word * 32 + __ffs(bal) - 1);
        }
        // links inside the word: each cell to one listed neighbour of a lower label here, then to that chain's end
        int up = lane;
        if (cand)
            for (int32_t r = m.cc_off[c]; r < m.cc_off[c + 1]; ++r) {
                const int32_t nb = m.ccl[r];
                if (nb < c && (nb >> 5) == word && ((bal >> (nb & 31)) & 1u)) { up = nb & 31; break; }
            }
#pragma unroll
        for (int k = 0; k < 5; ++k) up = __shfl_sync(0xffffffffu, up, up);
        int t = 1;
        if (cand) {
            if (n_in < np) {
                const double* C = m.Cc + 3 * (int64_t)c;
                const float hx = (float)C[0], hy = (float)C[1], hz = (float)C[2];
                int in = poly_inside32(sh, P, hx, hy, hz, (float)(C[0] - (double)hx), (float)(C[1] - (double)hy),
                                       (float)(C[2] - (double)hz));
                if (in == 2) in = inside64(sh, world2local(poly_vec(m.Cc, c), state_pos(st[s]), state_quat(st[s]))) ? 1 : 0;
                t = in ? 2 : 3;
            }
            w.parent[(int64_t)s * m.ncells + c] = word * 32 + up;
        }
        const unsigned b1 = __ballot_sync(0xffffffffu, cand && t == 1), b2 = __ballot_sync(0xffffffffu, cand && t == 2);
        if (lane == 0) {
            w.all_in[at + word] = b1;
            w.centre_in[at + word] = b2;
        }
    }
}

// root of cell c in a solid's forest; links on the way are shortened (every link leads to a lower label, so a lost update
// only leaves a longer path)
__device__ inline int32_t poly_root(int32_t* parent, int32_t c) {
    volatile int32_t* p = parent;
    int32_t up = p[c];
    while (up != c) {
        const int32_t next = p[up];
        if (next != up) p[c] = next;
        c = up;
        up = next;
    }
    return c;
}

// Union over the face neighbours of the listed words' cells (each pair from its higher label): the higher root is hung under
// the lower one by compare-and-swap.  A failed swap means that root has been hung meanwhile, so labels only fall and the loop
// ends.  A CTA takes up to 32 words at a time (fewer where that spreads them over more CTAs), a thread per cell, which finds its
// word in the prefix sums.
__global__ void __launch_bounds__(256) poly_link_kernel(PolyK m, PolyWork w) {
    __shared__ int s_word[32], s_end[32];
    __shared__ uint32_t s_bits[32];
    const int s = blockIdx.x, tid = threadIdx.x, n = (int)(w.wcount[s] >> 32);
    int32_t* parent = w.parent + (int64_t)s * m.ncells;
    const uint32_t* bits = w.visited + (int64_t)s * w.words;
    const int take = max(1, min(32, (n + (int)gridDim.y - 1) / (int)gridDim.y));
    for (int w0 = blockIdx.y * take; w0 < n; w0 += gridDim.y * take) {
        if (tid < 32) {
            const bool on = tid < take && w0 + tid < n;
            const int word = on ? w.wlist[(int64_t)s * w.words + w0 + tid].x : 0;
            const uint32_t b = on ? bits[word] : 0u;
            int end = __popc(b);
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, end, o);
                if (tid >= o) end += y;
            }
            s_word[tid] = word; s_bits[tid] = b; s_end[tid] = end;
        }
        __syncthreads();
        for (int e = tid; e < s_end[31]; e += blockDim.x) {
            int i = 0;
#pragma unroll
            for (int h = 16; h > 0; h >>= 1)
                if (s_end[i + h - 1] <= e) i += h;
            const uint32_t b = s_bits[i];
            const int32_t c = s_word[i] * 32 + nth_bit(b, e - s_end[i] + __popc(b));
            for (int32_t r = m.cc_off[c]; r < m.cc_off[c + 1]; ++r) {
                const int32_t nb = m.ccl[r];
                if (nb >= c || !((bits[nb >> 5] >> (nb & 31)) & 1u)) continue;
                int32_t a = poly_root(parent, c), d = poly_root(parent, nb);
                while (a != d) {
                    if (a < d) { const int32_t t = a; a = d; d = t; }
                    const int32_t seen = atomicCAS(parent + a, a, d);
                    if (seen == a) break;
                    a = poly_root(parent, seen);
                    d = poly_root(parent, d);
                }
            }
        }
        __syncthreads();
    }
}

// ---- fraction and forcing ---------------------------------------------------------------------------------------------
// GeometricTools::calcLineFraction (geometrictools.cpp:13-23)
__device__ inline double poly_line_fraction(double pa, double pb) {
    if (pa > 0 && pb > 0) return 0;
    if (pa <= 0 && pb <= 0) return 1;
    if (pa > 0) return -pb / (pa - pb);
    return -pa / (pb - pa);
}

// Distance in the reference's own operations.  A half space has no filter, and the geometry jumps by SMALL / h where its distance is
// zero or next to zero, so it is always taken from here; the other shapes' distances within 1e-8 are all -1e-8, and the matrix of
// the rotation serves, but for the ellipse and the ellipsoid at their centre, where it can be no number when the reference's is.
// Out of line: the others have no registers to spare for it.
static __device__ __noinline__ double poly_exact_phi(const PolyK& m, const ShapeK& sh, int32_t p, const sdfibm_solid_state& st) {
    return sdf64(sh, world2local(poly_point(m, p), state_pos(st), state_quat(st)));
}

constexpr int POLY_MAX_CELL_POINTS = 64;  // points of a cell whose distances are kept; later ones count as 0

// GeometricTools::calcApex over n points (geometrictools.cpp:25-45); point(i), phi(i)
template <class Point, class Phi>
__device__ inline D3 poly_apex(int n, const Point& point, const Phi& phi) {
    const D3 A = point(0);
    const double phiA = phi(0);
    D3 B{0.0, 0.0, 0.0};
    double phiB = 0.0;
    int at = 0;
    for (int i = 1; i < n; ++i) {
        at = i;
        phiB = phi(i);
        if (phiA * phiB <= 0) break;
    }
    if (at > 0) B = point(at);
    return A - fabs(phiA) / (SMALL_D + fabs(phiA) + fabs(phiB)) * (A - B);
}

// GeometricTools::calcCellVolume (geometrictools.cpp:47-72) with calcFaceAreaFraction / calcFaceArea (:74-116) of cell c
// by 8 lanes: a lane per vertex computes the distances (into phi, the group's shared memory), a lane per face its pyramid,
// and the pyramids are added in face order.  A thread per cell spent 169 us on the serial chain of one cylinder's cut
// cells (FP64 instructions issue every 16 cycles a warp and wait on each other); 8 lanes cut the chain to one distance
// and one face.  All lanes of the warp call it (c < 0: a group without a cell).
__device__ double poly_cell_volume8(const PolyK& m, int32_t c, const ShapeK& sh, const sdfibm_solid_state& st, const D3& x,
                                    const double* R, double* phi) {
    const int sub = threadIdx.x & 7;
    const int32_t p0 = c < 0 ? 0 : m.cp_off[c], np = c < 0 ? 0 : m.cp_off[c + 1] - p0;
    const int32_t* cp = m.cp + p0;
    for (int i = sub; i < np && i < POLY_MAX_CELL_POINTS; i += 8) {
        const D3 d = poly_point(m, cp[i]) - x;
        bool exact = sh.type == SDFIBM_SHAPE_PLANE;
        double v = 0.0;
        if (!exact) {
            v = sdf64(sh, D3{R[0] * d.x + R[1] * d.y + R[2] * d.z, R[3] * d.x + R[4] * d.y + R[5] * d.z,
                             R[6] * d.x + R[7] * d.y + R[8] * d.z});
            exact = (__double2hiint(v) & 0x7ff00000) == 0x7ff00000;
        }
        if (exact) v = poly_exact_phi(m, sh, cp[i], st);
        phi[i] = v;
    }
    __syncwarp();
    auto phi_at = [&](int slot) { return slot < POLY_MAX_CELL_POINTS ? phi[slot] : 0.0; };
    double volume = 0.0;
    const int32_t f0 = c < 0 ? 0 : m.cf_off[c], nf = c < 0 ? 0 : m.cf_off[c + 1] - f0;
    D3 apex{0, 0, 0};
    if (nf > 0) {
        apex = poly_apex(np, [&](int i) { return poly_point(m, cp[i]); }, phi_at);
        if (m.twod) apex.z = 0.0;
    }
    const int nf_max = __reduce_max_sync(0xffffffffu, nf);
    for (int r0 = 0; r0 < nf_max; r0 += 8) {
        double part = 0.0;
        if (r0 + sub < nf) {
            const int32_t r = f0 + r0 + sub, f = m.cf[r];
            const int32_t* fv = m.face_lab + m.face_off[f];
            const uint8_t* sl = m.cfv + m.cfv_off[r];
            const int nv = m.face_off[f + 1] - m.face_off[f];
            int sign_sum = 0;
            for (int i = 0; i < nv; ++i) sign_sum += phi_at(sl[i]) > 0 ? 1 : -1;
            double eps;
            if (sign_sum == nv) {
                eps = 0.0;
            } else if (sign_sum == -nv) {
                eps = 1.0;
            } else {
                const D3 fa = poly_apex(nv, [&](int i) { return poly_point(m, fv[i]); }, [&](int i) { return phi_at(sl[i]); });
                const bool fin = fabs(fa.x) + fabs(fa.y) + fabs(fa.z) < 1e150;
                double area = 0.0;
                const D3 first = poly_point(m, fv[0]);
                const double phi_first = phi_at(sl[0]);
                D3 O = first;
                double phiO = phi_first;
                for (int i = 0; i < nv; ++i) {
                    const bool last = i + 1 == nv;
                    const D3 A = last ? first : poly_point(m, fv[i + 1]);
                    const double phiA = last ? phi_first : phi_at(sl[i + 1]);
                    const double lf = poly_line_fraction(phiO, phiA);
                    // an edge outside adds nothing (unless the apex is not finite)
                    if (lf != 0.0 || !fin) area += fabs(0.5 * mag(cross(A - O, fa - O))) * lf;
                    O = A;
                    phiO = phiA;
                }
                eps = area / m.mSf[f];
            }
            part = (1.0 / 3.0) * eps * fabs(dot(apex - poly_vec(m.Cf, f), poly_vec(m.Sf, f)));
        }
        for (int i = 0; i < 8; ++i) {  // in face order, as the reference sums
            const double v = __shfl_sync(0xffffffffu, part, i, 8);
            if (r0 + i < nf) volume += v;
        }
    }
    __syncwarp();
    return volume;
}

// Touched cells of one solid (blockIdx.x), POLY_BATCH of them a CTA: linked, of the cells with an inside vertex in the order of
// their list of words those in the seed's set (the others are marked); else of the touched list.  The cut cells of a batch are
// spread over the CTA's 32 groups of 8 lanes, then a lane per cell does the forcing.  Bound by the FP64 pipe (about 2000
// operations a cut cell): 172 us for the 140 000-cell mesh's 40 solids, 360 us with a thread per cell; 33 us against 169 us for
// one cylinder.  (Batches of whole words, whose cells differ in number: 186 us.)  The solids run along grid.x, so that the first
// batches of all of them land on different SMs.
__global__ void __launch_bounds__(256, 2) poly_couple_kernel(PolyK m, const SolidK* __restrict__ sk,
                                                             const sdfibm_solid_state* __restrict__ st, PolyWork w,
                                                             const float* __restrict__ U, double* __restrict__ ftacc,
                                                             double dtINV, int linked) {
    __shared__ double s_phi[32][POLY_MAX_CELL_POINTS];
    __shared__ double s_alpha[POLY_BATCH], s_R[9];
    __shared__ int32_t s_cell[POLY_BATCH], s_cut[POLY_BATCH];
    __shared__ int8_t s_type[POLY_BATCH];
    __shared__ int s_ncut;
    const unsigned FULL = 0xffffffffu;
    const int s = blockIdx.x, tid = threadIdx.x, lane = tid & 31;
    const int64_t o = (int64_t)s * w.qcap, ow = (int64_t)s * w.words;
    const unsigned long long listed = linked ? w.wcount[s] : 0ull;
    const int32_t n = linked ? (int32_t)listed : w.count[s], nwords = (int32_t)(listed >> 32);
    int32_t* parent = w.parent + (int64_t)s * m.ncells;
    if ((int64_t)blockIdx.y * POLY_BATCH >= n) return;
    int32_t home = 0;
    if (tid < POLY_BATCH && linked) {
        const int32_t sd = w.seed[s];
        const bool on = sd < m.ncells && ((w.visited[ow + (sd >> 5)] >> (sd & 31)) & 1u);
        home = poly_root(parent, on ? sd : w.mincand[s]);
    }
    const ShapeK& sh = sk[s].shape;
    const D3 x = state_pos(st[s]);
    if (linked) {
        if (tid < 9) s_R[tid] = w.plan[s].R[tid];
    } else if (tid == 0) {
        local_matrix(state_quat(st[s]), s_R);
    }
    if (tid == 0) s_ncut = 0;
    __syncthreads();
    const D3 v{st[s].vel[0], st[s].vel[1], st[s].vel[2]};
    const D3 om{st[s].omega[0], st[s].omega[1], st[s].omega[2]};
    double acc[6] = {0, 0, 0, 0, 0, 0};
    for (int64_t b = blockIdx.y; b * POLY_BATCH < n; b += gridDim.y) {
        int32_t c = -1;
        int t = 0;
        if (linked) {
            // the words of the batch: at most POLY_BATCH from the one its first cell lies in, by other warps than those that
            // look for the seed's root meanwhile
            const int j = tid - POLY_BATCH;
            const int32_t first = (int32_t)b * POLY_BATCH, at = j >= 0 && j < POLY_BATCH ? w.wstart[s * w.batches + b] + j : nwords;
            if (at < nwords) {
                const int2 it = w.wlist[ow + at];
                if (it.y < first + POLY_BATCH) {
                    const uint32_t bits = w.visited[ow + it.x], in = w.all_in[ow + it.x], ci = w.centre_in[ow + it.x];
                    int to = it.y - first;
                    for (uint32_t left = bits; left; left &= left - 1, ++to) {
                        const int i = __ffs(left) - 1;
                        if (to >= 0 && to < POLY_BATCH) {
                            s_cell[to] = it.x * 32 + i;
                            s_type[to] = (in >> i) & 1u ? 1 : ((ci >> i) & 1u ? 2 : 3);
                        }
                    }
                }
            }
            __syncthreads();
        }
        if (tid < POLY_BATCH) {  // whole warps
            const int64_t e = b * POLY_BATCH + tid;
            if (e < n) {
                c = linked ? s_cell[tid] : w.queue[o + e];
                t = linked ? s_type[tid] : w.qtype[o + e];
                if (linked && poly_root(parent, c) != home) {  // left out of the touched cells: both types
                    atomicOr(w.all_in + ow + (c >> 5), 1u << (c & 31));
                    atomicOr(w.centre_in + ow + (c >> 5), 1u << (c & 31));
                    c = -1;
                }
            }
            const unsigned below = (1u << lane) - 1u;
            if (linked) {
                const unsigned bal = __ballot_sync(FULL, c >= 0);
                if (lane == 0 && bal) atomicAdd(w.count + s, __popc(bal));
            }
            const bool cut = c >= 0 && t != 1;
            const unsigned bal = __ballot_sync(FULL, cut);
            int base = 0;
            if (lane == 0 && bal) base = atomicAdd(&s_ncut, __popc(bal));
            base = __shfl_sync(FULL, base, 0) + __popc(bal & below);
            if (cut) s_cut[base] = tid;
            s_cell[tid] = c;
            s_alpha[tid] = 1.0;
        }
        __syncthreads();
        const int ncut = s_ncut;
        for (int g0 = 0; g0 + ((tid >> 5) << 2) < ncut; g0 += 32) {  // warp-uniform
            const int g = g0 + (tid >> 3);
            const int32_t cc = g < ncut ? s_cell[s_cut[g]] : -1;
            const double vol = poly_cell_volume8(m, cc, sh, st[s], x, s_R, s_phi[tid >> 3]);
            if (cc >= 0 && (tid & 7) == 0) s_alpha[s_cut[g]] = vol / m.Vc[cc];
        }
        __syncthreads();
        if (tid == 0) s_ncut = 0;
        if (c >= 0) {
            const double V = m.Vc[c], alpha = s_alpha[tid];
            const D3 C = poly_vec(m.Cc, c);
            const D3 uf{(double)U[c], (double)U[(int64_t)m.ncells + c], (double)U[2 * (int64_t)m.ncells + c]};
            const D3 us = v + cross(om, C - x);  // Solid::evalPointVelocity
            const D3 f = alpha * (uf - us);
            const D3 tq = cross(C - x, f);
            const D3 fv = f * V * dtINV, tv = tq * V * dtINV;
            acc[0] += fv.x; acc[1] += fv.y; acc[2] += fv.z;
            acc[3] += tv.x; acc[4] += tv.y; acc[5] += tv.z;
            double* a = w.acc + 5 * (int64_t)c;
            atomicAdd(a + 0, alpha);
            atomicAdd(a + 1, alpha);
            const D3 fd = f * dtINV;
            atomicAdd(a + 2, fd.x);
            atomicAdd(a + 3, fd.y);
            atomicAdd(a + 4, fd.z);
            atomicMax(w.claim + c, 4 * s + t);
        }
        __syncthreads();
    }
    if (tid < POLY_BATCH)
        for (int r = 0; r < 6; ++r) {
            double y = acc[r];
            for (int o2 = 16; o2 > 0; o2 >>= 1) y += __shfl_xor_sync(FULL, y, o2);
            if (lane == 0 && y != 0.0) atomicAdd(ftacc + 6 * s + r, y);
        }
}

// Fields of every cell from the sums (cells no solid touched hold zeros), the sums and claims of the touched cells cleared
// for the next call; the force and torque of every solid (force *= m_rhof, solidcloud.cpp:423) into ft and its state.
__global__ void poly_finalize_kernel(PolyWork w, int32_t N, float* __restrict__ As, float* __restrict__ Fs,
                                     float* __restrict__ Ts, int32_t* __restrict__ Ct, int S,
                                     const double* __restrict__ ftacc, double* __restrict__ ft, double rho_f,
                                     sdfibm_solid_state* __restrict__ st) {
    const int64_t tid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    for (int64_t c = tid; c < N; c += nt) {
        const int32_t k = w.claim[c];
        float f[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
        if (k >= 0) {
            double* a = w.acc + 5 * c;
            f[0] = (float)fmin(a[0], 1.0);
            for (int r = 1; r < 5; ++r) f[r] = (float)a[r];
            for (int r = 0; r < 5; ++r) a[r] = 0.0;
            w.claim[c] = -1;
        }
        As[c] = f[0];
        Ts[c] = f[1];
        Fs[c] = f[2];
        Fs[(int64_t)N + c] = f[3];
        Fs[2 * (int64_t)N + c] = f[4];
        Ct[c] = k < 0 ? 0 : ((k & 3) == 1 ? (k >> 2) + 4 : (k & 3));
    }
    for (int64_t e = tid; e < 6 * (int64_t)S; e += nt) {
        const int64_t s = e / 6, r = e - 6 * s;
        const double y = ftacc[e] * rho_f;
        ft[e] = y;
        if (r < 3) st[s].fluid_force[r] = y;
        else st[s].fluid_torque[r - 3] = y;
    }
    if (tid == 0) *w.nitems = 0;
}

// SolidCloud::fixInternal: U = velocity of solid Ct - 4 at the cell centre where Ct >= 4
__global__ void poly_fix_kernel(PolyK m, const sdfibm_solid_state* __restrict__ st, int S, const int32_t* __restrict__ Ct,
                                float* __restrict__ U) {
    const int32_t N = m.ncells;
    for (int32_t c = blockIdx.x * blockDim.x + threadIdx.x; c < N; c += gridDim.x * blockDim.x) {
        const int32_t k = Ct[c];
        if (k < 4 || k - 4 >= S) continue;
        const sdfibm_solid_state& x = st[k - 4];
        const D3 C = poly_vec(m.Cc, c);
        const D3 us = D3{x.vel[0], x.vel[1], x.vel[2]} +
                      cross(D3{x.omega[0], x.omega[1], x.omega[2]}, C - D3{x.pos[0], x.pos[1], x.pos[2]});
        U[c] = (float)us.x;
        U[(int64_t)N + c] = (float)us.y;
        U[2 * (int64_t)N + c] = (float)us.z;
    }
}

}  // namespace sdfibm_dev
