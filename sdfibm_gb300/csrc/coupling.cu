// Coupling kernels: the GB300 replacement of SolidCloud::interact (src/solidcloud.cpp:361-464) and
// SolidCloud::fixInternal (src/solidcloud.cpp:288-301).
//
// Pipeline of one interact (no host round trip until FT is read back):
//   plan      per solid: bbox origin in cell indices, FP32 world->local matrix, nearest cell (meshSearch), the
//             two-float forms used by the fraction and forcing kernels
//   classify  persistent CTAs pulling (solid, cell-tile) items from an atomic counter; each tile evaluates the
//             inside test once per vertex (FP32 with a guard band, FP64 re-check inside the band) and writes one
//             class byte per cell: 0 no inside vertex, 1 all inside, 2 centre inside, 3 centre outside
//             (CellEnumerator::_next, cellenumerator.cpp:6-34), and lists the cut cells for the fraction kernels
//   fraction  (classify.cu) REF-GEO a thread per listed cell; SUBSAMPLE a lane per listed cell, a warp where there are few;
//             LEARNED the network, then SUBSAMPLE on the cells outside its band; FP64 rechecks of undecided sample points
//   connect   on a side stream beside the fraction kernels: a CTA, 128 threads or a warp per solid; the cells with an inside
//             vertex as bitmaps, a proof that they hang together or a bit-parallel flood fill from the seed (the BFS of
//             CellEnumerator::intersect with its seed fallback, cellenumerator.cpp:47-78), then the reached cells appended to
//             the ALL_INSIDE list or the cut-cell list in ascending cell order
//   claim     of each touched cell, and marks of the 8-cell chunks they lie in
//   scan      the list entries on cells of several solids; reset of the cells the previous call touched and this one does not
//             (sparse form of solidcloud.cpp:438-441)
//   couple    warps over the marked chunks: alpha (1, or the fraction), direct forcing, the final fields of single-owner
//             cells, zeros for unclaimed ones, force and torque summed per solid in the warp, then by FP64 atomics
//   finalize  cells of several solids from the FP64 table: Ct of the last solid (as the serial loop), As = min(As,1)
//             (checkAlpha); FT = rho_f V / dt * sums
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace sdfibm_dev {


// ---- plan ---------------------------------------------------------------------------------------------------------
// bounding region and bbox origin (warp 0 of a plan CTA)
__device__ inline void plan_box(const MeshK& m, const SolidK& k, const Q4& q, const D3& x, SolidPlan& p, Counters* cnt) {
    int err = 0;
    const int32_t n[3] = {m.nx, m.ny, m.nz};
    int32_t vlo[3] = {0, 0, 0}, vhi[3] = {m.nx, m.ny, m.nz}, lo3[3] = {0, 0, 0};
    const double inv[3] = {1.0 / m.h[0], 1.0 / m.h[1], 1.0 / m.h[2]};
    if (k.infinite) {
        // the half space n . (v - x) < 0 over the mesh box bounds the inside vertices along every axis its normal has a
        // component of (a wall along an axis: one layer of cells), widened far beyond the rounding of the inside test
        const D3 nw = qtransform(q, D3{0, 1, 0});
        const double nv[3] = {nw.x, nw.y, nw.z}, xv[3] = {x.x, x.y, x.z};
        double low = 0.0, mag = 0.0, term[3];
        for (int a = 0; a < 3; ++a) {
            const double l = m.o[a], u = mesh_coord(m, a, n[a]);
            term[a] = dmin(nv[a] * (l - xv[a]), nv[a] * (u - xv[a]));
            low += term[a];
            mag += fabs(nv[a]) * (fabs(l) + fabs(u) + fabs(xv[a]));
        }
        for (int a = 0; a < 3; ++a) {
            if (nv[a] == 0.0) continue;
            const double bound = xv[a] - (low - term[a]) / nv[a], tol = 1e-12 * (mag / fabs(nv[a])) + 1e-12 * fabs(xv[a]);
            if (nv[a] > 0.0) vhi[a] = (int32_t)dmin(dmax(floor((bound + tol - m.o[a]) / m.h[a]) + 1, -1.0), (double)n[a]);
            else vlo[a] = (int32_t)dmin(dmax(ceil((bound - tol - m.o[a]) / m.h[a]) - 1, 0.0), (double)n[a] + 1);
        }
    } else {
        D3 cl{-k.shape.com[0], -k.shape.com[1], -k.shape.com[2]};
        if (k.shape.type == SDFIBM_SHAPE_ELLIPSOID) cl = D3{0, 0, 0};
        if (k.shape.prism) cl.z = 0.0;
        D3 cw = x;
        if (cl.x != 0.0 || cl.y != 0.0 || cl.z != 0.0) cw = x + qtransform(q, cl);
        const double r = k.shape.bound_r * (1.0 + 1e-9) + 1e-12;
        double rad[3] = {r, r, r};
        if (k.shape.prism && !(q.v.x == 0.0 && q.v.y == 0.0)) {
            // the inside region is a prism along the local z axis a; clip it to the mesh slab in z
            const double qq = q.w * q.w + magSqr(q.v);
            const D3 a = qtransform(q, D3{0, 0, 1}) / qq;
            const double sxy = sqrt(a.x * a.x + a.y * a.y), az = fabs(a.z);
            if (az < 0.3 && (k.ext[0] < n[0] + 2 || k.ext[1] < n[1] + 2)) err = DERR_BBOX;
            const double zlo = m.o[2], zhi = mesh_coord(m, 2, m.nz);
            const double zspan = dmax(fabs(zhi - cw.z), fabs(zlo - cw.z));
            // one that lies: no bound, the window spans the mesh
            const double rxy = az < 0.3 ? INFINITY : (sxy > 0 ? r + (zspan + r * sxy) / az * sxy : r);
            rad[0] = rad[1] = rxy * (1.0 + 1e-9);
        }
        // half extents of the oriented bounding box of the inside region along the world axes; FP32, widened
        float e[3] = {INFINITY, INFINITY, INFINITY};
        if (k.shape.type == SDFIBM_SHAPE_ELLIPSOID || k.shape.type == SDFIBM_SHAPE_BOX) {
            const float w = (float)q.w, qx = (float)q.v.x, qy = (float)q.v.y, qz = (float)q.v.z;
            const float qq = w * w + qx * qx + qy * qy + qz * qz, iq = 1.f / qq;
            const float size = (float)k.shape.bound_r, isize = 1.f / size;  // squares of the sizes stay in range
            const float Rm[3][3] = {{w * w + qx * qx - qy * qy - qz * qz, 2.f * (qx * qy - w * qz), 2.f * (qx * qz + w * qy)},
                                    {2.f * (qx * qy + w * qz), w * w - qx * qx + qy * qy - qz * qz, 2.f * (qy * qz - w * qx)},
                                    {2.f * (qx * qz - w * qy), 2.f * (qy * qz + w * qx), w * w - qx * qx - qy * qy + qz * qz}};
            const float* sp = k.shape.p32;
            const bool ell = k.shape.type == SDFIBM_SHAPE_ELLIPSOID;
            for (int a = 0; a < 3; ++a) {
                float t = 0.f;
                for (int c = 0; c < 3; ++c) {
                    const float v = fabsf(Rm[a][c]) * iq * (sp[c] * isize);
                    t += ell ? v * v : v;
                }
                // FP32 errors of R are relative to 1, not to the entry
                if (qq > 1e-6f && qq < 1e6f) e[a] = size * ((ell ? sqrtf(t) : t) + 3e-5f);
            }
        }
        const double c3[3] = {cw.x, cw.y, cw.z};
        for (int a = 0; a < 3; ++a) {
            if (k.shape.prism && a == 2) continue;  // all layers
            const double ea = dmin(rad[a], (double)e[a]) * (1.0 + 1e-9) + 1e-12;
            const double l = ceil((c3[a] - ea - m.o[a]) * inv[a]) - 1, u = floor((c3[a] + ea - m.o[a]) * inv[a]) + 1;
            vlo[a] = (int32_t)dmin(dmax(l, -1.0), (double)n[a] + 1);
            vhi[a] = (int32_t)dmin(dmax(u, -1.0), (double)n[a] + 1);
            if (k.ext[a] >= n[a] + 2) { lo3[a] = -1; continue; }  // the window spans the whole axis
            const double lo = floor((c3[a] - rad[a] - m.o[a]) * inv[a]) - 1, hi = floor((c3[a] + rad[a] - m.o[a]) * inv[a]) + 1;
            // only cells 0..n-1 matter: start the window no lower than -1 (this also keeps the int conversion
            // defined for solids far outside the mesh)
            const double lo_c = dmin(dmax(lo, -1.0), 1e9), hi_c = dmin(hi, (double)n[a]);
            lo3[a] = (int32_t)lo_c;
            if (hi_c >= lo_c && hi_c - lo_c + 1 > (double)k.ext[a]) err = DERR_BBOX;
        }
    }
    for (int a = 0; a < 3; ++a) { p.lo[a] = lo3[a]; p.vlo[a] = vlo[a]; p.vhi[a] = vhi[a]; }
    p.err = err;
    if (err) set_error(cnt, err);
    // FP64 origin of the tile frames and the local map (world2local of the bbox corner plus the images of the cell edge
    // vectors), so tiles build their frames without per-tile FP64 work
    const D3 p0 = mesh_point(m, lo3[0], lo3[1], lo3[2]);
    const D3 b = p0 - x;
    p.base32[0] = (float)b.x; p.base32[1] = (float)b.y; p.base32[2] = (float)b.z;
    double L[9];
    local_matrix(q, L);
    double l12[12];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        l12[r] = L[3 * r] * b.x + L[3 * r + 1] * b.y + L[3 * r + 2] * b.z;
#pragma unroll
        for (int a = 0; a < 3; ++a) l12[3 + 3 * a + r] = L[3 * r + a] * m.h[a];
    }
#pragma unroll
    for (int r = 0; r < 12; ++r) {
        p.lmap[r] = l12[r];
        p.lmap_hi[r] = (float)l12[r];
        p.lmap_lo[r] = (float)(l12[r] - (double)p.lmap_hi[r]);
    }
#pragma unroll
    for (int r = 0; r < 9; ++r) p.M[r] = (float)L[r];  // |q|^2 R(q)^T: the linear map of world2local
    float mag = 0.f;
    const float o3[3] = {(float)m.o[0], (float)m.o[1], (float)m.o[2]}, x3[3] = {(float)x.x, (float)x.y, (float)x.z};
    for (int a = 0; a < 3; ++a)
        mag += fabsf(o3[a] + (float)lo3[a] * m.h32[a]) + fabsf(o3[a] + (float)(lo3[a] + k.ext[a]) * m.h32[a]) + fabsf(x3[a]) +
               1e-6f * fabsf(o3[a]);
    p.e64 = 4.1e-15f * mag;
}

// nearest cell (warp 1): meshSearch::findNearestCell, ties to the lowest label, and the rigid-body velocity there.  The
// squared distance is (dx^2 + dy^2) + dz^2 with each sum rounded, which never falls when a term grows, so the minimum over
// the neighbourhood is at the axes' minima; the lowest label among equals is found axis by axis.
__device__ inline void plan_nearest(const MeshK& m, const Q4& q, const D3& x, const sdfibm_solid_state& st, SolidPlan& p) {
    const double pc[3] = {x.x, x.y, x.z};
    const int32_t n[3] = {m.nx, m.ny, m.nz};
    int lo[3], cnt3[3];
    double d[3][3], sq[3][3], least[3];
    for (int a = 0; a < 3; ++a) {
        const double t = floor((pc[a] - m.o[a]) / m.h[a]);
        const int e = !(t >= 0.0) ? 0 : (t > (double)(n[a] - 1) ? n[a] - 1 : (int)t);
        lo[a] = e > 0 ? e - 1 : 0;
        cnt3[a] = (e + 1 < n[a] ? e + 1 : n[a] - 1) - lo[a] + 1;
        for (int i = 0; i < 3; ++i) {
            d[a][i] = mesh_centre(m, a, lo[a] + i) - pc[a];
            sq[a][i] = i < cnt3[a] ? d[a][i] * d[a][i] : INFINITY;
        }
        least[a] = sq[a][0];
        for (int i = 1; i < 3; ++i) least[a] = sq[a][i] < least[a] ? sq[a][i] : least[a];
    }
    const double best = least[0] + least[1] + least[2];
    int at[3] = {0, 0, 0};
    for (int i = 2; i >= 0; --i) at[2] = least[0] + least[1] + sq[2][i] == best ? i : at[2];
    const double dz2 = at[2] == 0 ? sq[2][0] : (at[2] == 1 ? sq[2][1] : sq[2][2]);
    for (int i = 2; i >= 0; --i) at[1] = least[0] + sq[1][i] + dz2 == best ? i : at[1];
    const double dy2 = at[1] == 0 ? sq[1][0] : (at[1] == 1 ? sq[1][1] : sq[1][2]);
    for (int i = 2; i >= 0; --i) at[0] = sq[0][i] + dy2 + dz2 == best ? i : at[0];
    double cb[3];
    for (int a = 0; a < 3; ++a) {
        p.seed_ijk[a] = lo[a] + at[a];
        cb[a] = at[a] == 0 ? d[a][0] : (at[a] == 1 ? d[a][1] : d[a][2]);
        p.cb32[a] = (float)cb[a];
    }
    // us at a cell (i, j, k) = us0 + omega x ((i, j, k) - seed) h: us0 and the six per-step terms, split into
    // FP32 pairs (the couple kernel evaluates U - us in two-float arithmetic)
    const D3 vel{st.vel[0], st.vel[1], st.vel[2]}, om{st.omega[0], st.omega[1], st.omega[2]};
    const D3 us0 = vel + cross(om, D3{cb[0], cb[1], cb[2]});
    const double u3[3] = {us0.x, us0.y, us0.z};
    const double d6[6] = {-om.z * m.h[1], om.y * m.h[2], om.z * m.h[0], -om.x * m.h[2], -om.y * m.h[0], om.x * m.h[1]};
    for (int a = 0; a < 3; ++a) {
        p.us_hi[a] = (float)u3[a];
        p.us_lo[a] = (float)(u3[a] - (double)p.us_hi[a]);
    }
    for (int r = 0; r < 6; ++r) {
        p.ds_hi[r] = (float)d6[r];
        p.ds_lo[r] = (float)(d6[r] - (double)p.ds_hi[r]);
    }
}

// Head of an interact: the time-step block, the counters, the cleared sums and chunk marks, and the plan of every solid.  A
// CTA plans 32 solids, warp 0 their boxes, warp 1 their nearest cells, warp 2 the rest; the CTAs after those clear the marks.
// Bound by FP64 latency (one chain per solid): one thread a solid with the 27-cell search written out took 46 us for one
// solid and 55 for 4096, with two launches and three fills before it; this takes 12 and 15 (GB300).
__global__ void __launch_bounds__(96) plan_kernel(PrepArgs A) {
    const MeshK& m = A.m;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if ((int)blockIdx.x >= A.plan_ctas) {
        const int64_t t = (int64_t)(blockIdx.x - A.plan_ctas) * 96 + threadIdx.x, nt = (int64_t)(gridDim.x - A.plan_ctas) * 96;
        for (int64_t i = t; i < A.words; i += nt) {
            A.cbits[i] = 0u;
            A.sbits[i] = 0u;
        }
        return;
    }
    if (blockIdx.x == 0 && wid == 2 && lane == 0) {
        if (A.step) *A.step = A.sp;
        Counters* cnt = A.cnt;
        if (A.new_call) {  // the previous lengths are kept for the sparse reset
            cnt->prev_n_inside = cnt->n_inside;
            cnt->prev_n_cut = cnt->n_cut;
            cnt->classify_next = 0; cnt->classify_any_next = 0;
            cnt->n_inside = 0; cnt->n_cut = 0; cnt->n_shared = 0; cnt->shared_marks = 0;
            cnt->exact_rechecks = 0; cnt->bbox_cells = 0;
            cnt->n_feat = 0; cnt->n_fb = 0; cnt->n_recheck = 0; cnt->n_ovf = 0; cnt->n_shent = 0;
            cnt->n_inband = 0; cnt->n_small = 0; cnt->couple_next = 0;
        }
    }
    const int s = blockIdx.x * 32 + lane;
    if (s >= A.S) return;
    const SolidK& k = A.sk[s];
    SolidPlan& p = A.plan[s];
    const Q4 q = state_quat(A.st[s]);
    const D3 x = state_pos(A.st[s]);
    if (wid == 0) {
        plan_box(m, k, q, x, p, A.cnt);
    } else if (wid == 1) {
        plan_nearest(m, q, x, A.st[s], p);
    } else {
        // local box holding the inside region (widened far beyond FP32 rounding): tiles of the classify pass that lie
        // outside it hold no inside vertex
        p.cull_box = 0;
        p.radius_cells = (float)k.radiusB * (1.f / m.h32[0]);
        if (!k.shape.prism && !k.infinite &&
            (k.shape.type == SDFIBM_SHAPE_SPHERE || k.shape.type == SDFIBM_SHAPE_ELLIPSOID ||
             k.shape.type == SDFIBM_SHAPE_BOX)) {
            const double* sp = k.shape.p;
            const bool ell = k.shape.type == SDFIBM_SHAPE_ELLIPSOID;  // ignores com
            const bool sph = k.shape.type == SDFIBM_SHAPE_SPHERE;
            for (int a = 0; a < 3; ++a) {
                const double half = sph ? sp[0] : sp[a];
                p.lbox_c[a] = ell ? 0.f : (float)(-k.shape.com[a]);
                p.lbox_s[a] = (float)(half * (1.0 + 1e-4) + 1e-4 * fabs(k.shape.com[a]) + 1e-30);
            }
            p.cull_box = 1;
        }
        p.n_inside = p.n_cut = 0;
        if (A.ftacc)
            for (int r = 0; r < 6; ++r) A.ftacc[6 * (int64_t)s + r] = 0.0;
    }
}

// ---- claims ----------------------------------------------------------------------------------------------------------
// Ct during a call holds claim words CT_KEY_BASE | (solid << 2 | type); CT_SHARED is set once a second solid touches
// the cell and the low bits then keep the largest claim (the last solid of the reference's serial loop).  Any value
// below CT_KEY_BASE -- zero, or the decoded Ct a previous call left -- is an unclaimed cell.
// One atomicMax claims the cell (any previous value is below every claim word); seeing another claim of this call
// in its return value, the claimer raises the word to the larger claim with CT_SHARED set.

// set bit (c >> 3) of a chunk bitmap (one bit per 8 consecutive cells)
__device__ inline void mark_chunk(uint32_t* bits, int64_t c) { atomicOr(bits + (c >> 8), 1u << ((c >> 3) & 31)); }

// claim pass over this call's lists; marks the chunks of the claimed cells in cbits and, for a cell claimed more than
// once, in sbits (every claimer after the first sees an earlier claim, so each shared cell's chunk is marked).
// Bound by the latency of the claims (a returning atomic on a line in memory), so a thread has four in flight; neighbours in
// the lists are neighbours on the mesh, so the first lane of a run marks its chunk.  0.150 -> 0.099 ms at 512^3 and 16 384
// solids, 0.030 -> 0.018 at 256^3 and 4096 (GB300).
constexpr int CLAIM_BATCH = 4;
__global__ void __launch_bounds__(256) claim_kernel(const int32_t* __restrict__ in_cell, const int32_t* __restrict__ in_solid,
                                                    const int32_t* __restrict__ cut_cell, const int32_t* __restrict__ cut_solid,
                                                    int32_t* __restrict__ Ct, Counters* cnt, int64_t N,
                                                    uint32_t* __restrict__ cbits, uint32_t* __restrict__ sbits) {
    const int64_t n_in = clamp_len(cnt->n_inside, cnt->list_cap), n = n_in + clamp_len(cnt->n_cut, cnt->list_cap);
    const int lane = threadIdx.x & 31;
    const int64_t step = (int64_t)gridDim.x * blockDim.x * CLAIM_BATCH;
    // whole warps: a warp's entries of a batch are consecutive
    for (int64_t e0 = (int64_t)blockIdx.x * blockDim.x * CLAIM_BATCH + threadIdx.x; e0 - lane < n; e0 += step) {
        int32_t c[CLAIM_BATCH];
        uint32_t key[CLAIM_BATCH], old[CLAIM_BATCH];
#pragma unroll
        for (int u = 0; u < CLAIM_BATCH; ++u) {
            const int64_t e = e0 + u * (int64_t)blockDim.x;
            c[u] = -1;
            key[u] = 0u;
            if (e < n) {
                const bool cut = e >= n_in;
                const int64_t ee = cut ? e - n_in : e;
                c[u] = cut ? cut_cell[ee] : in_cell[ee];
                const int32_t sw = cut ? cut_solid[ee] : in_solid[ee];
                key[u] = CT_KEY_BASE | ((uint32_t)(sw & LIST_SOLID_MASK) << 2) | (uint32_t)list_type(sw);
                if (c[u] >= N) c[u] = -1;
            }
        }
#pragma unroll
        for (int u = 0; u < CLAIM_BATCH; ++u)
            old[u] = c[u] >= 0 ? atomicMax(reinterpret_cast<uint32_t*>(Ct) + c[u], key[u]) : 0u;
#pragma unroll
        for (int u = 0; u < CLAIM_BATCH; ++u) {
            const int32_t chunk = c[u] >> 3, before = __shfl_up_sync(0xffffffffu, chunk, 1);
            if (c[u] >= 0 && (lane == 0 || before != chunk)) mark_chunk(cbits, c[u]);
        }
#pragma unroll
        for (int u = 0; u < CLAIM_BATCH; ++u)
            if (old[u] >= CT_KEY_BASE) {  // claimed before in this call
                atomicMax(reinterpret_cast<uint32_t*>(Ct) + c[u], max(key[u], old[u] & ~CT_SHARED) | CT_SHARED);
                mark_chunk(sbits, c[u]);
                atomicAdd(&cnt->shared_marks, 1);
            }
    }
}

__device__ inline int32_t decode_claim(uint32_t w) {
    const uint32_t k = (w & ~CT_SHARED) - CT_KEY_BASE;
    const int32_t s = (int32_t)(k >> 2), code = (int32_t)(k & 3);
    return code == 1 ? s + 4 : code;
}

// ---- connect: the connected set of the seed, bit-parallel --------------------------------------------------------------------------------
constexpr int CON_THREADS = 512;       // a CTA: one solid, or CON_MID_GROUPS groups of CON_MID with a solid each, or 16 warps
constexpr int CON_MID = 128;
constexpr int CON_MID_GROUPS = CON_THREADS / CON_MID;
constexpr int CON_WARPS = CON_THREADS / 32;

// fill upward (towards higher bits) inside runs of c starting from seeds s (s subset of c)
__device__ inline uint32_t fill_up(uint32_t c, uint32_t s) { return (((c + s) ^ c) & c) | s; }
__device__ inline uint32_t fill_down(uint32_t c, uint32_t s) { return __brev(fill_up(__brev(c), __brev(s))); }

// The cells that can have an inside vertex: the bbox cells of the mesh next to the plan's vertex box (the classify pass
// writes class bytes for these only).  c0: lowest cell, n: cells per axis (0 on some axis: none).
struct ActiveBox {
    int c0[3], n[3];
};
__device__ inline ActiveBox active_box(const MeshK& m, const SolidK& k, const SolidPlan& pl) {
    const int nm[3] = {m.nx, m.ny, m.nz};
    ActiveBox b;
    for (int a = 0; a < 3; ++a) {
        const int lo = max(max(pl.vlo[a] - 1, 0), pl.lo[a]);
        const int64_t top = (int64_t)pl.lo[a] + k.ext[a] - 1;
        const int hi = (int)min((int64_t)min(pl.vhi[a], nm[a] - 1), top);
        b.c0[a] = lo;
        b.n[a] = max(0, hi - lo + 1);
    }
    return b;
}

// bit index (row * sx + x) in the active box of the solid's nearest cell; -1 outside it
__device__ inline int64_t seed_bit(const SolidPlan& pl, const ActiveBox& b) {
    const int64_t x = pl.seed_ijk[0] - b.c0[0], y = pl.seed_ijk[1] - b.c0[1], z = pl.seed_ijk[2] - b.c0[2];
    if (x < 0 || y < 0 || z < 0 || x >= b.n[0] || y >= b.n[1] || z >= b.n[2]) return -1;
    return x + (int64_t)b.n[0] * (y + (int64_t)b.n[1] * z);
}

// The reached cells of one solid by a group of NT threads (a warp, CON_MID threads or a CTA):
// bitmaps of the active box, rows along x of W words, C (an inside vertex), I (all inside) and T (centre inside) from the class
// bytes, then the connected set of the seed, then the lists in ascending label order.
//
// Nearly every set is connected, and that can be seen in one parallel pass: every row of candidates is one run, every
// non-empty row but the first of its layer shares a column with the row before it, and every non-empty layer but the
// first has such a pair with the layer below.  Then C is the answer.  Only sets that fail this (plates thinner than a
// cell, concave shapes) are flooded from the seed, in sweeps that carry serial chains along y and z.  Bound by issue and
// by the largest solids, which a launch cannot end without.  Measured (GB300): bitmaps by a byte a lane and a ballot, lists by a
// word at a time, 0.52 ms at 512^3 and 16 384 solids and 0.16 at 256^3 and 4096; 16 bytes a lane, and lists by a lane a cell,
// 0.26 and 0.059.
__device__ inline FastDiv device_fastdiv(uint32_t d) {  // make_fastdiv for d < 2^31
    const uint32_t l = d <= 1 ? 0 : 32 - __clz(d - 1);
    return FastDiv{((1ull << (32 + l)) + d - 1) / d, 32 + l, d};
}
struct ConnectShared {
    int bad, starts, base_in, base_cut;
    unsigned first;          // lowest word of C with a bit
    FastDiv div_sy, div_w;   // by the rows per layer and by the words per row
    int cnt[16][2];          // reached cells of each warp's words
};
// barrier of a solid's group: a warp, CON_MID threads (each group its own hardware barrier), or the CTA
template <int NT>
__device__ __forceinline__ void group_sync() {
    if (NT == 32) __syncwarp();
    else if (NT == CON_THREADS) __syncthreads();
    else asm volatile("bar.sync %0, %1;" ::"r"(1 + (int)threadIdx.x / NT), "n"(NT) : "memory");
}
template <int NT>
__device__ __forceinline__ bool group_any(bool p) {
    if (NT == 32) return __any_sync(0xffffffffu, p);
    if (NT == CON_THREADS) return __syncthreads_or(p) != 0;
    uint32_t r;
    asm volatile(
        "{\n .reg .pred a, b;\n setp.ne.u32 a, %1, 0;\n barrier.cta.red.or.pred b, %2, %3, a;\n selp.u32 %0, 1, 0, b;\n}"
        : "=r"(r)
        : "r"((uint32_t)p), "r"(1 + (int)threadIdx.x / NT), "n"(NT)
        : "memory");
    return r != 0;
}

// rows of the active box, W words each
struct ConnectRows {
    int sx, sy, W, rows;
    FastDiv dsy, dw;
};
// bits 0 and 1 of 16 class bytes as two 16-bit masks
__device__ __forceinline__ void class_bits(uint4 v, uint32_t& b0, uint32_t& b1) {
    const uint32_t x[4] = {v.x, v.y, v.z, v.w};
    b0 = b1 = 0u;
#pragma unroll
    for (int i = 0; i < 4; ++i) {  // the product gathers the bytes' low bits in bits 28..31
        b0 |= (((x[i] & 0x01010101u) * 0x10204080u) >> 28) << (4 * i);
        b1 |= ((((x[i] >> 1) & 0x01010101u) * 0x10204080u) >> 28) << (4 * i);
    }
}
// bitmaps of the rows: a thread per word, which reads the up to 32 class bytes as the aligned 16-byte pieces they lie in (the
// bytes around them, other rows' or stale, are shifted and masked away; a solid's bytes begin and end with whole pieces)
template <int NT>
__device__ __forceinline__ void connect_bitmaps(const SolidK& k, const uint8_t* cls, const int* off, const ConnectRows& q, uint32_t* C,
                                                uint32_t* I, uint32_t* T, int tid) {
    const int nwords = q.rows * q.W;
    for (int w = tid; w < nwords; w += NT) {
        const int r = q.W == 1 ? w : (int)fdiv((uint32_t)w, q.dw), x = (w - r * q.W) << 5;
        const int kk = (int)fdiv((uint32_t)r, q.dsy), jj = r - kk * q.sy, n = min(32, q.sx - x);
        const uint8_t* p = cls + off[0] + x + (int64_t)k.ext[0] * ((jj + off[1]) + (int64_t)k.ext[1] * (kk + off[2]));
        const int sh = (int)((uintptr_t)p & 15);
        const uint4* p4 = reinterpret_cast<const uint4*>(p - sh);
        const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
        const uint4 v0 = p4[0], v1 = sh + n > 16 ? p4[1] : zero, v2 = sh + n > 32 ? p4[2] : zero;
        uint32_t l0, l1, m0, m1, h0, h1;
        class_bits(v0, l0, l1);
        class_bits(v1, m0, m1);
        class_bits(v2, h0, h1);
        const uint32_t msk = n == 32 ? 0xffffffffu : (1u << n) - 1u;
        const uint32_t b0 = __funnelshift_r(l0 | (m0 << 16), h0, sh) & msk, b1 = __funnelshift_r(l1 | (m1 << 16), h1, sh) & msk;
        C[w] = b0 | b1;   // classes: 1 all inside, 2 centre inside, 3 cut
        I[w] = b0 & ~b1;
        T[w] = b1 & ~b0;
    }
}
// what the rows say of the set's connectivity, into sh.bad, sh.starts and the layer bitmaps
template <int NT>
__device__ __forceinline__ void connect_proof(const ConnectRows& q, const uint32_t* C, ConnectShared& sh, uint32_t* layers, int lw,
                                              int tid) {
    const unsigned FULL = 0xffffffffu;
    int bad = 0, starts = 0;
    for (int r = tid; r < q.rows; r += NT) {
        const uint32_t* c = C + r * q.W;
        const int kk = (int)fdiv((uint32_t)r, q.dsy), jj = r - kk * q.sy;
        int first = -1, last = -1, pop = 0;
        uint32_t along = 0, below = 0;
        for (int w = 0; w < q.W; ++w) {
            const uint32_t x = c[w];
            if (!x) continue;
            pop += __popc(x);
            if (first < 0) first = (w << 5) + __ffs(x) - 1;
            last = (w << 5) + 31 - __clz(x);
            if (jj > 0) along |= x & c[w - q.W];
            if (kk > 0) below |= x & c[w - q.W * q.sy];
        }
        if (pop == 0) continue;
        if (last - first + 1 != pop) ++bad;
        if (!along) ++starts;
        atomicOr(layers + (kk >> 5), 1u << (kk & 31));
        if (below) atomicOr(layers + lw + (kk >> 5), 1u << (kk & 31));
    }
    bad = __reduce_add_sync(FULL, bad);
    starts = __reduce_add_sync(FULL, starts);
    if ((tid & 31) == 0) {
        if (bad) atomicAdd(&sh.bad, bad);
        if (starts) atomicAdd(&sh.starts, starts);
    }
}
// the words [w0, w1) of warp tid / 32
template <int NT>
__device__ __forceinline__ void connect_share(int nwords, int tid, int& w0, int& w1) {
    constexpr int NW = NT / 32;
    const int per = (((nwords + NW - 1) / NW) + 31) & ~31;
    w0 = min(nwords, (tid >> 5) * per);
    w1 = min(nwords, w0 + per);
}
// reached cells: sh.cnt of every warp, then the sums before this warp and of the group
template <int NT>
__device__ __forceinline__ void connect_count(const uint32_t* C, const uint32_t* I, int nwords, ConnectShared& sh, int tid) {
    const unsigned FULL = 0xffffffffu;
    int w0, w1, nin = 0, ncut = 0;
    connect_share<NT>(nwords, tid, w0, w1);
    for (int w = w0 + (tid & 31); w < w1; w += 32) {
        const uint32_t bits = C[w], in = I[w];
        nin += __popc(bits & in);
        ncut += __popc(bits & ~in);
    }
    nin = __reduce_add_sync(FULL, nin);
    ncut = __reduce_add_sync(FULL, ncut);
    if ((tid & 31) == 0) { sh.cnt[tid >> 5][0] = nin; sh.cnt[tid >> 5][1] = ncut; }
}
template <int NT>
__device__ __forceinline__ void connect_sums(const ConnectShared& sh, int tid, int& before_in, int& before_cut, int& tot_in,
                                             int& tot_cut) {
    before_in = before_cut = tot_in = tot_cut = 0;
#pragma unroll
    for (int i = 0; i < NT / 32; ++i) {
        const int a = sh.cnt[i][0], c = sh.cnt[i][1];
        if (i < (tid >> 5)) { before_in += a; before_cut += c; }
        tot_in += a;
        tot_cut += c;
    }
}
// the lists of the rows from pin and pcut on: 32 words at a time, a lane per listed cell, which finds its word in the prefix
// sums and its bit in the word
template <int NT>
__device__ __forceinline__ void connect_emit(const ConnectArgs& A, int s, const int* c0, const ConnectRows& q, const uint32_t* C,
                                             const uint32_t* I, const uint32_t* T, int64_t pin, int64_t pcut, int tid) {
    const unsigned FULL = 0xffffffffu;
    const int lane = tid & 31;
    int w0, w1;
    connect_share<NT>(q.rows * q.W, tid, w0, w1);
    for (int wb = w0; wb < w1; wb += 32) {
        const int w = wb + lane;
        uint32_t bits = 0, in = 0, ci = 0;
        int label = 0;
        if (w < w1) {
            bits = C[w]; in = I[w]; ci = T[w];
            const int r = (int)fdiv((uint32_t)w, q.dw), kk = (int)fdiv((uint32_t)r, q.dsy), jj = r - kk * q.sy;
            label = (c0[0] + ((w - r * q.W) << 5)) + A.m.nx * ((c0[1] + jj) + A.m.ny * (c0[2] + kk));
        }
        const uint32_t mi = bits & in, mc = bits & ~in;
        const int a = __popc(mi), c = __popc(mc);
        int xa = a, xc = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int ya = __shfl_up_sync(FULL, xa, o), yc = __shfl_up_sync(FULL, xc, o);
            if (lane >= o) { xa += ya; xc += yc; }
        }
        const int na = __shfl_sync(FULL, xa, 31), nc = __shfl_sync(FULL, xc, 31);
        for (int t = lane; t - lane < na; t += 32) {
            int src = 0;
#pragma unroll
            for (int h = 16; h > 0; h >>= 1)
                if (__shfl_sync(FULL, xa, src + h - 1) <= t) src += h;
            const uint32_t m = __shfl_sync(FULL, mi, src);
            const int r = t - __shfl_sync(FULL, xa - a, src), l = __shfl_sync(FULL, label, src);
            if (t < na) {
                A.in_cell[pin + t] = l + nth_bit(m, r);
                A.in_solid[pin + t] = list_word(s, 1);
            }
        }
        for (int t = lane; t - lane < nc; t += 32) {
            int src = 0;
#pragma unroll
            for (int h = 16; h > 0; h >>= 1)
                if (__shfl_sync(FULL, xc, src + h - 1) <= t) src += h;
            const uint32_t m = __shfl_sync(FULL, mc, src), tt = __shfl_sync(FULL, ci, src);
            const int r = t - __shfl_sync(FULL, xc - c, src), l = __shfl_sync(FULL, label, src);
            if (t < nc) {
                const int p = nth_bit(m, r);
                A.cut_cell[pcut + t] = l + p;
                A.cut_solid[pcut + t] = list_word(s, ((tt >> p) & 1u) ? 2 : 3);
            }
        }
        pin += na;
        pcut += nc;
    }
}

constexpr int CON_MAX_LAYERS = 2048;
template <int NT>
__device__ __forceinline__ void connect_body(const ConnectArgs& A, const SolidK& k, int s, uint32_t* bitmaps, ConnectShared& sh,
                                             uint32_t* layers, int max_layers, int tid) {
    const unsigned FULL = 0xffffffffu;
    const int lane = tid & 31;
    SolidPlan& pl = A.plan[s];
    const ActiveBox b = active_box(A.m, k, pl);
    const int sx = b.n[0], sy = b.n[1], sz = b.n[2];
    if (tid == 0) {
        sh.first = ~0u;
        sh.bad = 0;
        sh.starts = 0;
        sh.div_sy = device_fastdiv((uint32_t)max(1, sy));
        sh.div_w = device_fastdiv((uint32_t)max(1, (sx + 31) >> 5));
    }
    const bool proof = sz <= max_layers;
    const int lw = (sz + 31) >> 5;  // words per layer bitmap: non-empty layers, then layers joined to the one below
    if (proof)
        for (int i = tid; i < 2 * lw; i += NT) layers[i] = 0u;
    group_sync<NT>();
    if (pl.err || sx == 0 || sy == 0 || sz == 0) {
        if (tid == 0) { pl.n_inside = 0; pl.n_cut = 0; }
        return;
    }
    const int W = (sx + 31) >> 5, rows = sy * sz, nwords = rows * W;
    const ConnectRows q{sx, sy, W, rows, sh.div_sy, sh.div_w};
    uint32_t* C = bitmaps;
    uint32_t* I = C + nwords;
    uint32_t* T = I + nwords;
    uint32_t* R = T + nwords;
    const int off[3] = {b.c0[0] - pl.lo[0], b.c0[1] - pl.lo[1], b.c0[2] - pl.lo[2]};
    connect_bitmaps<NT>(k, A.scratch + k.scratch_off, off, q, C, I, T, tid);
    group_sync<NT>();
    bool connected = false;
    if (proof) {
        connect_proof<NT>(q, C, sh, layers, lw, tid);
        group_sync<NT>();
        int nl = 0, links = 0;
        for (int i = 0; i < lw; ++i) {
            nl += __popc(layers[i]);
            links += __popc(layers[lw + i]);
        }
        connected = nl > 0 && sh.bad == 0 && sh.starts == nl && links == nl - 1;
    }
    if (!connected) {
        unsigned first = ~0u;
        for (int w = tid; w < nwords; w += NT) {
            R[w] = 0u;
            if (C[w]) first = min(first, (unsigned)w);
        }
        first = __reduce_min_sync(FULL, first);
        if (lane == 0 && first != ~0u) atomicMin(&sh.first, first);
        group_sync<NT>();
        if (sh.first == ~0u) {  // no cell has an inside vertex
            if (tid == 0) { pl.n_inside = 0; pl.n_cut = 0; }
            return;
        }
        // the flood's seed: the nearest cell when it has an inside vertex, else the lowest-label cell that has one (the seed
        // fallback scan of cellenumerator.cpp:52-63; rows are in label order)
        if (tid == 0) {
            const int64_t sb = seed_bit(pl, b);
            int w = (int)sh.first;
            uint32_t bit = C[w] & (0u - C[w]);
            if (sb >= 0) {
                const int srow = (int)(sb / sx), x = (int)(sb - (int64_t)srow * sx);
                if ((C[srow * W + (x >> 5)] >> (x & 31)) & 1u) { w = srow * W + (x >> 5); bit = 1u << (x & 31); }
            }
            R[w] = bit;
        }
        group_sync<NT>();
        // directional sweeps until nothing changes
        const int max_rounds = 8 + 2 * (sx + sy + sz);
        for (int round = 0;; ++round) {
            int changed = 0;
            // x: carry fill along each row
            for (int row = tid; row < rows; row += NT) {
                uint32_t* r = R + row * W;
                const uint32_t* c = C + row * W;
                uint32_t carry = 0;
                for (int w = 0; w < W; ++w) {
                    const uint32_t seeds = (r[w] | (carry & 1u)) & c[w];
                    const uint32_t f = fill_up(c[w], seeds);
                    if (f != r[w]) { changed = 1; r[w] = f; }
                    carry = f >> 31;
                }
                carry = 0;
                for (int w = W - 1; w >= 0; --w) {
                    const uint32_t seeds = (r[w] | (carry << 31)) & c[w];
                    const uint32_t f = fill_down(c[w], seeds);
                    if (f != r[w]) { changed = 1; r[w] = f; }
                    carry = f & 1u;
                }
            }
            group_sync<NT>();
            // y, then z: forward and backward scans along each column of words (the running value in a register)
            for (int axis = 1; axis < 3; ++axis) {
                const int len = axis == 1 ? sy : sz, ncol = axis == 1 ? sz * W : sy * W, stride = axis == 1 ? W : sy * W;
                for (int col = tid; col < ncol; col += NT) {
                    const int u = col / W, w = col - u * W;
                    const int o = axis == 1 ? u * sy * W + w : u * W + w;
                    uint32_t* r = R + o;
                    const uint32_t* c = C + o;
                    uint32_t prev = r[0];
                    for (int j = 1; j < len; ++j) {
                        const uint32_t cur = r[j * stride], f = cur | (prev & c[j * stride]);
                        if (f != cur) { changed = 1; r[j * stride] = f; }
                        prev = f;
                    }
                    for (int j = len - 2; j >= 0; --j) {
                        const uint32_t cur = r[j * stride], f = cur | (prev & c[j * stride]);
                        if (f != cur) { changed = 1; r[j * stride] = f; }
                        prev = f;
                    }
                }
                group_sync<NT>();
            }
            if (!group_any<NT>(changed != 0)) break;
            if (round >= max_rounds) {
                if (tid == 0) set_error(A.cnt, DERR_FLOOD_LIMIT);
                break;
            }
        }
        C = R;
    }
    connect_count<NT>(C, I, nwords, sh, tid);
    group_sync<NT>();
    int before_in, before_cut, tot_in, tot_cut;
    connect_sums<NT>(sh, tid, before_in, before_cut, tot_in, tot_cut);
    if (tid == 0) {
        sh.base_in = atomicAdd(&A.cnt->n_inside, tot_in);
        sh.base_cut = atomicAdd(&A.cnt->n_cut, tot_cut);
        pl.n_inside = tot_in;
        pl.n_cut = tot_cut;
    }
    group_sync<NT>();
    if ((int64_t)sh.base_in + tot_in > A.cap_in || (int64_t)sh.base_cut + tot_cut > A.cap_cut) {
        if (tid == 0) set_error(A.cnt, DERR_CAPACITY);
        return;
    }
    connect_emit<NT>(A, s, b.c0, q, C, I, T, (int64_t)sh.base_in + before_in, (int64_t)sh.base_cut + before_cut, tid);
}

// Solids in order of size, the largest first: n_big of them a CTA each (bitmaps in shared memory, or in global memory above a
// size: bitmap_global), then n_mid of them CON_MID threads each, then the others a warp each; one launch, so that the smaller
// ones fill the SMs while the last of the larger ones end.  (A cluster of 8 CTAs for the largest ones gained nothing: 0.053
// against 0.059 ms at 256^3, 0.29 against 0.28 at 512^3.)
__global__ void __launch_bounds__(CON_THREADS, 2) connect_kernel(ConnectArgs A) {
    extern __shared__ uint32_t dsm[];
    __shared__ ConnectShared sh[CON_WARPS];
    __shared__ uint32_t layers[CON_WARPS * 2 * (CON_SMALL_WORDS / 32)];
    static_assert(CON_WARPS * 2 * (CON_SMALL_WORDS / 32) >= 2 * (CON_MAX_LAYERS / 32) &&
                      CON_WARPS * (CON_SMALL_WORDS / 32) >= CON_MID_GROUPS * (CON_MID_WORDS / 32), "layer bitmaps");
    const int mid_ctas = (A.n_mid + CON_MID_GROUPS - 1) / CON_MID_GROUPS, tid = threadIdx.x;
    const int b = (int)blockIdx.x - A.n_big;
    if (b < 0) {
        const int s = A.solids ? A.solids[blockIdx.x] : (int)blockIdx.x;
        const SolidK& k = A.sk[s];
        connect_body<CON_THREADS>(A, k, s, k.bitmap_global ? A.gbitmaps + k.bitmap_off : dsm, sh[0], layers, CON_MAX_LAYERS, tid);
    } else if (b < mid_ctas) {
        const int g = tid / CON_MID, item = b * CON_MID_GROUPS + g;
        if (item >= A.n_mid) return;
        const int s = A.solids[A.n_big + item];
        connect_body<CON_MID>(A, A.sk[s], s, dsm + g * 4 * CON_MID_WORDS, sh[g], layers + g * 2 * (CON_MID_WORDS / 32), CON_MID_WORDS,
                              tid % CON_MID);
    } else {
        const int g = tid >> 5, item = (b - mid_ctas) * CON_WARPS + g;
        if (item >= A.n_small) return;
        const int s = A.solids[A.n_big + A.n_mid + item];
        connect_body<32>(A, A.sk[s], s, dsm + g * 4 * CON_SMALL_WORDS, sh[g], layers + g * 2 * (CON_SMALL_WORDS / 32),
                         CON_SMALL_WORDS, tid & 31);
    }
}

// ---- shared cells -----------------------------------------------------------------------------------------------------
// slot of cell c in the shared table, inserting it on first use; -1 (and an error flag) when the table is full
__device__ inline int shared_slot(const CoupleArgs& A, int32_t c) {
    uint32_t h = ((uint32_t)c * 2654435761u) & (uint32_t)A.sh_mask;
    for (int p = 0; p < SHARED_MAX_PROBES; ++p) {
        const int32_t k = atomicCAS(A.sh_keys + h, -1, c);
        if (k == -1) {
            const int u = atomicAdd(&A.cnt->n_shared, 1);
            if (u <= A.sh_mask) A.sh_used[u] = (int32_t)h;
            return (int)h;
        }
        if (k == c) return (int)h;
        h = (h + 1) & (uint32_t)A.sh_mask;
    }
    set_error(A.cnt, DERR_SHARED_TABLE);
    return -1;
}

// ---- couple ---------------------------------------------------------------------------------------------------------
constexpr int CPL_THREADS = 256;



// Reduce-scatter of 8 values over the warp in three xor steps: afterwards each lane holds slot (lane >> 2) & 7 summed
// over the 8 lanes that share its bits 0..1; warp_total4 then adds the 4 lanes that differ in those bits.
template <typename T>
__device__ __forceinline__ T reduce_scatter8(T* v, int lane) {
    {
        const bool up = (lane & 16) != 0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const T send = up ? v[i] : v[i + 4];
            const T keep = up ? v[i + 4] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
        }
    }
    {
        const bool up = (lane & 8) != 0;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const T send = up ? v[i] : v[i + 2];
            const T keep = up ? v[i + 2] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
        }
    }
    const bool up = (lane & 4) != 0;
    const T send = up ? v[0] : v[1];
    const T keep = up ? v[1] : v[0];
    return keep + __shfl_xor_sync(0xffffffffu, send, 4);
}
// sum over the 4 lanes that differ in bits 0..1 (FP64)
__device__ __forceinline__ double warp_total4(double x) {
    x += __shfl_xor_sync(0xffffffffu, x, 2);
    x += __shfl_xor_sync(0xffffffffu, x, 1);
    return x;
}

// Two-float arithmetic (Dekker / Knuth): a + b = s + e and a * b = p + e exactly, with explicit rounding intrinsics
// so that nothing is contracted or reassociated.
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}
// U - (u0 + a p + b q) with u0, p, q given as FP32 pairs hi + lo and a, b small integers, rounded once to FP32 after
// an error of about 2^-46 of the magnitudes
__device__ __forceinline__ float ff_u_minus_us(float U, float u0h, float u0l, float a, float ph, float pl, float b,
                                               float qh, float ql) {
    const float t1 = __fmul_rn(a, ph), e1 = __fmaf_rn(a, ph, -t1);
    const float t2 = __fmul_rn(b, qh), e2 = __fmaf_rn(b, qh, -t2);
    float s1, f1, s2, f2;
    two_sum(u0h, t1, s1, f1);
    two_sum(s1, t2, s2, f2);
    const float lo = __fadd_rn(__fadd_rn(__fadd_rn(u0l, __fadd_rn(e1, e2)), __fadd_rn(f1, f2)),
                               __fmaf_rn(a, pl, __fmul_rn(b, ql)));
    float d, g;
    two_sum(U, -s2, d, g);
    return __fadd_rn(d, __fsub_rn(g, lo));
}

// Conversions between the formats on the integer pipes: the FP64 pipe, which the exact forcing keeps busy, takes 64 issue slots
// for one.  Zeros and normal values (the others go to the instruction); double to float rounds to nearest even.
__device__ __forceinline__ double wide(float x) {
    const uint32_t b = __float_as_uint(x), m = b & 0x7fffffffu;
    double r = __hiloint2double((int)((b & 0x80000000u) | ((m >> 3) + 0x38000000u)), (int)(b << 29));
    if (m == 0u) r = __hiloint2double((int)b, 0);
    else if (m - 0x00800000u >= 0x7f000000u) r = (double)x;
    return r;
}
__device__ __forceinline__ float narrow(double x) {
    const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x), m = hi & 0x7fffffffu;
    const uint64_t v = ((uint64_t)m << 32) | lo, r = v + 0x0fffffffu + ((lo >> 29) & 1u);
    uint32_t b = (uint32_t)(r >> 29) + 0x40000000u;
    if ((m | lo) == 0u) b = 0u;
    else if (m - 0x38100000u >= 0x0fd00000u) return (float)x;  // outside 2^-126 .. 2^127
    return __uint_as_float(b | (hi & 0x80000000u));
}

// Per-cell forcing of solid s on cell c with fluid velocity U (pcHydrodynamicInteraction, solidcloud.cpp:384-390):
// alpha, the FP32 Fs and the cell's contributions to the force/torque sums (:411-421), FP64 in f6 (exact mode) or
// FP32 in g6.
template <bool EXACT>
__device__ __forceinline__ float cell_forcing(const CoupleArgs& A, int64_t c, int s, int type, float dtINV32,
                                              double dtINV, float fs[3], double f6[8], float g6[8], float Ux,
                                              float Uy, float Uz) {
    const MeshK& m = A.m;
    int i, j, k;
    cell_ijk(m, c, i, j, k);
    float alpha = 1.f;
    if (type != 1) {
        // computed by the fraction pass for every cut candidate of the solid's bbox
        const SolidK& ks = A.sk[s];
        const int32_t* lo = A.plan[s].lo;
        const int64_t li = (i - lo[0]) + (int64_t)ks.ext[0] * ((j - lo[1]) + (int64_t)ks.ext[1] * (k - lo[2]));
        alpha = A.alpha[ks.scratch_off + li];
        // a SUBSAMPLE count whose undecided points were rechecked on full warps
        if (alpha < 0.f) alpha = __fdiv_rn(-alpha - 1.f, (float)A.count_samples);
    }
    if (EXACT) {
        // FP64; the cross products as fused multiply-adds: 24 operations a cell for 43 as written out with conversions
        const sdfibm_solid_state& st = A.st[s];
        // mesh_C from its per-axis tables: the FP64 pipe also converts the indices, twelve of its instructions a cell
        const double dx = A.centres[i] - st.pos[0], dy = A.centres[m.nx + j] - st.pos[1],
                     dz = A.centres[m.nx + m.ny + k] - st.pos[2];
        const double ox = st.omega[0], oy = st.omega[1], oz = st.omega[2];
        double fx = __fma_rn(oz, dy, __fma_rn(-oy, dz, wide(Ux) - st.vel[0]));
        double fy = __fma_rn(ox, dz, __fma_rn(-oz, dx, wide(Uy) - st.vel[1]));
        double fz = __fma_rn(oy, dx, __fma_rn(-ox, dy, wide(Uz) - st.vel[2]));
        if (alpha != 1.f) {
            const double al = wide(alpha);
            fx *= al; fy *= al; fz *= al;
        }
        f6[0] = fx; f6[1] = fy; f6[2] = fz;
        f6[3] = __fma_rn(dy, fz, -(dz * fy)); f6[4] = __fma_rn(dz, fx, -(dx * fz)); f6[5] = __fma_rn(dx, fy, -(dy * fx));
        fs[0] = narrow(fx * dtINV); fs[1] = narrow(fy * dtINV); fs[2] = narrow(fz * dtINV);
    } else {
        // U - us in two-float arithmetic (the difference can cancel; about 2^-46 of the magnitudes, against 2^-24 of
        // the difference for the FP32 rounding that follows), FP32 after it.  The cell offsets from the seed are
        // exact small integers.
        const SolidPlan& pl = A.plan[s];
        const float di = (float)(i - pl.seed_ijk[0]), dj = (float)(j - pl.seed_ijk[1]), dk = (float)(k - pl.seed_ijk[2]);
        const float fx = alpha * ff_u_minus_us(Ux, pl.us_hi[0], pl.us_lo[0], dj, pl.ds_hi[0], pl.ds_lo[0], dk,
                                               pl.ds_hi[1], pl.ds_lo[1]);
        const float fy = alpha * ff_u_minus_us(Uy, pl.us_hi[1], pl.us_lo[1], di, pl.ds_hi[2], pl.ds_lo[2], dk,
                                               pl.ds_hi[3], pl.ds_lo[3]);
        const float fz = alpha * ff_u_minus_us(Uz, pl.us_hi[2], pl.us_lo[2], di, pl.ds_hi[4], pl.ds_lo[4], dj,
                                               pl.ds_hi[5], pl.ds_lo[5]);
        const float dx = __fmaf_rn(di, m.h32[0], pl.cb32[0]), dy = __fmaf_rn(dj, m.h32[1], pl.cb32[1]),
                    dz = __fmaf_rn(dk, m.h32[2], pl.cb32[2]);
        g6[0] = fx; g6[1] = fy; g6[2] = fz;
        g6[3] = dy * fz - dz * fy; g6[4] = dz * fx - dx * fz; g6[5] = dx * fy - dy * fx;
        fs[0] = fx * dtINV32; fs[1] = fy * dtINV32; fs[2] = fz * dtINV32;
    }
    return alpha;
}

// The cell's FP64 sums in the shared table (As, Ts, Fs of every solid on a cell several solids touch).
__device__ __forceinline__ void add_shared(const CoupleArgs& A, int64_t c, float alpha, const float fs[3]) {
    const int slot = shared_slot(A, (int32_t)c);
    if (slot >= 0) {
        double* v = A.sh_vals + 5 * (int64_t)slot;
        atomicAdd(v + 0, (double)alpha);
        atomicAdd(v + 1, (double)alpha);
        atomicAdd(v + 2, (double)fs[0]);
        atomicAdd(v + 3, (double)fs[1]);
        atomicAdd(v + 4, (double)fs[2]);
    }
}

// After the claims, on the side stream beside the fraction kernels.
// Shared cells: the list entries on cells that several solids claimed, compacted into shent (entry index into the in list
// then the cut list).  Only the chunks marked in sbits are looked at; nothing when no cell was claimed twice.
// Sparse reset (prev_in_cell not null): the cells the previous call touched and this call does not go back to zero -- the
// sparse form of solidcloud.cpp:438-441.  Cells in the chunks marked in cbits are left to couple_chunks_kernel, which writes
// every cell of those chunks.
__global__ void scan_reset_kernel(const int32_t* __restrict__ in_cell, const int32_t* __restrict__ cut_cell, Counters* cnt,
                                  int64_t N, const uint32_t* __restrict__ sbits, uint32_t* __restrict__ shent,
                                  int64_t shent_cap, const int32_t* __restrict__ prev_in_cell,
                                  const int32_t* __restrict__ prev_cut_cell, float* As, float* Fs, float* Ts, int32_t* Ct,
                                  const uint32_t* __restrict__ cbits) {
    constexpr int B = 4;  // entries of a thread in flight: bound by their latency
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    if (cnt->shared_marks != 0) {
        const int64_t n_in = clamp_len(cnt->n_inside, cnt->list_cap), n_cut = clamp_len(cnt->n_cut, cnt->list_cap);
        for (int64_t e0 = t0; e0 < n_in + n_cut; e0 += B * nt) {
            int32_t c[B];
            uint32_t w[B];
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const int64_t e = e0 + u * nt;
                c[u] = e >= n_in + n_cut ? -1 : (e < n_in ? in_cell[e] : cut_cell[e - n_in]);
                if (c[u] >= N) c[u] = -1;
            }
#pragma unroll
            for (int u = 0; u < B; ++u) w[u] = c[u] >= 0 ? sbits[c[u] >> 8] : 0u;
#pragma unroll
            for (int u = 0; u < B; ++u) {
                if (!((w[u] >> ((c[u] >> 3) & 31)) & 1u)) continue;  // no cell of this chunk is shared
                if (!(reinterpret_cast<const uint32_t*>(Ct)[c[u]] & CT_SHARED)) continue;
                const int32_t slot = atomicAdd(&cnt->n_shent, 1);
                if (slot < shent_cap) shent[slot] = (uint32_t)(e0 + u * nt);
                else set_error(cnt, DERR_SHARED_TABLE);
            }
        }
    }
    if (prev_in_cell) {
        const int64_t n_in = clamp_len(cnt->prev_n_inside, cnt->list_cap), n_cut = clamp_len(cnt->prev_n_cut, cnt->list_cap);
        for (int64_t e0 = t0; e0 < n_in + n_cut; e0 += B * nt) {
            int32_t cc[B];
            uint32_t w[B];
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const int64_t e = e0 + u * nt;
                cc[u] = e >= n_in + n_cut ? -1 : (e < n_in ? prev_in_cell[e] : prev_cut_cell[e - n_in]);
                if (cc[u] >= N) cc[u] = -1;
            }
#pragma unroll
            for (int u = 0; u < B; ++u) w[u] = cc[u] >= 0 ? cbits[cc[u] >> 8] : ~0u;
#pragma unroll
            for (int u = 0; u < B; ++u) {
                const int64_t c = cc[u];
                if ((w[u] >> ((c >> 3) & 31)) & 1u) continue;  // written by the chunked coupling
                if (reinterpret_cast<const uint32_t*>(Ct)[c] >= CT_KEY_BASE) continue;
                As[c] = 0.f; Ts[c] = 0.f; Ct[c] = 0;
                Fs[c] = 0.f; Fs[N + c] = 0.f; Fs[2 * N + c] = 0.f;
            }
        }
    }
}

// Shared cells, second half (after the fraction kernels): every compacted entry adds its solid's As / Ts / Fs to the
// cell's FP64 sums in the shared table (finalize_kernel writes them) and its force/torque contribution to the solid's sums.
template <bool EXACT>
__device__ __noinline__ void couple_shared(const CoupleArgs& A, int64_t n) {
    const int64_t N = A.m.ncells;
    const int64_t n_in = clamp_len(A.cnt->n_inside, A.cnt->list_cap);
    const double dtINV = A.step->dtINV;
    const float dtINV32 = (float)dtINV;
    for (int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; q < n; q += (int64_t)gridDim.x * blockDim.x) {
        const int64_t e = A.shent[q];
        const bool is_cut = e >= n_in;
        const int32_t c = is_cut ? A.cut_cell[e - n_in] : A.in_cell[e];
        const int32_t sw = is_cut ? A.cut_solid[e - n_in] : A.in_solid[e];
        const int s = sw & LIST_SOLID_MASK;
        double f6[8] = {0, 0, 0, 0, 0, 0, 0, 0};
        float g6[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        float fs[3];
        const float alpha = cell_forcing<EXACT>(A, c, s, list_type(sw), dtINV32, dtINV, fs, f6, g6, A.U[c],
                                                A.U[N + c], A.U[2 * N + c]);
        add_shared(A, c, alpha, fs);
        for (int r = 0; r < 6; ++r) atomicAdd(A.ftacc + 6 * s + r, EXACT ? f6[r] : (double)g6[r]);
    }
}

// Chunked coupling.  The claim pass marks in cbits every chunk of 8 consecutive cells that holds a claimed cell (and
// in sbits the chunks of cells claimed more than once).  This kernel runs over the marked chunks, a warp per 64 bits of the
// bitmap, four chunks at a time with 8 lanes each, and writes the four fields of every
// cell of a marked chunk: zero for an unclaimed cell (a cell that no solid touches, or one the previous call touched:
// the sparse reset inside these chunks), zero As / Ts / Fs and the claim word kept in Ct for a shared cell
// (finalize_kernel writes its sums and decodes its Ct), and for a cell claimed once the forcing of its solid.  The
// cells claimed once are queued per warp in shared memory and computed 32 at a time on full warps; their values
// land in the same sectors a few instructions after the zeros, so every 32-byte sector of a field is written whole
// while L2 holds it and DRAM takes no read-modify-write, and U / Ct sectors are read once whatever the lists' order.
// The force/torque sums are reduced per solid over the lanes of the warp (segmented by solid) before one FP64
// atomic per (solid, component).  The marks stay until the next interact clears them (sdfibm_cuda_apply_forcing
// visits the same chunks).
constexpr int CPL_WARPS = CPL_THREADS / 32;

// Force and torque sums of the FP64 forcing: the warp's contributions go through shared memory, and lane (g, r) of 5 x 6 adds
// component r of the cells 7 g .. 7 g + 6, seven additions a batch, keeping the sum of a run of cells of one solid (over
// batches too) until another solid follows.
struct FtSum {
    double acc;
    int solid;
};
constexpr int FT_GROUPS = 5, FT_CELLS = 7, FT_STRIDE = 33;
__device__ __forceinline__ void ft_flush(const CoupleArgs& A, FtSum& q, int r) {
    if (q.solid >= 0) atomicAdd(A.ftacc + 6 * q.solid + r, q.acc);
    q.acc = 0.0;
}

// forcing of the first `count` queued cells (lane l takes entry l), written to the fields, F/T summed per solid
template <bool EXACT>
__device__ __forceinline__ void couple_queued(const CoupleArgs& A, const int32_t* qc, const uint32_t* qk, double* sv, FtSum& ft,
                                              int count, float dtINV32, double dtINV) {
    const int lane = threadIdx.x & 31;
    const int64_t N = A.m.ncells;
    int s = -1;
    double f6[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    float g6[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (lane < count) {
        const int64_t c = qc[lane];
        const uint32_t key = qk[lane] - CT_KEY_BASE;
        s = (int)(key >> 2);
        const int type = (int)(key & 3u);
        float fs[3];
        const float alpha = cell_forcing<EXACT>(A, c, s, type, dtINV32, dtINV, fs, f6, g6, A.U[c], A.U[N + c],
                                                A.U[2 * N + c]);
        A.As[c] = fminf(alpha, 1.0f);
        A.Ts[c] = alpha;
        A.Fs[c] = fs[0];
        A.Fs[N + c] = fs[1];
        A.Fs[2 * N + c] = fs[2];
        A.Ct[c] = type == 1 ? s + 4 : type;
    }
    if (EXACT) {
#pragma unroll
        for (int r = 0; r < 6; ++r) sv[r * FT_STRIDE + lane] = f6[r];
        __syncwarp();
        const int g = lane / 6, r = lane - 6 * g;
        if (g < FT_GROUPS) {
            double v[FT_CELLS];
            int who[FT_CELLS];
#pragma unroll
            for (int i = 0; i < FT_CELLS; ++i) {
                const int e = min(FT_CELLS * g + i, 31);
                v[i] = sv[r * FT_STRIDE + e];
                who[i] = FT_CELLS * g + i < count ? (int)((qk[e] - CT_KEY_BASE) >> 2) : -1;
            }
#pragma unroll
            for (int i = 0; i < FT_CELLS; ++i) {
                if (who[i] < 0) break;
                if (who[i] != ft.solid) {
                    ft_flush(A, ft, r);
                    ft.solid = who[i];
                }
                ft.acc += v[i];
            }
        }
        return;
    }
    uint32_t pend = __ballot_sync(0xffffffffu, s >= 0);
    while (pend) {
        const int sl = __shfl_sync(0xffffffffu, s, __ffs(pend) - 1);
        const bool mine = s == sl;
        pend &= ~__ballot_sync(0xffffffffu, mine);
        float t[8];
#pragma unroll
        for (int r = 0; r < 8; ++r) t[r] = mine ? g6[r] : 0.f;
        const double v = warp_total4((double)reduce_scatter8(t, lane));
        const int slot = lane >> 2;
        if ((lane & 3) == 0 && slot < 6) atomicAdd(A.ftacc + 6 * sl + slot, v);
    }
}

// The FP32 forcing is bound by memory latency.  The FP64 forcing is bound by the FP64 pipe (1/64 of the FP32 rate): 24
// operations a cell and 7 a batch of 32 for the sums; its items are taken as warps get free, since their cells differ much in
// number.  Measured (GB300): FP64 at 256^3 and 4096 solids, 2.2 M cells, 0.34 -> 0.20 ms (the earlier form: 43 operations a
// cell and conversions on the same pipe, a reduction of nine additions for every distinct solid of a batch, about 3; chunks
// in patches of 64 x 8 cells paid then, now they take 0.21); FP32 at 512^3, 10.5 M cells, 0.56 ms.
template <bool EXACT>
__global__ void __launch_bounds__(CPL_THREADS, 4) couple_chunks_kernel(CoupleArgs A) {
    __shared__ int32_t s_qc[CPL_WARPS][64];   // per warp: queued cells claimed once, and their claim words
    __shared__ uint32_t s_qk[CPL_WARPS][64];
    const unsigned FULL = 0xffffffffu;
    const int64_t N = A.m.ncells;
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5, grp = lane >> 3, sub = lane & 7;
    int32_t* qc = s_qc[wib];
    uint32_t* qk = s_qk[wib];
    __shared__ double s_ft[EXACT ? CPL_WARPS : 1][6 * FT_STRIDE];
    double* sv = s_ft[EXACT ? wib : 0];
    FtSum ft{0.0, -1};
    const int64_t words = (N + 255) >> 8, items = (words + 1) >> 1;
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    const double dtINV = A.step->dtINV;
    const float dtINV32 = (float)dtINV;
    const uint32_t* C = reinterpret_cast<const uint32_t*>(A.Ct);
    const int64_t n_shared = min((int64_t)A.cnt->n_shent, A.shent_cap);
    if (n_shared > 0) couple_shared<EXACT>(A, n_shared);
    int nq = 0;  // warp-uniform
    // tickets of up to 32 items, about five tickets a warp; the items of a ticket lie far apart (a solid's cells spread over the
    // warps) and their marks are read by a lane each.  FP64: the next ticket is asked for while this one is done.
    const int64_t run = max((int64_t)1, min((int64_t)32, items / (5 * nw))), tickets = (items + run - 1) / run;
    for (int64_t t = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < tickets;) {
        const int64_t first = t;
        int asked = 0;
        if (EXACT && lane == 0) asked = atomicAdd(&A.cnt->couple_next, 1);
        uint64_t marks = 0;
        const int64_t w = 2 * (first + lane * tickets);
        if (w < words) {
            marks = A.cbits[w];
            if (w + 1 < words) marks |= (uint64_t)A.cbits[w + 1] << 32;
        }
        for (unsigned some = __ballot_sync(FULL, marks != 0); some; some &= some - 1) {
            const int64_t cur = first + (__ffs(some) - 1) * tickets;
            uint64_t rem = __shfl_sync(FULL, marks, __ffs(some) - 1);  // bit: chunk
            auto cell_of = [&](uint64_t left) {  // this lane's cell of the next four chunks of `left`, -1: none
                for (int q = 0; q < grp; ++q) left &= left - 1;
                const int at = __ffsll((long long)left) - 1;
                if (at < 0) return (int64_t)-1;
                const int64_t c = (cur << 9) + (at << 3) + sub;
                return c < N ? c : (int64_t)-1;
            };
            int64_t c = cell_of(rem);
            uint32_t claim = c >= 0 ? C[c] : 0u;
            while (rem) {  // warp-uniform: four marked chunks per pass, the claims of the next pass loaded ahead
#pragma unroll
                for (int q = 0; q < 4; ++q) rem &= rem - 1;
                const int64_t c_next = cell_of(rem);
                const uint32_t claim_next = c_next >= 0 ? C[c_next] : 0u;
                const bool single = claim >= CT_KEY_BASE && !(claim & CT_SHARED);
                if (c >= 0 && !single) {
                    A.As[c] = 0.f;
                    A.Ts[c] = 0.f;
                    A.Fs[c] = 0.f;
                    A.Fs[N + c] = 0.f;
                    A.Fs[2 * N + c] = 0.f;
                    A.Ct[c] = (claim & CT_SHARED) ? (int32_t)claim : 0;
                }
                const uint32_t m = __ballot_sync(FULL, single);
                if (single) {
                    const int pos = nq + __popc(m & ((1u << lane) - 1u));
                    qc[pos] = (int32_t)c;
                    qk[pos] = claim;
                }
                nq += __popc(m);
                __syncwarp();
                if (nq >= 32) {
                    couple_queued<EXACT>(A, qc, qk, sv, ft, 32, dtINV32, dtINV);
                    __syncwarp();
                    if (lane < nq - 32) {
                        qc[lane] = qc[32 + lane];
                        qk[lane] = qk[32 + lane];
                    }
                    nq -= 32;
                    __syncwarp();
                }
                c = c_next;
                claim = claim_next;
            }
        }
        t = nw + (EXACT ? (int64_t)__shfl_sync(FULL, asked, 0) : t);
    }
    if (nq > 0) couple_queued<EXACT>(A, qc, qk, sv, ft, nq, dtINV32, dtINV);
    if (EXACT && lane < 6 * FT_GROUPS) ft_flush(A, ft, lane % 6);
}
void launch_couple_chunks(const CoupleArgs& A, bool exact, int grid, cudaStream_t st) {
    if (exact) couple_chunks_kernel<true><<<grid, CPL_THREADS, 0, st>>>(A);
    else couple_chunks_kernel<false><<<grid, CPL_THREADS, 0, st>>>(A);
}
int couple_occupancy(bool exact) {  // resident CTAs per SM
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        &occ, exact ? (const void*)couple_chunks_kernel<true> : (const void*)couple_chunks_kernel<false>, CPL_THREADS, 0);
    return occ;
}

// FP64 cell centres per axis, x then y then z (mesh_C), once per context
__global__ void centres_kernel(MeshK m, double* __restrict__ out) {
    const int64_t n = (int64_t)m.nx + m.ny + m.nz;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = i < m.nx ? mesh_centre(m, 0, i)
                          : (i < (int64_t)m.nx + m.ny ? mesh_centre(m, 1, i - m.nx) : mesh_centre(m, 2, i - m.nx - m.ny));
}

// Forcing applied to a GPU-resident fluid (main.cpp:70-77, its cell fields): U = U - Fs dt and T = (1 - As) T + Ts,
// in FP64 and rounded once to the FP32 fields, over the chunks the last interact marked in cbits.  Every other cell
// has As = Fs = Ts = 0 there and keeps its values, as in the dense update.  With cbits == nullptr (unstructured
// meshes) every cell is visited.  A warp reads its words, a lane each, and queues the cells of the marked chunks that change (a
// cell without force and solid keeps U and T), 32 consecutive cells at a time; they are updated on full warps.
// Bound by the FP64 pipe: 6 operations a cell.  Early steps of 1800 solids at 256 x 288 x 224 166 -> 87 us (15 operations,
// with the conversions, for every cell of a marked chunk, 13 of 32 lanes active), 100 circles at 1024^2 31 -> 25 (GB300).
constexpr int APPLY_THREADS = 256;
__device__ __forceinline__ void apply_queued(int64_t N, const int32_t* q, int count, double dt, const float* __restrict__ As,
                                             const float* __restrict__ Fs, const float* __restrict__ Ts, float* __restrict__ U,
                                             float* __restrict__ T) {
    const int lane = threadIdx.x & 31;
    if (lane >= count) return;
    const int64_t c = q[lane];
    float f[3], u[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) { f[a] = Fs[a * N + c]; u[a] = U[a * N + c]; }
    // separate roundings, as the solver's own field operations (no contraction into FMAs)
#pragma unroll
    for (int a = 0; a < 3; ++a) U[a * N + c] = narrow(__dsub_rn(wide(u[a]), __dmul_rn(wide(f[a]), dt)));
    if (T) T[c] = narrow(__dadd_rn(__dmul_rn(__dsub_rn(1.0, wide(As[c])), wide(T[c])), wide(Ts[c])));
}
__global__ void __launch_bounds__(APPLY_THREADS) apply_forcing_kernel(int64_t N, const uint32_t* __restrict__ cbits, double dt,
                                                                      const float* __restrict__ As, const float* __restrict__ Fs,
                                                                      const float* __restrict__ Ts, float* __restrict__ U,
                                                                      float* __restrict__ T) {
    __shared__ int32_t s_q[APPLY_THREADS / 32][64];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int32_t* q = s_q[threadIdx.x >> 5];
    const int64_t words = (N + 255) >> 8;
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    const int64_t run = max((int64_t)1, min((int64_t)32, words / (8 * nw)));
    const int64_t tickets = (words + run - 1) / run;  // of up to 32 words, far apart
    const bool finite = fabs(dt) < INFINITY;          // else every cell changes
    int nq = 0;                                       // warp-uniform
    for (int64_t t0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; t0 < tickets; t0 += nw) {
        const int64_t w0 = t0 + lane * tickets;
        const uint32_t marks = w0 >= words ? 0u : (cbits ? cbits[w0] : 0xffffffffu);
        for (unsigned some = __ballot_sync(FULL, marks != 0u); some; some &= some - 1) {
            const int src = __ffs(some) - 1;
            const int64_t w = t0 + src * tickets;
            const uint32_t word = __shfl_sync(FULL, marks, src);
            unsigned change = 0;  // bit t: this lane's cell of 32 t .. 32 t + 31
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const int idx = 32 * t + lane;
                const int64_t c = (w << 8) + idx;
                if (((word >> (idx >> 3)) & 1u) && c < N &&
                    (!finite || Fs[c] != 0.f || Fs[N + c] != 0.f || Fs[2 * N + c] != 0.f || (T && (As[c] != 0.f || Ts[c] != 0.f))))
                    change |= 1u << t;
            }
#pragma unroll
            for (int t = 0; t < 8; ++t) {
                const bool on = (change >> t) & 1u;
                const unsigned m = __ballot_sync(FULL, on);
                if (!m) continue;
                if (on) q[nq + __popc(m & ((1u << lane) - 1u))] = (int32_t)((w << 8) + 32 * t + lane);
                nq += __popc(m);
                __syncwarp();
                if (nq >= 32) {
                    apply_queued(N, q, 32, dt, As, Fs, Ts, U, T);
                    __syncwarp();
                    nq -= 32;
                    const int32_t keep = q[32 + lane];
                    __syncwarp();
                    if (lane < nq) q[lane] = keep;
                    __syncwarp();
                }
            }
        }
    }
    if (nq > 0) apply_queued(N, q, nq, dt, As, Fs, Ts, U, T);
}

// ---- finalize: cells shared by several solids, forces ------------------------------------------------------------------
// FP64 sums rounded once to the FP32 fields, Ct decoded from the largest claim, As = min(As, 1) (checkAlpha); the slot
// is cleared for the next call.  F = rho_f * V / dt * sum f, T = rho_f * V / dt * sum (C - x) x f  (solidcloud.cpp:411-421),
// into ft and the solid's state (Solid::setFluidForceAndTorque).
__global__ void finalize_kernel(float* __restrict__ As, float* __restrict__ Ts, float* __restrict__ Fs,
                                int32_t* __restrict__ Ct, const Counters* cnt, int64_t N, int32_t* __restrict__ sh_keys,
                                double* __restrict__ sh_vals, const int32_t* __restrict__ sh_used, int32_t sh_mask,
                                const double* __restrict__ ftacc, double* __restrict__ ft, int S, const StepParams* step,
                                sdfibm_solid_state* __restrict__ st) {
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    const double scale = step->ft_scale;
    for (int64_t e = t0; e < 6 * (int64_t)S; e += nt) {
        const int64_t s = e / 6, r = e - 6 * s;
        const double y = ftacc[e] * scale;
        ft[e] = y;
        if (r < 3) st[s].fluid_force[r] = y;
        else st[s].fluid_torque[r - 3] = y;
    }
    const int n_sh = min(cnt->n_shared, sh_mask + 1);
    uint32_t* C = reinterpret_cast<uint32_t*>(Ct);
    for (int64_t e = t0; e < n_sh; e += nt) {
        const int slot = sh_used[e];
        const int32_t c = sh_keys[slot];
        double* v = sh_vals + 5 * (int64_t)slot;
        if (c >= 0 && c < N) {
            Ct[c] = decode_claim(C[c]);
            As[c] = (float)fmin(v[0], 1.0);
            Ts[c] = (float)v[1];
            Fs[c] = (float)v[2];
            Fs[N + c] = (float)v[3];
            Fs[2 * N + c] = (float)v[4];
        }
        for (int r = 0; r < 5; ++r) v[r] = 0.0;
        sh_keys[slot] = -1;
    }
}

// n doubles (forces, solid states) and the counters into page-locked host memory, read after the stream is synchronised: one
// launch instead of two copies
__global__ void export_host_kernel(const double* __restrict__ src, int64_t n, const Counters* __restrict__ cnt,
                                   double* __restrict__ dst, Counters* __restrict__ h_cnt) {
    const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, nt = (int64_t)gridDim.x * blockDim.x;
    for (int64_t e = t0; e < n; e += nt) dst[e] = src[e];
    const uint32_t* a = reinterpret_cast<const uint32_t*>(cnt);
    uint32_t* b = reinterpret_cast<uint32_t*>(h_cnt);
    if (t0 < (int64_t)(sizeof(Counters) / 4)) b[t0] = a[t0];
}

__global__ void set_step_kernel(StepParams* p, StepParams v, EvolveCtrl* ctrl) {
    if (ctrl) *ctrl = EvolveCtrl{};
    *p = v;
}

// interact_host on page-locked host fields.  The host fields held the previous call's values; the cells this call or
// the previous one touched (the current and the previous lists) are the ones that changed.  mark_export_kernel sets
// their chunks of EXPORT_CHUNK consecutive cells in a bitmap (one bit per chunk); export_kernel then copies every
// marked chunk from the device fields to the host fields through the mapped host pointers, a warp per bitmap word so
// that each store instruction covers 32 consecutive cells of a host array, and clears the word.
constexpr int EXPORT_LG = 3;  // log2 of the cells per chunk
constexpr int EXPORT_CHUNK = 1 << EXPORT_LG;
int export_chunk_cells() { return EXPORT_CHUNK; }

__global__ void mark_export_kernel(const int32_t* __restrict__ in_cell, const int32_t* __restrict__ cut_cell,
                                   const int32_t* __restrict__ prev_in_cell, const int32_t* __restrict__ prev_cut_cell,
                                   const Counters* cnt, int64_t N, uint32_t* __restrict__ dirty) {
    const int64_t n0 = clamp_len(cnt->n_inside, cnt->list_cap), n1 = clamp_len(cnt->n_cut, cnt->list_cap);
    const int64_t n2 = clamp_len(cnt->prev_n_inside, cnt->list_cap), n3 = clamp_len(cnt->prev_n_cut, cnt->list_cap);
    const int64_t total = n0 + n1 + n2 + n3;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total; e += (int64_t)gridDim.x * blockDim.x) {
        int64_t c;
        if (e < n0) c = in_cell[e];
        else if (e < n0 + n1) c = cut_cell[e - n0];
        else if (e < n0 + n1 + n2) c = prev_in_cell[e - n0 - n1];
        else c = prev_cut_cell[e - n0 - n1 - n2];
        if (c < 0 || c >= N) continue;
        const uint32_t bit = 1u << ((c >> EXPORT_LG) & 31);
        uint32_t* word = dirty + (c >> (EXPORT_LG + 5));
        if (!(*word & bit)) atomicOr(word, bit);
    }
}

__global__ void export_kernel(Counters* cnt, int64_t N, uint32_t* __restrict__ dirty, const float* __restrict__ As,
                              const float* __restrict__ Fs, const float* __restrict__ Ts,
                              const int32_t* __restrict__ Ct, float* hAs, float* hFs, float* hTs, int32_t* hCt) {
    const int lane = threadIdx.x & 31;
    const int64_t words = (N + 32 * EXPORT_CHUNK - 1) >> (EXPORT_LG + 5);
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    int chunks = 0;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < words; w += nw) {
        const uint32_t word = dirty[w];
        if (!word) continue;
        chunks += __popc(word);
#pragma unroll
        for (int t = 0; t < EXPORT_CHUNK; ++t) {
            const int64_t c = (w << (EXPORT_LG + 5)) + 32 * t + lane;
            if (((word >> ((32 * t + lane) >> EXPORT_LG)) & 1u) && c < N) {
                hAs[c] = As[c]; hTs[c] = Ts[c]; hCt[c] = Ct[c];
                hFs[c] = Fs[c]; hFs[N + c] = Fs[N + c]; hFs[2 * N + c] = Fs[2 * N + c];
            }
        }
        __syncwarp();
        if (lane == 0) dirty[w] = 0u;
    }
    if (lane == 0 && chunks) atomicAdd(&cnt->n_export, chunks);
}

// ---- FP64 host fields in OpenFOAM's own layout (sdfibm_cuda_interact_host64) -------------------------------------
// U is a volVectorField (one x,y,z triple per cell), As / Ts / Ct volScalarFields and Fs a volVectorField, all FP64
// in page-locked host memory.  gather_u64_kernel reads U at the coupling cells only (24 contiguous bytes per cell)
// into the FP32 device plane layout the coupling kernel reads; export64_kernel writes the marked 8-cell chunks of
// the four result fields back in FP64.
__global__ void gather_u64_kernel(const int32_t* __restrict__ in_cell, const int32_t* __restrict__ cut_cell,
                                  const Counters* cnt, int64_t N, const double* __restrict__ hU,
                                  float* __restrict__ U) {
    const int64_t n0 = clamp_len(cnt->n_inside, cnt->list_cap), n1 = clamp_len(cnt->n_cut, cnt->list_cap);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n0 + n1; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = e < n0 ? in_cell[e] : cut_cell[e - n0];
        if (c < 0 || c >= N) continue;
        const double x = hU[3 * c], y = hU[3 * c + 1], z = hU[3 * c + 2];
        U[c] = (float)x;
        U[N + c] = (float)y;
        U[2 * N + c] = (float)z;
    }
}

// all chunks marked (the first call on a set of host fields writes every cell)
__global__ void mark_all_kernel(uint32_t* __restrict__ dirty, int64_t words) {
    for (int64_t w = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; w < words; w += (int64_t)gridDim.x * blockDim.x)
        dirty[w] = 0xffffffffu;
}

// A warp per bitmap word (256 cells, 32 chunks).  An FP64 chunk of a scalar field is 64 bytes and of Fs 192 bytes,
// whole host cache lines: the scalar fields go out one cell per lane, Fs as the interleaved x,y,z sequence of the
// word's cells, element e of it at lane e mod 32, so that every store instruction writes 256 contiguous bytes (a lane
// per cell and a store per component would leave each instruction a third of each line).  The device values of a
// group of stores are loaded before the first of them.
__global__ void __launch_bounds__(256, 3) export64_kernel(Counters* cnt, int64_t N, uint32_t* __restrict__ dirty,
                                                      const float* __restrict__ As, const float* __restrict__ Fs,
                                                      const float* __restrict__ Ts, const int32_t* __restrict__ Ct,
                                                      double* __restrict__ hAs, double* __restrict__ hFs,
                                                      double* __restrict__ hTs, double* __restrict__ hCt) {
    const int lane = threadIdx.x & 31;
    const int64_t words = (N + 32 * EXPORT_CHUNK - 1) >> (EXPORT_LG + 5);
    const int64_t nw = (int64_t)gridDim.x * (blockDim.x >> 5);
    int chunks = 0;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < words; w += nw) {
        const uint32_t word = dirty[w];
        if (!word) continue;
        chunks += __popc(word);
        const int64_t base = w << (EXPORT_LG + 5);
        {
            float a[EXPORT_CHUNK], t[EXPORT_CHUNK];
            int32_t k[EXPORT_CHUNK];
            bool on[EXPORT_CHUNK];
#pragma unroll
            for (int q = 0; q < EXPORT_CHUNK; ++q) {
                const int64_t c = base + 32 * q + lane;
                on[q] = ((word >> ((32 * q + lane) >> EXPORT_LG)) & 1u) && c < N;
                a[q] = on[q] ? As[c] : 0.f;
                t[q] = on[q] ? Ts[c] : 0.f;
                k[q] = on[q] ? Ct[c] : 0;
            }
#pragma unroll
            for (int q = 0; q < EXPORT_CHUNK; ++q) {
                const int64_t c = base + 32 * q + lane;
                if (on[q]) {
                    hAs[c] = (double)a[q];
                    hTs[c] = (double)t[q];
                    hCt[c] = (double)k[q];
                }
            }
        }
        // Fs: 3 x 256 elements, 24 stores per lane in three groups of eight
#pragma unroll 1
        for (int g = 0; g < 3; ++g) {
            float v[8];
            bool on[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int e = 32 * (8 * g + q) + lane;      // element of the word's interleaved sequence
                const int cl = (int)((unsigned)e / 3u), comp = e - 3 * cl;
                const int64_t c = base + cl;
                on[q] = ((word >> (cl >> EXPORT_LG)) & 1u) && c < N;
                v[q] = on[q] ? Fs[comp * N + c] : 0.f;
            }
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (on[q]) hFs[3 * base + 32 * (8 * g + q) + lane] = (double)v[q];
        }
        __syncwarp();
        if (lane == 0) dirty[w] = 0u;
    }
    if (lane == 0 && chunks) atomicAdd(&cnt->n_export, chunks);
}

// whole-field conversions of the FP64 path for host memory the GPU cannot address (staged through device copies)
__global__ void u64_to_planes_kernel(const double* __restrict__ U64, int64_t N, float* __restrict__ U) {
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < N; c += (int64_t)gridDim.x * blockDim.x) {
        U[c] = (float)U64[3 * c];
        U[N + c] = (float)U64[3 * c + 1];
        U[2 * N + c] = (float)U64[3 * c + 2];
    }
}
__global__ void fields_to_f64_kernel(int64_t N, const float* __restrict__ As, const float* __restrict__ Fs,
                                     const float* __restrict__ Ts, const int32_t* __restrict__ Ct,
                                     double* __restrict__ out) {
    // out: As[N], Fs[N][3], Ts[N], Ct[N]
    for (int64_t c = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; c < N; c += (int64_t)gridDim.x * blockDim.x) {
        out[c] = (double)As[c];
        out[N + 3 * c] = (double)Fs[c];
        out[N + 3 * c + 1] = (double)Fs[N + c];
        out[N + 3 * c + 2] = (double)Fs[2 * N + c];
        out[4 * N + c] = (double)Ts[c];
        out[5 * N + c] = (double)Ct[c];
    }
}

// SolidCloud::fixInternal over the ALL_INSIDE list: U = rigid velocity of the solid that owns the cell.  Bound by the FP64 pipe:
// 12 operations a cell (30 with the centres and the roundings computed on it).
// 36 -> 18 us in the same steps, 21 -> 10 for the circles (GB300).
__global__ void fix_internal_kernel(MeshK m, const double* __restrict__ centres, const sdfibm_solid_state* __restrict__ st,
                                    const int32_t* __restrict__ in_cell, const int32_t* __restrict__ in_solid,
                                    const int32_t* __restrict__ Ct, float* __restrict__ U, const Counters* cnt) {
    const int n_in = clamp_len(cnt->n_inside, cnt->list_cap);
    const int64_t N = m.ncells;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n_in; e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t c = in_cell[e];
        const int32_t s = in_solid[e] & LIST_SOLID_MASK;
        if (c < 0 || c >= N) continue;
        if (Ct[c] != s + 4) continue;
        int i, j, k;
        cell_ijk(m, c, i, j, k);
        const sdfibm_solid_state& x = st[s];
        const double dx = centres[i] - x.pos[0], dy = centres[m.nx + j] - x.pos[1], dz = centres[m.nx + m.ny + k] - x.pos[2];
        const double ox = x.omega[0], oy = x.omega[1], oz = x.omega[2];
        U[c] = narrow(__fma_rn(oy, dz, __fma_rn(-oz, dy, x.vel[0])));
        U[N + c] = narrow(__fma_rn(oz, dx, __fma_rn(-ox, dz, x.vel[1])));
        U[2 * N + c] = narrow(__fma_rn(ox, dy, __fma_rn(-oy, dx, x.vel[2])));
    }
}

}  // namespace sdfibm_dev
