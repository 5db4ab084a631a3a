// Enumeration and cut-cell solid fraction: one pass over (solid, cell-tile) work items, then per-cell kernels.
//
// Each persistent CTA pulls tiles from an atomic counter.  For a tile it
//   1. skips tiles whose box cannot meet the solid's bounding sphere (prism: bounding disc) and zero-fills them;
//   2. evaluates the inside test once per tile vertex (FP32 with a rigorous error bound, FP64 re-check inside the
//      band -- identical answers to the reference's FP64 Solid::phi01) and writes one class byte per cell
//      (CellEnumerator::_next, src/cellenumerator.cpp:6-34): 0 no inside vertex, 1 all inside, 2 centre inside,
//      3 centre outside;
//   3. lists every cut candidate (class 2/3) for the fraction kernels:
//      REF-GEO   as (solid, fraction index), with the signed distances of its 8 vertices in FP64 numerators (sdf_mixed) for
//                all shapes but 3-D spheres, ellipsoids and boxes; refgeo_cells_kernel computes those (two-float, sdf_ff_at)
//                and runs GeometricTools::calcCellVolume (src/geometrictools.cpp:13-116) in FP32 in cell-local
//                coordinates (vertices on {0,1}^3, every term a product of non-negative factors), a thread per cell;
//      SUBSAMPLE as (solid, fraction index); subsample_cells_kernel counts the n^3 (2-D: n^2) midpoint lattice of
//                each listed cell, a lane per cell (a warp for few cells), with the same exact inside test as the vertices
//                (run counting along lattice columns for the convex shapes), undecided points rechecked in FP64 by
//                recheck_kernel;
//      LEARNED   as (solid, fraction index); learned_stencil_kernel (stencil.cu) computes the network's inputs and
//                band, the cells outside the band go to subsample_cells_kernel.
// The allocation-free entry point wants the classes only.  Candidates that the flood fill later leaves out simply have their
// alpha ignored.
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"
#include "mlp.cuh"

namespace sdfibm_dev {


// ---- REF-GEO geometry in cell-local FP32 coordinates -------------------------------------------------------------------
// Vertex slots: 0:(i,j,k) 1:(i+1,j,k) 2:(i,j+1,k) 3:(i+1,j+1,k) 4..7 the same at k+1 (ascending point label); the face
// vertex orders are the ones the mesh stores (owner's hex-model face for internal faces, the cell's own for boundary
// faces), which fix the apex of each face.
struct FaceSlots {
    int8_t v[9][4];
};
constexpr FaceSlots FACE_SLOTS = {{
    {1, 3, 7, 5},  // x-max, owner order (internal +x face and x-max boundary face)
    {2, 6, 7, 3},  // y-max
    {4, 5, 7, 6},  // z-max
    {0, 4, 6, 2},  // x-min boundary face
    {0, 1, 5, 4},  // y-min boundary face
    {0, 2, 3, 1},  // z-min boundary face
    {0, 2, 6, 4},  // -x internal face (owner is the lower neighbour)
    {0, 4, 5, 1},  // -y internal face
    {0, 1, 3, 2},  // -z internal face
}};
__constant__ FaceSlots c_face_slots = FACE_SLOTS;  // for runtime indices

__device__ inline float lfrac32(float pa, float pb) {
    if (pa > 0.f && pb > 0.f) return 0.f;
    if (pa <= 0.f && pb <= 0.f) return 1.f;
    if (pa > 0.f) return -pb / (pa - pb);
    return -pa / (pb - pa);
}

// A point of the unit cell carried as, per axis, its coordinate v and 1 - v, both computed without cancellation:
// the apex of calcApex lies on the segment between two vertices of {0,1}^3, so each coordinate is 0, 1, t or 1 - t
// with t = |phiA| / (SMALL + |phiA| + |phiB|) and 1 - t = (SMALL + |phiB|) / (same), and every later use (pyramid
// heights, the in-face cross product) only needs the distance of the apex to a face plane 0 or 1 along one axis.
struct ApexPair {
    float v[3], w[3];
    __device__ float dist(int axis, int plane) const { return plane ? w[axis] : v[axis]; }
};

// GeometricTools::calcApex: first vertex A, first later vertex B of opposite (or zero) sign
__device__ inline ApexPair apex_pair(const float* ph, const int8_t* idx, int n) {
    const int A = idx[0];
    const float phiA = ph[A];
    int B = A;
    float phiB = 0.f;
    for (int i = 1; i < n; ++i) {
        B = idx[i];
        phiB = ph[B];
        // the sign of the reference's FP64 product phiA*phiB, without FP32 underflow of tiny values
        if (phiA == 0.f || phiB == 0.f || ((phiA > 0.f) != (phiB > 0.f))) break;
    }
    const float den = (float)SMALL_D + fabsf(phiA) + fabsf(phiB);
    const float t = fabsf(phiA) / den, u = ((float)SMALL_D + fabsf(phiB)) / den;
    ApexPair p;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const int ca = (A >> a) & 1, cb = (B >> a) & 1;
        if (ca == cb) { p.v[a] = (float)ca; p.w[a] = (float)(1 - ca); }
        else if (ca) { p.v[a] = u; p.w[a] = t; }   // 1 - t(1 - 0)
        else { p.v[a] = t; p.w[a] = u; }           // 0 - t(0 - 1)
    }
    return p;
}

// GeometricTools::calcFaceAreaFraction in units of the face area; `axis` is the face normal.  Each edge O->A runs
// along one in-face axis e; |(A-O) x (apex-O)| is then the apex's distance from O along the other in-face axis.
__device__ inline float face_fraction32(const float* ph, const int8_t* f, int axis) {
    int sign_sum = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) sign_sum += (ph[f[i]] > 0.f) ? 1 : -1;
    if (sign_sum == 4) return 0.f;
    if (sign_sum == -4) return 1.f;
    const ApexPair ap = apex_pair(ph, f, 4);
    float area = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int o = f[e], a = f[(e + 1) & 3];
        const int diff = o ^ a;                       // one bit: the edge axis
        const int eax = diff == 1 ? 0 : (diff == 2 ? 1 : 2);
        const int oax = 3 - axis - eax;               // the other in-face axis
        const float c = ap.dist(oax, (o >> oax) & 1);
        area += 0.5f * c * lfrac32(ph[o], ph[a]);
    }
    return area;
}

// GeometricTools::calcCellVolume / V.  apz/apz1: local z of the 2-D apex plane and 1 minus it
// (geometrictools.cpp:57-58), unused in 3-D.
static __device__ __noinline__ float refgeo32(const MeshK& m, const float* ph, int64_t i, int64_t j, int64_t k, float apz, float apz1) {
    const int8_t order[8] = {0, 1, 2, 3, 4, 5, 6, 7};
    ApexPair ap = apex_pair(ph, order, 8);
    if (m.twod) { ap.v[2] = apz; ap.w[2] = apz1; }
    float vol = 0.f;
    auto acc = [&](int slot, int axis, int plane) {
        const float eps = face_fraction32(ph, c_face_slots.v[slot], axis);
        vol += (1.0f / 3.0f) * eps * ap.dist(axis, plane);
    };
    // mesh.cells()[c] order: owned internal (+x,+y,+z), boundary faces by patch, then -z,-y,-x
    if (i + 1 < m.nx) acc(0, 0, 1);
    if (j + 1 < m.ny) acc(1, 1, 1);
    if (k + 1 < m.nz) acc(2, 2, 1);
    if (i == 0) acc(3, 0, 0);
    if (i == m.nx - 1) acc(0, 0, 1);
    if (j == 0) acc(4, 1, 0);
    if (j == m.ny - 1) acc(1, 1, 1);
    if (k == 0) acc(5, 2, 0);
    if (k == m.nz - 1) acc(2, 2, 1);
    if (k > 0) acc(8, 2, 0);
    if (j > 0) acc(7, 1, 0);
    if (i > 0) acc(6, 0, 0);
    return vol;
}

// The same for a cell whose faces are known (inside the mesh in x and y, and in z too unless the mesh has one layer): operation
// for operation what refgeo32 does, with every vertex, edge and face at a compile-time place.  refgeo32 keeps its cells' arrays
// in local memory, as its faces pick from them, and divides twice for every edge.
__device__ __forceinline__ constexpr int face_vertex(int slot, int q) { return FACE_SLOTS.v[slot][q]; }
__device__ __forceinline__ constexpr int edge_axis(int o, int a) { return (o ^ a) == 1 ? 0 : ((o ^ a) == 2 ? 1 : 2); }
// edge from the lower vertex v along an axis: 4 * axis + the other two bits of v
__device__ __forceinline__ constexpr int edge_slot(int o, int a) {
    const int v = o & a, x = edge_axis(o, a);
    return 4 * x + (x == 0 ? v >> 1 : (x == 1 ? (v & 1) | ((v >> 1) & 2) : v & 3));
}
__device__ __forceinline__ bool apex_stop(float phiA, float phiB) {
    return phiA == 0.f || phiB == 0.f || ((phiA > 0.f) != (phiB > 0.f));
}
template <int SLOT, int AXIS>
__device__ __forceinline__ float face_fraction_at(const float (&ph)[8], const float (&ef)[12]) {
    constexpr int f0 = face_vertex(SLOT, 0), f1 = face_vertex(SLOT, 1), f2 = face_vertex(SLOT, 2), f3 = face_vertex(SLOT, 3);
    const int npos = (ph[f0] > 0.f) + (ph[f1] > 0.f) + (ph[f2] > 0.f) + (ph[f3] > 0.f);
    const float phiA = ph[f0];
    const bool s1 = apex_stop(phiA, ph[f1]), s2 = apex_stop(phiA, ph[f2]);
    const float phiB = s1 ? ph[f1] : (s2 ? ph[f2] : ph[f3]);
    const float den = (float)SMALL_D + fabsf(phiA) + fabsf(phiB);
    const float t = fabsf(phiA) / den, u = ((float)SMALL_D + fabsf(phiB)) / den;
    // the segment A..B runs along the axis of the edge f0 f1 unless B = f3, and along that of f0 f3 unless B = f1
    constexpr int e1 = edge_axis(f0, f1), e3 = edge_axis(f0, f3);
    const bool along1 = s1 || s2, along3 = !s1;
    float v[3], w[3];
    constexpr int c1 = (f0 >> e1) & 1, c3 = (f0 >> e3) & 1;
    v[e1] = along1 ? (c1 ? u : t) : (float)c1;
    w[e1] = along1 ? (c1 ? t : u) : (float)(1 - c1);
    v[e3] = along3 ? (c3 ? u : t) : (float)c3;
    w[e3] = along3 ? (c3 ? t : u) : (float)(1 - c3);
    constexpr int f[4] = {f0, f1, f2, f3};
    float area = 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const int o = f[e], a = f[(e + 1) & 3], oax = 3 - AXIS - edge_axis(o, a);
        area += 0.5f * (((o >> oax) & 1) ? w[oax] : v[oax]) * ef[edge_slot(o, a)];
    }
    return npos == 4 ? 0.f : (npos == 0 ? 1.f : area);
}
template <bool LAYER>
static __device__ __forceinline__ float refgeo_inner(const MeshK& m, const float (&ph)[8], float apz, float apz1) {
    float ef[12];
#pragma unroll
    for (int x = 0; x < 3; ++x)
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int o = x == 0 ? r << 1 : (x == 1 ? (r & 1) | ((r & 2) << 1) : r);
            ef[4 * x + r] = lfrac32(ph[o], ph[o | (1 << x)]);
        }
    int B = 7;
    float phiB = ph[7];
#pragma unroll
    for (int i = 6; i >= 1; --i) {
        const bool s = apex_stop(ph[0], ph[i]);
        B = s ? i : B;
        phiB = s ? ph[i] : phiB;
    }
    const float den = (float)SMALL_D + fabsf(ph[0]) + fabsf(phiB);
    const float t = fabsf(ph[0]) / den, u = ((float)SMALL_D + fabsf(phiB)) / den;
    float v[3], w[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        v[a] = (B >> a) & 1 ? t : 0.f;
        w[a] = (B >> a) & 1 ? u : 1.f;
    }
    if (m.twod) { v[2] = apz; w[2] = apz1; }
    float vol = 0.f;
    vol += (1.0f / 3.0f) * face_fraction_at<0, 0>(ph, ef) * w[0];
    vol += (1.0f / 3.0f) * face_fraction_at<1, 1>(ph, ef) * w[1];
    if (LAYER) {  // both z faces are boundary faces
        vol += (1.0f / 3.0f) * face_fraction_at<5, 2>(ph, ef) * v[2];
        vol += (1.0f / 3.0f) * face_fraction_at<2, 2>(ph, ef) * w[2];
    } else {
        vol += (1.0f / 3.0f) * face_fraction_at<2, 2>(ph, ef) * w[2];
        vol += (1.0f / 3.0f) * face_fraction_at<8, 2>(ph, ef) * v[2];
    }
    vol += (1.0f / 3.0f) * face_fraction_at<7, 1>(ph, ef) * v[1];
    vol += (1.0f / 3.0f) * face_fraction_at<6, 0>(ph, ef) * v[0];
    return vol;
}

// the oracle's FP64 sample point (i + (2a+1)/(2n), ...) and the reference's inside test, out of line (see
// exact_inside_point)
static __device__ __noinline__ int exact_inside_sample(const ShapeK& sh, const MeshK& m, int64_t i, int64_t j, int64_t k,
                                                int a, int b, int c3, int n, const D3& x, const Q4& q) {
    const double ta64 = (double)(2 * a + 1) / (double)(2 * n), tb64 = (double)(2 * b + 1) / (double)(2 * n);
    const double tc64 = m.twod ? 0.5 : (double)(2 * c3 + 1) / (double)(2 * n);
    const D3 p{m.o[0] + ((double)i + ta64) * m.h[0], m.o[1] + ((double)j + tb64) * m.h[1],
               m.o[2] + ((double)k + tc64) * m.h[2]};
    return inside64(sh, world2local(p, x, q)) ? 1 : 0;
}

// Where an undecided SUBSAMPLE point goes: appended to the recheck list (counted later by recheck_kernel) when there
// is room, else re-evaluated here.  DEFER_ONLY kernels carry no FP64 path: a point the full list cannot take sets the
// warp's overflow flag instead, and the cell is recounted by recount_kernel.
struct Defer {
    Recheck* rq;
    int64_t cap;
    int32_t* count;
    int64_t idx;
    int32_t solid;
    int32_t* overflow;  // DEFER_ONLY: the warp's flag in shared memory
};
template <bool DEFER_ONLY>
static __device__ __forceinline__ int undecided_sample(const Defer* df, const ShapeK& sh, const MeshK& m, int64_t i,
                                                       int64_t j, int64_t k, int a, int b, int c3, int n, const D3& x,
                                                       const Q4& q) {
    if (df) {
        const int slot = atomicAdd(df->count, 1);
        if (slot < df->cap) {
            df->rq[slot] = Recheck{df->idx, df->solid,
                                   (uint32_t)a | ((uint32_t)b << 8) | ((uint32_t)c3 << 16) | ((uint32_t)n << 24)};
            return 0;
        }
        if (DEFER_ONLY) {
            *(volatile int32_t*)df->overflow = 1;
            return 0;
        }
    }
    if (DEFER_ONLY) return 0;  // DEFER_ONLY callers always pass a Defer
    return exact_inside_sample(sh, m, i, j, k, a, b, c3, n, x, q);
}

// the reference's FP64 Solid::phi of mesh point (I,J,K), out of line
static __device__ __noinline__ float exact_phi_point(const ShapeK& sh, const MeshK& m, int64_t I, int64_t J, int64_t K,
                                              const D3& x, const Q4& q) {
    const D3 p{m.o[0] + (double)I * m.h[0], m.o[1] + (double)J * m.h[1], m.o[2] + (double)K * m.h[2]};
    return (float)sdf64(sh, world2local(p, x, q));
}

// ---- SUBSAMPLE: a warp per cut cell -----------------------------------------------------------------------------------
// Each lane owns (a,b) columns of the n x n x n midpoint lattice and walks its column in z.  Local coordinates step by
// three precomputed vectors (the columns of the world->local map times h).  One error bound E covers every sample
// coordinate of the cell; for the convex shapes the bound of the inside function is also taken once per cell, from
// the largest coordinate any sample can have, so a sample costs a few FMAs and two compares.  Undecided samples are
// re-evaluated with the oracle's FP64 point formula.

// sample frame of one cell: corner point p (shape centre offset folded in for the convex shapes), steps s*, bounds
struct SampleFrame {
    float px, py, pz;
    float sxx, sxy, sxz, syx, syy, syz, szx, szy, szz;
    float E;   // bound of |computed - exact| of every sample coordinate (without the folded offset)
    float Eg;  // bound of |computed - exact| of the inside function (convex shapes, offset folded)
    float k0, k1, k2, k3;  // quadric X^2 k0 + Y^2 k1 + Z^2 k2 - k3, or box half extents k0..k2
};

__device__ __forceinline__ int band(float g, float Eg) { return g < -Eg ? 1 : (g > Eg ? 0 : 2); }

constexpr int SS_QUADRIC = 0, SS_BOX = 1, SS_GENERIC = 2;

// inside function of the convex shapes at a local point (negative inside), within f.Eg of its exact value
template <int T>
__device__ __forceinline__ float sample_g(const SampleFrame& f, float X, float Y, float Z) {
    if (T == SS_QUADRIC) return __fmaf_rn(X * X, f.k0, __fmaf_rn(Y * Y, f.k1, (Z * Z) * f.k2)) - f.k3;
    return fmaxf(fmaxf(fabsf(X) - f.k0, fabsf(Y) - f.k1), fabsf(Z) - f.k2);
}

template <int T>
__device__ __forceinline__ int sample_inside(const ShapeK& sh, const SampleFrame& f, float X, float Y, float Z) {
    if (T == SS_QUADRIC || T == SS_BOX) return band(sample_g<T>(f, X, Y, Z), f.Eg);
    return inside32(sh, X, Y, Z, f.E);  // tails and planes: the general test with its per-sample bound
}

template <int T, bool DEFER_ONLY>
__device__ __forceinline__ int subsample_count(const MeshK& m, const ShapeK& sh, const SampleFrame& f, int64_t i,
                                               int64_t j, int64_t k, int n, const D3& x, const Q4& q,
                                               unsigned long long* rechecks, const Defer* df) {
    const int lane = threadIdx.x & 31;
    const int nzs = m.twod ? 1 : n;
    const float inv2n = 1.0f / (float)(2 * n);
    int cnt = 0;
#pragma unroll 1
    for (int col = lane; col < n * n; col += 32) {
        const int ia = col % n, ib = col / n;
        const float ta = (float)(2 * ia + 1) * inv2n, tb = (float)(2 * ib + 1) * inv2n;
        const float bx = __fmaf_rn(tb, f.syx, __fmaf_rn(ta, f.sxx, f.px));
        const float by = __fmaf_rn(tb, f.syy, __fmaf_rn(ta, f.sxy, f.py));
        const float bz = __fmaf_rn(tb, f.syz, __fmaf_rn(ta, f.sxz, f.pz));
        float odd = 1.f;  // 2*c3 + 1, exact
#pragma unroll 2
        for (int c3 = 0; c3 < nzs; ++c3) {
            const float tc = m.twod ? 0.5f : odd * inv2n;
            odd += 2.f;
            int r = sample_inside<T>(sh, f, __fmaf_rn(tc, f.szx, bx), __fmaf_rn(tc, f.szy, by),
                                     __fmaf_rn(tc, f.szz, bz));
            if (r == 2) {
                ++*rechecks;
                r = undecided_sample<DEFER_ONLY>(df, sh, m, i, j, k, ia, ib, c3, n, x, q);
            }
            cnt += r;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    return cnt;
}

// Block-skipping count for the quadrics and boxes: the lattice is split into B x B x B blocks (B x B x 1 on one-layer
// meshes).  For each block the inside function is bounded over the box of local coordinates that holds the block's
// samples (centre +- half the block's span along the three step vectors, widened by the coordinate error bound Ep);
// a block whose upper bound is below -Eg has every sample inside in the reference's FP64 evaluation, one whose
// lower bound is above Eg has none, and only the remaining blocks are sampled, with the same coordinate sequence
// and per-sample bound as subsample_count.  The count is therefore the exhaustive lattice count.
template <int T>
__device__ __forceinline__ void block_bounds(const SampleFrame& f, float X, float Y, float Z, float hx, float hy,
                                             float hz, float& gmin, float& gmax) {
    const float xl = X - hx, xh = X + hx, yl = Y - hy, yh = Y + hy, zl = Z - hz, zh = Z + hz;
    const float ax = fmaxf(fabsf(xl), fabsf(xh)), ay = fmaxf(fabsf(yl), fabsf(yh)), az = fmaxf(fabsf(zl), fabsf(zh));
    const float bx = (xl <= 0.f && xh >= 0.f) ? 0.f : fminf(fabsf(xl), fabsf(xh));
    const float by = (yl <= 0.f && yh >= 0.f) ? 0.f : fminf(fabsf(yl), fabsf(yh));
    const float bz = (zl <= 0.f && zh >= 0.f) ? 0.f : fminf(fabsf(zl), fabsf(zh));
    if (T == SS_QUADRIC) {
        gmax = __fmaf_rn(ax * ax, f.k0, __fmaf_rn(ay * ay, f.k1, (az * az) * f.k2)) - f.k3;
        gmin = __fmaf_rn(bx * bx, f.k0, __fmaf_rn(by * by, f.k1, (bz * bz) * f.k2)) - f.k3;
    } else {
        gmax = fmaxf(fmaxf(ax - f.k0, ay - f.k1), az - f.k2);
        gmin = fmaxf(fmaxf(bx - f.k0, by - f.k1), bz - f.k2);
    }
}

template <int T, bool DEFER_ONLY>
__device__ __noinline__ int subsample_blocks(const MeshK& m, const ShapeK& sh, const SampleFrame& f, int64_t i,
                                             int64_t j, int64_t k, int n, int lb, float Ep, const D3& x, const Q4& q,
                                             unsigned long long* rechecks, const Defer* df) {
    __shared__ uint16_t s_und[8][128];  // undecided blocks of each warp, (ba, bb, bc) packed 5 bits each
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    uint16_t* list = s_und[(threadIdx.x >> 5) & 7];
    const bool flat = m.twod != 0;
    const int B = 1 << lb, nb = n >> lb, nbz = flat ? 1 : nb;
    const int lsz = flat ? 2 * lb : 3 * lb;  // log2 of the samples per block
    const int nblocks = nb * nb * nbz;
    const float inv2n = 1.0f / (float)(2 * n);
    // half span of a block along each step vector (t from its first to its last sample), widened by a relative 1e-6
    const float half = 0.5f * (float)(2 * (B - 1)) * inv2n * 1.000001f;
    const float halfz = flat ? 0.f : half;
    const float hx = half * (fabsf(f.sxx) + fabsf(f.syx)) + halfz * fabsf(f.szx) + Ep;
    const float hy = half * (fabsf(f.sxy) + fabsf(f.syy)) + halfz * fabsf(f.szy) + Ep;
    const float hz = half * (fabsf(f.sxz) + fabsf(f.syz)) + halfz * fabsf(f.szz) + Ep + U32 * fabsf(f.pz);
    int cnt = 0, nund = 0;
    for (int base = 0; base < nblocks; base += 32) {
        const int blk = base + lane;
        bool undecided = false;
        int packed = 0;
        if (blk < nblocks) {
            const int ba = blk % nb, bb = (blk / nb) % nb, bc = blk / (nb * nb);
            packed = ba | (bb << 5) | (bc << 10);
            const float ta = (float)(2 * ba * B + B) * inv2n, tb = (float)(2 * bb * B + B) * inv2n;
            const float tc = flat ? 0.5f : (float)(2 * bc * B + B) * inv2n;
            const float X = __fmaf_rn(tc, f.szx, __fmaf_rn(tb, f.syx, __fmaf_rn(ta, f.sxx, f.px)));
            const float Y = __fmaf_rn(tc, f.szy, __fmaf_rn(tb, f.syy, __fmaf_rn(ta, f.sxy, f.py)));
            const float Z = __fmaf_rn(tc, f.szz, __fmaf_rn(tb, f.syz, __fmaf_rn(ta, f.sxz, f.pz)));
            float gmin, gmax;
            block_bounds<T>(f, X, Y, Z, hx, hy, hz, gmin, gmax);
            if (gmax < -f.Eg) cnt += 1 << lsz;
            else if (!(gmin > f.Eg)) undecided = true;
        }
        const unsigned mask = __ballot_sync(FULL, undecided);
        if (undecided) list[nund + __popc(mask & ((1u << lane) - 1u))] = (uint16_t)packed;
        nund += __popc(mask);
    }
    __syncwarp();
    // the undecided blocks' columns: one (block, a, b) column per slot, walked along c as subsample_count does
    const int lcol = 2 * lb;  // log2 of the columns per block
    const int slots = nund << lcol;
    const int Bz = flat ? 1 : B;
    for (int e = lane; e < slots; e += 32) {
        const int pk = list[e >> lcol], col = e & ((1 << lcol) - 1);
        const int ia = ((pk & 31) << lb) + (col & (B - 1)), ib = (((pk >> 5) & 31) << lb) + (col >> lb);
        const int ic0 = ((pk >> 10) & 31) << lb;
        const float ta = (float)(2 * ia + 1) * inv2n, tb = (float)(2 * ib + 1) * inv2n;
        const float bx = __fmaf_rn(tb, f.syx, __fmaf_rn(ta, f.sxx, f.px));
        const float by = __fmaf_rn(tb, f.syy, __fmaf_rn(ta, f.sxy, f.py));
        const float bz = __fmaf_rn(tb, f.syz, __fmaf_rn(ta, f.sxz, f.pz));
        float odd = (float)(2 * ic0 + 1);  // 2*ic + 1, exact
        for (int dc = 0; dc < Bz; ++dc, odd += 2.f) {
            const float tc = flat ? 0.5f : odd * inv2n;
            int res = sample_inside<T>(sh, f, __fmaf_rn(tc, f.szx, bx), __fmaf_rn(tc, f.szy, by),
                                       __fmaf_rn(tc, f.szz, bz));
            if (res == 2) {
                ++*rechecks;
                res = undecided_sample<DEFER_ONLY>(df, sh, m, i, j, k, ia, ib, flat ? 0 : ic0 + dc, n, x, q);
            }
            cnt += res;
        }
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(FULL, cnt, o);
    return cnt;
}

// log2 of the block edge for block skipping (power of two of at least 4 dividing n, at most 128 blocks), 0: sample
// every point (blocks of 2 samples per axis cost more to test than they save)
__device__ inline int block_log2(int n, bool flat) {
    for (int lb = 2; lb <= 3; ++lb) {
        const int B = 1 << lb;
        if (n % B) continue;
        const int nb = n / B;
        if ((flat ? nb * nb : nb * nb * nb) <= 128) return lb;
    }
    return 0;
}

// Run counting for the convex shapes (3-D): the inside samples of a lattice column (a, b) are one run.  Along the column the
// local coordinates are w + c d (c the sample index), so the inside function q is the quadric polynomial A c^2 + 2 B c + C or
// the box maximum of three |w + c d| - k.  Two intervals of c decide the column: I, where q <= -E, holds certain samples only,
// and P, where q <= E, all possible ones (E >= every rounding between the real q of the reference's sample and the interval's
// ends).  If both hold the same samples, that is the column's count, and it is 0 if P holds none; else the column is walked
// sample by sample with the coordinates, bound and deferral of subsample_count.  The count is therefore the exhaustive
// lattice count.
//
// E.  Quadric, M = sum k X^2 + k3 over the cell: w, d and the coefficients give the polynomial's value to a few units of
// roundoff u of M.  An end is (-B -+ s) / A with s = sqrt(B^2 - A (C -+ E)); B^2 <= A M and s^2 <= A M, so B^2 - A C is
// good to 3 u A M and the ends to an error that changes q by at most 16 u M (2^-22 for the approximate root included);
// sample_frame adds 128 u M to Eg.  Box, m = max |X| + max k: the ends err by a few u m; sample_frame adds 64 u m, and a slab
// the column hardly moves against (|d| < E / 4 n) takes that d with its own sign (slab_step), which shifts a coordinate by E / 4
// at most: 1.3 E in all.
struct RunFrame {
    float kdx, kdy, kdz, A, minvA, AE;               // quadric (minvA: -1 / A)
    float ix, iy, iz, px, py, pz, cx, cy, cz;        // box: -1 / d, half widths of P and of I
    float last;                                      // n - 1
};
template <int T>
__device__ __forceinline__ RunFrame run_frame(const SampleFrame& f, float Egh, int n, float invn) {
    RunFrame r;
    r.last = (float)(n - 1);
    const float dx = f.szx * invn, dy = f.szy * invn, dz = f.szz * invn;
    if (T == SS_QUADRIC) {
        r.kdx = f.k0 * dx; r.kdy = f.k1 * dy; r.kdz = f.k2 * dz;
        r.A = __fmaf_rn(dx, r.kdx, __fmaf_rn(dy, r.kdy, dz * r.kdz));
        r.minvA = -__frcp_rn(r.A);
        // a leading coefficient that is no normal number: no column is decided (E = NaN)
        r.AE = r.A > 1e-36f ? r.A * Egh : NAN;
    } else {
        const float least = 0.25f * Egh * invn, E = 1.3f * Egh;
        const float ix = __frcp_rn(slab_step(dx, least)), iy = __frcp_rn(slab_step(dy, least)), iz = __frcp_rn(slab_step(dz, least));
        r.ix = -ix; r.iy = -iy; r.iz = -iz;
        r.px = (f.k0 + E) * fabsf(ix); r.py = (f.k1 + E) * fabsf(iy); r.pz = (f.k2 + E) * fabsf(iz);
        r.cx = (f.k0 - E) * fabsf(ix); r.cy = (f.k1 - E) * fabsf(iy); r.cz = (f.k2 - E) * fabsf(iz);
    }
    return r;
}
__device__ __forceinline__ float sqrt_fast(float x) {
    float y;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
// inside samples of the column whose sample c has the local coordinates w + c d, or -1: to be walked (as is whatever is not a
// number here)
template <int T>
__device__ __forceinline__ float run_column(const SampleFrame& f, const RunFrame& r, float wx, float wy, float wz) {
    float p1, p2, c1, c2;  // P and I
    bool none, some = true;  // P is empty, I is not
    if (T == SS_QUADRIC) {
        const float B = __fmaf_rn(wx, r.kdx, __fmaf_rn(wy, r.kdy, wz * r.kdz));
        const float C = __fmaf_rn(wx * wx, f.k0, __fmaf_rn(wy * wy, f.k1, __fmaf_rn(wz * wz, f.k2, -f.k3)));
        const float disc = __fmaf_rn(B, B, r.A * -C), dp = disc + r.AE, dc = disc - r.AE;
        const float mid = B * r.minvA, sp = sqrt_fast(dp), sc = sqrt_fast(dc);  // NaN below zero
        p1 = __fmaf_rn(sp, r.minvA, mid); p2 = __fmaf_rn(-sp, r.minvA, mid);
        c1 = __fmaf_rn(sc, r.minvA, mid); c2 = __fmaf_rn(-sc, r.minvA, mid);
        none = dp <= 0.f;
    } else {
        const float mx = wx * r.ix, my = wy * r.iy, mz = wz * r.iz;
        p1 = fmaxf(fmaxf(mx - r.px, my - r.py), mz - r.pz); p2 = fminf(fminf(mx + r.px, my + r.py), mz + r.pz);
        c1 = fmaxf(fmaxf(mx - r.cx, my - r.cy), mz - r.cz); c2 = fminf(fminf(mx + r.cx, my + r.cy), mz + r.cz);
        none = p1 > p2;
        some = mx + my + mz == mx + my + mz;
    }
    some = some && c1 <= c2;
    // the first and the last sample of each in the column, plus 3 2^22 (the sum's last place is 1: its directed rounding is
    // the ceiling or the floor); an end beyond the column's is the column's, however uncertain it is
    const float R = 12582912.f;
    const float pa = __fadd_ru(fmaxf(p1, 0.f), R), pb = __fadd_rd(fminf(p2, r.last), R), cnt = pb - pa + 1.f;
    const bool same = pa == __fadd_ru(fmaxf(c1, 0.f), R) && pb == __fadd_rd(fminf(c2, r.last), R);
    return none || cnt <= 0.f ? 0.f : (same && some ? cnt : -1.f);
}
template <int T, bool DEFER_ONLY>
__device__ __forceinline__ int subsample_runs_body(const MeshK& m, const ShapeK& sh, const SampleFrame& f, float Egh,
                                                   int64_t i, int64_t j, int64_t k, int n, const D3& x, const Q4& q,
                                                   unsigned long long* rechecks, const Defer* df) {
    __shared__ uint16_t s_walk[8][128];  // columns of each warp left to the sample-by-sample walk
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    uint16_t* walk_list = s_walk[(threadIdx.x >> 5) & 7];
    // correctly rounded reciprocals (the same values as 1.0f / x, without the division sequence)
    const float inv2n = __frcp_rn((float)(2 * n)), invn = __frcp_rn((float)n);
    const RunFrame rf = run_frame<T>(f, Egh, n, invn);
    auto column_base = [&](int col, int& ia, int& ib, float& bx, float& by, float& bz) {
        ib = __float2int_rz(((float)col + 0.5f) * invn);
        ia = col - ib * n;
        const float ta = (float)(2 * ia + 1) * inv2n, tb = (float)(2 * ib + 1) * inv2n;
        bx = __fmaf_rn(tb, f.syx, __fmaf_rn(ta, f.sxx, f.px));
        by = __fmaf_rn(tb, f.syy, __fmaf_rn(ta, f.sxy, f.py));
        bz = __fmaf_rn(tb, f.syz, __fmaf_rn(ta, f.sxz, f.pz));
    };
    // the walk's sample: the same coordinates, bound and deferral as subsample_count
    auto walk_sample = [&](int ia, int ib, int c3, float bx, float by, float bz) {
        const float tc = (float)(2 * c3 + 1) * inv2n;
        int r = band(sample_g<T>(f, __fmaf_rn(tc, f.szx, bx), __fmaf_rn(tc, f.szy, by), __fmaf_rn(tc, f.szz, bz)),
                     f.Eg);
        if (r == 2) {
            ++*rechecks;
            r = undecided_sample<DEFER_ONLY>(df, sh, m, i, j, k, ia, ib, c3, n, x, q);
        }
        return r;
    };
    int cnt = 0, nwalk = 0;
#pragma unroll 1
    for (int base = 0; base < n * n; base += 32) {
        const int col = base + lane;
        float res = 0.f;
        int ia = 0, ib = 0;
        float bx = 0.f, by = 0.f, bz = 0.f;
        if (col < n * n) {
            column_base(col, ia, ib, bx, by, bz);
            // coordinates of sample c: w + c d
            res = run_column<T>(f, rf, __fmaf_rn(f.szx, inv2n, bx), __fmaf_rn(f.szy, inv2n, by), __fmaf_rn(f.szz, inv2n, bz));
        }
        const bool walk = res < 0.f;
        const unsigned mask = __ballot_sync(FULL, walk);
        const int pos = nwalk + __popc(mask & ((1u << lane) - 1u));
        nwalk += __popc(mask);
        if (walk) {
            if (pos < 128) {
                walk_list[pos] = (uint16_t)col;
            } else {  // list full: walk here
                for (int c3 = 0; c3 < n; ++c3) cnt += walk_sample(ia, ib, c3, bx, by, bz);
            }
        } else {
            cnt += (int)res;
        }
    }
    __syncwarp();
    // the listed columns' samples spread over the lanes
    const int listed = min(nwalk, 128);
#pragma unroll 1
    for (int e = lane; e < listed * n; e += 32) {
        const int w = __float2int_rz(((float)e + 0.5f) * invn), c3 = e - w * n;
        int ia, ib;
        float bx, by, bz;
        column_base(walk_list[w], ia, ib, bx, by, bz);
        cnt += walk_sample(ia, ib, c3, bx, by, bz);
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(FULL, cnt, o);
    return cnt;
}

// out of line for the recount (FP64 path included); subsample_cells_kernel inlines the body (DEFER_ONLY, no FP64 path)
template <int T, bool DEFER_ONLY>
__device__ __noinline__ int subsample_runs(const MeshK& m, const ShapeK& sh, const SampleFrame& f, float Egh, int64_t i,
                                           int64_t j, int64_t k, int n, const D3& x, const Q4& q,
                                           unsigned long long* rechecks, const Defer* df) {
    return subsample_runs_body<T, DEFER_ONLY>(m, sh, f, Egh, i, j, k, n, x, q, rechecks, df);
}

// The frame of a cell's lattice (cell (a0, b0, c0) of the tile) and its bounds: Ep of the coordinates with the offset, Egh of the
// columns' intervals (E above).
__device__ __forceinline__ int sample_frame(const MeshK& m, const ShapeK& sh, const float* M, const TileFrame& tf, int a0, int b0,
                                            int c0, SampleFrame& f, float& Ep, float& Egh) {
    const float u = U32;
    const float hx = m.h32[0], hy = m.h32[1], hz = m.h32[2];
    const float ox = (float)a0 * hx, oy = (float)b0 * hy, oz = (float)c0 * hz;  // cell corner within the tile
    const float dx = tf.bx + ox, dy = tf.by + oy, dz = tf.bz + oz;
    f.px = __fmaf_rn(M[0], dx, __fmaf_rn(M[1], dy, M[2] * dz));
    f.py = __fmaf_rn(M[3], dx, __fmaf_rn(M[4], dy, M[5] * dz));
    f.pz = __fmaf_rn(M[6], dx, __fmaf_rn(M[7], dy, M[8] * dz));
    f.sxx = M[0] * hx; f.sxy = M[3] * hx; f.sxz = M[6] * hx;
    f.syx = M[1] * hy; f.syy = M[4] * hy; f.syz = M[7] * hy;
    f.szx = M[2] * hz; f.szy = M[5] * hz; f.szz = M[8] * hz;
    const float sabs = fabsf(f.sxx) + fabsf(f.sxy) + fabsf(f.sxz) + fabsf(f.syx) + fabsf(f.syy) + fabsf(f.syz) +
                       fabsf(f.szx) + fabsf(f.szy) + fabsf(f.szz);
    f.E = 8.f * u * (tf.babs + fabsf(ox) + fabsf(oy) + fabsf(oz) + 2.f * (fabsf(dx) + fabsf(dy) + fabsf(dz)) +
                     3.f * (hx + hy + hz)) +
          8.f * u * (fabsf(f.px) + fabsf(f.py) + fabsf(f.pz) + sabs) + tf.e64 + 1e-30f;
    const int type = sh.type;
    const bool prism = sh.prism;
    const float* a = sh.p32;
    int kind = SS_GENERIC;
    if (type == SDFIBM_SHAPE_CIRCLE || type == SDFIBM_SHAPE_SPHERE || type == SDFIBM_SHAPE_ELLIPSE ||
        type == SDFIBM_SHAPE_ELLIPSOID)
        kind = SS_QUADRIC;
    else if (type == SDFIBM_SHAPE_RECTANGLE || type == SDFIBM_SHAPE_BOX)
        kind = SS_BOX;
    Ep = f.E;
    Egh = 0.f;
    if (kind == SS_GENERIC) return kind;
    {
        // sample = (corner + com) + steps: one more rounding of the corner, the conversion of com to FP32, and the
        // stepping FMAs now run at magnitudes up to |com| larger (the ellipsoid ignores com, as the reference does)
        const bool use_com = type != SDFIBM_SHAPE_ELLIPSOID;
        const float c0x = use_com ? sh.com32[0] : 0.f, c0y = use_com ? sh.com32[1] : 0.f;
        f.px += c0x;
        f.py += c0y;
        if (prism) {
            // 2-D shapes: the local z is the FP32 com z for every sample (exact steps of zero)
            f.pz = sh.com32[2];
            f.sxz = 0.f; f.syz = 0.f; f.szz = 0.f;
        } else if (use_com) {
            f.pz += sh.com32[2];
        }
        const float cabs = use_com ? fabsf(sh.com32[0]) + fabsf(sh.com32[1]) + fabsf(sh.com32[2]) : 0.f;
        Ep = f.E + 2.f * u * (fabsf(f.px) + fabsf(f.py) + fabsf(f.pz) + sabs) + 5.f * u * cabs;
    }
    // largest |coordinate| any sample of the cell can reach
    const float mx = fabsf(f.px) + fabsf(f.sxx) + fabsf(f.syx) + fabsf(f.szx) + Ep;
    const float my = fabsf(f.py) + fabsf(f.sxy) + fabsf(f.syy) + fabsf(f.szy) + Ep;
    const float mz = fabsf(f.pz) + fabsf(f.sxz) + fabsf(f.syz) + fabsf(f.szz) + Ep;
    if (kind == SS_QUADRIC) {
        switch (type) {
            case SDFIBM_SHAPE_CIRCLE:
            case SDFIBM_SHAPE_SPHERE: f.k0 = 1.f; f.k1 = 1.f; f.k2 = 1.f; f.k3 = a[1]; break;
            case SDFIBM_SHAPE_ELLIPSE: f.k0 = a[2]; f.k1 = a[3]; f.k2 = 0.f; f.k3 = 1.f; break;
            default: f.k0 = a[3]; f.k1 = a[4]; f.k2 = a[5]; f.k3 = 1.f; break;
        }
        f.Eg = (2.f * (mx * f.k0 + my * f.k1 + mz * f.k2) + Ep * (f.k0 + f.k1 + f.k2)) * Ep +
               10.f * u * (mx * mx * f.k0 + my * my * f.k1 + mz * mz * f.k2 + f.k3);
        Egh = f.Eg + 128.f * u * (mx * mx * f.k0 + my * my * f.k1 + mz * mz * f.k2 + f.k3);
    } else {
        f.k0 = a[0]; f.k1 = a[1];
        f.k2 = prism ? INFINITY : a[2];  // the rectangle has no z extent
        f.k3 = 0.f;
        f.Eg = Ep + 2.f * u * (fmaxf(mx, fmaxf(my, prism ? 0.f : mz)) + fmaxf(a[0], fmaxf(a[1], prism ? 0.f : a[2])));
        Egh = f.Eg + 64.f * u * (fmaxf(mx, fmaxf(my, mz)) + fmaxf(a[0], fmaxf(a[1], a[2])));
    }
    return kind;
}

// Inside count of the cell's n^3 (n^2 on one-layer meshes) lattice; with a Defer the undecided points are not counted
// here but appended to the recheck list.  DEFER_ONLY: x, q and (i, j, k) only feed the FP64 path, which it lacks.
template <bool DEFER_ONLY>
static __device__ __forceinline__ int subsample_warp_body(const MeshK& m, const ShapeK& sh, const float* M,
                                                          const TileFrame& tf, int a0, int b0, int c0, const D3& x,
                                                          const Q4& q, int64_t i, int64_t j, int64_t k, int n,
                                                          unsigned long long* rechecks, const Defer* df) {
    SampleFrame f;
    float Ep, Egh;
    const int kind = sample_frame(m, sh, M, tf, a0, b0, c0, f, Ep, Egh);
    // 3-D convex shapes count runs along columns from 5 samples per axis; in the recount lattices of 16 and more skip
    // 4 x 4 x 4 blocks instead
    const bool use_runs = !m.twod && !sh.prism && n >= 5 && (DEFER_ONLY || n < 16);
    int cnt;
    if (kind == SS_QUADRIC) {
        const int lb = block_log2(n, m.twod != 0);
        if (use_runs && DEFER_ONLY)
            cnt = subsample_runs_body<SS_QUADRIC, true>(m, sh, f, Egh, i, j, k, n, x, q, rechecks, df);
        else if (use_runs)
            cnt = subsample_runs<SS_QUADRIC, DEFER_ONLY>(m, sh, f, Egh, i, j, k, n, x, q, rechecks, df);
        else if (lb)
            cnt = subsample_blocks<SS_QUADRIC, DEFER_ONLY>(m, sh, f, i, j, k, n, lb, Ep, x, q, rechecks, df);
        else
            cnt = subsample_count<SS_QUADRIC, DEFER_ONLY>(m, sh, f, i, j, k, n, x, q, rechecks, df);
    } else if (kind == SS_BOX) {
        const int lb = block_log2(n, m.twod != 0);
        if (use_runs && DEFER_ONLY)
            cnt = subsample_runs_body<SS_BOX, true>(m, sh, f, Egh, i, j, k, n, x, q, rechecks, df);
        else if (use_runs)
            cnt = subsample_runs<SS_BOX, DEFER_ONLY>(m, sh, f, Egh, i, j, k, n, x, q, rechecks, df);
        else if (lb)
            cnt = subsample_blocks<SS_BOX, DEFER_ONLY>(m, sh, f, i, j, k, n, lb, Ep, x, q, rechecks, df);
        else
            cnt = subsample_count<SS_BOX, DEFER_ONLY>(m, sh, f, i, j, k, n, x, q, rechecks, df);
    } else {
        cnt = subsample_count<SS_GENERIC, DEFER_ONLY>(m, sh, f, i, j, k, n, x, q, rechecks, df);
    }
    return cnt;
}

// the out-of-line form of the recount (FP64 path included)
static __device__ __noinline__ int subsample_warp(const MeshK& m, const ShapeK& sh, const float* M, const TileFrame& tf,
                                                  int a0, int b0, int c0, const D3& x, const Q4& q, int64_t i,
                                                  int64_t j, int64_t k, int n, unsigned long long* rechecks,
                                                  const Defer* df) {
    return subsample_warp_body<false>(m, sh, M, tf, a0, b0, c0, x, q, i, j, k, n, rechecks, df);
}

// ---- signed distance for REF-GEO: FP64 where it decides, FP32 where it only scales ------------------------------------
// The geometry consumes phi in FP32, so phi needs ~1e-7 relative accuracy and the reference's exact sign and filter
// (|phi| < 1e-8 -> -1e-8).  The local point and every cancelling difference (|p|^2 - r^2, |x| - a, ...) are FP64; the
// square roots and the final division only scale a non-cancelling quantity and run in FP32.  Values within 1e-6 of
// the filter threshold are recomputed with the reference's full FP64 sequence by the caller.  2-D shapes and half spaces: 3-D
// spheres, ellipsoids and boxes have sdf_ff_at.
__device__ inline float rect_mixed(double x, double y, double ra, double rb) {
    const double dx = fabs(x) - ra, dy = fabs(y) - rb;
    const double dxp = dmax(0.0, dx), dyp = dmax(0.0, dy);
    return sqrtf((float)(dxp * dxp + dyp * dyp)) + (float)dmin(0.0, dmax(dx, dy));
}
static __device__ __noinline__ float sdf_mixed(const ShapeK& s, const D3& p) {
    const double* a = s.p;
    const D3 com{s.com[0], s.com[1], s.com[2]};
    switch (s.type) {
        case SDFIBM_SHAPE_CIRCLE: {
            const D3 q = com + D3{p.x, p.y, 0.0};
            const double qq = magSqr(q);
            return (float)(qq - a[1]) / (sqrtf((float)qq) + (float)a[0]);
        }
        case SDFIBM_SHAPE_ELLIPSE: {
            const D3 q = com + p;
            const double xa = q.x * q.x * a[2], yb = q.y * q.y * a[3];
            return (float)(0.5 * (xa + yb - 1.0)) / sqrtf((float)(xa * a[2] + yb * a[3]));
        }
        case SDFIBM_SHAPE_RECTANGLE: {
            const D3 q = com + p;
            return rect_mixed(q.x, q.y, a[0], a[1]);
        }
        case SDFIBM_SHAPE_PLANE: return (float)p.y;
        case SDFIBM_SHAPE_CIRCLE_TAIL: {
            const D3 q = com + p;
            const double qq = q.x * q.x + q.y * q.y;
            const float d1 = (float)(qq - a[3]) / (sqrtf((float)qq) + (float)a[0]);
            const float d2 = rect_mixed(q.x - a[4], q.y, a[4], a[2]);
            return fminf(d1, d2);
        }
        case SDFIBM_SHAPE_CIRCLE_TWOTAIL: {
            const D3 q = com + p;
            const double qq = q.x * q.x + q.y * q.y;
            const float dc = (float)(qq - a[3]) / (sqrtf((float)qq) + (float)a[0]);
            const D3 r1 = rot30_64(D3{q.x, q.y, 0.0}), r2 = rot30_64(D3{q.x, -q.y, 0.0});
            const float d1 = rect_mixed(r1.x - a[4], r1.y, a[4], a[2]);
            const float d2 = rect_mixed(r2.x - a[4], r2.y, a[4], a[2]);
            return fminf(dc, fminf(d1, d2));
        }
    }
    return 0.f;
}

// ---- two-float vertex distances (REF-GEO, 3-D spheres, ellipsoids and boxes) ---------------------------------------
// Pairs hi + lo with error-free sums and products (Dekker, Knuth), explicit rounding intrinsics so that nothing is
// contracted or reassociated; each operation errs by a few 2^-48 of its operands' magnitudes.  GB300 issues FP32 at 64
// times the FP64 rate, so the pairs replace the FP64 local point and the cancelling differences of sdf_mixed.
struct FF {
    float hi, lo;
};
__device__ __forceinline__ FF ff_fast(float a, float b) {  // |a| >= |b|, or the pair carries the rounding of b
    const float s = __fadd_rn(a, b);
    return FF{s, __fsub_rn(b, __fsub_rn(s, a))};
}
__device__ __forceinline__ FF ff_sum(float a, float b) {
    const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
    return FF{s, __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb))};
}
__device__ __forceinline__ FF ff_add(FF x, FF y) {
    const FF t = ff_sum(x.hi, y.hi);
    return ff_fast(t.hi, __fadd_rn(t.lo, __fadd_rn(x.lo, y.lo)));
}
__device__ __forceinline__ FF ff_mul(FF x, FF y) {
    const float p = __fmul_rn(x.hi, y.hi);
    return ff_fast(p, __fmaf_rn(x.hi, y.lo, __fmaf_rn(x.lo, y.hi, __fmaf_rn(x.hi, y.hi, -p))));
}
__device__ __forceinline__ FF ff_scale(FF x, float n) {  // n: a small integer, exact in FP32
    const float p = __fmul_rn(x.hi, n);
    return ff_fast(p, __fmaf_rn(x.lo, n, __fmaf_rn(x.hi, n, -p)));
}
__device__ __forceinline__ FF ff_abs(FF x) { return x.hi < 0.f ? FF{-x.hi, -x.lo} : x; }

// component r of the local point of bbox vertex (da, db, dc) from the plan's two-float map; mag: the sum of the magnitudes
__device__ __forceinline__ FF ff_local(const SolidPlan& pl, int r, float da, float db, float dc, float& mag) {
    const float f3[3] = {da, db, dc};
    FF v{pl.lmap_hi[r], pl.lmap_lo[r]};
    mag = fabsf(pl.lmap_hi[r]);
#pragma unroll
    for (int t = 0; t < 3; ++t) {
        const int i = 3 + 3 * t + r;
        v = ff_add(v, ff_scale(FF{pl.lmap_hi[i], pl.lmap_lo[i]}, f3[t]));
        mag += fabsf(f3[t] * pl.lmap_hi[i]);
    }
    return v;
}
// Solid::phi at local point P as sdf_mixed computes it (the same FP32 formula after the cancelling differences); err / den
// bounds the difference to the exact value with a factor of 4 to spare over the operations' roundoff (2^-44 of the magnitudes,
// ml those of the local point).
__device__ inline float sdf_ff_at(const ShapeK& s, const FF (&P)[3], float ml, float& err, float& den) {
    const float U44 = 5.6843418860808015e-14f;  // 2^-44
    const float* a = s.p32;
    if (s.type == SDFIBM_SHAPE_ELLIPSOID) {  // the reference's ellipsoid ignores com
        const FF xa = ff_mul(ff_mul(P[0], P[0]), FF{a[3], s.p_lo[3]});
        const FF yb = ff_mul(ff_mul(P[1], P[1]), FF{a[4], s.p_lo[4]});
        const FF zc = ff_mul(ff_mul(P[2], P[2]), FF{a[5], s.p_lo[5]});
        const FF sum = ff_add(ff_add(ff_add(xa, yb), zc), FF{-1.f, 0.f});
        den = sqrtf(xa.hi * a[3] + yb.hi * a[4] + zc.hi * a[5]);
        const float am = fmaxf(a[3], fmaxf(a[4], a[5]));
        const float pm = fmaxf(fabsf(P[0].hi), fmaxf(fabsf(P[1].hi), fabsf(P[2].hi)));
        err = 4.f * U44 * (xa.hi + yb.hi + zc.hi + 1.f + 6.f * am * pm * (ml + pm));
        return (0.5f * __fadd_rn(sum.hi, sum.lo)) / den;
    }
    FF q[3];
    float qm = 0.f;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        q[r] = P[r];
        if (s.com32[r] != 0.f) q[r] = ff_add(P[r], FF{s.com32[r], s.com_lo[r]});  // (adding zero changes nothing)
        qm = fmaxf(qm, fabsf(q[r].hi));
    }
    const float mag = ml + fabsf(s.com32[0]) + fabsf(s.com32[1]) + fabsf(s.com32[2]) + qm;
    if (s.type == SDFIBM_SHAPE_SPHERE) {
        const FF qq = ff_add(ff_add(ff_mul(q[0], q[0]), ff_mul(q[1], q[1])), ff_mul(q[2], q[2]));
        const FF num = ff_add(qq, FF{-a[1], -s.p_lo[1]});
        den = sqrtf(qq.hi) + a[0];
        err = 4.f * U44 * (qq.hi + a[1] + 6.f * qm * mag);
        return __fadd_rn(num.hi, num.lo) / den;
    }
    // box
    float d[3];
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        const FF t = ff_add(ff_abs(q[r]), FF{-a[r], -s.p_lo[r]});
        d[r] = __fadd_rn(t.hi, t.lo);
    }
    err = 4.f * U44 * (mag + a[0] + a[1] + a[2]);
    den = 1.f;
    const float dxp = fmaxf(0.f, d[0]), dyp = fmaxf(0.f, d[1]), dzp = fmaxf(0.f, d[2]);
    return sqrtf(dxp * dxp + dyp * dyp + dzp * dzp) + fminf(0.f, fmaxf(d[2], fmaxf(d[0], d[1])));
}

// the filter of sdf.h:147-150 on such a value; false: its decision is not certain, as where den is 0 or the value no number (an
// ellipsoid's distance next to its centre)
__device__ __forceinline__ bool ff_filter(float& phi, float err, float den) {
    const float a = fabsf(phi);
    if (a < 1e-8f) phi = -1e-8f;
    return (fabsf(a - 1e-8f) - 1e-14f) * den > err;
}
__device__ inline float sdf_ff(const ShapeK& s, const SolidPlan& pl, float da, float db, float dc, float& err,
                               float& den) {
    FF P[3];
    float ml = 0.f;
#pragma unroll
    for (int r = 0; r < 3; ++r) {
        float mag;
        P[r] = ff_local(pl, r, da, db, dc, mag);
        ml = fmaxf(ml, mag);
    }
    return sdf_ff_at(s, P, ml, err, den);
}

// filter of sdf.h:147-150 applied to a value of sdf_mixed; *exact_needed set when the value sits on the threshold or is no number (an
// ellipse's next to its axis)
__device__ inline float filter_mixed(const ShapeK& s, float phi, bool* exact_needed) {
    if (s.type == SDFIBM_SHAPE_PLANE) return phi;  // the plane's distance is unfiltered and exact
    const float a = fabsf(phi);
    if (!(fabsf(a - 1e-8f) > 1e-14f && a < INFINITY)) *exact_needed = true;
    return a < 1e-8f ? -1e-8f : phi;
}

// REF-GEO: the tile's cut cells (one warp) appended to the cell list with the distances of their 8 vertices; out of line to keep
// the tile loop small.  tile0 = fraction index of the tile's cell (0,0,0).
template <int TX, int TY, int TZ>
static __device__ __noinline__ void write_refgeo_list(const ClassifyArgs& A, const uint8_t* cutlist, int ncut,
                                                      const float* vphi, int s, int64_t tile0, int ext0, int ext1) {
    constexpr int VX = TX + 1, VY = TY + 1;
    const int lane = threadIdx.x & 31;
    for (int u0 = 0; u0 < ncut; u0 += 32) {
        int base = 0;
        if (lane == 0) base = atomicAdd(&A.cnt->n_feat, min(32, ncut - u0));
        base = __shfl_sync(0xffffffffu, base, 0);
        const int u = u0 + lane;
        if (u < ncut) {
            const int e = cutlist[u];
            const int a = e % TX, b = (e / TX) % TY, c = e / (TX * TY);
            const int v0 = a + VX * (b + VY * c);
            const int64_t slot = (int64_t)base + lane;
            if (slot < A.feat_cap) {
                const int vo[8] = {0, 1, VX, VX + 1, VX * VY, VX * VY + 1, VX * VY + VX, VX * VY + VX + 1};
#pragma unroll
                for (int q = 0; q < 8; ++q) A.rg_phi[q * A.feat_cap + slot] = vphi[v0 + vo[q]];
                A.fref_solid[slot] = s;
                A.fref_index[slot] = tile0 + a + (int64_t)ext0 * (b + (int64_t)ext1 * c);
            } else {
                set_error(A.cnt, DERR_CAPACITY);
            }
        }
    }
}

// SUBSAMPLE and LEARNED: the tile's cut cells (one warp) appended to the cell list as (solid, fraction index)
template <int TX, int TY, int TZ>
static __device__ __noinline__ void write_cut_list(const ClassifyArgs& A, const uint8_t* cutlist, int ncut, int s,
                                                   int64_t tile0, int ext0, int ext1) {
    const int lane = threadIdx.x & 31;
    // LEARNED, a solid under rho_min cells: from the back of the list, for the fallback
    const bool back = A.method == SDFIBM_FRACTION_LEARNED && A.plan[s].radius_cells < A.rho_min;
    for (int u0 = 0; u0 < ncut; u0 += 32) {
        int base = 0;
        if (lane == 0) base = atomicAdd(back ? &A.cnt->n_small : &A.cnt->n_feat, min(32, ncut - u0));
        base = __shfl_sync(0xffffffffu, base, 0);
        const int u = u0 + lane;
        if (u < ncut) {
            const int e = cutlist[u];
            const int a = e % TX, b = (e / TX) % TY, c = e / (TX * TY);
            const int64_t slot = back ? A.feat_cap - 1 - ((int64_t)base + lane) : (int64_t)base + lane;
            if (slot >= 0 && slot < A.feat_cap) {
                A.fref_solid[slot] = s;
                A.fref_index[slot] = tile0 + a + (int64_t)ext0 * (b + (int64_t)ext1 * c);
            } else {
                set_error(A.cnt, DERR_CAPACITY);
            }
        }
    }
}

// ---- the tile kernel: one warp per chunk of consecutive tiles of one solid ------------------------------------------
constexpr int CLS_WARPS = 8;

// one chunk of any shape: a test per vertex with its own error bound
template <int TX, int TY, int TZ, int METHOD>
__device__ __forceinline__ void classify_any(const ClassifyArgs& A, const int2 ch, unsigned long long& rechecks,
                                             unsigned long long& valid_cells) {
    constexpr int VX = TX + 1, VY = TY + 1, VZ = TZ + 1, NV = VX * VY * VZ, NC = TX * TY * TZ;
    constexpr bool FLAT = TZ == 2;  // only there 3-D spheres, ellipsoids and boxes come here
    __shared__ uint8_t s_vin[CLS_WARPS][NV];
    __shared__ uint8_t s_need[CLS_WARPS][NV];
    __shared__ float s_phi[CLS_WARPS][NV];
    __shared__ uint8_t s_cut[CLS_WARPS][NC];
    __shared__ uint8_t s_vlist[CLS_WARPS][NV];
    const MeshK& m = A.m;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint8_t* vin = s_vin[w];
    uint8_t* vneed = s_need[w];
    float* vphi = s_phi[w];
    uint8_t* cutlist = s_cut[w];
    {
        const int s = ch.x;
        const SolidK& k = A.sk[s];
        const SolidPlan& pl = A.plan[s];
        const int ntile_all = k.ntile[0] * k.ntile[1] * k.ntile[2];
        const int t_end = min(ch.y + (k.infinite ? A.wall_tiles : A.finite_tiles), ntile_all);
        const Q4 q = state_quat(A.st[s]);
        const D3 x = state_pos(A.st[s]);
        const ShapeK& sh = k.shape;
        float M[9];
#pragma unroll
        for (int r = 0; r < 9; ++r) M[r] = pl.M[r];
        const int32_t vlo0 = pl.vlo[0], vlo1 = pl.vlo[1], vlo2 = pl.vlo[2];
        const int32_t vhi0 = pl.vhi[0], vhi1 = pl.vhi[1], vhi2 = pl.vhi[2];
        uint8_t* out = A.cls + k.scratch_off;
        const float sb[3] = {pl.base32[0], pl.base32[1], pl.base32[2]};
        for (int t = ch.y; t < t_end; ++t) {
            const int tx = t % k.ntile[0], ty = (t / k.ntile[0]) % k.ntile[1], tz = t / (k.ntile[0] * k.ntile[1]);
            const int cx = min(TX, k.ext[0] - tx * TX);
            const int cy = min(TY, k.ext[1] - ty * TY);
            const int cz = min(TZ, k.ext[2] - tz * TZ);
            const int64_t I0 = (int64_t)pl.lo[0] + tx * TX;
            const int64_t J0 = (int64_t)pl.lo[1] + ty * TY;
            const int64_t K0 = (int64_t)pl.lo[2] + tz * TZ;
            auto local_index = [&](int a, int b, int c) {
                return (int64_t)(tx * TX + a) + (int64_t)k.ext[0] * ((ty * TY + b) + (int64_t)k.ext[1] * (tz * TZ + c));
            };
            // whole tile outside the mesh or outside the solid's oriented bounding box: no cell has an inside vertex
            // (nobody reads the class bytes of such a tile)
            if (pl.err != 0 || I0 + cx <= 0 || J0 + cy <= 0 || K0 + cz <= 0 || I0 >= m.nx || J0 >= m.ny || K0 >= m.nz ||
                I0 + cx < vlo0 || I0 > vhi0 || J0 + cy < vlo1 || J0 > vhi1 || K0 + cz < vlo2 || K0 > vhi2)
                continue;
            bool cull = false;
            if (FLAT && pl.cull_box) {
                // separating axes of the solid's local box: the tile's centre and half extents seen in the local
                // frame (FP32 with a relative margin of 1e-4 on both sides of every comparison)
                const float hx = 0.5f * (float)cx * m.h32[0], hy = 0.5f * (float)cy * m.h32[1],
                            hz = 0.5f * (float)cz * m.h32[2];
                const float tcx = sb[0] + (float)(tx * TX) * m.h32[0] + hx;
                const float tcy = sb[1] + (float)(ty * TY) * m.h32[1] + hy;
                const float tcz = sb[2] + (float)(tz * TZ) * m.h32[2] + hz;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const float lc = __fmaf_rn(M[3 * a], tcx, __fmaf_rn(M[3 * a + 1], tcy, M[3 * a + 2] * tcz));
                    const float rad = fabsf(M[3 * a]) * hx + fabsf(M[3 * a + 1]) * hy + fabsf(M[3 * a + 2]) * hz;
                    const float gap = fabsf(lc - pl.lbox_c[a]) - pl.lbox_s[a] - rad;
                    cull = cull || gap > 1e-4f * (fabsf(lc) + fabsf(pl.lbox_c[a]) + pl.lbox_s[a] + rad) + 1e-30f;
                }
            }
            if (cull) {
                for (int e = lane; e < NC; e += 32) {
                    const int a = e % TX, b = (e / TX) % TY, c = e / (TX * TY);
                    if (a < cx && b < cy && c < cz) out[local_index(a, b, c)] = 0;
                }
                continue;
            }
            // tile frame in FP32: the solid's FP64 base plus the tile's cell offset; babs covers both roundings
            TileFrame tf;
            {
                const float ofx = (float)(tx * TX) * m.h32[0], ofy = (float)(ty * TY) * m.h32[1],
                            ofz = (float)(tz * TZ) * m.h32[2];
                tf.bx = sb[0] + ofx; tf.by = sb[1] + ofy; tf.bz = sb[2] + ofz;
                tf.babs = fabsf(sb[0]) + fabsf(sb[1]) + fabsf(sb[2]) + 2.f * (fabsf(ofx) + fabsf(ofy) + fabsf(ofz)) +
                          fabsf(tf.bx) + fabsf(tf.by) + fabsf(tf.bz);
                tf.e64 = pl.e64;
            }
            for (int v = lane; v < NV; v += 32) {
                const int a = v % VX, b = (v / VX) % VY, c = v / (VX * VY);
                const int64_t I = I0 + a, J = J0 + b, K = K0 + c;
                uint8_t r = 0;
                if (a <= cx && b <= cy && c <= cz && I >= vlo0 && I <= vhi0 && J >= vlo1 && J <= vhi1 && K >= vlo2 &&
                    K <= vhi2 && I >= 0 && J >= 0 && K >= 0 && I <= m.nx && J <= m.ny && K <= m.nz) {
                    const float ox = (float)a * m.h32[0], oy = (float)b * m.h32[1], oz = (float)c * m.h32[2];
                    r = (uint8_t)classify_point(sh, M, tf, ox, oy, oz, m, I, J, K, 0, x, q, &rechecks);
                }
                vin[v] = r;
                vneed[v] = 0;
            }
            __syncwarp();
            int ncut = 0;
#pragma unroll 1
            for (int base = 0; base < NC; base += 32) {
                const int e = base + lane;
                const int a = e % TX, b = (e / TX) % TY, c = e / (TX * TY);
                uint8_t cls = 0;
                const bool in_tile = e < NC && a < cx && b < cy && c < cz;
                if (in_tile) {
                    const int64_t I = I0 + a, J = J0 + b, K = K0 + c;
                    if (I >= 0 && J >= 0 && K >= 0 && I < m.nx && J < m.ny && K < m.nz) {
                        ++valid_cells;
                        const int v0 = a + VX * (b + VY * c);
                        const int cntv = vin[v0] + vin[v0 + 1] + vin[v0 + VX] + vin[v0 + VX + 1] + vin[v0 + VX * VY] +
                                         vin[v0 + VX * VY + 1] + vin[v0 + VX * VY + VX] + vin[v0 + VX * VY + VX + 1];
                        if (cntv == 8) {
                            cls = 1;
                        } else if (cntv > 0) {
                            const float ox = ((float)a + 0.5f) * m.h32[0], oy = ((float)b + 0.5f) * m.h32[1],
                                        oz = ((float)c + 0.5f) * m.h32[2];
                            const int ci = classify_point(sh, M, tf, ox, oy, oz, m, I, J, K, 1, x, q, &rechecks);
                            cls = ci ? 2 : 3;
                        }
                    }
                    out[local_index(a, b, c)] = cls;
                }
                // compact the cut candidates of this pass
                const bool is_cut = (cls == 2 || cls == 3) && METHOD >= 0;
                const unsigned bal = __ballot_sync(FULL, is_cut);
                if (is_cut) {
                    cutlist[ncut + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)e;
                    if (METHOD == SDFIBM_FRACTION_REFGEO) {
                        const int v0 = a + VX * (b + VY * c);
                        vneed[v0] = 1; vneed[v0 + 1] = 1; vneed[v0 + VX] = 1; vneed[v0 + VX + 1] = 1;
                        vneed[v0 + VX * VY] = 1; vneed[v0 + VX * VY + 1] = 1; vneed[v0 + VX * VY + VX] = 1;
                        vneed[v0 + VX * VY + VX + 1] = 1;
                    }
                }
                ncut += __popc(bal);
            }
            if (ncut == 0) continue;
            __syncwarp();
            if (METHOD == SDFIBM_FRACTION_REFGEO) {
                // Solid::phi once per vertex next to a cut candidate.  The needed vertices are compacted first so
                // every FP64 instruction runs on a full warp; the local point is the solid's FP64 local map applied to
                // small integer offsets from the bbox corner.
                uint8_t* vlist = s_vlist[w];
                int nneed = 0;
                for (int base = 0; base < NV; base += 32) {
                    const int v = base + lane;
                    const bool need = v < NV && vneed[v];
                    const unsigned bal = __ballot_sync(FULL, need);
                    if (need) vlist[nneed + __popc(bal & ((1u << lane) - 1u))] = (uint8_t)v;
                    nneed += __popc(bal);
                }
                __syncwarp();
                const double* L = pl.lmap;
                // 3-D spheres, ellipsoids and boxes: two-float distances (FP32 pipe); others: sdf_mixed (FP64)
                const bool ff_shape = FLAT && !sh.prism && (sh.type == SDFIBM_SHAPE_SPHERE ||
                                                    sh.type == SDFIBM_SHAPE_ELLIPSOID || sh.type == SDFIBM_SHAPE_BOX);
                for (int u = lane; u < nneed; u += 32) {
                    const int v = vlist[u];
                    const int a = v % VX, b = (v / VX) % VY, c = v / (VX * VY);
                    bool exact = false;
                    float ph;
                    if (ff_shape) {
                        float err, den;
                        ph = sdf_ff(sh, pl, (float)(tx * TX + a), (float)(ty * TY + b), (float)(tz * TZ + c), err, den);
                        exact = !ff_filter(ph, err, den);
                    } else {
                        const double da = (double)(tx * TX + a), db = (double)(ty * TY + b),
                                     dc = (double)(tz * TZ + c);
                        const D3 plc{L[0] + da * L[3] + db * L[6] + dc * L[9],
                                     L[1] + da * L[4] + db * L[7] + dc * L[10],
                                     L[2] + da * L[5] + db * L[8] + dc * L[11]};
                        ph = filter_mixed(sh, sdf_mixed(sh, plc), &exact);
                    }
                    if (exact || sh.type == SDFIBM_SHAPE_PLANE) ph = exact_phi_point(sh, m, I0 + a, J0 + b, K0 + c, x, q);
                    vphi[v] = ph;
                }
                __syncwarp();
                // the cut cells and their vertex distances are listed; refgeo_cells_kernel computes the fractions
                write_refgeo_list<TX, TY, TZ>(A, cutlist, ncut, vphi, s, k.scratch_off + local_index(0, 0, 0), k.ext[0],
                                              k.ext[1]);
            } else if (METHOD >= 0) {
                // SUBSAMPLE and LEARNED: the cut cells are listed; subsample_cells_kernel samples them (LEARNED:
                // learned_stencil_kernel computes the model's inputs, a thread per cell), a warp per cell
                write_cut_list<TX, TY, TZ>(A, cutlist, ncut, s, k.scratch_off + local_index(0, 0, 0), k.ext[0],
                                           k.ext[1]);
            }
            __syncwarp();
        }
    }
}

// ---- the same for the shapes nearly every cloud is made of: 3-D spheres, ellipsoids and boxes, and on one- and two-layer
// meshes circles, ellipses, rectangles and half spaces that turn about z.  One error bound covers every vertex of the solid's bounding box,
// so a vertex costs a few multiply-adds and two comparisons; a tile's answers are ballots, and cells are read off them with
// shifts.  Tiles are culled 32 at a time, a lane each.  Bound by instruction issue.  Measured against a test per vertex with
// its own bound (GB300, 512^3, 16 384 solids): LEARNED 1.13 -> 0.43 ms, REF-GEO 1.63 -> 0.44 (0.92 while it computed the
// vertex distances too, which refgeo_cells_kernel does now).
//
// The bound.  A local coordinate is M (b + v h) + com from FP32 roundings of the base b (bbox corner minus centre), M, h and
// com, added in a chain of at most 12 roundings of partial sums no larger than A = max|M| (|b|_1 + sum_a ext_a h_a) + |com|_1:
// 16 u A, plus the FP64 reference's own rounding e64, holds its error (E).  For the inside function the bounds are those of
// the sampling kernels (SampleFrame::Eg, and 64 units of roundoff of the magnitudes where a column's polynomial is used), with
// the largest coordinates of the whole box.  Values within the bound go to the point's own bound and then to the FP64 test,
// so the classes are the reference's.
struct FastFrame {
    float px, py, pz;  // local coordinates of the bbox corner (com added)
    float sxx, sxy, sxz, syx, syy, syz, szx, szy, szz;  // local images of the cell edges
    float k0, k1, k2, k3;  // quadric X^2 k0 + Y^2 k1 + Z^2 k2 - k3, or box half extents k0..k2
    float Eg;
    float A2;          // quadric: the polynomial's leading coefficient along z
    bool quadric, half_space;
};
__device__ __forceinline__ FastFrame fast_frame(const MeshK& m, const SolidK& k, const SolidPlan& pl, bool prism) {
    FastFrame f;
    const ShapeK& sh = k.shape;
    const float* M = pl.M;
    const float hx = m.h32[0], hy = m.h32[1], hz = m.h32[2];
    const float bx = pl.base32[0], by = pl.base32[1], bz = pl.base32[2];
    const bool use_com = sh.type != SDFIBM_SHAPE_ELLIPSOID;  // the reference's ellipsoid ignores com
    const float c0 = use_com ? sh.com32[0] : 0.f, c1 = use_com ? sh.com32[1] : 0.f, c2 = use_com ? sh.com32[2] : 0.f;
    f.px = __fmaf_rn(M[0], bx, __fmaf_rn(M[1], by, M[2] * bz)) + c0;
    f.py = __fmaf_rn(M[3], bx, __fmaf_rn(M[4], by, M[5] * bz)) + c1;
    f.pz = __fmaf_rn(M[6], bx, __fmaf_rn(M[7], by, M[8] * bz)) + c2;
    f.sxx = M[0] * hx; f.sxy = M[3] * hx; f.sxz = M[6] * hx;
    f.syx = M[1] * hy; f.syy = M[4] * hy; f.syz = M[7] * hy;
    f.szx = M[2] * hz; f.szy = M[5] * hz; f.szz = M[8] * hz;
    if (prism) {  // 2-D shapes: the local z is com's for every point
        f.pz = c2;
        f.sxz = 0.f; f.syz = 0.f; f.szz = 0.f;
    }
    const float ex = (float)k.ext[0] + 4.f, ey = (float)k.ext[1] + 4.f, ez = (float)k.ext[2] + 4.f;
    float mm = 1.f;
    for (int r = 0; r < 9; ++r) mm = fmaxf(mm, fabsf(M[r]));
    const float A = mm * (fabsf(bx) + fabsf(by) + fabsf(bz) + ex * hx + ey * hy + ez * hz) + fabsf(c0) + fabsf(c1) + fabsf(c2);
    const float E = 16.f * U32 * A + pl.e64 + 1e-30f;
    // largest |coordinate| of any vertex or centre of the box (and of the tiles that reach beyond it)
    const float mx = fabsf(f.px) + ex * fabsf(f.sxx) + ey * fabsf(f.syx) + ez * fabsf(f.szx) + E;
    const float my = fabsf(f.py) + ex * fabsf(f.sxy) + ey * fabsf(f.syy) + ez * fabsf(f.szy) + E;
    const float mz = fabsf(f.pz) + ex * fabsf(f.sxz) + ey * fabsf(f.syz) + ez * fabsf(f.szz) + E;
    const float* a = sh.p32;
    f.quadric = true;
    f.half_space = false;
    switch (sh.type) {
        case SDFIBM_SHAPE_CIRCLE:
        case SDFIBM_SHAPE_SPHERE: f.k0 = 1.f; f.k1 = 1.f; f.k2 = 1.f; f.k3 = a[1]; break;
        case SDFIBM_SHAPE_ELLIPSE: f.k0 = a[2]; f.k1 = a[3]; f.k2 = 0.f; f.k3 = 1.f; break;
        case SDFIBM_SHAPE_ELLIPSOID: f.k0 = a[3]; f.k1 = a[4]; f.k2 = a[5]; f.k3 = 1.f; break;
        case SDFIBM_SHAPE_PLANE: f.quadric = false; f.half_space = true; f.k0 = f.k1 = f.k2 = f.k3 = 0.f; break;
        default: f.quadric = false; f.k0 = a[0]; f.k1 = a[1]; f.k2 = prism ? INFINITY : a[2]; f.k3 = 0.f; break;
    }
    if (f.quadric) {
        const float mag = mx * mx * f.k0 + my * my * f.k1 + mz * mz * f.k2 + f.k3;
        f.Eg = (2.f * (mx * f.k0 + my * f.k1 + mz * f.k2) + E * (f.k0 + f.k1 + f.k2)) * E + 74.f * U32 * mag;
        f.A2 = __fmaf_rn(f.szx, f.szx * f.k0, __fmaf_rn(f.szy, f.szy * f.k1, f.szz * f.szz * f.k2));
    } else if (f.half_space) {  // inside: local y < 0
        f.Eg = E + 2.f * U32 * my;
        f.A2 = 0.f;
    } else {
        f.Eg = E + 34.f * U32 * (fmaxf(mx, fmaxf(my, prism ? 0.f : mz)) + fmaxf(a[0], fmaxf(a[1], prism ? 0.f : a[2])));
        f.A2 = 0.f;
    }
    return f;
}
// inside function at a local point (negative inside), within f.Eg of its exact value
__device__ __forceinline__ float fast_g(const FastFrame& f, float X, float Y, float Z) {
    if (f.quadric) return __fmaf_rn(X * X, f.k0, __fmaf_rn(Y * Y, f.k1, (Z * Z) * f.k2)) - f.k3;
    if (f.half_space) return Y;
    return fmaxf(fmaxf(fabsf(X) - f.k0, fabsf(Y) - f.k1), fabsf(Z) - f.k2);
}
// the answer for a value the box's bound does not decide: the point's own bound (a few times tighter), then FP64
static __device__ __noinline__ bool fast_exact(const MeshK& m, const SolidK& k, const SolidPlan& pl,
                                               const sdfibm_solid_state& st, int I, int J, int K, int centre,
                                               unsigned& rechecks) {
    const float half = centre ? 0.5f : 0.f;
    TileFrame tf;
    tf.bx = pl.base32[0]; tf.by = pl.base32[1]; tf.bz = pl.base32[2];
    tf.babs = fabsf(tf.bx) + fabsf(tf.by) + fabsf(tf.bz);
    tf.e64 = pl.e64;
    unsigned long long n = 0;
    const int in = classify_point(k.shape, pl.M, tf, ((float)(I - pl.lo[0]) + half) * m.h32[0],
                                  ((float)(J - pl.lo[1]) + half) * m.h32[1], ((float)(K - pl.lo[2]) + half) * m.h32[2], m, I, J,
                                  K, centre, state_pos(st), state_quat(st), &n);
    rechecks += (unsigned)n;
    return in != 0;
}

// vertex distance for REF-GEO of a 2-D shape (see classify_any) at bbox vertex (da, db, dc)
static __device__ __forceinline__ float flat_phi(const MeshK& m, const SolidK& k, const SolidPlan& pl, const sdfibm_solid_state& st,
                                                 int da, int db, int dc) {
    const ShapeK& sh = k.shape;
    bool exact = sh.type == SDFIBM_SHAPE_PLANE;  // unfiltered, FP64
    float ph = 0.f;
    if (!exact) {
        const double* L = pl.lmap;
        const double a = da, b = db, c = dc;
        const D3 plc{L[0] + a * L[3] + b * L[6] + c * L[9], L[1] + a * L[4] + b * L[7] + c * L[10],
                     L[2] + a * L[5] + b * L[8] + c * L[11]};
        ph = filter_mixed(sh, sdf_mixed(sh, plc), &exact);
    }
    if (exact) ph = exact_phi_point(sh, m, (int64_t)pl.lo[0] + da, (int64_t)pl.lo[1] + db, (int64_t)pl.lo[2] + dc,
                                    state_pos(st), state_quat(st));
    return ph;
}

// FLAT: tiles of 8 x 8 x 2 cells, the vertex answers the same on every layer; else 4 x 4 x 4.  Lanes: vertex (lane % V,
// lane / V) of a layer (flat: of three rows), cells lane, lane + 32, ...
template <bool FLAT, int METHOD>
__device__ __forceinline__ void classify_fast(const ClassifyArgs& A, const int2 ch, unsigned& rechecks,
                                              unsigned& valid_cells) {
    constexpr int TX = FLAT ? 8 : 4, TY = TX, TZ = FLAT ? 2 : 4;
    constexpr int V = TX + 1, NPASS = FLAT ? 4 : 2, NL = FLAT ? 3 : 5;  // passes over the cells, ballots of vertices
    constexpr int NVERT = METHOD == SDFIBM_FRACTION_REFGEO && FLAT ? V * V : 1;
    __shared__ float s_phi[CLS_WARPS][NVERT];
    __shared__ uint8_t s_list[CLS_WARPS][NVERT];
    const unsigned FULL = 0xffffffffu;
    const MeshK& m = A.m;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const unsigned below = (1u << lane) - 1u;
    const int s = ch.x;
    const SolidK& k = A.sk[s];
    const SolidPlan& pl = A.plan[s];
    if (pl.err) return;
    const sdfibm_solid_state& st = A.st[s];
    const FastFrame f = fast_frame(m, k, pl, FLAT);
    const int e0 = k.ext[0], e1 = k.ext[1], e2 = k.ext[2], lo0 = pl.lo[0], lo1 = pl.lo[1], lo2 = pl.lo[2];
    const int nt0 = k.ntile[0], nt01 = k.ntile[0] * k.ntile[1];
    const int t_end = min(ch.y + (k.infinite ? A.wall_tiles : A.finite_tiles), nt01 * k.ntile[2]);
    uint8_t* out = A.cls + k.scratch_off;
    // LEARNED, a solid under rho_min cells: listed from the back, for the fallback
    const bool back = METHOD == SDFIBM_FRACTION_LEARNED && pl.radius_cells < A.rho_min;
    // this lane's vertex and cell within a tile
    const int va = lane % V, vb = lane / V;
    const int ca = lane & (TX - 1), cb = (lane / TX) & (TY - 1);  // pass p adds rows (flat) or layers
    const float fva = (float)va;
    for (int t0 = ch.y; t0 < t_end; t0 += 32) {
        // cull 32 tiles, a lane each: 0 nobody reads its class bytes, 1 no inside vertex (zeros), 2 to be looked at
        int tx = 0, ty = 0, tz = 0, state = 0;
        if (t0 + lane < t_end) {
            const int t = t0 + lane;
            tz = t / nt01;
            ty = (t - tz * nt01) / nt0;
            tx = t - tz * nt01 - ty * nt0;
            const int cx = min(TX, e0 - tx * TX), cy = min(TY, e1 - ty * TY), cz = min(TZ, e2 - tz * TZ);
            const int I0 = lo0 + tx * TX, J0 = lo1 + ty * TY, K0 = lo2 + tz * TZ;
            if (!(I0 + cx <= 0 || J0 + cy <= 0 || K0 + cz <= 0 || I0 >= m.nx || J0 >= m.ny || K0 >= m.nz ||
                  I0 + cx < pl.vlo[0] || I0 > pl.vhi[0] || J0 + cy < pl.vlo[1] || J0 > pl.vhi[1] || K0 + cz < pl.vlo[2] ||
                  K0 > pl.vhi[2])) {
                state = 2;
                if (!FLAT) {  // separating axes of the solid's local box (margins of 1e-4, see classify_any)
                    const float hx = 0.5f * (float)cx, hy = 0.5f * (float)cy, hz = 0.5f * (float)cz;
                    const float ux = (float)(tx * TX) + hx, uy = (float)(ty * TY) + hy, uz = (float)(tz * TZ) + hz;
                    const float lc[3] = {f.px + f.sxx * ux + f.syx * uy + f.szx * uz,
                                         f.py + f.sxy * ux + f.syy * uy + f.szy * uz,
                                         f.pz + f.sxz * ux + f.syz * uy + f.szz * uz};
                    const float rad[3] = {fabsf(f.sxx) * hx + fabsf(f.syx) * hy + fabsf(f.szx) * hz,
                                          fabsf(f.sxy) * hx + fabsf(f.syy) * hy + fabsf(f.szy) * hz,
                                          fabsf(f.sxz) * hx + fabsf(f.syz) * hy + fabsf(f.szz) * hz};
#pragma unroll
                    for (int a = 0; a < 3; ++a) {  // com is part of the coordinates here: the box is centred
                        const float gap = fabsf(lc[a]) - pl.lbox_s[a] - rad[a];
                        if (gap > 1e-4f * (fabsf(lc[a]) + pl.lbox_s[a] + rad[a] + fabsf(pl.lbox_c[a])) + 1e-30f) state = 1;
                    }
                }
            }
        }
        unsigned zero = __ballot_sync(FULL, state == 1), act = __ballot_sync(FULL, state == 2);
        auto cell_offset = [&](int x, int y, int z, int p) {  // bbox index of this lane's cell of pass p
            const int b = FLAT ? cb + 4 * (p & 1) : cb, c = FLAT ? p >> 1 : (lane >> 4) + 2 * p;
            return (int64_t)(x * TX + ca) + (int64_t)e0 * ((y * TY + b) + (int64_t)e1 * (z * TZ + c));
        };
        auto in_box = [&](int x, int y, int z, int p) {
            const int b = FLAT ? cb + 4 * (p & 1) : cb, c = FLAT ? p >> 1 : (lane >> 4) + 2 * p;
            return x * TX + ca < e0 && y * TY + b < e1 && z * TZ + c < e2;
        };
        while (zero) {
            const int src = __ffs(zero) - 1;
            zero &= zero - 1;
            const int x = __shfl_sync(FULL, tx, src), y = __shfl_sync(FULL, ty, src), z = __shfl_sync(FULL, tz, src);
#pragma unroll
            for (int p = 0; p < NPASS; ++p)
                if (in_box(x, y, z, p)) out[cell_offset(x, y, z, p)] = 0;
        }
        while (act) {
            const int src = __ffs(act) - 1;
            act &= act - 1;
            const int x = __shfl_sync(FULL, tx, src), y = __shfl_sync(FULL, ty, src), z = __shfl_sync(FULL, tz, src);
            const int I0 = lo0 + x * TX, J0 = lo1 + y * TY, K0 = lo2 + z * TZ;
            const float ux = (float)(x * TX), uy = (float)(y * TY), uz = (float)(z * TZ);
            const float Lx = __fmaf_rn(ux, f.sxx, __fmaf_rn(uy, f.syx, __fmaf_rn(uz, f.szx, f.px)));
            const float Ly = __fmaf_rn(ux, f.sxy, __fmaf_rn(uy, f.syy, __fmaf_rn(uz, f.szy, f.py)));
            const float Lz = __fmaf_rn(ux, f.sxz, __fmaf_rn(uy, f.syz, __fmaf_rn(uz, f.szz, f.pz)));
            // vertices: bit lane of bits[l] = vertex (va, vb) of layer l (flat: of rows 3 l ..) is inside
            unsigned bits[NL];
            if (FLAT) {
#pragma unroll
                for (int l = 0; l < NL; ++l) {
                    const float fb = (float)(vb + 3 * l);
                    const float g = fast_g(f, __fmaf_rn(fva, f.sxx, __fmaf_rn(fb, f.syx, Lx)),
                                           __fmaf_rn(fva, f.sxy, __fmaf_rn(fb, f.syy, Ly)), Lz);
                    bool in = g < -f.Eg;
                    if (lane < 27 && !in && !(g > f.Eg))
                        in = fast_exact(m, k, pl, st, I0 + va, J0 + vb + 3 * l, K0, 0, rechecks);
                    bits[l] = __ballot_sync(FULL, in) & 0x7ffffffu;
                }
            } else {
                const float fb = (float)vb;
                const float wx = __fmaf_rn(fva, f.sxx, __fmaf_rn(fb, f.syx, Lx)),
                            wy = __fmaf_rn(fva, f.sxy, __fmaf_rn(fb, f.syy, Ly)),
                            wz = __fmaf_rn(fva, f.sxz, __fmaf_rn(fb, f.syz, Lz));
                float B2 = 0.f, C0 = 0.f;
                if (f.quadric) {
                    const float kx = f.k0 * wx, ky = f.k1 * wy, kz = f.k2 * wz;
                    B2 = 2.f * __fmaf_rn(kx, f.szx, __fmaf_rn(ky, f.szy, kz * f.szz));
                    C0 = __fmaf_rn(kx, wx, __fmaf_rn(ky, wy, kz * wz)) - f.k3;
                }
#pragma unroll
                for (int l = 0; l < NL; ++l) {
                    const float c = (float)l;
                    float g;
                    if (f.quadric) g = __fmaf_rn(__fmaf_rn(f.A2, c, B2), c, C0);
                    else g = fast_g(f, __fmaf_rn(c, f.szx, wx), __fmaf_rn(c, f.szy, wy), __fmaf_rn(c, f.szz, wz));
                    bool in = g < -f.Eg;
                    if (lane < 25 && !in && !(g > f.Eg))
                        in = fast_exact(m, k, pl, st, I0 + va, J0 + vb, K0 + l, 0, rechecks);
                    bits[l] = __ballot_sync(FULL, in) & 0x1ffffffu;
                }
            }
            // cells: all and any of the eight vertices, this lane's cells of each pass
            unsigned all_p = 0, any_p = 0;  // bit p: pass p
            if (FLAT) {
                const int r = lane < 9 ? lane : 0;
                const unsigned row = ((r < 3 ? bits[0] : (r < 6 ? bits[1] : bits[2])) >> (9 * (r % 3))) & 0x1ffu;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const unsigned r0 = __shfl_sync(FULL, row, cb + 4 * h) >> ca, r1 = __shfl_sync(FULL, row, cb + 4 * h + 1) >> ca;
                    const unsigned al = r0 & (r0 >> 1) & r1 & (r1 >> 1) & 1u, an = (r0 | (r0 >> 1) | r1 | (r1 >> 1)) & 1u;
                    all_p |= al * (5u << h);  // passes h and h + 2 (the second layer)
                    any_p |= an * (5u << h);
                }
            } else {
                const int pos = ca + 5 * cb;
                unsigned al0 = bits[0] & (bits[0] >> 1), an0 = bits[0] | (bits[0] >> 1);
                al0 &= al0 >> 5;
                an0 |= an0 >> 5;
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    unsigned al1 = bits[c + 1] & (bits[c + 1] >> 1), an1 = bits[c + 1] | (bits[c + 1] >> 1);
                    al1 &= al1 >> 5;
                    an1 |= an1 >> 5;
                    const unsigned al = al0 & al1, an = an0 | an1;
                    if ((lane >> 4) == (c & 1)) {
                        all_p |= ((al >> pos) & 1u) << (c >> 1);
                        any_p |= ((an >> pos) & 1u) << (c >> 1);
                    }
                    al0 = al1;
                    an0 = an1;
                }
            }
            unsigned cut_b[NPASS];
            int ncut = 0;
            uint8_t cls[NPASS];
#pragma unroll
            for (int p = 0; p < NPASS; ++p) {
                const int b = FLAT ? cb + 4 * (p & 1) : cb, c = FLAT ? p >> 1 : (lane >> 4) + 2 * p;
                const bool box = in_box(x, y, z, p);
                const bool valid = box && (unsigned)(I0 + ca) < (unsigned)m.nx && (unsigned)(J0 + b) < (unsigned)m.ny &&
                                   (unsigned)(K0 + c) < (unsigned)m.nz;
                valid_cells += valid;
                const bool al = (all_p >> p) & 1u, cut = valid && ((any_p >> p) & 1u) && !al;
                cls[p] = valid && al ? 1 : 0;
                cut_b[p] = __ballot_sync(FULL, cut);
                if (cut_b[p]) {
                    if (cut) {
                        const float fa = (float)ca + 0.5f, fb = (float)b + 0.5f, fc = (float)c + 0.5f;
                        const float g = fast_g(f, __fmaf_rn(fa, f.sxx, __fmaf_rn(fb, f.syx, __fmaf_rn(fc, f.szx, Lx))),
                                               __fmaf_rn(fa, f.sxy, __fmaf_rn(fb, f.syy, __fmaf_rn(fc, f.szy, Ly))),
                                               __fmaf_rn(fa, f.sxz, __fmaf_rn(fb, f.syz, __fmaf_rn(fc, f.szz, Lz))));
                        bool in = g < -f.Eg;
                        if (!in && !(g > f.Eg)) in = fast_exact(m, k, pl, st, I0 + ca, J0 + b, K0 + c, 1, rechecks);
                        cls[p] = in ? 2 : 3;
                    }
                    ncut += __popc(cut_b[p]);
                }
                if (box) out[cell_offset(x, y, z, p)] = cls[p];
            }
            if (METHOD < 0 || ncut == 0) continue;
            if (METHOD == SDFIBM_FRACTION_REFGEO && FLAT) {
                // Solid::phi once per vertex next to a cut cell, the needed vertices compacted: rows of cut cells (any
                // layer, any pass), widened to their vertices.  (In 3-D refgeo_cells_kernel computes them.)
                uint8_t* list = s_list[w];
                int n = 0;
                unsigned need_row = 0;  // lane r < 9: vertex row r
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const unsigned c2 = cut_b[h] | cut_b[(h + 2) % NPASS];
#pragma unroll
                    for (int r = 0; r < 4; ++r) {
                        const unsigned row = (c2 >> (8 * r)) & 0xffu, wide = row | (row << 1);
                        if (lane == 4 * h + r || lane == 4 * h + r + 1) need_row |= wide;
                    }
                }
#pragma unroll
                for (int l = 0; l < NL; ++l) {
                    const unsigned row = __shfl_sync(FULL, need_row, min(vb + 3 * l, 8));
                    const bool need = lane < 27 && ((row >> va) & 1u);
                    const unsigned bal = __ballot_sync(FULL, need);
                    if (need) list[n + __popc(bal & below)] = (uint8_t)(lane + 27 * l);
                    n += __popc(bal);
                }
                __syncwarp();
                for (int u = lane; u < n; u += 32) {
                    const int v = list[u];
                    s_phi[w][v] = flat_phi(m, k, pl, st, x * TX + v % V, y * TY + v / V, z * TZ);
                }
                __syncwarp();
            }
            // the cut cells listed for the fraction kernels
            int base = 0;
            if (lane == 0) base = atomicAdd(back ? &A.cnt->n_small : &A.cnt->n_feat, ncut);
            base = __shfl_sync(FULL, base, 0);
#pragma unroll
            for (int p = 0; p < NPASS; ++p) {
                if ((cut_b[p] >> lane) & 1u) {
                    const int64_t at = (int64_t)base + __popc(cut_b[p] & below);
                    const int64_t slot = back ? A.feat_cap - 1 - at : at;
                    if (slot >= 0 && slot < A.feat_cap) {
                        if (METHOD == SDFIBM_FRACTION_REFGEO && FLAT) {  // the layers' distances are the same
                            const int v0 = ca + V * (cb + 4 * (p & 1));
                            const int vo[4] = {0, 1, V, V + 1};
#pragma unroll
                            for (int q = 0; q < 8; ++q) A.rg_phi[q * A.feat_cap + slot] = s_phi[w][v0 + vo[q & 3]];
                        }
                        A.fref_solid[slot] = s;
                        A.fref_index[slot] = k.scratch_off + cell_offset(x, y, z, p);
                    } else {
                        set_error(A.cnt, DERR_CAPACITY);
                    }
                }
                base += __popc(cut_b[p]);
            }
            __syncwarp();
        }
    }
}

// The shapes classify_fast takes.  Tilted 2-D shapes, half spaces in 3-D and the tailed circles go to classify_any, and so do 2-D
// shapes on meshes of more than two layers.
template <bool FLAT>
__device__ __forceinline__ bool fast_shape(const SolidK& k, const sdfibm_solid_state& st) {
    const int t = k.shape.type;
    if (FLAT)
        return (t == SDFIBM_SHAPE_CIRCLE || t == SDFIBM_SHAPE_ELLIPSE || t == SDFIBM_SHAPE_RECTANGLE ||
                t == SDFIBM_SHAPE_PLANE) &&
               st.quat[1] == 0.0 && st.quat[2] == 0.0;
    return t == SDFIBM_SHAPE_SPHERE || t == SDFIBM_SHAPE_ELLIPSOID || t == SDFIBM_SHAPE_BOX;
}

// FAST: the chunks classify_fast takes; else the others.  Chunks are taken one at a time with an atomic; on flat meshes the
// other kernel first looks at the chunks before fast_chunks, nearly all of which are the first kernel's: 32 together, which
// lie a grid of warps apart, since those of a tilted solid are neighbours (32 neighbours a warp, all shapes: one tailed circle of
// 81 items 165 us, now 22; 1500 of them 893, now 143; 300 3-D shapes on two layers 248, now 31; GB300).
template <bool FLAT, int METHOD, bool FAST>
__device__ __forceinline__ void classify_body(const ClassifyArgs& A) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    unsigned long long rechecks = 0, valid_cells = 0;
    unsigned rechecks32 = 0, valid32 = 0;
    constexpr bool LOOK = FLAT && !FAST;
    const int nw = gridDim.x * CLS_WARPS;
    int64_t look = blockIdx.x * CLS_WARPS + (threadIdx.x >> 5);
    int2 seen = make_int2(-1, 0);  // chunk look + lane * nw
    unsigned mine = 0;             // of those, the ones to be done here
    for (;;) {
        int2 ch;
        if (LOOK && mine) {
            const int src = __ffs(mine) - 1;
            mine &= mine - 1;
            ch = make_int2(__shfl_sync(FULL, seen.x, src), __shfl_sync(FULL, seen.y, src));
        } else if (LOOK && look < A.fast_chunks) {
            const int64_t at = look + lane * (int64_t)nw;
            look += 32 * (int64_t)nw;
            seen = at < A.fast_chunks ? A.chunks[at] : make_int2(-1, 0);
            mine = __ballot_sync(FULL, seen.x >= 0 && !fast_shape<FLAT>(A.sk[max(seen.x, 0)], A.st[max(seen.x, 0)]));
            continue;
        } else if (LOOK && A.fast_chunks >= A.total_chunks) {
            break;  // nothing in the queue: no warp asks
        } else {
            int chunk = 0;
            if (lane == 0) chunk = FAST ? atomicAdd(&A.cnt->classify_next, 1) : atomicAdd(&A.cnt->classify_any_next, 1) + A.fast_chunks;
            chunk = __shfl_sync(FULL, chunk, 0);
            if (chunk >= (FAST ? A.fast_chunks : A.total_chunks)) break;
            ch = A.chunks[chunk];
            if (FAST && !fast_shape<FLAT>(A.sk[ch.x], A.st[ch.x])) continue;
        }
        if (FAST) classify_fast<FLAT, METHOD>(A, ch, rechecks32, valid32);
        else classify_any<FLAT ? 8 : 4, FLAT ? 8 : 4, FLAT ? 2 : 4, METHOD>(A, ch, rechecks, valid_cells);
    }
    rechecks += rechecks32;
    valid_cells += valid32;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        rechecks += __shfl_xor_sync(FULL, rechecks, o);
        valid_cells += __shfl_xor_sync(FULL, valid_cells, o);
    }
    if (lane == 0) {
        if (rechecks) atomicAdd(&A.cnt->exact_rechecks, rechecks);
        if (valid_cells) atomicAdd(&A.cnt->bbox_cells, valid_cells);
    }
}

// FP32 frame of the listed cell idx of a solid, built as the classify pass builds a tile's: the solid's rounded base plus a
// whole number of cells; the cell's place in the bbox
__device__ __forceinline__ int3 cell_frame(const FallbackArgs& A, const SolidK& k, const SolidPlan& pl, int64_t idx, TileFrame& tf) {
    const uint32_t local = (uint32_t)(idx - k.scratch_off);  // < bbox cells of one solid (< 2^31)
    const int row = (int)fdiv(local, k.div_e0), lc = (int)fdiv(local, k.div_e01);
    const int la = (int)local - row * k.ext[0], lb = row - lc * k.ext[1];
    const float sbx = pl.base32[0], sby = pl.base32[1], sbz = pl.base32[2];
    const float ofx = (float)la * A.m.h32[0], ofy = (float)lb * A.m.h32[1], ofz = (float)lc * A.m.h32[2];
    tf.bx = sbx + ofx; tf.by = sby + ofy; tf.bz = sbz + ofz;
    tf.babs = fabsf(sbx) + fabsf(sby) + fabsf(sbz) + 2.f * (fabsf(ofx) + fabsf(ofy) + fabsf(ofz)) +
              fabsf(tf.bx) + fabsf(tf.by) + fabsf(tf.bz);
    tf.e64 = pl.e64;
    return make_int3(la, lb, lc);
}
// SUBSAMPLE count of one listed cell (bbox index idx of solid s) by a warp
template <bool DEFER_ONLY>
__device__ __forceinline__ int count_listed_cell(const FallbackArgs& A, int s, int64_t idx, unsigned long long* rechecks,
                                                 const Defer* df) {
    const SolidK& k = A.sk[s];
    const SolidPlan& pl = A.plan[s];
    TileFrame tf;
    const int3 at = cell_frame(A, k, pl, idx, tf);
    float M[9];
#pragma unroll
    for (int r = 0; r < 9; ++r) M[r] = pl.M[r];
    if (DEFER_ONLY) {  // inlined; the FP64 state is not needed
        return subsample_warp_body<true>(A.m, k.shape, M, tf, 0, 0, 0, D3{0, 0, 0}, Q4{1, D3{0, 0, 0}}, 0, 0, 0, A.n,
                                         rechecks, df);
    }
    const Q4 q = state_quat(A.st[s]);
    const D3 x = state_pos(A.st[s]);
    return subsample_warp(A.m, k.shape, M, tf, 0, 0, 0, x, q, pl.lo[0] + at.x, pl.lo[1] + at.y, pl.lo[2] + at.z, A.n,
                          rechecks, df);
}

// The same of 32 listed cells at once, a lane each: all lanes do the same column of their own cells, so nothing of a cell's
// frame is computed 32 times and no lane is without a column.  Columns left to the walk are listed and their samples spread
// over the lanes, which take the frame of the sample's cell from its lane.  Lanes with `mine` have cells of kind T.
constexpr int WALK_CAP = 96;
constexpr int SUB_WINDOW = 256;  // cells of a warp sorted by kind
struct ThreadWalk {
    uint32_t list[WALK_CAP];  // lane of the cell | column << 5
    int32_t inside[32];       // walked samples found inside, per lane
    int32_t overflow[32];
};
template <int T>
__device__ __forceinline__ int thread_runs(const FallbackArgs& A, const ShapeK& sh, const SampleFrame& f, float Egh, bool mine,
                                           int s, int64_t idx, ThreadWalk& tw, unsigned long long* rechecks) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, n = A.n;
    const float inv2n = __frcp_rn((float)(2 * n)), invn = __frcp_rn((float)n);
    const RunFrame rf = run_frame<T>(f, Egh, n, invn);
    float cnt = 0.f;
    int nwalk = 0;
    auto flush = [&]() {
        __syncwarp();
        for (int e0 = 0; e0 < nwalk * n; e0 += 32) {
            const int e = min(e0 + lane, nwalk * n - 1), w = __float2int_rz(((float)e + 0.5f) * invn), c3 = e - w * n;
            const uint32_t it = tw.list[w];
            const int from = (int)(it & 31u), col = (int)(it >> 5), ib = __float2int_rz(((float)col + 0.5f) * invn), ia = col - ib * n;
            SampleFrame g;
            auto of = [&](float v) { return __shfl_sync(FULL, v, from); };
            g.px = of(f.px); g.py = of(f.py); g.pz = of(f.pz);
            g.sxx = of(f.sxx); g.sxy = of(f.sxy); g.sxz = of(f.sxz);
            g.syx = of(f.syx); g.syy = of(f.syy); g.syz = of(f.syz);
            g.szx = of(f.szx); g.szy = of(f.szy); g.szz = of(f.szz);
            g.k0 = of(f.k0); g.k1 = of(f.k1); g.k2 = of(f.k2); g.k3 = of(f.k3);
            g.Eg = of(f.Eg);
            const int so = __shfl_sync(FULL, s, from);
            const int64_t io = __shfl_sync(FULL, idx, from);
            const float ta = (float)(2 * ia + 1) * inv2n, tb = (float)(2 * ib + 1) * inv2n, tc = (float)(2 * c3 + 1) * inv2n;
            const float bx = __fmaf_rn(tb, g.syx, __fmaf_rn(ta, g.sxx, g.px)), by = __fmaf_rn(tb, g.syy, __fmaf_rn(ta, g.sxy, g.py)),
                        bz = __fmaf_rn(tb, g.syz, __fmaf_rn(ta, g.sxz, g.pz));
            if (e0 + lane < nwalk * n) {
                int r = band(sample_g<T>(g, __fmaf_rn(tc, g.szx, bx), __fmaf_rn(tc, g.szy, by), __fmaf_rn(tc, g.szz, bz)), g.Eg);
                if (r == 2) {
                    ++*rechecks;
                    const Defer df{A.rq, A.rq_cap, &A.cnt->n_recheck, io, so, &tw.overflow[from]};
                    r = undecided_sample<true>(&df, sh, A.m, 0, 0, 0, ia, ib, c3, n, D3{0, 0, 0}, Q4{1, D3{0, 0, 0}});
                }
                if (r) atomicAdd(&tw.inside[from], r);
            }
        }
        nwalk = 0;
        __syncwarp();
    };
    // coordinates of a column's sample 0
    const float qx = __fmaf_rn(f.szx, inv2n, f.px), qy = __fmaf_rn(f.szy, inv2n, f.py), qz = __fmaf_rn(f.szz, inv2n, f.pz);
    float oa = 1.f;  // 2 ia + 1, exact
#pragma unroll 1
    for (int ia = 0; ia < n; ++ia, oa += 2.f) {
        const float ta = oa * inv2n;
        const float ux = __fmaf_rn(ta, f.sxx, qx), uy = __fmaf_rn(ta, f.sxy, qy), uz = __fmaf_rn(ta, f.sxz, qz);
        float ob = 1.f;
        for (int ib0 = 0; ib0 < n; ib0 += 32) {
            uint32_t walk = 0;  // columns ib0 + bit of this row
            const int m = min(32, n - ib0);
#pragma unroll 2
            for (int b = 0; b < m; ++b, ob += 2.f) {
                const float tb = ob * inv2n;
                const float res = run_column<T>(f, rf, __fmaf_rn(tb, f.syx, ux), __fmaf_rn(tb, f.syy, uy), __fmaf_rn(tb, f.syz, uz));
                if (res < 0.f) walk |= 1u << b;
                cnt += fmaxf(res, 0.f);
            }
            if (!mine) walk = 0;
            while (__any_sync(FULL, walk != 0)) {
                const unsigned mask = __ballot_sync(FULL, walk != 0);
                if (walk) {
                    tw.list[nwalk + __popc(mask & ((1u << lane) - 1u))] = (uint32_t)lane | (uint32_t)(ia + (ib0 + __ffs(walk) - 1) * n) << 5;
                    walk &= walk - 1;
                }
                nwalk += __popc(mask);
                if (nwalk > WALK_CAP - 32) flush();
            }
        }
    }
    flush();
    return (int)cnt;
}

// SUBSAMPLE of listed cells: the cut cells of the classify pass (SUBSAMPLE, fb_list == nullptr)
// or the cells outside the network's band (LEARNED fallback).  Undecided points always go to the recheck list (this
// kernel holds no FP64 path, which keeps its register count and so its occupancy); a cell some of whose points found
// the list full is listed for recount_kernel.
// 3-D convex shapes on lattices of 5 samples and more are done a lane per cell from A.lane_min cells on, everything else a
// warp per cell.  Bound by issue.  Measured (GB300): 1.32 M cells of 10^3 samples, 1.32 -> 0.33 ms (a warp per cell with four
// evaluations of q to verify each column's run: 984 instructions a cell, now 226); 1.2 M cells of 16^3, 2.11 -> 0.75 ms.  A warp
// per cell took 32 cells each however few there were: 1092 cells 98 -> 12 us.
__global__ void __launch_bounds__(256, 3) subsample_cells_kernel(FallbackArgs A) {
    __shared__ int32_t s_overflow[8];
    const int lane = threadIdx.x & 31;
    int32_t* overflow = s_overflow + ((threadIdx.x >> 5) & 7);
    // LEARNED: the band's rejects (fb_list), then the cells listed from the back; a front and a back that overlap
    // (more cut cells than the list holds) are a capacity error
    const int64_t n_fb = A.fb_list ? min((int64_t)A.cnt->n_fb, A.cap) : 0;
    const int64_t n_back = A.fb_list ? (int64_t)A.cnt->n_small : 0;
    if (A.fb_list && (int64_t)A.cnt->n_feat + n_back > A.cap && threadIdx.x == 0 && blockIdx.x == 0)
        set_error(A.cnt, DERR_CAPACITY);
    const int64_t nfb = A.fb_list ? min(n_fb + n_back, A.cap) : min((int64_t)A.cnt->n_feat, A.cap);
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    unsigned long long rechecks = 0;
    __shared__ ThreadWalk tw[8];
    __shared__ uint8_t s_order[8][SUB_WINDOW];
    const bool lanes = nfb >= A.lane_min && A.n >= 5 && !A.m.twod;
    if (lane == 0) *overflow = 0;
    __syncwarp();
    auto entry = [&](int64_t q, int& s, int64_t& idx) {  // q-th listed cell
        const int64_t slot = !A.fb_list ? q : (q < n_fb ? (int64_t)A.fb_list[q] : A.cap - 1 - (q - n_fb));
        s = A.fref_solid[slot];
        idx = A.fref_index[slot];
    };
    // each warp takes consecutive list entries, as many as give every warp some: a lane per cell, up to SUB_WINDOW of them,
    // sorted by kind so that the lanes of a batch are alike, else up to 32, one after the other
    const int64_t share = (nfb + warps - 1) / warps;
    const int window = lanes ? (int)min((int64_t)SUB_WINDOW, (share + 31) & ~(int64_t)31) : (int)min((int64_t)32, share);
    for (int64_t base = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * window; base < nfb; base += warps * window) {
        const int count = (int)min((int64_t)window, nfb - base);
        int rest = count, first = 0;  // entries left to the warp loop: order[first ..] (lanes), else all
        uint8_t* order = s_order[(threadIdx.x >> 5) & 7];
        if (lanes) {
            // order: quadrics from the front, then boxes, then the others
            int n_kind[3] = {0, 0, 0};
            unsigned kinds = 0;  // two bits a batch
            for (int t = 0; t < count; t += 32) {
                int kind = 3, s = 0;
                int64_t idx = 0;
                if (t + lane < count) {
                    entry(base + t + lane, s, idx);
                    const ShapeK& sh = A.sk[s].shape;
                    kind = sh.prism ? 2 : (sh.type == SDFIBM_SHAPE_SPHERE || sh.type == SDFIBM_SHAPE_ELLIPSOID ? 0
                                                                      : (sh.type == SDFIBM_SHAPE_BOX ? 1 : 2));
                }
                kinds |= (unsigned)kind << (t >> 4);
#pragma unroll
                for (int v = 0; v < 3; ++v) n_kind[v] += __popc(__ballot_sync(0xffffffffu, kind == v));
            }
            int at[3] = {0, n_kind[0], n_kind[0] + n_kind[1]};
            for (int t = 0; t < count; t += 32) {
                const int kind = (kinds >> (t >> 4)) & 3;
#pragma unroll
                for (int v = 0; v < 3; ++v) {
                    const unsigned m = __ballot_sync(0xffffffffu, kind == v);
                    if (kind == v) order[at[v] + __popc(m & ((1u << lane) - 1u))] = (uint8_t)(t + lane);
                    at[v] += __popc(m);
                }
            }
            __syncwarp();
            ThreadWalk& w = tw[(threadIdx.x >> 5) & 7];
            first = n_kind[0] + n_kind[1];
            rest = count - first;
            for (int v = 0; v < 2; ++v) {
                const int lo = v == 0 ? 0 : n_kind[0], hi = lo + n_kind[v];
                for (int e0 = lo; e0 < hi; e0 += 32) {
                    const bool mine = e0 + lane < hi;
                    int s = 0;
                    int64_t idx = 0;
                    if (mine) entry(base + order[e0 + lane], s, idx);
                    const SolidK& k = A.sk[s];
                    SampleFrame f{};
                    float Egh = 0.f;
                    if (mine) {
                        TileFrame tf;
                        cell_frame(A, k, A.plan[s], idx, tf);
                        float Ep;
                        sample_frame(A.m, k.shape, A.plan[s].M, tf, 0, 0, 0, f, Ep, Egh);
                    }
                    w.inside[lane] = 0;
                    w.overflow[lane] = 0;
                    const int cnt = v == 0 ? thread_runs<SS_QUADRIC>(A, k.shape, f, Egh, mine, s, idx, w, &rechecks)
                                           : thread_runs<SS_BOX>(A, k.shape, f, Egh, mine, s, idx, w, &rechecks);
                    if (mine) {
                        A.alpha[idx] = -1.f - (float)(cnt + w.inside[lane]);
                        if (w.overflow[lane]) {
                            const int slot = atomicAdd(&A.cnt->n_ovf, 1);
                            if (slot < A.ovf_cap) A.ovf[slot] = Recheck{idx, s, 0u};
                            else set_error(A.cnt, DERR_CAPACITY);
                        }
                    }
                    __syncwarp();
                }
            }
        }
        for (int t0 = 0; t0 < rest; t0 += 32) {
            int s_l = 0;
            int64_t idx_l = 0;
            if (t0 + lane < rest) entry(base + (lanes ? order[first + t0 + lane] : t0 + lane), s_l, idx_l);
            for (int t = 0; t < min(32, rest - t0); ++t) {
                const int s = __shfl_sync(0xffffffffu, s_l, t);
                const int64_t idx = __shfl_sync(0xffffffffu, idx_l, t);
                const Defer df{A.rq, A.rq_cap, &A.cnt->n_recheck, idx, s, overflow};
                const int cnt = count_listed_cell<true>(A, s, idx, &rechecks, &df);
                __syncwarp();
                if (lane == 0) {
                    A.alpha[idx] = -1.f - (float)cnt;
                    if (*(volatile int32_t*)overflow) {
                        *overflow = 0;
                        const int slot = atomicAdd(&A.cnt->n_ovf, 1);
                        if (slot < A.ovf_cap) A.ovf[slot] = Recheck{idx, s, 0u};
                        else set_error(A.cnt, DERR_CAPACITY);
                    }
                }
                __syncwarp();
            }
        }
        __syncwarp();
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rechecks += __shfl_xor_sync(0xffffffffu, rechecks, o);
    if (lane == 0 && rechecks) atomicAdd(&A.cnt->exact_rechecks, rechecks);
}

// Cells of the fallback whose undecided points overflowed the recheck list: counted again from scratch, undecided
// points in FP64 in place, after recheck_kernel (whose updates of these cells the new count replaces).
__global__ void __launch_bounds__(256) recount_kernel(FallbackArgs A) {
    const int lane = threadIdx.x & 31;
    const int64_t n = min((int64_t)A.cnt->n_ovf, A.ovf_cap);
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    unsigned long long rechecks = 0;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < n; w += warps) {
        const Recheck r = A.ovf[w];
        const int cnt = count_listed_cell<false>(A, r.solid, r.idx, &rechecks, nullptr);
        if (lane == 0) A.alpha[r.idx] = -1.f - (float)cnt;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) rechecks += __shfl_xor_sync(0xffffffffu, rechecks, o);
    if (lane == 0 && rechecks) atomicAdd(&A.cnt->exact_rechecks, rechecks);
}

// REF-GEO fraction of the listed cut cells, one thread per cell (GeometricTools::calcCellVolume on the cell's vertex
// distances, see refgeo32): the tile pass lists the cells, so every lane here has a cell.  Cells at the mesh boundary, whose
// face lists differ, take refgeo32; the others refgeo_inner.  In 3-D (!FLAT) the distances of the shapes of
// classify_fast are computed here, eight a cell, rather than once a vertex in the classify pass: that pass then fits its
// instruction cache and this one runs beside the connected sets.  Bound by issue.  Measured (GB300), with the classify pass:
// 512^3 and 16 384 solids 0.92 + 0.54 ms with table-driven fractions, 0.92 + 0.23 unrolled, 0.44 + 0.77 with the distances here
// (the interact 2.09 -> 2.05); 256^3 and 4096 0.23 + 0.12, 0.23 + 0.065, 0.12 + 0.18 (0.65 -> 0.63); one cylinder 18 -> 8 us,
// where the chain of one cell counts.
template <bool FLAT>
__global__ void __launch_bounds__(256, FLAT ? 4 : 3) refgeo_cells_kernel(MeshK m, const SolidK* __restrict__ sk,
                                                           const sdfibm_solid_state* __restrict__ st,
                                                           const SolidPlan* __restrict__ plan,
                                                           const int32_t* __restrict__ fref_solid,
                                                           const int64_t* __restrict__ fref_index,
                                                           const float* __restrict__ rg_phi, int64_t cap,
                                                           const Counters* cnt, float* __restrict__ alpha) {
    __shared__ float s_ph[FLAT ? 1 : 8][256];
    const int64_t n = min((int64_t)cnt->n_feat, cap);
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const int s = fref_solid[e];
        const int64_t idx = fref_index[e];
        const SolidK& k = sk[s];
        const SolidPlan& pl = plan[s];
        const uint32_t local = (uint32_t)(idx - k.scratch_off);
        const int row = (int)fdiv(local, k.div_e0), lc = (int)fdiv(local, k.div_e01);
        const int la = (int)local - row * k.ext[0], lb = row - lc * k.ext[1];
        float ph[8];
        const int type = k.shape.type;
        if (!FLAT && (type == SDFIBM_SHAPE_SPHERE || type == SDFIBM_SHAPE_ELLIPSOID || type == SDFIBM_SHAPE_BOX)) {
            // the shapes of classify_fast: the corners' local points as ff_local computes them, its sums shared (x, then y,
            // then z)
            auto step = [&](const FF (&from)[3], const float (&mf)[3], FF (&to)[3], float (&mt)[3], int axis, float n) {
#pragma unroll
                for (int r = 0; r < 3; ++r) {
                    const int i = 3 + 3 * axis + r;
                    to[r] = ff_add(from[r], ff_scale(FF{pl.lmap_hi[i], pl.lmap_lo[i]}, n));
                    mt[r] = mf[r] + fabsf(n * pl.lmap_hi[i]);
                }
            };
            FF P[3];
            float mp[3];
#pragma unroll
            for (int r = 0; r < 3; ++r) {
                P[r] = FF{pl.lmap_hi[r], pl.lmap_lo[r]};
                mp[r] = fabsf(pl.lmap_hi[r]);
            }
#pragma unroll 1
            for (int a = 0; a < 2; ++a) {
                FF X[3];
                float mx[3];
                step(P, mp, X, mx, 0, (float)(la + a));
#pragma unroll 1
                for (int b = 0; b < 2; ++b) {
                    FF Y[3];
                    float my[3];
                    step(X, mx, Y, my, 1, (float)(lb + b));
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        FF Z[3];
                        float mz[3], err, den;
                        step(Y, my, Z, mz, 2, (float)(lc + c));
                        float p = sdf_ff_at(k.shape, Z, fmaxf(fmaxf(mz[0], mz[1]), mz[2]), err, den);
                        if (!ff_filter(p, err, den))
                            p = exact_phi_point(k.shape, m, (int64_t)pl.lo[0] + la + a, (int64_t)pl.lo[1] + lb + b,
                                                (int64_t)pl.lo[2] + lc + c, state_pos(st[s]), state_quat(st[s]));
                        s_ph[FLAT ? 0 : a + 2 * b + 4 * c][threadIdx.x] = p;
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) ph[q] = s_ph[FLAT ? 0 : q][threadIdx.x];
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) ph[q] = rg_phi[q * cap + e];
        }
        const int I = pl.lo[0] + la, J = pl.lo[1] + lb, K = pl.lo[2] + lc;
        float apz = 0.f, apz1 = 0.f;
        if (m.twod) {
            apz = (float)((0.0 - mesh_coord(m, 2, K)) / m.h[2]);
            apz1 = (float)((mesh_coord(m, 2, K + 1) - 0.0) / m.h[2]);
        }
        const bool inner = I > 0 && J > 0 && I + 1 < m.nx && J + 1 < m.ny;
        float a;
        if (inner && K > 0 && K + 1 < m.nz) a = refgeo_inner<false>(m, ph, apz, apz1);
        else if (inner && m.nz == 1) a = refgeo_inner<true>(m, ph, apz, apz1);
        else {
            float pc[8];  // refgeo32 indexes its copy
#pragma unroll
            for (int q = 0; q < 8; ++q) pc[q] = ph[q];
            a = refgeo32(m, pc, I, J, K, apz, apz1);
        }
        alpha[idx] = a;
    }
}

void launch_refgeo_cells(const MeshK& m, const SolidK* sk, const sdfibm_solid_state* st, const SolidPlan* plan,
                         const int32_t* fref_solid, const int64_t* fref_index, const float* rg_phi, int64_t cap, const Counters* cnt,
                         float* alpha, int grid, cudaStream_t stream) {
    if (m.nz <= 2)
        refgeo_cells_kernel<true><<<grid, 256, 0, stream>>>(m, sk, st, plan, fref_solid, fref_index, rg_phi, cap, cnt, alpha);
    else refgeo_cells_kernel<false><<<grid, 256, 0, stream>>>(m, sk, st, plan, fref_solid, fref_index, rg_phi, cap, cnt, alpha);
}

// The deferred SUBSAMPLE points: one per thread, the reference's FP64 point and inside test, an inside point lowers the
// cell's encoded count (-(1 + count)) by one.
__global__ void __launch_bounds__(256) recheck_kernel(MeshK m, const SolidK* __restrict__ sk,
                                                      const sdfibm_solid_state* __restrict__ st,
                                                      const SolidPlan* __restrict__ plan,
                                                      const Recheck* __restrict__ rq, int64_t cap, Counters* cnt,
                                                      float* __restrict__ alpha) {
    const int64_t n = min((int64_t)cnt->n_recheck, cap);
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
        const Recheck r = rq[e];
        const SolidK& k = sk[r.solid];
        const SolidPlan& pl = plan[r.solid];
        const int local = (int)(r.idx - k.scratch_off);
        const int la = local % k.ext[0], lb = (local / k.ext[0]) % k.ext[1], lc = local / (k.ext[0] * k.ext[1]);
        const int a = r.sample & 255, b = (r.sample >> 8) & 255, c = (r.sample >> 16) & 255, ns = r.sample >> 24;
        const int in = exact_inside_sample(k.shape, m, pl.lo[0] + la, pl.lo[1] + lb, pl.lo[2] + lc, a, b, c, ns,
                                           state_pos(st[r.solid]), state_quat(st[r.solid]));
        if (in) atomicAdd(alpha + r.idx, -1.f);
    }
}

// 3-D meshes: 4x4x4-cell tiles; one- and two-layer meshes: 8x8x2.  One instantiation per fraction method (-1: classification
// only), so each kernel carries only its own path, and one per set of shapes.  CTAs per SM: as many as their registers allow
// without spilling much.
template <bool FLAT, int METHOD>
__global__ void __launch_bounds__(CLS_WARPS * 32, METHOD == SDFIBM_FRACTION_REFGEO && FLAT ? 3 : 4) classify_kernel(ClassifyArgs A) {
    classify_body<FLAT, METHOD, true>(A);
}
template <bool FLAT, int METHOD>
__global__ void __launch_bounds__(CLS_WARPS * 32, 2) classify_any_kernel(ClassifyArgs A) {
    classify_body<FLAT, METHOD, false>(A);
}

template <bool FLAT, int METHOD>
static int launch_classify_as(const ClassifyArgs& A, int grid, cudaStream_t st) {
    const bool fast = A.fast_chunks > 0, any = any_chunks(A, FLAT) > 0;
    if (fast) classify_kernel<FLAT, METHOD><<<grid, CLS_WARPS * 32, 0, st>>>(A);
    if (any) classify_any_kernel<FLAT, METHOD><<<A.any_grid, CLS_WARPS * 32, 0, st>>>(A);
    return (int)fast + (int)any;
}
template <bool FLAT>
static int launch_classify_flat(const ClassifyArgs& A, int grid, cudaStream_t st) {
    switch (A.method) {
        case SDFIBM_FRACTION_REFGEO: return launch_classify_as<FLAT, SDFIBM_FRACTION_REFGEO>(A, grid, st);
        case SDFIBM_FRACTION_SUBSAMPLE: return launch_classify_as<FLAT, SDFIBM_FRACTION_SUBSAMPLE>(A, grid, st);
        case SDFIBM_FRACTION_LEARNED: return launch_classify_as<FLAT, SDFIBM_FRACTION_LEARNED>(A, grid, st);
        default: return launch_classify_as<FLAT, -1>(A, grid, st);
    }
}
// host side: the instantiations for a method and a tile shape; the kernels launched
int launch_classify(const ClassifyArgs& A, bool flat, int grid, cudaStream_t st) {
    return flat ? launch_classify_flat<true>(A, grid, st) : launch_classify_flat<false>(A, grid, st);
}

// Shapes whose chunks classify_kernel may take (0) and those it never takes (1): the chunk table holds them in this order.
// On flat meshes the first kind is decided per call by the orientation, and both kernels look at those chunks (any_chunks).
int classify_kind(int shape_type, bool flat) {
    if (flat)
        return shape_type == SDFIBM_SHAPE_CIRCLE || shape_type == SDFIBM_SHAPE_ELLIPSE ||
                       shape_type == SDFIBM_SHAPE_RECTANGLE || shape_type == SDFIBM_SHAPE_PLANE
                   ? 0 : 1;
    return shape_type == SDFIBM_SHAPE_SPHERE || shape_type == SDFIBM_SHAPE_ELLIPSOID || shape_type == SDFIBM_SHAPE_BOX ? 0 : 1;
}

// resident CTAs per SM of the instantiation a launch would use
template <bool FLAT>
static const void* classify_function(int method) {
    switch (method) {
        case SDFIBM_FRACTION_REFGEO: return (const void*)classify_kernel<FLAT, SDFIBM_FRACTION_REFGEO>;
        case SDFIBM_FRACTION_SUBSAMPLE: return (const void*)classify_kernel<FLAT, SDFIBM_FRACTION_SUBSAMPLE>;
        case SDFIBM_FRACTION_LEARNED: return (const void*)classify_kernel<FLAT, SDFIBM_FRACTION_LEARNED>;
        default: return (const void*)classify_kernel<FLAT, -1>;
    }
}
int classify_occupancy(int method, bool flat) {
    int occ = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, flat ? classify_function<true>(method) : classify_function<false>(method),
                                                  CLS_WARPS * 32, 0);
    return occ;
}

}  // namespace sdfibm_dev
