// Device view of an explicit polyMesh (poly.hpp) and the per-call work space of the unstructured coupling path
// (poly.cu), shared with the C ABI (capi.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

#include "kernels.cuh"

namespace sdfibm_dev {

struct PolyK {
    int32_t ncells, npoints, nfaces, twod;
    const double* points;     // [npoints][3]
    const int32_t* face_off;  // face -> points
    const int32_t* face_lab;
    const int32_t* cf_off;    // cell -> faces (owned, then neighbour faces)
    const int32_t* cf;
    const int32_t* cp_off;    // cell -> points, ascending
    const int32_t* cp;
    const int32_t* cc_off;    // cell -> face neighbours
    const int32_t* ccl;
    const double* Cf;         // [nfaces][3] face centres
    const double* Sf;         // [nfaces][3] face area vectors
    const double* Cc;         // [ncells][3] cell centres
    const double* Vc;         // [ncells] cell volumes
    const float4* pt32;       // [npoints][2]: points as FP32 pairs (hi.x, hi.y, hi.z, lo.x), (lo.y, lo.z, -, -)
    const int32_t* cfv_off;   // entry of cf -> its vertices' slots in cfv
    const uint8_t* cfv;       // position of each face vertex in the cell's point list (255: beyond the 255th)
    const float4* cell32;     // [ncells]: centre and a radius that holds the cell's points (FP32, widened)
    const double* mSf;        // [nfaces] |Sf|
    const float* blk;         // [nblocks][12]: boxes of the points and of the centres of POLY_BLOCK consecutive cells
    int32_t nblocks;          //   (lo, hi, lo, hi; widened)
    int32_t uniform_np;       // 1: every cell has the same number of points
};
constexpr int POLY_BLOCK = 128;  // cells per block: four bitmap words
constexpr int POLY_BATCH = 64;   // cells a CTA of poly_couple_kernel takes at a time

// Per-call record of a solid (poly_plan_kernel): FP32 map to the local frame and the region its inside points lie in.
struct PolySolid {
    float M[9];        // |q|^2 R^T
    float xh[3], xl[3];  // solid centre as FP32 pairs
    float mn;          // bound of the row sums of |M|
    float xabs;        // |centre|_1
    float pad;
    double R[9];       // the map in FP64 (distances)
    float c[3], r;     // bounding sphere (2-D shapes: the axis point and the radius), widened
    float axis[3];     // 2-D shapes: direction of the prism
    int32_t kind;      // 0 sphere, 1 prism along z, 2 prism, 3 half space
};

struct PolyWork {
    uint32_t* visited;  // [S][words]: cells the search of each solid has reached; uniform_np: cells with an inside vertex
    int64_t words;
    int32_t* count;     // [S]: touched cells of each solid
    // the breadth-first search
    int32_t* queue;     // [S][ncells]: touched cells of each solid in search order
    int8_t* qtype;      // [S][ncells]: their types (1 ALL_INSIDE, 2 CENTER_INSIDE, 3 CENTER_OUTSIDE)
    int64_t qcap;       // ncells
    double* acc;        // [N][5]: sums over the solids of As, Ts, Fs.x, Fs.y, Fs.z
    int32_t* claim;     // [N]: largest 4 * solid + type over the solids touching the cell (-1: none)
    int32_t* err;       // first device error (DeviceError)
    // meshes whose cells all have the same point count: cells with an inside vertex and their connected sets.  Lists of words
    // of the bitmap, not of cells: 4.8 bytes a solid and cell (the search takes 5.1), where lists of cells, their types and the
    // touched ones beside the forest would take 14
    PolySolid* plan;    // [S]
    int2* items;        // (solid, block) pairs whose boxes meet the solid
    int32_t* nitems;    // their count (left zero by poly_finalize_kernel)
    int32_t* parent;    // [S][ncells]: union-find forest (parent label <= own label) of the cells with an inside vertex
    uint32_t *all_in, *centre_in;  // [S][words]: of those, the cells of type 1 and of type 2 (none: type 3; both: not touched)
    int2* wlist;        // [S][words]: words of visited that hold such cells, and the number of cells before each
    int32_t* wstart;    // [S][batches]: place in wlist of the word that holds cell POLY_BATCH * i of the list
    int64_t batches;
    unsigned long long* wcount;  // [S]: words << 32 | cells of the list
    int32_t* seed;      // [S]: nearest cell
    int32_t* mincand;   // [S]: lowest label of the cells with an inside vertex
};

__global__ void poly_enum_kernel(PolyK m, const SolidK* sk, const sdfibm_solid_state* st, PolyWork w);
__global__ void poly_setup_kernel(PolyK m, float4* pt32, float4* cell32, double* mSf, float* blk);
__global__ void poly_plan_kernel(PolyK m, const SolidK* sk, const sdfibm_solid_state* st, PolyWork w, double* ftacc);
__global__ void poly_classify_kernel(PolyK m, const SolidK* sk, const sdfibm_solid_state* st, PolyWork w, int S);
__global__ void poly_link_kernel(PolyK m, PolyWork w);
__global__ void poly_couple_kernel(PolyK m, const SolidK* sk, const sdfibm_solid_state* st, PolyWork w, const float* U,
                                   double* ftacc, double dtINV, int linked);
__global__ void poly_finalize_kernel(PolyWork w, int32_t N, float* As, float* Fs, float* Ts, int32_t* Ct, int S,
                                     const double* ftacc, double* ft, double rho_f, sdfibm_solid_state* st);
__global__ void poly_fix_kernel(PolyK m, const sdfibm_solid_state* st, int S, const int32_t* Ct, float* U);

}  // namespace sdfibm_dev
