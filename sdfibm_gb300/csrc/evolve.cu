// Rigid-body side of the time step: the GB300 replacement of SolidCloud::evolve (src/solidcloud.cpp:521-562) with
// Solid::applyForcer / addMidFluidForceAndTorque / addAcceleration / move / storeOldForce (src/solid.h:126-202),
// addMidEnvironment (solidcloud.cpp:466-475), the motions (src/libmotion) and forcers (src/libforcer), and the
// uniform-grid collision of solidSolidInteract / solidSolidCollision (solidcloud.cpp:477-519,
// src/libcollision/ugrid.cpp:5-77, collision.cpp:7-57).
//
// Without collisions every solid is independent, so one thread runs all sub-steps of one solid in a single launch.
// With collisions up to 20 solids per SM run all sub-steps in one cooperative launch (evolve_contacts_kernel); for more, each
// sub-step is: forces + grid hash, counting sort of solid ids by grid cell, pair forces (each solid sums its own side of
// every pair: no atomics, the pair law is evaluated once per side), move.
#include <cstdint>
#include <cuda_runtime.h>

#include "common.cuh"

namespace sdfibm_dev {

__device__ inline D3 ld3(const double* a) { return D3{a[0], a[1], a[2]}; }
__device__ inline void st3(double* a, const D3& v) { a[0] = v.x; a[1] = v.y; a[2] = v.z; }

// IMotion::constraint of each registered motion
__device__ inline void motion_constraint(const SolidK& k, double time, D3& velocity, D3& omega) {
    const double* p = k.motion_p;
    switch (k.motion_type) {
        case SDFIBM_MOTION_000002: velocity = D3{0, 0, 0}; omega = D3{0, 0, 0}; omega.z = p[1]; return;
        case SDFIBM_MOTION_110002: velocity.z = 0.0; omega = D3{0, 0, 0}; omega.z = p[1]; return;
        case SDFIBM_MOTION_222000: velocity = D3{p[0], p[1], p[2]}; omega = D3{0, 0, 0}; return;
        case SDFIBM_MOTION_SINEDIRECTIONAL:
            velocity = p[0] * p[2] * cos(p[2] * time) * D3{p[3], p[4], p[5]};
            omega = D3{0, 0, 0};
            return;
        case SDFIBM_MOTION_01MASK:
            velocity = D3{velocity.x * p[0], velocity.y * p[1], velocity.z * p[2]};
            omega = D3{omega.x * p[3], omega.y * p[4], omega.z * p[5]};
            return;
        case SDFIBM_MOTION_ROTOR:
            velocity = D3{0, 0, 0};
            velocity.x = -p[2] * p[1] * sin(p[1] * time + p[3]);
            velocity.y = p[2] * p[1] * cos(p[1] * time + p[3]);
            omega = D3{0, 0, 0};
            omega.z = p[4];
            return;
        case SDFIBM_MOTION_OPENCLOSE: {
            const double t = fmod(time, 5.0);
            double v = 0.0;
            if (t > 1 && t < 2) v = -1.0;
            if (t > 3 && t < 4) v = 1.0;
            velocity = D3{0, v, 0};
            omega = D3{0, 0, 0};
            return;
        }
        default: return;
    }
}

// IForcer::generate of each registered forcer
__device__ inline void forcer_generate(const SolidK& k, const sdfibm_solid_state& s, double time, D3& f, D3& t) {
    const double* p = k.forcer_p;
    f = D3{0, 0, 0};
    t = D3{0, 0, 0};
    switch (k.forcer_type) {
        case SDFIBM_FORCER_CONSTANT: f = D3{p[0], p[1], p[2]}; t = D3{p[3], p[4], p[5]}; return;
        case SDFIBM_FORCER_SPRING: {
            const D3 r = ld3(s.pos) - D3{p[0], p[1], p[2]};
            if (mag(r) > SMALL_D) f = -p[3] * r * (1.0 - p[4] / mag(r));
            return;
        }
        case SDFIBM_FORCER_MAGNETIC: {
            const D3 m_original = (1.0) * (D3{0.0, 0.0, 1.0});
            const D3 B = p[3] * cos(p[4] * time) * D3{p[0], p[1], p[2]};
            const Q4 q{s.quat[0], D3{s.quat[1], s.quat[2], s.quat[3]}};
            const D3 m = qtransform(qconj(q), m_original);
            t = cross(m, B);
            return;
        }
        default: return;
    }
}

// clearForceAndTorque, applyForcer, addMidFluidForceAndTorque, addMidEnvironment for one solid
__device__ inline void pre_forces(const SolidK& k, sdfibm_solid_state& s, double time, double rho_f, const D3& g) {
    D3 force{0, 0, 0}, torque{0, 0, 0};
    if (k.forcer_type != SDFIBM_FORCER_NONE) {
        D3 f_, t_;
        forcer_generate(k, s, time, f_, t_);
        st3(s.forcer_force, f_);
        st3(s.forcer_torque, t_);
        if (s.first_forcer_step) {
            st3(s.forcer_force_old, f_);
            st3(s.forcer_torque_old, t_);
            s.first_forcer_step = 0;
        }
        force = force + (1.5 * ld3(s.forcer_force) - 0.5 * ld3(s.forcer_force_old));
        torque = torque + (1.5 * ld3(s.forcer_torque) - 0.5 * ld3(s.forcer_torque_old));
    }
    if (s.first_fluid_step) {
        for (int a = 0; a < 3; ++a) { s.fluid_force_old[a] = s.fluid_force[a]; s.fluid_torque_old[a] = s.fluid_torque[a]; }
        s.first_fluid_step = 0;
    }
    force = force + (1.5 * ld3(s.fluid_force) - 0.5 * ld3(s.fluid_force_old));
    torque = torque + (1.5 * ld3(s.fluid_torque) - 0.5 * ld3(s.fluid_torque_old));
    const double rhos = k.rho;
    const D3 gprime = ((rhos - rho_f) / rhos) * g;
    force = force + k.mass * gprime;
    st3(s.force, force);
    st3(s.torque, torque);
}

// Solid::move, its rotation half (which needs no force): the new angular velocity and orientation
__device__ inline void move_rotation(const SolidK& k, const Q4& q, const D3& omega_old, const D3& T, double time, double dt,
                                     D3& om, Q4& qn) {
    const double w2 = q.w * q.w, x2 = q.v.x * q.v.x, y2 = q.v.y * q.v.y, z2 = q.v.z * q.v.z;
    const double txy = 2 * q.v.x * q.v.y, twz = 2 * q.w * q.v.z, txz = 2 * q.v.x * q.v.z;
    const double twy = 2 * q.w * q.v.y, tyz = 2 * q.v.y * q.v.z, twx = 2 * q.w * q.v.x;
    const double R[9] = {w2 + x2 - y2 - z2, txy - twz, txz + twy, txy + twz, w2 - x2 + y2 - z2,
                         tyz - twx, txz - twy, tyz + twx, w2 - x2 - y2 + z2};
    const double* I = k.moi_inv;
    double RI[9], W[9];
    for (int r = 0; r < 3; ++r)
        for (int c = 0; c < 3; ++c) RI[3 * r + c] = R[3 * r] * I[c] + R[3 * r + 1] * I[3 + c] + R[3 * r + 2] * I[6 + c];
    for (int r = 0; r < 3; ++r)  // (R & I) & R^T
        for (int c = 0; c < 3; ++c) W[3 * r + c] = RI[3 * r] * R[3 * c] + RI[3 * r + 1] * R[3 * c + 1] + RI[3 * r + 2] * R[3 * c + 2];
    const D3 WT{W[0] * T.x + W[1] * T.y + W[2] * T.z, W[3] * T.x + W[4] * T.y + W[5] * T.z,
                W[6] * T.x + W[7] * T.y + W[8] * T.z};
    om = omega_old + WT * dt;
    if (k.motion_type != SDFIBM_MOTION_FREE) {
        D3 unused{0, 0, 0};
        motion_constraint(k, time, unused, om);
    }
    const Q4 h{0.5 * 0.0, 0.5 * (0.5 * (om + omega_old))};
    const Q4 dq0 = qmul(h, q);
    const Q4 dq{dq0.w * dt, dq0.v * dt};
    qn = Q4{q.w + dq.w, q.v + dq.v};
    const double mq = sqrt(qn.w * qn.w + magSqr(qn.v));
    qn = Q4{qn.w / mq, qn.v / mq};
}

// its translation half: velocity and position
__device__ inline void move_translation(const SolidK& k, const D3& force, double time, double dt, D3& vel, D3& pos) {
    const D3 velocity_old = vel;
    vel = velocity_old + force * k.mass_inv * dt;
    if (k.motion_type != SDFIBM_MOTION_FREE) {
        D3 unused{0, 0, 0};
        motion_constraint(k, time, vel, unused);
    }
    pos = pos + 0.5 * (vel + velocity_old) * dt;
}

__device__ inline void move_solid(const SolidK& k, sdfibm_solid_state& s, double time, double dt) {
    D3 om, vel = ld3(s.vel), pos = ld3(s.pos);
    Q4 qn;
    move_rotation(k, Q4{s.quat[0], D3{s.quat[1], s.quat[2], s.quat[3]}}, ld3(s.omega), ld3(s.torque), time, dt, om, qn);
    move_translation(k, ld3(s.force), time, dt, vel, pos);
    st3(s.vel, vel);
    st3(s.omega, om);
    st3(s.pos, pos);
    s.quat[0] = qn.w; s.quat[1] = qn.v.x; s.quat[2] = qn.v.y; s.quat[3] = qn.v.z;
}

__device__ inline void store_old(sdfibm_solid_state& s) {
    for (int a = 0; a < 3; ++a) {
        s.fluid_force_old[a] = s.fluid_force[a];
        s.fluid_torque_old[a] = s.fluid_torque[a];
        s.forcer_force_old[a] = s.forcer_force[a];
        s.forcer_torque_old[a] = s.forcer_torque[a];
    }
}

// all sub-steps of one solid (no solid-solid interaction)
__global__ void evolve_independent_kernel(const SolidK* __restrict__ sk, sdfibm_solid_state* st, int S, int nsub,
                                          StepParams step, double rho_f, D3 g) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const double time = step.time, dt_sub = step.dt_sub;
    const SolidK& k = sk[s];
    sdfibm_solid_state x = st[s];
    for (int it = 0; it < nsub; ++it) {
        pre_forces(k, x, time, rho_f, g);
        move_solid(k, x, time, dt_sub);
    }
    store_old(x);
    st[s] = x;
}



__device__ inline int64_t grid_hash(const GridK& gk, const D3& c) {
    const int i = (int)floor((c.x - gk.low[0]) * gk.dINV);
    const int j = (int)floor((c.y - gk.low[1]) * gk.dINV);
    const int k = (int)floor((c.z - gk.low[2]) * gk.dINV);
    return (int64_t)i * gk.nynz + (int64_t)j * gk.nz + k;
}

// collision id of the pair-law table: SPHERES mode treats every non-plane solid as its bounding sphere
__device__ inline int coll_id(const SolidK& k, int mode) {
    return mode == SDFIBM_COLLISION_SPHERES ? (k.infinite ? 0 : 2) : k.collision_id;
}

// fine-grid cell range of a bounding box, clamped to the grid
__device__ inline void fine_range(const FineGridK& fg, const D3& c, double r, int lo[3], int hi[3]) {
    const double cc[3] = {c.x, c.y, c.z};
    for (int a = 0; a < 3; ++a) {
        const double l = floor((cc[a] - r - fg.low[a]) * fg.inv), h = floor((cc[a] + r - fg.low[a]) * fg.inv);
        lo[a] = (int)fmin(fmax(l, 0.0), (double)(fg.n[a] - 1));
        hi[a] = (int)fmin(fmax(h, 0.0), (double)(fg.n[a] - 1));
    }
}
__device__ inline int64_t fine_index(const FineGridK& fg, int i, int j, int k) {
    return (int64_t)i + (int64_t)fg.n[0] * ((int64_t)j + (int64_t)fg.n[1] * k);
}

// forces of one sub-step, the UGrid key of every solid (UGrid::insert, ugrid.h:31-34) with the coarse counts (only
// needed by plane-like solids, which search their 27 coarse neighbours), the fine-grid counts of the sphere-like
// solids whose key is on the grid (the reference never pairs the others) and the solid's collision record
__global__ void evolve_pre_kernel(const SolidK* __restrict__ sk, sdfibm_solid_state* st, int S,
                                  const StepParams* step, double rho_f, D3 g, GridK gk, int64_t* __restrict__ hashes,
                                  int32_t* __restrict__ counts, FineGridK fg, int32_t* __restrict__ fcounts, int mode,
                                  int coarse_needed, CollRec* __restrict__ recs, int move_first) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    if (move_first) move_solid(sk[s], st[s], step->time, step->dt_sub);  // Solid::move of the previous sub-step
    pre_forces(sk[s], st[s], step->time, rho_f, g);
    const D3 c = ld3(st[s].pos);
    const int64_t h = grid_hash(gk, c);
    hashes[s] = h;
    CollRec rec{};
    rec.id = -1;
    if (h >= 0 && h < gk.ncell) {
        if (coarse_needed) atomicAdd(counts + h, 1);
        const double rB = sk[s].radiusB;
        rec.id = coll_id(sk[s], mode);
        rec.c[0] = (int32_t)(h / gk.nynz);
        rec.c[1] = (int32_t)((h / gk.nz) % gk.ny);
        rec.c[2] = (int32_t)(h % gk.nz);
        rec.x = (float)c.x; rec.y = (float)c.y; rec.z = (float)c.z; rec.r = (float)rB;
        if (rec.id == 1 || rec.id == 2) {
            fine_range(fg, c, rB, rec.lo, rec.hi);
            for (int k = rec.lo[2]; k <= rec.hi[2]; ++k)
                for (int j = rec.lo[1]; j <= rec.hi[1]; ++j)
                    for (int i = rec.lo[0]; i <= rec.hi[0]; ++i) atomicAdd(fcounts + fine_index(fg, i, j, k), 1);
        }
    }
    recs[s] = rec;
}

__global__ void fine_scatter_kernel(const CollRec* __restrict__ recs, int S, FineGridK fg, int32_t* __restrict__ fcursor,
                                    int32_t* __restrict__ flist, Counters* cnt) {
    // one warp per solid: the lanes split its fine cells, so a large solid's claims do not run one after another
    const int lane = threadIdx.x & 31;
    const int s = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (s >= S) return;
    const CollRec& r = recs[s];
    if (r.id != 1 && r.id != 2) return;
    const int nx = r.hi[0] - r.lo[0] + 1, ny = r.hi[1] - r.lo[1] + 1, nz = r.hi[2] - r.lo[2] + 1;
    for (int e = lane; e < nx * ny * nz; e += 32) {
        const int i = r.lo[0] + e % nx, j = r.lo[1] + (e / nx) % ny, k = r.lo[2] + e / (nx * ny);
        const int32_t slot = atomicAdd(fcursor + fine_index(fg, i, j, k), 1);
        if (slot < fg.cap) flist[slot] = s;
        else set_error(cnt, DERR_CAPACITY);
    }
}

// exclusive scan of the per-cell counts (single block), zeroing them as they are read
__global__ void grid_scan_kernel(int32_t* __restrict__ counts, int32_t* __restrict__ start,
                                 int32_t* __restrict__ cursor, int64_t ncell) {
    __shared__ int32_t warp_tot[32];
    __shared__ int32_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
    for (int64_t base = 0; base < ncell; base += blockDim.x) {
        const int64_t i = base + threadIdx.x;
        const int32_t v = i < ncell ? counts[i] : 0;
        if (i < ncell) counts[i] = 0;  // read once: left zeroed for the next sub-step's counts
        int32_t x = v;
        for (int o = 1; o < 32; o <<= 1) {
            int32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_tot[wid] = x;
        __syncthreads();
        if (wid == 0) {
            int32_t w = lane < nw ? warp_tot[lane] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                int32_t y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            if (lane < nw) warp_tot[lane] = w;
        }
        __syncthreads();
        const int32_t excl = carry + (wid > 0 ? warp_tot[wid - 1] : 0) + x - v;
        if (i < ncell) { start[i] = excl; cursor[i] = excl; }
        __syncthreads();
        if (threadIdx.x == 0) carry += warp_tot[nw - 1];
        __syncthreads();
    }
    if (threadIdx.x == 0) start[ncell] = carry;
}

// exclusive scan of large count arrays in three launches: per-1024-block scans, a scan of the block sums, offsets;
// the counts are zeroed as they are read
__global__ void __launch_bounds__(1024) scan_blocks_kernel(int32_t* __restrict__ counts, int32_t* __restrict__ start,
                                                           int32_t* __restrict__ sums, int64_t ncell) {
    __shared__ int32_t warp_tot[32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t i = (int64_t)blockIdx.x * 1024 + threadIdx.x;
    const int32_t v = i < ncell ? counts[i] : 0;
    if (i < ncell) counts[i] = 0;  // read once: left zeroed for the next sub-step's counts
    int32_t x = v;
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) warp_tot[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int32_t w = warp_tot[lane];
        for (int o = 1; o < 32; o <<= 1) {
            const int32_t y = __shfl_up_sync(0xffffffffu, w, o);
            if (lane >= o) w += y;
        }
        warp_tot[lane] = w;
    }
    __syncthreads();
    if (i < ncell) start[i] = (wid > 0 ? warp_tot[wid - 1] : 0) + x - v;
    if (threadIdx.x == 1023) sums[blockIdx.x] = warp_tot[31];
}

__global__ void __launch_bounds__(1024) scan_add_kernel(int32_t* __restrict__ start, int32_t* __restrict__ cursor,
                                                        const int32_t* __restrict__ sums_excl, int64_t ncell,
                                                        int64_t nblocks) {
    const int64_t i = (int64_t)blockIdx.x * 1024 + threadIdx.x;
    if (i < ncell) {
        const int32_t v = start[i] + sums_excl[blockIdx.x];
        start[i] = v;
        cursor[i] = v;
    }
    if (i == 0) start[ncell] = sums_excl[nblocks];  // the scan of the sums holds the total at nblocks
}

__global__ void grid_scatter_kernel(const int64_t* __restrict__ hashes, int32_t* __restrict__ cursor,
                                    int32_t* __restrict__ list, int S, int64_t ncell) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    const int64_t h = hashes[s];
    if (h >= 0 && h < ncell) list[atomicAdd(cursor + h, 1)] = s;
}

// the collision laws of collision.cpp:7-35 (positions of the sub-step start)
__device__ inline double plane_sphere(const sdfibm_solid_state& p, const sdfibm_solid_state& s, double rB_s, D3& cN) {
    const Q4 qp{p.quat[0], D3{p.quat[1], p.quat[2], p.quat[3]}};
    const D3 s_center = qtransform(qconj(qp), ld3(s.pos) - ld3(p.pos));
    const double p2s = s_center.y;
    cN = qtransform(qp, D3{0, 1, 0});
    return rB_s - p2s;
}
__device__ inline double sphere_sphere(const sdfibm_solid_state& s1, const sdfibm_solid_state& s2, double r1,
                                       double r2, D3& cN) {
    const D3 s2s = ld3(s2.pos) - ld3(s1.pos);
    const double m = mag(s2s);
    cN = m < 1e-150 ? D3{0, 0, 0} : s2s / m;
    return r1 + r2 - mag(s2s);
}

// contact force on s2 (s1 receives the opposite); returns false when the pair has no law or no overlap
__device__ inline bool pair_force(const SolidK& k1, const sdfibm_solid_state& s1, int id1, const SolidK& k2,
                                  const sdfibm_solid_state& s2, int id2, D3& f) {
    double cd;
    D3 cN;
    if ((id1 == 1 || id1 == 2) && id2 == 0) cd = plane_sphere(s2, s1, k1.radiusB, cN);
    else if (id1 == 0 && (id2 == 1 || id2 == 2)) cd = plane_sphere(s1, s2, k2.radiusB, cN);
    else if ((id1 == 1 && id2 == 1) || (id1 == 2 && id2 == 2)) cd = sphere_sphere(s1, s2, k1.radiusB, k2.radiusB, cN);
    else return false;
    if (cd < 0) return false;
    f = 1e4 * cd * cN;
    return true;
}

// the 27 coarse cells around key a contain key b (the neighbour loops of ugrid.cpp:50-77)
__device__ inline bool coarse_neighbours(const GridK& gk, int64_t a, int64_t b) {
    const int64_t ai = a / gk.nynz, aj = (a / gk.nz) % gk.ny, ak = a % gk.nz;
    const int64_t bi = b / gk.nynz, bj = (b / gk.nz) % gk.ny, bk = b % gk.nz;
    return llabs(ai - bi) <= 1 && llabs(aj - bj) <= 1 && llabs(ak - bk) <= 1;
}
__device__ inline bool coarse_neighbours(const CollRec& a, const CollRec& b) {
    return abs(a.c[0] - b.c[0]) <= 1 && abs(a.c[1] - b.c[1]) <= 1 && abs(a.c[2] - b.c[2]) <= 1;
}

// FP32 screen of a sphere pair: false only when the bounding spheres are certainly apart, i.e. the FP64 contact depth
// r1 + r2 - |x2 - x1| is negative.  The FP32 values carry relative errors of a few 2^-24; the margin is 2^-16 of the
// magnitudes involved, far above them.
__device__ inline bool sphere_screen(const CollRec& a, const CollRec& b) {
    const float dx = b.x - a.x, dy = b.y - a.y, dz = b.z - a.z;
    const float mag = fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fabsf(a.z)) + fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fabsf(b.z));
    const float reach = a.r + b.r + 1.52587890625e-5f * (mag + a.r + b.r);
    return dx * dx + dy * dy + dz * dz <= reach * reach;
}

// Pair forces of one sub-step, each solid summing its own side of every pair the reference's UGrid would form
// (27 coarse neighbours of its key, keys on the grid) that has a contact law and overlaps.  Sphere-like pairs come
// from the fine grid: a pair is taken in the one fine cell holding the corner max(lo_p, lo_q) of the two bounding
// boxes' intersection, then kept only when the coarse keys are neighbours, so the contacts are exactly the
// reference's.  Plane-like solids (law id 0) search the coarse grid; sphere-like solids test the plane list.
__global__ void collide_kernel(const SolidK* __restrict__ sk, sdfibm_solid_state* st, int S, GridK gk,
                               const int64_t* __restrict__ hashes, const int32_t* __restrict__ start,
                               const int32_t* __restrict__ list, int mode, FineGridK fg,
                               const int32_t* __restrict__ fstart, const int32_t* __restrict__ flist,
                               const int32_t* __restrict__ planes, int nplanes, const CollRec* __restrict__ recs) {
    // one warp per solid: lanes split the solid's fine cells (a large solid spans thousands), the plane list, or the
    // entries of its coarse cells; the warp sums the force
    const int lane = threadIdx.x & 31;
    const int p = (int)(((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5);
    if (p >= S) return;
    const CollRec rp = recs[p];
    if (rp.id < 0) return;
    const SolidK& kp = sk[p];
    const int idp = rp.id;
    D3 fsum{0, 0, 0};
    const sdfibm_solid_state& sp = st[p];
    auto add_pair = [&](int q, int idq) {
        D3 f;
        if (p < q) {
            if (pair_force(kp, sp, idp, sk[q], st[q], idq, f)) fsum = fsum + (-f);
        } else {
            if (pair_force(sk[q], st[q], idq, kp, sp, idp, f)) fsum = fsum + f;
        }
    };
    if (idp == 1 || idp == 2) {
        const int nx = rp.hi[0] - rp.lo[0] + 1, ny = rp.hi[1] - rp.lo[1] + 1, nz = rp.hi[2] - rp.lo[2] + 1;
        const int ncells = nx * ny * nz;
        for (int e = lane; e < ncells; e += 32) {
            const int i = rp.lo[0] + e % nx, j = rp.lo[1] + (e / nx) % ny, k = rp.lo[2] + e / (nx * ny);
            const int64_t cell = fine_index(fg, i, j, k);
            for (int f = fstart[cell]; f < fstart[cell + 1]; ++f) {
                const int q = flist[f];
                if (q == p) continue;
                const CollRec rq = recs[q];
                if (rq.id != idp) continue;  // (1,1) and (2,2) have a law, (1,2) has none
                // the pair's home cell: the corner max(lo_p, lo_q) of the two cell ranges' intersection (both solids
                // compute it from the same indices, so exactly one of p's and one of q's visits holds the pair)
                if (max(rp.lo[0], rq.lo[0]) != i || max(rp.lo[1], rq.lo[1]) != j || max(rp.lo[2], rq.lo[2]) != k)
                    continue;
                if (i > rq.hi[0] || j > rq.hi[1] || k > rq.hi[2]) continue;  // ranges do not intersect
                if (!coarse_neighbours(rp, rq) || !sphere_screen(rp, rq)) continue;
                add_pair(q, idp);
            }
        }
        for (int e = lane; e < nplanes; e += 32) {
            const int q = planes[e];
            const CollRec& rq = recs[q];
            if (rq.id < 0 || !coarse_neighbours(rp, rq)) continue;
            add_pair(q, 0);
        }
    } else {
        const int ci = rp.c[0], cj = rp.c[1], ck = rp.c[2];
        for (int a = ci - 1; a <= ci + 1; ++a) {
            if (a < 0 || a > gk.nx - 1) continue;
            for (int b = cj - 1; b <= cj + 1; ++b) {
                if (b < 0 || b > gk.ny - 1) continue;
                for (int c = ck - 1; c <= ck + 1; ++c) {
                    if (c < 0 || c > gk.nz - 1) continue;
                    const int64_t nb = (int64_t)a * gk.nynz + (int64_t)b * gk.nz + c;
                    for (int e = start[nb] + lane; e < start[nb + 1]; e += 32) {
                        const int q = list[e];
                        if (q != p) add_pair(q, recs[q].id);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        fsum.x += __shfl_xor_sync(0xffffffffu, fsum.x, o);
        fsum.y += __shfl_xor_sync(0xffffffffu, fsum.y, o);
        fsum.z += __shfl_xor_sync(0xffffffffu, fsum.z, o);
    }
    // force += -f / +f in pair order (reordered sum); torque += -0 leaves it unchanged
    if (lane == 0) {
        st[p].force[0] += fsum.x;
        st[p].force[1] += fsum.y;
        st[p].force[2] += fsum.z;
    }
}

// ---- all sub-steps of a cloud with contacts in one cooperative launch --------------------------------------------------
// The sub-steps are short chains of dependent FP64 work (a solid's move is about 250 operations) with a search between
// them; as six launches each (forces, counts, scan, scatter, pairs) they took 1.26 ms for 104 solids and 1.4 ms for 1800,
// launch and memory latency.  Here CTA b keeps solids [b per, (b + 1) per): a thread per solid holds its state in
// registers over all sub-steps, the other warps test its pairs meanwhile, and one grid barrier a sub-step publishes the
// new positions (two buffers).  The pairs come from lists built once, by testing all solids in FP32, of the solids nearer
// than the contact distance plus a skin.  A solid that has moved half the skin is hot from then on: it tests every solid, the
// others test the hot ones beside their lists (a solid that left its stable step size does not make everybody search again);
// past EV_HOT of them every CTA lists its pairs in every sub-step, without a skin.  Pairs go through the FP32 screen, the
// reference's 27-cell rule on the UGrid keys and the FP64 contact law, as in collide_kernel, so the contacts are the same.
// The rotation half of a move needs no pair and runs in warps of its own beside the barrier and the pairs.  Plane-like solids
// (law 0) test every sphere, spheres every plane: for up to EV_MAX_PLANES.
// Bound by latency: 9 us a sub-step (barrier, two dependent L2 reads, the FP64 chains of a contact and a move).  Measured
// (GB300), 20 sub-steps: 104 solids 1.26 -> 0.20 ms, 1800 solids 1.05 -> 0.19 ms, all of them crossing the skin in every
// sub-step 1.18 -> 0.61 ms (2.6 with room for 256 hot ones and one record a lane in flight).
constexpr int EV_THREADS = 256, EV_WARPS = EV_THREADS / 32;
constexpr int EV_SOLIDS = 32;             // most solids of a CTA: their rotations take half of its warps
static_assert(EV_PER_SM <= EV_SOLIDS && EV_SOLIDS * 4 <= EV_THREADS / 2, "solids of a CTA");
constexpr int EV_LIST = 128;              // listed neighbours of a solid; more: it tests every solid every sub-step
constexpr int EV_HOT = 32;                // solids beyond half the skin before the lists are made in every sub-step
constexpr int EV_BATCH = 4;               // records of a lane in flight when a warp tests many solids
int evolve_contacts_threads() { return EV_THREADS; }
int evolve_contacts_list() { return EV_LIST; }
int evolve_contacts_hot() { return EV_HOT; }
constexpr long long EV_WAIT_CYCLES = 4000000000LL;  // about two seconds

// Grid barrier in two halves: one thread arrives after a __syncthreads, one waits.  The wait gives up after its limit.
__device__ inline void ev_arrive(EvolveWork w) {
    __threadfence();
    atomicAdd(&w.ctrl->arrived, 1u);
}
__device__ inline bool ev_wait(EvolveWork w, unsigned target) {
    const long long t0 = clock64();
    volatile unsigned* a = &w.ctrl->arrived;
    while (*a < target)
        if (clock64() - t0 > EV_WAIT_CYCLES) return false;
    __threadfence();
    return true;
}
__device__ inline void ev_bar(int id, int threads) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory"); }

// Position record of a solid for the pair tests: x, y, z and the radius, signed by the contact law (1: positive, 2:
// negative, zero included, others: NaN), so that two records have a sphere law when their radii have the same sign.
__device__ inline float4 ev_record(const D3& x, int id, double rB) {
    const float r = (float)rB;
    return make_float4((float)x.x, (float)x.y, (float)x.z, id == 1 ? r : (id == 2 ? -r : NAN));
}

// the UGrid key of a position, decomposed as its neighbour loops do; w = 1 when it is on the grid
__device__ inline int4 ev_key(const GridK& gk, const D3& x) {
    const int i = (int)floor((x.x - gk.low[0]) * gk.dINV), j = (int)floor((x.y - gk.low[1]) * gk.dINV),
              k = (int)floor((x.z - gk.low[2]) * gk.dINV);
    if (i >= 0 && i < gk.nx && j >= 0 && j < gk.ny && k >= 0 && k < gk.nz) return make_int4(i, j, k, 1);
    const int64_t h = (int64_t)i * gk.nynz + (int64_t)j * gk.nz + k;
    if (h < 0 || h >= gk.ncell) return make_int4(0, 0, 0, 0);
    return make_int4((int)(h / gk.nynz), (int)((h / gk.nz) % gk.ny), (int)(h % gk.nz), 1);
}
__device__ inline bool ev_neighbours(const int4& a, const int4& b) {
    return a.w && b.w && abs(a.x - b.x) <= 1 && abs(a.y - b.y) <= 1 && abs(a.z - b.z) <= 1;
}

__device__ inline D3 ev_pos(const EvolveWork& w, int buf, int S, int q) {
    const double2* p = reinterpret_cast<const double2*>(w.x + 4 * ((int64_t)buf * S + q));
    const double2 a = __ldcg(p), b = __ldcg(p + 1);
    return D3{a.x, a.y, b.x};
}

// FP32 screens: false only when the FP64 contact depth is certainly negative (margins of 2^-16 of the magnitudes)
__device__ inline bool ev_sphere_near(const float4& a, const float4& b, float skin) {
    const float dx = b.x - a.x, dy = b.y - a.y, dz = b.z - a.z;
    const float mag = fmaxf(fmaxf(fabsf(a.x), fabsf(a.y)), fabsf(a.z)) + fmaxf(fmaxf(fabsf(b.x), fabsf(b.y)), fabsf(b.z));
    const float rr = fabsf(a.w) + fabsf(b.w);
    const float reach = rr + skin + 1.52587890625e-5f * (mag + rr);
    return (__float_as_int(a.w) ^ __float_as_int(b.w)) >= 0 && dx * dx + dy * dy + dz * dz <= reach * reach;
}
__device__ inline bool ev_plane_near(const float4& n, const float4& xp, const float4& xs) {
    const float d = n.x * (xs.x - xp.x) + n.y * (xs.y - xp.y) + n.z * (xs.z - xp.z), r = fabsf(xs.w);
    const float mag = fabsf(xs.x) + fabsf(xs.y) + fabsf(xs.z) + fabsf(xp.x) + fabsf(xp.y) + fabsf(xp.z);
    return xs.w == xs.w && !(r - d < -1.52587890625e-5f * (mag + r));  // a position that is not finite goes to the law
}

// force on solid p of its contact with q, and of a plane-like solid's contact on the sphere (collision.cpp:7-35)
__device__ inline D3 ev_sphere_force(const D3& xp, const D3& xq, double rp, double rq) {
    const D3 d = xp - xq;
    const double m = mag(d);
    const D3 cN = m < 1e-150 ? D3{0, 0, 0} : d / m;
    const double cd = rp + rq - m;
    return cd < 0 ? D3{0, 0, 0} : 1e4 * cd * cN;
}
// record of a plane-like solid: orientation, then the normal qtransform(q, (0, 1, 0))
__device__ inline D3 ev_plane_force(const double* rec, const D3& xp, const D3& xs, double rB_s) {
    const double2* r = reinterpret_cast<const double2*>(rec);
    const double2 a = __ldcg(r), b = __ldcg(r + 1), c = __ldcg(r + 2), d = __ldcg(r + 3);
    const D3 l = qtransform(qconj(Q4{a.x, D3{a.y, b.x, b.y}}), xs - xp);
    const double cd = rB_s - l.y;
    return cd < 0 ? D3{0, 0, 0} : 1e4 * cd * D3{c.x, c.y, d.x};
}

// move_rotation by four lanes: lane r of the group computes row r of R I R^T and component r of the products (3: the scalar
// part of the quaternion).  The same operations in the same order, about 120 instructions a lane instead of 290.
// All lanes of the warp call it; w receives component r of the quaternion (x, y, z, w), o of the angular velocity.
__device__ inline void move_rotation4(const SolidK& k, const double* q4, const double* o3, const double* T, double time,
                                      double dt, double& o, double& qn) {
    const unsigned FULL = 0xffffffffu;
    const int r = threadIdx.x & 3;
    const Q4 q{q4[0], D3{q4[1], q4[2], q4[3]}};
    const D3 oo{o3[0], o3[1], o3[2]};
    const double w2 = q.w * q.w, x2 = q.v.x * q.v.x, y2 = q.v.y * q.v.y, z2 = q.v.z * q.v.z;
    const double txy = 2 * q.v.x * q.v.y, twz = 2 * q.w * q.v.z, txz = 2 * q.v.x * q.v.z;
    const double twy = 2 * q.w * q.v.y, tyz = 2 * q.v.y * q.v.z, twx = 2 * q.w * q.v.x;
    const double R[9] = {w2 + x2 - y2 - z2, txy - twz, txz + twy, txy + twz, w2 - x2 + y2 - z2,
                         tyz - twx, txz - twy, tyz + twx, w2 - x2 - y2 + z2};
    double row[3], RI[3], W[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) row[c] = r == 0 ? R[c] : (r == 1 ? R[3 + c] : R[6 + c]);
    const double* I = k.moi_inv;
#pragma unroll
    for (int c = 0; c < 3; ++c) RI[c] = row[0] * I[c] + row[1] * I[3 + c] + row[2] * I[6 + c];
#pragma unroll
    for (int c = 0; c < 3; ++c) W[c] = RI[0] * R[3 * c] + RI[1] * R[3 * c + 1] + RI[2] * R[3 * c + 2];
    o = (r == 0 ? oo.x : (r == 1 ? oo.y : oo.z)) + (W[0] * T[0] + W[1] * T[1] + W[2] * T[2]) * dt;
    D3 om{__shfl_sync(FULL, o, 0, 4), __shfl_sync(FULL, o, 1, 4), __shfl_sync(FULL, o, 2, 4)};
    if (k.motion_type != SDFIBM_MOTION_FREE) {
        D3 unused{0, 0, 0};
        motion_constraint(k, time, unused, om);
        o = r == 0 ? om.x : (r == 1 ? om.y : om.z);
    }
    const Q4 h{0.5 * 0.0, 0.5 * (0.5 * (om + oo))};
    double d;
    if (r == 3) {
        d = h.w * q.w - dot(h.v, q.v);
    } else {
        // component r of h.w q.v + q.w h.v + h.v x q.v: the cross product from the two cyclically next components
        const double hr = r == 0 ? h.v.x : (r == 1 ? h.v.y : h.v.z), qr = r == 0 ? q.v.x : (r == 1 ? q.v.y : q.v.z);
        const double h1 = r == 0 ? h.v.y : (r == 1 ? h.v.z : h.v.x), q1 = r == 0 ? q.v.y : (r == 1 ? q.v.z : q.v.x);
        const double h2 = r == 0 ? h.v.z : (r == 1 ? h.v.x : h.v.y), q2 = r == 0 ? q.v.z : (r == 1 ? q.v.x : q.v.y);
        d = h.w * qr + q.w * hr + (h1 * q2 - h2 * q1);
    }
    const double e = (r == 3 ? q.w : (r == 0 ? q.v.x : (r == 1 ? q.v.y : q.v.z))) + d * dt;
    const double ex = __shfl_sync(FULL, e, 0, 4), ey = __shfl_sync(FULL, e, 1, 4), ez = __shfl_sync(FULL, e, 2, 4),
                 ew = __shfl_sync(FULL, e, 3, 4);
    qn = e / sqrt(ew * ew + magSqr(D3{ex, ey, ez}));
}

// Sum of the sphere contacts q[0..n) of solid p over the warp (result on every lane): a lane per contact.  Up to two commute;
// more are added as collide_kernel adds them (lane and order by the pair's home cell in the fine grid), so that both paths
// give the same bits.
__device__ inline D3 ev_contact_sum(const EvolveWork& w, const SolidK* sk, int buf, int S, const FineGridK& fg, int p, int n,
                                    const int32_t* q, double (*fc)[3], int32_t* home) {
    const int lane = threadIdx.x & 31;
    D3 f{0, 0, 0};
    const D3 xp = ev_pos(w, buf, S, p);
    if (lane < n) f = ev_sphere_force(xp, ev_pos(w, buf, S, q[lane]), sk[p].radiusB, sk[q[lane]].radiusB);
    if (n > 2) {
        if (lane < n) {
            int lp[3], hp[3], lq[3], hq[3];
            fine_range(fg, xp, sk[p].radiusB, lp, hp);
            fine_range(fg, ev_pos(w, buf, S, q[lane]), sk[q[lane]].radiusB, lq, hq);
            const int nx = hp[0] - lp[0] + 1, ny = hp[1] - lp[1] + 1;
            home[lane] = (max(lp[0], lq[0]) - lp[0]) +
                         nx * ((max(lp[1], lq[1]) - lp[1]) + ny * (max(lp[2], lq[2]) - lp[2]));
            fc[lane][0] = f.x; fc[lane][1] = f.y; fc[lane][2] = f.z;
        }
        __syncwarp();
        f = D3{0, 0, 0};
        int64_t done = -1;  // cell and solid last added
        for (int t = 0; t < n; ++t) {
            int at = -1;
            int64_t next = INT64_MAX;
            for (int i = 0; i < n; ++i) {
                const int64_t key = ((int64_t)home[i] << 32) | (uint32_t)q[i];
                if ((home[i] & 31) == lane && key > done && key < next) { next = key; at = i; }
            }
            if (at < 0) break;
            f = f + D3{fc[at][0], fc[at][1], fc[at][2]};
            done = next;
        }
        __syncwarp();
    }
    return f;
}

__global__ void __launch_bounds__(EV_THREADS, 1) evolve_contacts_kernel(const SolidK* __restrict__ sk,
                                                                        sdfibm_solid_state* st, int S, int per, int nsub,
                                                                        const StepParams* step, double rho_f, D3 g,
                                                                        GridK gk, FineGridK fg, int mode,
                                                                        const int32_t* __restrict__ planes, int nplanes,
                                                                        float skin, EvolveWork w, Counters* cnt) {
    __shared__ double s_f[EV_SOLIDS][3];
    __shared__ double s_q[EV_SOLIDS][4], s_om[EV_SOLIDS][3], s_T[EV_SOLIDS][3], s_qn[EV_SOLIDS][4], s_omn[EV_SOLIDS][3];
    __shared__ double s_fc[EV_WARPS][32][3];
    __shared__ int32_t s_cq[EV_WARPS][32], s_ce[EV_WARPS][32], s_cn[EV_WARPS];
    __shared__ int32_t s_n[EV_SOLIDS];   // listed neighbours, -1: more than the list holds
    __shared__ int s_hot[EV_SOLIDS];
    __shared__ int s_ok, s_move, s_build, s_storm;
    const unsigned FULL = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const int s0 = blockIdx.x * per, own = min(per, S - s0);  // 1 .. EV_SOLIDS
    const double time = step->time, dt = step->dt_sub;
    unsigned arrive = 0;
    // warps 0 .. nrot - 1 do the rotations (four lanes a solid) while the others wait for the barrier and test the pairs
    const int nrot = (own + 7) >> 3, ncw = EV_WARPS - nrot;
    // this thread's solid
    const int s = s0 + tid;
    const bool mine = tid < own;
    D3 pos{0, 0, 0}, vel{0, 0, 0}, om{0, 0, 0}, force{0, 0, 0}, at{0, 0, 0};
    Q4 q{1, D3{0, 0, 0}};
    int id = -1, plane = -1;
    double rB = 0.0;
    auto publish = [&](int buf) {  // true when the solid is on the grid
        double2* xo = reinterpret_cast<double2*>(w.x + 4 * ((int64_t)buf * S + s));
        __stcg(xo, make_double2(pos.x, pos.y));
        __stcg(xo + 1, make_double2(pos.z, 0.0));
        __stcg(w.rec + (int64_t)buf * S + s, ev_record(pos, id, rB));
        const int4 key = ev_key(gk, pos);
        __stcg(w.key + (int64_t)buf * S + s, key);
        if (plane >= 0) {
            const D3 n = qtransform(q, D3{0, 1, 0});
            __stcg(w.pn + buf * nplanes + plane, make_float4((float)n.x, (float)n.y, (float)n.z, 0.f));
            double2* qo = reinterpret_cast<double2*>(w.pq + 8 * ((int64_t)buf * nplanes + plane));
            __stcg(qo, make_double2(q.w, q.v.x));
            __stcg(qo + 1, make_double2(q.v.y, q.v.z));
            __stcg(qo + 2, make_double2(n.x, n.y));
            __stcg(qo + 3, make_double2(n.z, 0.0));
        }
        s_q[tid][0] = q.w; s_q[tid][1] = q.v.x; s_q[tid][2] = q.v.y; s_q[tid][3] = q.v.z;
        s_om[tid][0] = om.x; s_om[tid][1] = om.y; s_om[tid][2] = om.z;
        return key.w != 0;
    };
    if (mine) {
        const SolidK& k = sk[s];
        const sdfibm_solid_state& x = st[s];
        pos = ld3(x.pos); vel = ld3(x.vel); om = ld3(x.omega);
        q = state_quat(x);
        id = coll_id(k, mode);
        rB = k.radiusB;
        if (id == 0)
            for (int i = 0; i < nplanes; ++i)
                if (planes[i] == s) plane = i;
        publish(0);
    }
    if (tid < EV_SOLIDS) s_hot[tid] = 0;
    if (blockIdx.x == 0 && tid < EV_HOT) __stcg(w.hot + tid, make_int2(0, 0x7fffffff));
    // the forces that need no pair (clearForceAndTorque, applyForcer, addMidFluidForceAndTorque, addMidEnvironment: the
    // same in every sub-step without a forcer) and the rotation half of the move
    auto rotate = [&](bool first) {
        if (mine) {
            const SolidK& k = sk[s];
            if (first || k.forcer_type != SDFIBM_FORCER_NONE) {
                sdfibm_solid_state& x = st[s];
                if (!first) {  // the forcers look at the pose
                    st3(x.pos, pos);
                    x.quat[0] = q.w; x.quat[1] = q.v.x; x.quat[2] = q.v.y; x.quat[3] = q.v.z;
                }
                pre_forces(k, x, time, rho_f, g);
                force = ld3(x.force);
                s_T[tid][0] = x.torque[0]; s_T[tid][1] = x.torque[1]; s_T[tid][2] = x.torque[2];
            }
        }
        ev_bar(2, 32 * nrot);
        const int i = min(tid >> 2, own - 1), r = tid & 3;
        double o, e;
        move_rotation4(sk[s0 + i], s_q[i], s_om[i], s_T[i], time, dt, o, e);
        if ((tid >> 2) < own) {
            s_qn[i][(r + 1) & 3] = e;
            if (r < 3) s_omn[i][r] = o;
        }
    };
    if (tid == 0) { s_build = 1; s_move = 0; s_storm = 0; }
    __syncthreads();
    if (tid == 0) ev_arrive(w);
    for (int it = 0; it < nsub; ++it) {
        const int buf = it & 1;
        const float4* rec = w.rec + (int64_t)buf * S;
        const int4* key = w.key + (int64_t)buf * S;
        ++arrive;
        if (wid < nrot) rotate(it == 0);
        if (wid >= nrot) {
            if (tid == 32 * nrot) {
                s_ok = ev_wait(w, gridDim.x * arrive) ? 1 : 0;
                if (it > 0 && !s_storm) s_storm = __ldcg(&w.ctrl->rebuild[(it - 1) & 1]) == it;
                s_build = it == 0 || s_storm;
            }
            ev_bar(1, 32 * ncw);
            if (s_ok && s_build) {  // lists of the CTA's solids, four of them per pass over the records
                for (int i0 = (wid - nrot) * 4; i0 < own; i0 += ncw * 4) {
                    float4 a[4];
                    int n[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        a[u] = i0 + u < own ? __ldcg(rec + s0 + i0 + u) : make_float4(0.f, 0.f, 0.f, NAN);
                        n[u] = 0;
                    }
                    const float reach = s_storm ? 0.f : skin;
                    for (int q0 = 0; q0 < S; q0 += 32 * EV_BATCH) {
                        float4 b[EV_BATCH];
#pragma unroll
                        for (int v = 0; v < EV_BATCH; ++v) {
                            const int qq = q0 + 32 * v + lane;
                            b[v] = qq < S ? __ldcg(rec + qq) : make_float4(0.f, 0.f, 0.f, NAN);
                        }
#pragma unroll
                        for (int v = 0; v < EV_BATCH; ++v) {
                            const int qq = q0 + 32 * v + lane;
#pragma unroll
                            for (int u = 0; u < 4; ++u) {
                                const bool hit = ev_sphere_near(a[u], b[v], reach) && qq != s0 + i0 + u;
                                const unsigned bal = __ballot_sync(FULL, hit);
                                if (bal) {
                                    const int to = n[u] + __popc(bal & ((1u << lane) - 1u));
                                    if (hit && to < EV_LIST) w.list[(int64_t)(s0 + i0 + u) * EV_LIST + to] = qq;
                                    n[u] += __popc(bal);
                                }
                            }
                        }
                    }
                    if (lane == 0)
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if (i0 + u < own) s_n[i0 + u] = n[u] <= EV_LIST ? n[u] : -1;
                }
                ev_bar(1, 32 * ncw);
            }
            // pair forces, a warp per solid; entries of the hot list hold the step they count from (a CTA ahead of this one
            // may add to it meanwhile)
            const int nhot = s_ok && !s_storm ? min(__ldcg(&w.ctrl->nhot), EV_HOT) : 0;
            for (int i = wid - nrot; i < (s_ok ? own : 0); i += ncw) {
                const int p = s0 + i;
                const int4 kp = __ldcg(key + p);
                const float4 rp = __ldcg(rec + p);
                D3 f{0, 0, 0};
                bool any = false;
                if (kp.w) {
                    if (rp.w == rp.w) {  // a sphere law
                        const int n = s_n[i];
                        const int32_t* list = w.list + (int64_t)p * EV_LIST;
                        const bool all = n < 0 || (s_hot[i] && !s_storm);
                        if (lane == 0) s_cn[wid] = 0;
                        __syncwarp();
                        auto near = [&](int qq) {
                            return qq != p && ev_sphere_near(rp, __ldcg(rec + qq), 0.f) && ev_neighbours(kp, __ldcg(key + qq));
                        };
                        auto is_hot = [&](int qq) {
                            for (int h = 0; h < nhot; ++h) {
                                const int2 hs = __ldcg(w.hot + h);
                                if (hs.x == qq && hs.y <= it) return true;
                            }
                            return false;
                        };
                        auto add = [&](int qq) {
                            const int slot = atomicAdd(&s_cn[wid], 1);
                            if (slot < 32) s_cq[wid][slot] = qq;
                        };
                        for (int e0 = lane; e0 < (all ? S : n); e0 += 32 * EV_BATCH) {
                            int qq[EV_BATCH];
                            float4 b[EV_BATCH];
#pragma unroll
                            for (int v = 0; v < EV_BATCH; ++v) {
                                const int e = e0 + 32 * v;
                                qq[v] = e < (all ? S : n) ? (all ? e : list[e]) : p;
                            }
#pragma unroll
                            for (int v = 0; v < EV_BATCH; ++v) b[v] = __ldcg(rec + qq[v]);
#pragma unroll
                            for (int v = 0; v < EV_BATCH; ++v)
                                if (qq[v] != p && ev_sphere_near(rp, b[v], 0.f) && ev_neighbours(kp, __ldcg(key + qq[v])) &&
                                    (all || !is_hot(qq[v])))
                                    add(qq[v]);
                        }
                        if (!all)
                            for (int h = lane; h < nhot; h += 32) {
                                const int2 hs = __ldcg(w.hot + h);
                                if (hs.y <= it && near(hs.x)) add(hs.x);
                            }
                        __syncwarp();
                        const int nc = s_cn[wid];
                        if (nc > 32) {  // a crowd: no room, summed as found
                            auto sum = [&](int qq) {
                                f = f + ev_sphere_force(ev_pos(w, buf, S, p), ev_pos(w, buf, S, qq), sk[p].radiusB,
                                                        sk[qq].radiusB);
                            };
                            for (int e = lane; e < (all ? S : n); e += 32) {
                                const int qq = all ? e : list[e];
                                if (near(qq) && (all || !is_hot(qq))) sum(qq);
                            }
                            if (!all)
                                for (int h = lane; h < nhot; h += 32) {
                                    const int2 hs = __ldcg(w.hot + h);
                                    if (hs.y <= it && near(hs.x)) sum(hs.x);
                                }
                            any = true;
                        } else if (nc > 0) {
                            f = ev_contact_sum(w, sk, buf, S, fg, p, nc, s_cq[wid], s_fc[wid], s_ce[wid]);
                            any = true;
                        }
                        for (int e = lane; e < nplanes; e += 32) {
                            const int qq = planes[e];
                            if (!ev_plane_near(__ldcg(w.pn + buf * nplanes + e), __ldcg(rec + qq), rp) ||
                                !ev_neighbours(kp, __ldcg(key + qq)))
                                continue;
                            const D3 fp = ev_plane_force(w.pq + 8 * ((int64_t)buf * nplanes + e), ev_pos(w, buf, S, qq),
                                                         ev_pos(w, buf, S, p), sk[p].radiusB);
                            f = p < qq ? f + (-fp) : f + fp;
                            any = true;
                        }
                    } else if (coll_id(sk[p], mode) == 0) {
                        int e = 0;
                        while (e < nplanes && planes[e] != p) ++e;
                        const float4 n = __ldcg(w.pn + buf * nplanes + e);
                        for (int qq = lane; qq < S; qq += 32) {
                            if (!ev_plane_near(n, rp, __ldcg(rec + qq)) || !ev_neighbours(kp, __ldcg(key + qq))) continue;
                            const D3 fp = ev_plane_force(w.pq + 8 * ((int64_t)buf * nplanes + e), ev_pos(w, buf, S, p),
                                                         ev_pos(w, buf, S, qq), sk[qq].radiusB);
                            f = p < qq ? f + (-fp) : f + fp;
                            any = true;
                        }
                    }
                }
                if (__any_sync(FULL, any)) {
#pragma unroll
                    for (int o = 16; o > 0; o >>= 1) {
                        f.x += __shfl_xor_sync(FULL, f.x, o);
                        f.y += __shfl_xor_sync(FULL, f.y, o);
                        f.z += __shfl_xor_sync(FULL, f.z, o);
                    }
                }
                if (lane == 0) { s_f[i][0] = f.x; s_f[i][1] = f.y; s_f[i][2] = f.z; }
            }
        }
        __syncthreads();
        if (!s_ok) {
            if (tid == 0) set_error(cnt, DERR_EVOLVE_TIMEOUT);
            return;
        }
        const bool last = it + 1 == nsub;
        if (mine) {
            const SolidK& k = sk[s];
            if (s_build) at = pos;
            const D3 ft{force.x + s_f[tid][0], force.y + s_f[tid][1], force.z + s_f[tid][2]};
            move_translation(k, ft, time, dt, vel, pos);
            om = D3{s_omn[tid][0], s_omn[tid][1], s_omn[tid][2]};
            q = Q4{s_qn[tid][0], D3{s_qn[tid][1], s_qn[tid][2], s_qn[tid][3]}};
            if (last) {
                sdfibm_solid_state& x = st[s];
                st3(x.force, ft);
                st3(x.vel, vel);
                st3(x.omega, om);
                st3(x.pos, pos);
                x.quat[0] = q.w; x.quat[1] = q.v.x; x.quat[2] = q.v.y; x.quat[3] = q.v.z;
                store_old(x);
            } else {
                const bool on = publish(buf ^ 1);
                const D3 d = pos - at;
                // beyond half the skin, with room.  Off the grid, or not finite, a solid has no sphere pair; back on the grid
                // it counts from then on
                if (on && !s_storm && !s_hot[tid] && magSqr(d) > 0.24 * (double)skin * (double)skin) {
                    const int slot = atomicAdd(&w.ctrl->nhot, 1);
                    if (slot < EV_HOT) {
                        __stcg(w.hot + slot, make_int2(s, it + 1));
                        s_hot[tid] = 1;
                    } else {
                        s_move = 1;
                    }
                }
            }
        }
        if (last) break;
        __syncthreads();
        if (tid == 0) {
            // no room among the hot ones: every CTA lists again, without a skin, from the next sub-step to the last.  Two
            // slots by step, since a CTA ahead of this one may already ask for the next step (but not for the one after it)
            if (s_move) atomicMax(&w.ctrl->rebuild[it & 1], it + 1);
            s_move = 0;
            ev_arrive(w);
        }
    }
}

__global__ void move_kernel(const SolidK* __restrict__ sk, sdfibm_solid_state* st, int S, const StepParams* step) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    move_solid(sk[s], st[s], step->time, step->dt_sub);
}

__global__ void store_old_kernel(sdfibm_solid_state* st, int S) {
    const int s = blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= S) return;
    store_old(st[s]);
}

}  // namespace sdfibm_dev
