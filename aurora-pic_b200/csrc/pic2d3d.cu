// Structured 2D3V / 3D3V periodic electrostatic PIC step on one B200 (FP64 form).
//
// Replaces Simulation2D::step / Simulation3D::step for fully periodic meshes
// (src/Simulation2D.cpp:1337-1364, src/Simulation3D.cpp:342-365) and what they
// call: interpolate_electric(Mesh2D&/Mesh3D&) (src/FieldSolver.cpp:926-1038),
// kick_boris / kick_leapfrog / drift_leapfrog (src/Pusher.cpp:82-186), the
// periodic particle boundaries (src/Simulation2D.cpp:57-97),
// deposit_charge_cic (src/Mesh2D.cpp:90-144, src/Mesh3D.cpp:62-126) and
// solve_periodic_spectral (src/FieldSolver.cpp:442-499, :659-731).
//
// One step: a push kernel per species (gather from an interleaved E grid,
// Boris or leapfrog kick, drift, periodic wrap, CIC deposit into a 64-bit
// fixed-point density with global atomics), then the spectral solve as line
// FFTs in shared memory: forward along x (reading and clearing the fixed-point
// density), [forward along y,] forward along the last axis fused with the
// k-space multiply and the first inverse transform, [inverse along y,] and an
// inverse along x that writes phi and the interleaved E field.  Particles are
// re-sorted by cell every `sort_interval` steps so gathers and atomics stay
// local.  Compiled with --fmad=false: particle arithmetic follows the
// reference operation by operation.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <functional>
#include <memory>
#include <mutex>
#include <set>
#include <string>
#include <thread>
#include <vector>

#include "apic_common.cuh"
#include "apic_rng.cuh"

namespace apic {
namespace nd {

constexpr int kThreads = 256;
constexpr int kMaxLine = 1024;

struct Cplx {
    double re, im;
};

struct SpeciesND {
    double qm;
    double dep;   // charge * weight (/ depth in 2D) times the inverse cell area/volume
    double hmw;   // 0.5 * mass * weight
    unsigned n;
    double* pos[2][3];
    double* vh[2][3];
    unsigned* id[2];
    double* v[3];  // runs with walls: in load order (an absorbed particle keeps its last v through sorts)
    // FP32 form: packed cell (10 bits per axis), in-cell offsets in [0, 1) and
    // float velocities; the FP64 arrays above then only stage loads/read-backs
    unsigned* cell[2];
    float* off[2][3];
    float* vel[2][3];
    float hqmdt;       // 0.5 * qm * dt
    float qmdt;        // qm * dt
    float tb[3], sb[3];  // Boris t = hqmdt B and s = 2 t / (1 + t^2)
    float drift[3];    // dt / d_a: cell units per unit velocity
    float dep_fixed;   // dep * rho_scale
    // runs with walls and an absorbing side: Particle::alive (null: all alive)
    uint8_t* alive[2];
    unsigned* live_end;  // particles alive at the last sort, which moved the others behind them (null: none absorb)
    // FP64 form: Boris h = 0.5 qm dt, t = h B and s = 2 t / (1 + t^2) of a full step in the uniform B
    double bh, bt[3], bs[3];
    int index;         // species index (loss ledger row)
    // 3D, sorted tile by tile (kTileCells^3 cells each, cells in order inside):
    // the push takes whole tiles through shared memory
    int tiled;
    uint4* chunk;      // work items: (tile, first particle, one past the last, -)
    unsigned* extra;   // items past the one of every tile
};

// Tiles of the 3D push.
constexpr int kTileCells = 8, kTileLog = 3;
constexpr unsigned kTileVolume = kTileCells * kTileCells * kTileCells;
// from 2 particles a cell: 128^3 x 2, 258 -> 243 us; 128^3 x 4, 525 -> 404; 64^3 x 12, 192 -> 150
constexpr double kTileMinPpc = 2.0;
// and from as many work items (one per tile, or per 2048 particles) as keep the chip busy, or
// with so many particles a cell that the untiled push's atomics queue at the few nodes.  Step in us
// of both species, by tiles against without: 128 items, 32^3 x 8 59 / 51, 64 x 32 x 32 x 4 62 / 51;
// 256 items, 32^3 x 16 67 / 74, 64 x 32 x 32 x 8 69 / 70, 64 x 64 x 32 x 4 74 / 73; 512, 64^3 x 4
// 106 / 113.  8^3 x 40 41 / 35, 16^3 x 16 54 / 37, 16^3 x 64 56 / 76, 8^3 x 200 47 / 94.
constexpr size_t kTileMinItems = 256;
constexpr double kTileCrowdedPpc = 64.0;
constexpr size_t kTileMinTarget = 2048;  // particles of a work item, at least

struct ParamsND {
    int dims;
    int n[3];
    double L[3], d[3];
    double rd[3];  // 1 / d (cells_of)
    double dt, eps;
    double B[3];
    double rho_scale, inv_rho_scale;
    const double* E;  // interleaved: 2 doubles per node (2D) or 4 (3D)
    const float* E32; // FP32 form: float copy of E
    unsigned long long* rho_acc;
    // magnetic_field_profile: B piecewise linear along prof_axis (prof_rows = 0: uniform B)
    int prof_axis, prof_rows;
    const double* prof_c;  // coordinates
    const double* prof_v;  // rows x 3
    // walls: Dirichlet axes, particle boundaries (left, right, bottom, top,
    // back, front: 0 periodic, 1 absorbing, 2 reflecting) and the absorbed
    // counts [species][6]
    int wall[3];
    int pbc[6];
    unsigned long long* losses;
};

// TabulatedVectorField1D::evaluate, src/PrescribedField.cpp:89-113, at coordinate
// q inside the table (create checks that the table covers the domain).  A particle
// loaded outside the domain, or at a NaN, takes the nearest (the last) bracket.
__device__ __forceinline__ void profile_b(const ParamsND& p, double q, double B[3]) {
    const double* c = p.prof_c;
    const int n = p.prof_rows;
    if (q == __ldg(c)) {
        for (int a = 0; a < 3; ++a) B[a] = __ldg(p.prof_v + a);
        return;
    }
    if (q == __ldg(c + n - 1)) {
        for (int a = 0; a < 3; ++a) B[a] = __ldg(p.prof_v + 3 * (n - 1) + a);
        return;
    }
    int lo = 0, hi = n;  // std::upper_bound
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (q < __ldg(c + mid)) hi = mid; else lo = mid + 1;
    }
    const int right = min(max(lo, 1), n - 1);
    const int left = right - 1;
    const double f = (q - __ldg(c + left)) / (__ldg(c + right) - __ldg(c + left));
    for (int a = 0; a < 3; ++a) {
        const double l = __ldg(p.prof_v + 3 * left + a), r = __ldg(p.prof_v + 3 * right + a);
        B[a] = l + f * (r - l);
    }
}

// magnetic_field(cfg, position), src/Simulation2D.cpp:121-132, src/Simulation3D.cpp:109-118
__device__ __forceinline__ void field_b(const ParamsND& p, const double pos[3], double B[3]) {
    if (!p.prof_rows) {
        B[0] = p.B[0]; B[1] = p.B[1]; B[2] = p.B[2];
        return;
    }
    const int a = p.prof_axis;
    profile_b(p, a < p.dims ? (a == 0 ? pos[0] : (a == 1 ? pos[1] : pos[2])) : 0.0, B);
}

// FP32 form: each CIC weight is rounded to a multiple of 2^-23 and summed per
// species in 64-bit integers (runs of particles in one cell first add theirs in
// 32-bit registers and warp reductions: 8 particles per lane x 32 lanes x 2^23
// stays below 2^32), so the density does not depend on particle order.
constexpr float kWeightScale = 8388608.0f;  // 2^23

// wrap_periodic, src/FieldSolver.cpp:15-17, with the exact fast branch for
// |x| < 2L; a position already inside [0, L) stays as it is (the reference's
// (x + L) - L rounds its last bits away)
__device__ __forceinline__ double wrap_periodic(double x, double L) {
    if (x >= 0.0 && x < L) return x;
    if (!(fabs(x) < 2.0 * L)) return fmod(fmod(x, L) + L, L);
    const double r = x >= L ? x - L : (x <= -L ? x + L : x);
    const double y = r + L;
    return y >= 2.0 * L ? 0.0 : (y >= L ? y - L : y);
}

struct Axis {
    int i0, i1;
    double f;
};

// One axis of the periodic CIC stencil, src/Mesh2D.cpp:96-114, src/FieldSolver.cpp:936-960.
// The wrap leaves 0 <= x <= L, so the cell is at most n and i % n is a
// compare (a NaN, which converts to INT_MIN, lands in cell 0 through it); 64-bit
// remainders here were most of the FP64 push's instructions.
__device__ __forceinline__ Axis axis(double x, double L, double d, double rd, int n) {
    const double xp = wrap_periodic(x, L);
    const double g = cells_of(xp, d, rd);
    const int i = (int)floor(g);
    Axis a;
    a.f = g - (double)i;
    a.i0 = (unsigned)i < (unsigned)n ? i : 0;
    a.i1 = a.i0 + 1 == n ? 0 : a.i0 + 1;
    return a;
}

// One axis of the CIC stencil on a wall axis: clamp into [0, L], cell
// min(floor, n - 2), fraction clamped to [0, 1], src/Mesh2D.cpp:96-129,
// src/FieldSolver.cpp:926-960.  A NaN position lands on the lower wall: the
// conversion of a NaN to int is INT_MIN, which no index may come from.
__device__ __forceinline__ Axis axis_wall(double x, double L, double d, double rd, int n) {
    const double c = !(x >= 0.0) ? 0.0 : (L < x ? L : x);
    const double g = cells_of(c, d, rd);
    int i = (int)floor(g);
    if ((unsigned)i > (unsigned)(n - 2)) i = n - 2;
    double f = g - (double)i;
    f = f < 0.0 ? 0.0 : (f > 1.0 ? 1.0 : f);
    Axis a;
    a.i0 = i;
    a.i1 = i + 1;
    a.f = f;
    return a;
}

template <bool WALLS>
__device__ __forceinline__ Axis axis2(const ParamsND& p, int a, double x) {
    return (WALLS && p.wall[a]) ? axis_wall(x, p.L[a], p.d[a], p.rd[a], p.n[a])
                                : axis(x, p.L[a], p.d[a], p.rd[a], p.n[a]);
}

// 1 / node_area (node_volume) relative to an interior node: 2 on each
// wall-axis wall node (Mesh2D::node_area and Mesh3D::node_volume halve the
// cell there, src/Mesh2D.cpp:77-88, src/Mesh3D.cpp:52-60)
template <bool WALLS>
__device__ __forceinline__ double area_factor(const ParamsND& p, int a, int i) {
    return (WALLS && p.wall[a] && (i == 0 || i == p.n[a] - 1)) ? 2.0 : 1.0;
}

template <int DIM, bool WALLS = false>
__device__ __forceinline__ void gather(const ParamsND& p, const double pos[3], double e[3]) {
    const Axis ax = axis2<WALLS>(p, 0, pos[0]);
    const Axis ay = axis2<WALLS>(p, 1, pos[1]);
    const int nx = p.n[0];
    if (DIM == 2) {
        const double fx = ax.f, fy = ay.f;
        const double w00 = (1.0 - fx) * (1.0 - fy), w10 = fx * (1.0 - fy);
        const double w01 = (1.0 - fx) * fy, w11 = fx * fy;
        const double2* E2 = reinterpret_cast<const double2*>(p.E);
        const double2 e00 = __ldg(E2 + ay.i0 * nx + ax.i0), e10 = __ldg(E2 + ay.i0 * nx + ax.i1);
        const double2 e01 = __ldg(E2 + ay.i1 * nx + ax.i0), e11 = __ldg(E2 + ay.i1 * nx + ax.i1);
        e[0] = e00.x * w00 + e10.x * w10 + e01.x * w01 + e11.x * w11;
        e[1] = e00.y * w00 + e10.y * w10 + e01.y * w01 + e11.y * w11;
        e[2] = 0.0;
    } else {
        // interpolate_electric(Mesh3D&), src/FieldSolver.cpp:978-1038: loops z, y, x
        const Axis az = axis2<WALLS>(p, 2, pos[2]);
        const double wx[2] = {1.0 - ax.f, ax.f}, wy[2] = {1.0 - ay.f, ay.f}, wz[2] = {1.0 - az.f, az.f};
        const int ii[2] = {ax.i0, ax.i1}, jj[2] = {ay.i0, ay.i1}, kk[2] = {az.i0, az.i1};
        const double4* E4 = reinterpret_cast<const double4*>(p.E);
        e[0] = e[1] = e[2] = 0.0;
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int b = 0; b < 2; ++b)
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const double shape = wx[a] * wy[b] * wz[c];
                    const double4 ev = E4[((size_t)kk[c] * p.n[1] + jj[b]) * nx + ii[a]];
                    e[0] += ev.x * shape;
                    e[1] += ev.y * shape;
                    e[2] += ev.z * shape;
                }
    }
}

// boris_advance, src/Pusher.cpp:20-29
__device__ __forceinline__ void boris(double v[3], const double E[3], const double B[3], double qm, double dt) {
    const double h = 0.5 * qm * dt;
    const double vm0 = v[0] + h * E[0], vm1 = v[1] + h * E[1], vm2 = v[2] + h * E[2];
    const double t0 = h * B[0], t1 = h * B[1], t2v = h * B[2];
    const double t2 = t0 * t0 + t1 * t1 + t2v * t2v;
    const double sf = 2.0 / (1.0 + t2);
    const double s0 = sf * t0, s1 = sf * t1, s2 = sf * t2v;
    const double vp0 = vm0 + (vm1 * t2v - vm2 * t1);
    const double vp1 = vm1 + (vm2 * t0 - vm0 * t2v);
    const double vp2 = vm2 + (vm0 * t1 - vm1 * t0);
    const double vq0 = vm0 + (vp1 * s2 - vp2 * s1);
    const double vq1 = vm1 + (vp2 * s0 - vp0 * s2);
    const double vq2 = vm2 + (vp0 * s1 - vp1 * s0);
    v[0] = vq0 + h * E[0];
    v[1] = vq1 + h * E[1];
    v[2] = vq2 + h * E[2];
}

// CIC deposit of a warp's particles with one atomic per node per run of lanes
// that share a cell: particles are sorted by cell, so neighbouring lanes mostly
// hit the same 2^DIM nodes.  Each lane's fixed-point contributions are summed
// over its run with a segmented shuffle scan (integer, so the total does not
// depend on the order), and the run's last lane commits them.  All 32 lanes
// must call this; `valid` marks lanes that carry a particle.
template <int DIM, bool WALLS = false>
__device__ __forceinline__ void deposit_warp(const ParamsND& p, const SpeciesND& S, const double pos[3], bool valid) {
    constexpr int K = DIM == 2 ? 4 : 8;
    const int lane = threadIdx.x & 31;
    long long a[K];
    size_t node[K];
    unsigned cell = 0xFFFFFFFFu;
    if (valid) {
        const Axis ax = axis2<WALLS>(p, 0, pos[0]);
        const Axis ay = axis2<WALLS>(p, 1, pos[1]);
        const int nx = p.n[0];
        if (DIM == 2 && WALLS) {
            // q shape / node_area over the wall nodes' half cells, src/Mesh2D.cpp:131-142
            const double fx = ax.f, fy = ay.f;
            const double x0 = area_factor<WALLS>(p, 0, ax.i0), x1 = area_factor<WALLS>(p, 0, ax.i1);
            const double y0 = area_factor<WALLS>(p, 1, ay.i0), y1 = area_factor<WALLS>(p, 1, ay.i1);
            a[0] = to_fixed(S.dep * (1.0 - fx) * (1.0 - fy) * (x0 * y0), p.rho_scale);
            a[1] = to_fixed(S.dep * fx * (1.0 - fy) * (x1 * y0), p.rho_scale);
            a[2] = to_fixed(S.dep * (1.0 - fx) * fy * (x0 * y1), p.rho_scale);
            a[3] = to_fixed(S.dep * fx * fy * (x1 * y1), p.rho_scale);
            node[0] = (size_t)ay.i0 * nx + ax.i0;
            node[1] = (size_t)ay.i0 * nx + ax.i1;
            node[2] = (size_t)ay.i1 * nx + ax.i0;
            node[3] = (size_t)ay.i1 * nx + ax.i1;
            cell = (unsigned)node[0];
        } else if (DIM == 2) {
            const double fx = ax.f, fy = ay.f;
            a[0] = to_fixed(S.dep * (1.0 - fx) * (1.0 - fy), p.rho_scale);
            a[1] = to_fixed(S.dep * fx * (1.0 - fy), p.rho_scale);
            a[2] = to_fixed(S.dep * (1.0 - fx) * fy, p.rho_scale);
            a[3] = to_fixed(S.dep * fx * fy, p.rho_scale);
            node[0] = (size_t)ay.i0 * nx + ax.i0;
            node[1] = (size_t)ay.i0 * nx + ax.i1;
            node[2] = (size_t)ay.i1 * nx + ax.i0;
            node[3] = (size_t)ay.i1 * nx + ax.i1;
            cell = (unsigned)node[0];
        } else {
            const Axis az = axis2<WALLS>(p, 2, pos[2]);
            const double wx[2] = {1.0 - ax.f, ax.f}, wy[2] = {1.0 - ay.f, ay.f}, wz[2] = {1.0 - az.f, az.f};
            const int ii[2] = {ax.i0, ax.i1}, jj[2] = {ay.i0, ay.i1}, kk[2] = {az.i0, az.i1};
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int b = 0; b < 2; ++b)
#pragma unroll
                    for (int q = 0; q < 2; ++q) {
                        const int k = (c * 2 + b) * 2 + q;
                        if (WALLS) {
                            // q shape / node_volume over the wall nodes' half cells, src/Mesh3D.cpp:110-122
                            const double f = area_factor<WALLS>(p, 0, ii[q]) * area_factor<WALLS>(p, 1, jj[b]) *
                                             area_factor<WALLS>(p, 2, kk[c]);
                            a[k] = to_fixed(S.dep * (wx[q] * wy[b] * wz[c]) * f, p.rho_scale);
                        } else {
                            a[k] = to_fixed(S.dep * (wx[q] * wy[b] * wz[c]), p.rho_scale);
                        }
                        node[k] = ((size_t)kk[c] * p.n[1] + jj[b]) * nx + ii[q];
                    }
            cell = (unsigned)node[0];
        }
    } else {
#pragma unroll
        for (int k = 0; k < K; ++k) { a[k] = 0; node[k] = 0; }
    }
    const unsigned up = __shfl_up_sync(0xffffffffu, cell, 1);
    const bool head = (lane & 7) == 0 || up != cell;  // runs capped at 8 lanes: three scan steps
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const int start = 31 - __clz(heads & (0xFFFFFFFFu >> (31 - lane)));
    const bool tail = lane == 31 || ((heads >> (lane + 1)) & 1u);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        long long v = a[k];
#pragma unroll
        for (int d = 1; d < 8; d <<= 1) {
            const long long t = __shfl_up_sync(0xffffffffu, v, d);
            if (lane - d >= start) v += t;
        }
        if (tail && valid) atomicAdd(p.rho_acc + node[k], (unsigned long long)v);
    }
}

enum : int { kPushStep = 0, kPushDepositOnly = 1, kPushInitHalf = 2, kPushSync = 3 };

// reflect_coordinate, src/Simulation2D.cpp:43-54 (a particle crosses at most a
// few domain lengths per step; the bound only guards against runaway input)
__device__ __forceinline__ void reflect_coordinate(double& c, double& v, double L) {
    for (int guard = 0; guard < (1 << 20) && (c < 0.0 || c > L); ++guard) {
        if (c < 0.0) { c = -c; v = -v; }
        else { c = 2.0 * L - c; v = -v; }
    }
}

// Simulation2D::apply_particle_boundaries, src/Simulation2D.cpp:1309-1335, and
// Simulation3D::apply_particle_boundaries, src/Simulation3D.cpp:309-340, with
// apply_lower/upper_boundary (src/Simulation2D.cpp:57-97, src/Simulation3D.cpp:42-83):
// sides left, right, bottom, top (, back, front); returns the absorbing side, or -1.
template <int DIM>
__device__ __forceinline__ int apply_walls(const ParamsND& p, double x[3], double v[3]) {
#pragma unroll
    for (int side = 0; side < 2 * DIM; ++side) {
        const int a = side >> 1;
        double& c = x[a];
        const double L = p.L[a];
        if ((side & 1) == 0 ? c >= 0.0 : c <= L) continue;
        const int kind = p.pbc[side];
        if (kind == 1) return side;
        if (kind == 2) reflect_coordinate(c, v[a], L);
        else c = wrap_periodic(c, L);
    }
    return -1;
}

// One particle per thread.  Modes: deposit only (initialize/resume), half-step
// initialisation from v (initialize_{boris,leapfrog}_half_step) and
// synchronisation into v.  (The full step is k_push_run.)
template <int DIM, bool BORIS, int MODE, bool WALLS = false>
__global__ void __launch_bounds__(kThreads) k_push(ParamsND p, SpeciesND S, int buf) {
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    const bool valid = i < S.n && (!WALLS || !S.alive[buf] || S.alive[buf][i]);
    if (MODE == kPushInitHalf || MODE == kPushSync) {
        if (!valid) return;
    } else if (blockIdx.x * kThreads + (threadIdx.x & ~31u) >= S.n) {
        return;  // whole warp past the end
    }
    const unsigned j = valid ? i : 0u;
    double pos[3] = {S.pos[buf][0][j], S.pos[buf][1][j], DIM == 3 ? S.pos[buf][2][j] : 0.0};
    if (MODE == kPushDepositOnly) {
        deposit_warp<DIM, WALLS>(p, S, pos, valid);
        return;
    }
    double e[3];
    gather<DIM, WALLS>(p, pos, e);
    const unsigned vi = WALLS && (MODE == kPushInitHalf || MODE == kPushSync) ? S.id[buf][j] : j;
    if (MODE == kPushInitHalf) {
        double v[3] = {S.v[0][vi], S.v[1][vi], S.v[2][vi]};
        if (BORIS) {
            double Bp[3];
            field_b(p, pos, Bp);
            boris(v, e, Bp, S.qm, -0.5 * p.dt);
        } else {
            // initialize_leapfrog_half_step, src/Pusher.cpp:88-92, :152-156
            for (int a = 0; a < DIM; ++a) v[a] = v[a] - 0.5 * S.qm * e[a] * p.dt;
        }
        for (int a = 0; a < 3; ++a) S.vh[buf][a][i] = v[a];
        return;
    }
    double vh[3] = {S.vh[buf][0][j], S.vh[buf][1][j], S.vh[buf][2][j]};
    if (MODE == kPushSync) {
        if (BORIS) {
            double Bp[3];
            field_b(p, pos, Bp);
            boris(vh, e, Bp, S.qm, 0.5 * p.dt);
        } else {
            // synchronize_leapfrog, src/Pusher.cpp:131-135, :176-180
            for (int a = 0; a < DIM; ++a) vh[a] = vh[a] + 0.5 * S.qm * e[a] * p.dt;
        }
        for (int a = 0; a < 3; ++a) S.v[a][vi] = vh[a];
        return;
    }
}

// boris_advance with the species' precomputed h, t and s (uniform B): the same
// operations as boris(), whose t, s and division depend on B only
__device__ __forceinline__ void boris_uniform(double v[3], const double E[3], const SpeciesND& S) {
    const double h = S.bh;
    const double vm0 = v[0] + h * E[0], vm1 = v[1] + h * E[1], vm2 = v[2] + h * E[2];
    const double vp0 = vm0 + (vm1 * S.bt[2] - vm2 * S.bt[1]);
    const double vp1 = vm1 + (vm2 * S.bt[0] - vm0 * S.bt[2]);
    const double vp2 = vm2 + (vm0 * S.bt[1] - vm1 * S.bt[0]);
    const double vq0 = vm0 + (vp1 * S.bs[2] - vp2 * S.bs[1]);
    const double vq1 = vm1 + (vp2 * S.bs[0] - vp0 * S.bs[2]);
    const double vq2 = vm2 + (vp0 * S.bs[1] - vp1 * S.bs[0]);
    v[0] = vq0 + h * E[0];
    v[1] = vq1 + h * E[1];
    v[2] = vq2 + h * E[2];
}

enum : int { kNoField = 0, kUniformField = 1, kProfileField = 2 };

// The FP64 step push: kick, drift, particle boundaries and CIC deposit of
// ITEMS consecutive particles per thread (1, or kRunItems).  Particles are sorted by cell,
// so the fixed-point contributions of a run of equal cells are summed in registers,
// a run that ends inside the thread is committed with one atomic per node, and each lane's
// last run joins a segmented sum over the lanes that end in the same cell.  The
// field is read from L1 for each particle: keeping a cell's nodes for the next particle
// took 48 registers and a third of the warps (64^3: 436 us a step against 384).
// The state moves as 16-byte vectors.  Contributions are integers, so the
// density does not depend on how particles are grouped.
// Against one particle per thread with 64-bit index remainders (both species, per
// step): 2 x 1 M particles on 256 x 128, 81 -> 63 us; 2 x 4.2 M on 64^3,
// 483 -> 384 us (bound by load latency and, between sorts, by the
// deposit's global atomics); walls, 2 x 2 M on 512 x 513, 161 -> 113 us and
// 2 x 4.2 M on 129^3, 680 -> 490 us (these also sorted by cell now).
constexpr int kRunItems = 2;
// Up to this many particles each has its own thread: all of them are resident at once, and
// two particles in a thread only lengthen its chain.  Push of both species, us a step, one
// against two a thread: 16^3 x 4 16.5 / 21.1, 256 x 128 x 8 on the line's far side 23.0 / 23.6,
// walls 9 x 8 x 10 15.2 / 18.3, 17^3 x 2 19.7 / 28.5, 33^3 x 2 23.3 / 29.9, 33^3 x 4 38.0 / 36.1.
constexpr unsigned kOneItemMax = 148 * 3 * kThreads;

// One buffer of the FP64 state, by kernel argument (an index into the species'
// arrays costs every access its pointer's load).
struct State64 {
    double* pos[3];
    double* vh[3];
    uint8_t* alive;
    const unsigned* live_end;
};

template <int DIM, int BKIND, bool WALLS, int ITEMS>
__global__ void __launch_bounds__(kThreads, DIM == 2 ? 4 : 3) k_push_run(ParamsND p, SpeciesND S, State64 A) {
    constexpr int NN = DIM == 2 ? 4 : 8;
    const unsigned first = (blockIdx.x * kThreads + threadIdx.x) * ITEMS;
    const int lane = threadIdx.x & 31;
    // whole warp past the end, or past the particles that were alive at the last sort
    const unsigned warp_first = (blockIdx.x * kThreads + (threadIdx.x & ~31u)) * ITEMS;
    if (warp_first >= (WALLS && A.live_end ? min(S.n, *A.live_end) : S.n)) return;
    const int nx = p.n[0], ny = p.n[1];
    double x[ITEMS][3], v[ITEMS][3];
    bool live[ITEMS];
    const bool full = ITEMS == 2 && first + ITEMS <= S.n;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        double2 q{0.0, 0.0}, w{0.0, 0.0};
        if (full) {
            if (a < DIM) q = __ldcs(reinterpret_cast<const double2*>(A.pos[a] + first));
            w = __ldcs(reinterpret_cast<const double2*>(A.vh[a] + first));
        } else if (first < S.n) {
            if (a < DIM) q.x = A.pos[a][first];
            w.x = A.vh[a][first];
        }
        x[0][a] = q.x;
        v[0][a] = w.x;
        if (ITEMS == 2) { x[ITEMS - 1][a] = q.y; v[ITEMS - 1][a] = w.y; }
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k)
        live[k] = first + k < S.n && (!WALLS || !A.alive || A.alive[first + k]);
    const unsigned kNoCell = 0xFFFFFFFFu;
    unsigned rcell = kNoCell;  // cell of the current deposit run
    long long racc[NN];
    unsigned rnode[3] = {0u, 0u, 0u};  // steps from the run's first node to its upper x, y, z neighbours
#pragma unroll
    for (int j = 0; j < NN; ++j) racc[j] = 0;
    auto commit = [&]() {
#pragma unroll
        for (int j = 0; j < NN; ++j) {
            const unsigned node = rcell + ((j & 1) ? rnode[0] : 0u) + ((j & 2) ? rnode[1] : 0u) + ((j & 4) ? rnode[2] : 0u);
            if (racc[j]) atomicAdd(p.rho_acc + node, (unsigned long long)racc[j]);
        }
    };
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if (!live[k]) continue;
        const Axis gx = axis2<WALLS>(p, 0, x[k][0]), gy = axis2<WALLS>(p, 1, x[k][1]);
        const Axis gz = DIM == 3 ? axis2<WALLS>(p, 2, x[k][DIM - 1]) : Axis{0, 0, 0.0};
        // field at node j of the cell
        auto node_field = [&](int j, double* out) {
            const unsigned g = ((unsigned)((j & 4) ? gz.i1 : gz.i0) * ny + ((j & 2) ? gy.i1 : gy.i0)) * nx +
                               ((j & 1) ? gx.i1 : gx.i0);
            if (DIM == 2) {
                const double2 q = __ldg(reinterpret_cast<const double2*>(p.E) + g);
                out[0] = q.x; out[1] = q.y;
            } else {
                const double2* E = reinterpret_cast<const double2*>(p.E) + 2 * (size_t)g;
                const double2 q = __ldg(E);
                out[0] = q.x; out[1] = q.y;
                out[DIM - 1] = __ldg(reinterpret_cast<const double*>(E + 1));
            }
        };
        double e[3] = {0.0, 0.0, 0.0};
        if (DIM == 2) {
            double en[NN][DIM];
#pragma unroll
            for (int j = 0; j < NN; ++j) node_field(j, en[j]);
            const double fx = gx.f, fy = gy.f;
            const double w00 = (1.0 - fx) * (1.0 - fy), w10 = fx * (1.0 - fy), w01 = (1.0 - fx) * fy, w11 = fx * fy;
            e[0] = en[0][0] * w00 + en[1][0] * w10 + en[2][0] * w01 + en[3][0] * w11;
            e[1] = en[0][1] * w00 + en[1][1] * w10 + en[2][1] * w01 + en[3][1] * w11;
        } else {
            // interpolate_electric(Mesh3D&), src/FieldSolver.cpp:978-1038: loops z, y, x
            const double wx[2] = {1.0 - gx.f, gx.f}, wy[2] = {1.0 - gy.f, gy.f}, wz[2] = {1.0 - gz.f, gz.f};
#pragma unroll
            for (int j = 0; j < NN; ++j) {
                const double shape = wx[j & 1] * wy[(j >> 1) & 1] * wz[(j >> 2) & 1];
                double q[3];
                node_field(j, q);
#pragma unroll
                for (int a = 0; a < DIM; ++a) e[a] += q[a] * shape;
            }
        }
        // kick_boris / kick_leapfrog + drift_leapfrog, src/Pusher.cpp:109-128, :162-174
        if (BKIND == kUniformField) {
            boris_uniform(v[k], e, S);
        } else if (BKIND == kProfileField) {
            double Bp[3];
            field_b(p, x[k], Bp);
            boris(v[k], e, Bp, S.qm, p.dt);
        } else {
#pragma unroll
            for (int a = 0; a < DIM; ++a) v[k][a] += S.qm * e[a] * p.dt;
        }
        if (WALLS) {
#pragma unroll
            for (int a = 0; a < DIM; ++a) x[k][a] = x[k][a] + v[k][a] * p.dt;
            const int side = apply_walls<DIM>(p, x[k], v[k]);
            if (side >= 0) {
                A.alive[first + k] = 0;
                atomicAdd(p.losses + 6 * S.index + side, 1ull);
                continue;
            }
        } else {
#pragma unroll
            for (int a = 0; a < DIM; ++a) {
                const double c = x[k][a] + v[k][a] * p.dt;
                // periodic particle boundary: wrap only outside [0, L], src/Simulation2D.cpp:57-97
                x[k][a] = (c >= 0.0 && c <= p.L[a]) ? c : wrap_periodic(c, p.L[a]);
            }
        }
        // deposit at the pushed position into the run of its cell (the contributions of deposit_warp)
        const Axis ax = axis2<WALLS>(p, 0, x[k][0]), ay = axis2<WALLS>(p, 1, x[k][1]);
        const Axis az = DIM == 3 ? axis2<WALLS>(p, 2, x[k][DIM - 1]) : Axis{0, 0, 0.0};
        const unsigned c1 = ((unsigned)az.i0 * ny + ay.i0) * nx + ax.i0;
        if (c1 != rcell) {
            if (rcell != kNoCell) commit();
            rcell = c1;
            rnode[0] = (unsigned)(ax.i1 - ax.i0);
            rnode[1] = (unsigned)((ay.i1 - ay.i0) * nx);
            if (DIM == 3) rnode[2] = (unsigned)((az.i1 - az.i0) * ny * nx);
#pragma unroll
            for (int j = 0; j < NN; ++j) racc[j] = 0;
        }
        const double ux[2] = {1.0 - ax.f, ax.f}, uy[2] = {1.0 - ay.f, ay.f}, uz[2] = {1.0 - az.f, az.f};
        // a cell on a wall (the volume factors are 1 elsewhere)
        const bool edge = WALLS && (ax.i0 == 0 || ax.i1 == nx - 1 || ay.i0 == 0 || ay.i1 == ny - 1 ||
                                    (DIM == 3 && (az.i0 == 0 || az.i1 == p.n[2] - 1)));
#pragma unroll
        for (int j = 0; j < NN; ++j) {
            double c = DIM == 2 ? S.dep * ux[j & 1] * uy[(j >> 1) & 1]
                                : S.dep * (ux[j & 1] * uy[(j >> 1) & 1] * uz[(j >> 2) & 1]);
            if (WALLS && edge) {  // q shape / node volume over the wall nodes' half cells
                double f = area_factor<WALLS>(p, 0, (j & 1) ? ax.i1 : ax.i0) *
                           area_factor<WALLS>(p, 1, (j & 2) ? ay.i1 : ay.i0);
                if (DIM == 3) f *= area_factor<WALLS>(p, 2, (j & 4) ? az.i1 : az.i0);
                c *= f;
            }
            racc[j] += to_fixed(c, p.rho_scale);
        }
    }
    // the state back, in place
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        if (WALLS && !live[0] && !live[ITEMS - 1]) break;  // nothing of absorbed particles changed
        if (full) {
            if (a < DIM) __stcs(reinterpret_cast<double2*>(A.pos[a] + first), make_double2(x[0][a], x[ITEMS - 1][a]));
            __stcs(reinterpret_cast<double2*>(A.vh[a] + first), make_double2(v[0][a], v[ITEMS - 1][a]));
        } else if (first < S.n) {
            if (a < DIM) A.pos[a][first] = x[0][a];
            A.vh[a][first] = v[0][a];
        }
    }
    // Each lane's last run, summed over segments of at most RSEG lanes that end in the same
    // cell; a warp with few runs (hundreds of particles a cell) sums whole runs, or
    // neighbouring warps' commits queue up at the same few nodes (32 x 32 periodic,
    // 2 x 500,000 particles: push 112 -> 106 us a step).
    constexpr int RSEG = DIM == 3 ? 4 : 8;
    constexpr unsigned kSegments = DIM == 3 ? 0x11111111u : 0x01010101u;  // the segments' first lanes
    constexpr int kFewRuns = 8;
    const unsigned prev = __shfl_up_sync(0xffffffffu, rcell, 1);
    const unsigned runs = __ballot_sync(0xffffffffu, lane == 0 || prev != rcell);
    const bool few = __popc(runs) <= kFewRuns;
    const unsigned heads = few ? runs : runs | kSegments;
    const int start = 31 - __clz(heads & (0xFFFFFFFFu >> (31 - lane)));
    const bool tail = lane == 31 || ((heads >> (lane + 1)) & 1u);
    auto add_up = [&](int d) {
#pragma unroll
        for (int j = 0; j < NN; ++j) {
            const long long t = __shfl_up_sync(0xffffffffu, racc[j], d);
            if (lane - d >= start) racc[j] += t;
        }
    };
#pragma unroll
    for (int d = 1; d < RSEG; d <<= 1) add_up(d);
    if (few)  // the same for the whole warp
#pragma unroll
        for (int d = RSEG; d < 32; d <<= 1) add_up(d);
    if (tail && rcell != kNoCell) commit();
}

// walls: fixed-point density to FP64 (the accumulator is cleared for the
// next deposit)
__global__ void k_walls_rho(unsigned long long* __restrict__ acc, double* __restrict__ rho, size_t N,
                            double inv_scale) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        rho[i] = (double)(long long)acc[i] * inv_scale;
        acc[i] = 0ull;
    }
}

// ---- FP32 particle form ---------------------------------------------------------
//
// A particle is a packed cell index (10 bits per axis), float offsets in
// [0, 1) inside that cell and float velocities: 24 B (2D3V) or 28 B (3D3V) of
// state instead of 40/48 B.  Positions never leave cell units, so the gather and
// the deposit need no division and no wrap; the field solve, the fixed-point
// density and the diagnostics stay FP64.

__device__ __forceinline__ void unpack_cell(unsigned c, int& ix, int& iy, int& iz) {
    ix = (int)(c & 1023u);
    iy = (int)((c >> 10) & 1023u);
    iz = (int)(c >> 20);
}
__device__ __forceinline__ unsigned pack_cell(int ix, int iy, int iz) {
    return (unsigned)ix | ((unsigned)iy << 10) | ((unsigned)iz << 20);
}

template <int DIM>
__device__ __forceinline__ void gather32(const ParamsND& p, int ix, int iy, int iz, const float f[3], float e[3]) {
    const int nx = p.n[0], ny = p.n[1];
    const int ix1 = (ix + 1) & (nx - 1), iy1 = (iy + 1) & (ny - 1);
    const float wx[2] = {1.0f - f[0], f[0]}, wy[2] = {1.0f - f[1], f[1]};
    if (DIM == 2) {
        const float2* E = reinterpret_cast<const float2*>(p.E32);
        const float2 a = __ldg(E + iy * nx + ix), b = __ldg(E + iy * nx + ix1), c = __ldg(E + iy1 * nx + ix),
                     d = __ldg(E + iy1 * nx + ix1);
        const float w00 = wx[0] * wy[0], w10 = wx[1] * wy[0], w01 = wx[0] * wy[1], w11 = wx[1] * wy[1];
        e[0] = fmaf(a.x, w00, fmaf(b.x, w10, fmaf(c.x, w01, d.x * w11)));
        e[1] = fmaf(a.y, w00, fmaf(b.y, w10, fmaf(c.y, w01, d.y * w11)));
        e[2] = 0.0f;
    } else {
        const int iz1 = (iz + 1) & (p.n[2] - 1);
        const float wz[2] = {1.0f - f[2], f[2]};
        const int xx[2] = {ix, ix1}, yy[2] = {iy, iy1}, zz[2] = {iz, iz1};
        const float4* E = reinterpret_cast<const float4*>(p.E32);
        e[0] = e[1] = e[2] = 0.0f;
#pragma unroll
        for (int c = 0; c < 2; ++c)
#pragma unroll
            for (int b = 0; b < 2; ++b) {
                const float wyz = wy[b] * wz[c];
                const size_t row = ((size_t)zz[c] * ny + yy[b]) * nx;
#pragma unroll
                for (int a = 0; a < 2; ++a) {
                    const float w = wx[a] * wyz;
                    const float4 v = __ldg(E + row + xx[a]);
                    e[0] = fmaf(v.x, w, e[0]);
                    e[1] = fmaf(v.y, w, e[1]);
                    e[2] = fmaf(v.z, w, e[2]);
                }
            }
    }
}

// Boris rotation in float (same algebra as boris_advance, src/Pusher.cpp:20-29)
__device__ __forceinline__ void boris32(float v[3], const float e[3], float h, const float t[3], const float s[3]) {
    const float vm0 = fmaf(h, e[0], v[0]), vm1 = fmaf(h, e[1], v[1]), vm2 = fmaf(h, e[2], v[2]);
    const float vp0 = vm0 + fmaf(vm1, t[2], -vm2 * t[1]);
    const float vp1 = vm1 + fmaf(vm2, t[0], -vm0 * t[2]);
    const float vp2 = vm2 + fmaf(vm0, t[1], -vm1 * t[0]);
    v[0] = fmaf(h, e[0], vm0 + fmaf(vp1, s[2], -vp2 * s[1]));
    v[1] = fmaf(h, e[1], vm1 + fmaf(vp2, s[0], -vp0 * s[2]));
    v[2] = fmaf(h, e[2], vm2 + fmaf(vp0, s[1], -vp1 * s[0]));
}

// FP32 form: the Boris rotation vectors t = (q/m dt/2) B and s = 2 t / (1 + t^2)
// of a particle, from its cell and offset when B is tabulated (the species'
// precomputed pair otherwise), in the same FP64 expression as the species' pair.
__device__ __forceinline__ void boris_ts32(const ParamsND& p, const SpeciesND& S, int ix, int iy, int iz,
                                           const float f[3], float tb[3], float sb[3]) {
    if (!p.prof_rows) {
        for (int a = 0; a < 3; ++a) { tb[a] = S.tb[a]; sb[a] = S.sb[a]; }
        return;
    }
    const int a = p.prof_axis;
    double q = 0.0;
    if (a < p.dims) {
        const int cell = a == 0 ? ix : (a == 1 ? iy : iz);
        const float off = a == 0 ? f[0] : (a == 1 ? f[1] : f[2]);
        q = ((double)cell + (double)off) * p.d[a];
    }
    double B[3];
    profile_b(p, q, B);
    const double hq = 0.5 * S.qm * p.dt;
    double t2 = 0.0;
    for (int c = 0; c < 3; ++c) t2 += (hq * B[c]) * (hq * B[c]);
    for (int c = 0; c < 3; ++c) {
        tb[c] = (float)(hq * B[c]);
        sb[c] = (float)(2.0 * hq * B[c] / (1.0 + t2));
    }
}

// Moves one axis by `disp` cells: integer carry into the periodic cell index.
__device__ __forceinline__ void advance(float& f, int& i, float disp, int n) {
    float g = f + disp;
    const float k = floorf(g);
    g -= k;
    int ki = (int)k;
    if (g >= 1.0f) { g -= 1.0f; ki += 1; }
    f = g;
    i = (i + ki) & (n - 1);
}

// Runs of lanes that share a cell (particles are sorted by cell) add their
// 2^-25-quantised weights with a converged segmented shuffle scan; runs are
// capped at SEG lanes (32 x 2^25 < 2^32, so a run's sum fits 32 bits): SEG = 32
// where a warp usually sits in one or two cells (2D, 64 particles per cell),
// 8 where it spans several (3D).  The last lane of each run commits its sums
// with one 64-bit atomic per node.
template <int DIM>
__device__ __forceinline__ void deposit32_warp(const ParamsND& p, unsigned long long* acc, bool valid, int ix, int iy,
                                               int iz, const float f[3]) {
    constexpr int SEG = DIM == 2 ? 32 : 8;
    const int lane = threadIdx.x & 31;
    const int nx = p.n[0], ny = p.n[1];
    const unsigned key = valid ? (((unsigned)iz * ny + iy) * nx + ix) : 0xFFFFFFFFu;
    const unsigned prev = __shfl_up_sync(0xffffffffu, key, 1);
    const bool head = (lane & (SEG - 1)) == 0 || prev != key;
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const int start = 31 - __clz(heads & (0xFFFFFFFFu >> (31 - lane)));
    const bool tail = lane == 31 || ((heads >> (lane + 1)) & 1u);
    const int ix1 = (ix + 1) & (nx - 1), iy1 = (iy + 1) & (ny - 1);
    const int iz1 = DIM == 3 ? (iz + 1) & (p.n[2] - 1) : 0;
    const int xx[2] = {ix, ix1}, yy[2] = {iy, iy1}, zz[2] = {iz, iz1};
    const float wx[2] = {1.0f - f[0], f[0]}, wy[2] = {1.0f - f[1], f[1]};
    const float wz[2] = {DIM == 3 ? 1.0f - f[2] : 1.0f, DIM == 3 ? f[2] : 0.0f};
#pragma unroll
    for (int c = 0; c < (DIM == 3 ? 2 : 1); ++c)
#pragma unroll
        for (int b = 0; b < 2; ++b)
#pragma unroll
            for (int a = 0; a < 2; ++a) {
                unsigned q = valid ? (unsigned)__float2int_rn(wx[a] * wy[b] * wz[c] * kWeightScale) : 0u;
#pragma unroll
                for (int d = 1; d < SEG; d <<= 1) {
                    const unsigned t = __shfl_up_sync(0xffffffffu, q, d);
                    if (lane - d >= start) q += t;
                }
                if (tail && valid && q)
                    atomicAdd(acc + ((size_t)zz[c] * ny + yy[b]) * nx + xx[a], (unsigned long long)q);
            }
}

template <int DIM, bool BORIS, int MODE>
__global__ void __launch_bounds__(kThreads) k_push32(ParamsND p, SpeciesND S, int buf, unsigned long long* acc) {
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    const bool valid = i < S.n;
    if ((MODE == kPushStep || MODE == kPushDepositOnly) && blockIdx.x * kThreads + (threadIdx.x & ~31u) >= S.n)
        return;  // whole warp past the end
    int ix = 0, iy = 0, iz = 0;
    float f[3] = {0.0f, 0.0f, 0.0f}, v[3] = {0.0f, 0.0f, 0.0f};
    if (valid) {  // streamed once per step: evict-first, so L1 keeps the field
        unpack_cell(__ldcs(&S.cell[buf][i]), ix, iy, iz);
        for (int a = 0; a < DIM; ++a) f[a] = __ldcs(&S.off[buf][a][i]);
        for (int a = 0; a < 3; ++a) v[a] = __ldcs(&S.vel[buf][a][i]);
    }
    if (MODE == kPushStep || MODE == kPushInitHalf || MODE == kPushSync) {
        float e[3] = {0.0f, 0.0f, 0.0f};
        if (valid) gather32<DIM>(p, ix, iy, iz, f, e);
        if (MODE == kPushInitHalf || MODE == kPushSync) {
            if (!valid) return;
            float w[3] = {(float)S.v[0][i], (float)S.v[1][i], (float)S.v[2][i]};
            float* vv = MODE == kPushInitHalf ? w : v;
            const float h = MODE == kPushInitHalf ? -0.5f * S.hqmdt : 0.5f * S.hqmdt;
            if (BORIS) {
                float t[3], sb[3], tp[3], sp[3];
                boris_ts32(p, S, ix, iy, iz, f, tp, sp);
                float t2 = 0.0f;
                for (int a = 0; a < 3; ++a) { t[a] = tp[a] * (MODE == kPushInitHalf ? -0.5f : 0.5f); t2 = fmaf(t[a], t[a], t2); }
                for (int a = 0; a < 3; ++a) sb[a] = 2.0f * t[a] / (1.0f + t2);
                boris32(vv, e, h, t, sb);
            } else {
                for (int a = 0; a < DIM; ++a) vv[a] = fmaf(2.0f * h, e[a], vv[a]);
            }
            if (MODE == kPushInitHalf) {
                for (int a = 0; a < 3; ++a) S.vel[buf][a][i] = vv[a];
            } else {
                for (int a = 0; a < 3; ++a) S.v[a][i] = (double)vv[a];
            }
            return;
        }
        // kick + drift
        if (BORIS) {
            float tp[3], sp[3];
            boris_ts32(p, S, ix, iy, iz, f, tp, sp);
            boris32(v, e, S.hqmdt, tp, sp);
        } else {
            for (int a = 0; a < DIM; ++a) v[a] = fmaf(S.qmdt, e[a], v[a]);
        }
        int* idx[3] = {&ix, &iy, &iz};
        for (int a = 0; a < DIM; ++a) advance(f[a], *idx[a], v[a] * S.drift[a], p.n[a]);
        if (valid) {
            __stcs(&S.cell[buf][i], pack_cell(ix, iy, iz));
            for (int a = 0; a < DIM; ++a) __stcs(&S.off[buf][a][i], f[a]);
            for (int a = 0; a < 3; ++a) __stcs(&S.vel[buf][a][i], v[a]);
        }
    }
    // ---- deposit ----
    deposit32_warp<DIM>(p, acc, valid, ix, iy, iz, f);
}

// The step push of the FP32 form with ITEMS particles per thread: all of the
// thread's particle loads are issued before the first gather, so each warp
// keeps ITEMS times the bytes in flight (the single-particle form leaves HBM
// latency-bound).  Slice k of the CTA is the contiguous block of kThreads
// particles at base + k * kThreads, so each warp still deposits runs of
// consecutive (cell-sorted) particles.
// PROF: B tabulated along one axis (a separate instantiation, so the uniform-B
// kernels keep their register budget).
template <int DIM, bool BORIS, int ITEMS, bool PROF>
__global__ void __launch_bounds__(kThreads) k_push32_step(ParamsND p, SpeciesND S, int buf, unsigned long long* acc) {
    const unsigned base = blockIdx.x * (ITEMS * kThreads);
    const unsigned tid = threadIdx.x;
    unsigned cl[ITEMS];
    float fo[ITEMS][3], vv[ITEMS][3];
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const unsigned i = base + k * kThreads + tid;
        const bool ok = i < S.n;
        cl[k] = ok ? __ldcs(&S.cell[buf][i]) : 0u;
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            fo[k][a] = (ok && a < DIM) ? __ldcs(&S.off[buf][a][i]) : 0.0f;
            vv[k][a] = ok ? __ldcs(&S.vel[buf][a][i]) : 0.0f;
        }
    }
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        const unsigned i = base + k * kThreads + tid;
        if (base + k * kThreads + (tid & ~31u) >= S.n) continue;  // whole warp past the end
        const bool valid = i < S.n;
        int ix = 0, iy = 0, iz = 0;
        unpack_cell(cl[k], ix, iy, iz);
        float* f = fo[k];
        float* v = vv[k];
        float e[3] = {0.0f, 0.0f, 0.0f};
        if (valid) gather32<DIM>(p, ix, iy, iz, f, e);
        // kick + drift, src/Pusher.cpp:109-128, :162-174
        if (BORIS && PROF) {
            float tp[3], sp[3];
            boris_ts32(p, S, ix, iy, iz, f, tp, sp);
            boris32(v, e, S.hqmdt, tp, sp);
        } else if (BORIS) {
            boris32(v, e, S.hqmdt, S.tb, S.sb);
        } else {
            for (int a = 0; a < DIM; ++a) v[a] = fmaf(S.qmdt, e[a], v[a]);
        }
        int* idx[3] = {&ix, &iy, &iz};
        for (int a = 0; a < DIM; ++a) advance(f[a], *idx[a], v[a] * S.drift[a], p.n[a]);
        if (valid) {
            __stcs(&S.cell[buf][i], pack_cell(ix, iy, iz));
            for (int a = 0; a < DIM; ++a) __stcs(&S.off[buf][a][i], f[a]);
            for (int a = 0; a < 3; ++a) __stcs(&S.vel[buf][a][i], v[a]);
        }
        deposit32_warp<DIM>(p, acc, valid, ix, iy, iz, f);
    }
}

// One buffer of the FP32 state, by kernel argument (an index into the species'
// arrays costs every access its pointer's load) ...
struct State32 {
    unsigned* cell;
    float* off[3];
    float* vel[3];
    __device__ __forceinline__ unsigned* cells() const { return cell; }
    __device__ __forceinline__ float* offs(int a) const { return off[a]; }
    __device__ __forceinline__ float* vels(int a) const { return vel[a]; }
};
// ... or by that index, for the 3D run push, where the pointers' registers cost more: 64 registers
// and no spills against 80 (128^3, 2 x 3.1 M particles: push 214 against 227 us a step)
struct Buffer32 {
    const SpeciesND& S;
    int buf;
    __device__ __forceinline__ unsigned* cells() const { return S.cell[buf]; }
    __device__ __forceinline__ float* offs(int a) const { return S.off[buf][a]; }
    __device__ __forceinline__ float* vels(int a) const { return S.vel[buf][a]; }
};

// 2D: the CTA's deposit into a box of nodes in shared memory (kDBoxX cells
// along x from x0 and the cell rows y0 .. y0 + 2 around the CTA's middle
// particle), flushed with one 64-bit global atomic per touched node: a
// particle that left its sorted neighbours then adds into shared memory
// instead of committing its own global atomics (which, on the few nodes a CTA
// touches, serialise in L2).  Each node's weight sum is one 32-bit word (native
// shared atomics); an add that wraps it carries 2^32 into the global sum at once, so
// the sums are exact.  Commits outside the box go to global memory as before.
// (512^2, 2 x 16.8 M particles, per step: 368 us with two 16-bit halves and the box's place
// broadcast by one thread, 336 now.)
// (In 3D the box around a CTA's 64 cells needs 1552 nodes; zeroing and
// flushing them and the kernel's extra registers cost more than the atomics
// saved, so 3D commits straight to global memory.)
constexpr int kDBoxX = 48;
constexpr int kDBoxNodes = (kDBoxX + 1) * 4;
struct DepositBox {
    unsigned* sum;
    int x0, y0;
};

// The step push of the FP32 form with ITEMS consecutive particles per thread
// (loaded and stored as vectors).  Particles are sorted by cell, so a thread's
// particles mostly share a cell: the field at the cell's nodes is fetched once
// per run of equal cells, and the CIC weights of a run are summed in registers
// (the deposit of src/Mesh2D.cpp:90-144 / src/Mesh3D.cpp:62-126 at the pushed
// positions).  A run that ends inside the thread is committed with one 64-bit
// atomic per node; each lane's last run joins a warp-segmented sum over the
// lanes holding the same cell, whose last lane commits it.
template <int DIM, bool BORIS, int ITEMS, bool PROF, class State>
__device__ __forceinline__ void push_run(const ParamsND& p, const SpeciesND& S, const State& A,
                                         unsigned long long* acc, const DepositBox& box) {
    constexpr int NN = DIM == 2 ? 4 : 8;  // nodes of a cell
    const unsigned first = (blockIdx.x * kThreads + threadIdx.x) * ITEMS;
    const int lane = threadIdx.x & 31;
    if ((blockIdx.x * kThreads + (threadIdx.x & ~31u)) * ITEMS >= S.n) {  // whole warp past the end
        if (DIM == 2) __syncthreads();
        return;
    }
    const int nx = p.n[0], ny = p.n[1], nz = DIM == 3 ? p.n[2] : 1;
    unsigned cl[ITEMS];
    float fo[ITEMS][3], vv[ITEMS][3];
    const bool full = first + ITEMS <= S.n;
    if (full) {
        if (ITEMS == 4) {
            const uint4 c = __ldcs(reinterpret_cast<const uint4*>(A.cells() + first));
            cl[0] = c.x; cl[1] = c.y; cl[2 % ITEMS] = c.z; cl[3 % ITEMS] = c.w;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (a < DIM) {
                    const float4 f = __ldcs(reinterpret_cast<const float4*>(A.offs(a) + first));
                    fo[0][a] = f.x; fo[1][a] = f.y; fo[2 % ITEMS][a] = f.z; fo[3 % ITEMS][a] = f.w;
                } else {
#pragma unroll
                    for (int k = 0; k < ITEMS; ++k) fo[k][a] = 0.0f;
                }
                const float4 v = __ldcs(reinterpret_cast<const float4*>(A.vels(a) + first));
                vv[0][a] = v.x; vv[1][a] = v.y; vv[2 % ITEMS][a] = v.z; vv[3 % ITEMS][a] = v.w;
            }
        } else {
            const uint2 c = __ldcs(reinterpret_cast<const uint2*>(A.cells() + first));
            cl[0] = c.x; cl[1 % ITEMS] = c.y;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (a < DIM) {
                    const float2 f = __ldcs(reinterpret_cast<const float2*>(A.offs(a) + first));
                    fo[0][a] = f.x; fo[1 % ITEMS][a] = f.y;
                } else {
                    fo[0][a] = 0.0f; fo[1 % ITEMS][a] = 0.0f;
                }
                const float2 v = __ldcs(reinterpret_cast<const float2*>(A.vels(a) + first));
                vv[0][a] = v.x; vv[1 % ITEMS][a] = v.y;
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const unsigned i = first + k;
            const bool ok = i < S.n;
            cl[k] = ok ? A.cells()[i] : 0u;
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                fo[k][a] = (ok && a < DIM) ? A.offs(a)[i] : 0.0f;
                vv[k][a] = ok ? A.vels(a)[i] : 0.0f;
            }
        }
    }
    // 2D: the box is clear and its place read in every thread; the state's loads are under way
    if (DIM == 2) __syncthreads();
    const unsigned kNoCell = 0xFFFFFFFFu;
    // 3D: the field lines of each later new cell in the thread's run are
    // prefetched into L1 before the first push: a cell change inside the run
    // then finds them there instead of waiting a whole L2 round trip between
    // two pushes (no registers are held for them).  The 2D field (8 B a node)
    // mostly sits in L1 already; prefetching it measured within noise.
#pragma unroll
    for (int k = 1; k < ITEMS; ++k) {
        if (DIM == 2 || first + k >= S.n || cl[k] == cl[k - 1]) continue;
        int ix, iy, iz;
        unpack_cell(cl[k], ix, iy, iz);
        const int iy1 = (iy + 1) & (ny - 1);
        {
            const int iz1 = (iz + 1) & (nz - 1);
            const float4* E = reinterpret_cast<const float4*>(p.E32);
            asm volatile("prefetch.global.L1 [%0];" ::"l"(E + ((size_t)iz * ny + iy) * nx + ix));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(E + ((size_t)iz * ny + iy1) * nx + ix));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(E + ((size_t)iz1 * ny + iy) * nx + ix));
            asm volatile("prefetch.global.L1 [%0];" ::"l"(E + ((size_t)iz1 * ny + iy1) * nx + ix));
        }
    }
    unsigned gcell = kNoCell;   // cell whose node fields are cached
    float en[NN][3];            // the field at its nodes
    unsigned rcell = kNoCell;   // cell of the current deposit run
    unsigned racc[NN];          // its summed quantised weights
#pragma unroll
    for (int j = 0; j < NN; ++j) racc[j] = 0u;
    auto commit = [&](unsigned c, const unsigned* w) {
        int ix, iy, iz;
        unpack_cell(c, ix, iy, iz);
        if (DIM == 2) {
            const int bx = (ix - box.x0) & (nx - 1), by = (iy - box.y0) & (ny - 1);
            if (bx < kDBoxX && by < 3) {
                const int b = by * (kDBoxX + 1) + bx;
                unsigned old[NN], high = 0u;
#pragma unroll
                for (int j = 0; j < NN; ++j) old[j] = atomicAdd(box.sum + b + (j & 1) + (j >> 1) * (kDBoxX + 1), w[j]);
#pragma unroll
                for (int j = 0; j < NN; ++j) high |= old[j];
                if (high >> 31)  // an add (at most 2^28) can only wrap a word that is past its half
                    for (int j = 0; j < NN; ++j)
                        if (old[j] + w[j] < old[j])
                            atomicAdd(acc + (size_t)((iy + (j >> 1)) & (ny - 1)) * nx + ((ix + (j & 1)) & (nx - 1)), 1ull << 32);
                return;
            }
        }
        const int ix1 = (ix + 1) & (nx - 1), iy1 = (iy + 1) & (ny - 1);
        const int iz1 = DIM == 3 ? (iz + 1) & (nz - 1) : 0;
#pragma unroll
        for (int j = 0; j < NN; ++j) {
            if (!w[j]) continue;
            const int xx = (j & 1) ? ix1 : ix, yy = (j & 2) ? iy1 : iy, zz = (j & 4) ? iz1 : iz;
            atomicAdd(acc + ((size_t)zz * ny + yy) * nx + xx, (unsigned long long)w[j]);
        }
    };
#pragma unroll
    for (int k = 0; k < ITEMS; ++k) {
        if (first + k >= S.n) continue;
        int ix, iy, iz;
        unpack_cell(cl[k], ix, iy, iz);
        float* f = fo[k];
        float* v = vv[k];
        if (cl[k] != gcell) {  // the field at the new cell's nodes
            gcell = cl[k];
            const int ix1 = (ix + 1) & (nx - 1), iy1 = (iy + 1) & (ny - 1);
            if (DIM == 2) {
                const float2* E = reinterpret_cast<const float2*>(p.E32);
                const float2 a = __ldg(E + iy * nx + ix), b = __ldg(E + iy * nx + ix1),
                             c = __ldg(E + iy1 * nx + ix), d = __ldg(E + iy1 * nx + ix1);
                en[0][0] = a.x; en[0][1] = a.y; en[1][0] = b.x; en[1][1] = b.y;
                en[2][0] = c.x; en[2][1] = c.y; en[3][0] = d.x; en[3][1] = d.y;
#pragma unroll
                for (int j = 0; j < NN; ++j) en[j][2] = 0.0f;
            } else {
                const int iz1 = (iz + 1) & (nz - 1);
                const float4* E = reinterpret_cast<const float4*>(p.E32);
#pragma unroll
                for (int j = 0; j < NN; ++j) {
                    const int xx = (j & 1) ? ix1 : ix, yy = (j & 2) ? iy1 : iy, zz = (j & 4) ? iz1 : iz;
                    const float4 q = __ldg(E + ((size_t)zz * ny + yy) * nx + xx);
                    en[j][0] = q.x; en[j][1] = q.y; en[j][2] = q.z;
                }
            }
        }
        // bilinear / trilinear gather, src/FieldSolver.cpp:925-1038 (the
        // arithmetic of gather32, so every particles-per-thread choice gives
        // the same bits)
        const float wx[2] = {1.0f - f[0], f[0]}, wy[2] = {1.0f - f[1], f[1]};
        float e[3] = {0.0f, 0.0f, 0.0f};
        if (DIM == 2) {
            const float w00 = wx[0] * wy[0], w10 = wx[1] * wy[0], w01 = wx[0] * wy[1], w11 = wx[1] * wy[1];
            e[0] = fmaf(en[0][0], w00, fmaf(en[1][0], w10, fmaf(en[2][0], w01, en[3][0] * w11)));
            e[1] = fmaf(en[0][1], w00, fmaf(en[1][1], w10, fmaf(en[2][1], w01, en[3][1] * w11)));
        } else {
            const float wz[2] = {1.0f - f[2], f[2]};
#pragma unroll
            for (int j = 0; j < NN; ++j) {
                const float w = wx[j & 1] * (wy[(j >> 1) & 1] * wz[(j >> 2) & 1]);
                e[0] = fmaf(en[j][0], w, e[0]);
                e[1] = fmaf(en[j][1], w, e[1]);
                e[2] = fmaf(en[j][2], w, e[2]);
            }
        }
        // kick + drift, src/Pusher.cpp:109-128, :162-174
        if (BORIS && PROF) {
            float tp[3], sp[3];
            boris_ts32(p, S, ix, iy, iz, f, tp, sp);
            boris32(v, e, S.hqmdt, tp, sp);
        } else if (BORIS) {
            boris32(v, e, S.hqmdt, S.tb, S.sb);
        } else {
            for (int a = 0; a < DIM; ++a) v[a] = fmaf(S.qmdt, e[a], v[a]);
        }
        advance(f[0], ix, v[0] * S.drift[0], nx);
        advance(f[1], iy, v[1] * S.drift[1], ny);
        if (DIM == 3) advance(f[2], iz, v[2] * S.drift[2], nz);
        cl[k] = pack_cell(ix, iy, iz);
        // deposit at the pushed position into the run of its cell
        if (cl[k] != rcell) {
            if (rcell != kNoCell) commit(rcell, racc);
            rcell = cl[k];
#pragma unroll
            for (int j = 0; j < NN; ++j) racc[j] = 0u;
        }
        // (units of 2^-23 to nearest even: adding 2^23 leaves the integer in the low
        // bits of the float; the scale, a power of two, is exact on any factor)
        const float ux[2] = {(1.0f - f[0]) * kWeightScale, f[0] * kWeightScale}, uy[2] = {1.0f - f[1], f[1]};
        const float uz[2] = {DIM == 3 ? 1.0f - f[2] : 1.0f, DIM == 3 ? f[2] : 0.0f};
#pragma unroll
        for (int j = 0; j < NN; ++j) {
            const float w = DIM == 3 ? ux[j & 1] * uy[(j >> 1) & 1] * uz[(j >> 2) & 1] : ux[j & 1] * uy[(j >> 1) & 1];
            // (a particle of infinite or NaN velocity keeps its cell and has a NaN offset: the
            // maximum makes its weights 0 instead of 106 particles' charge)
            racc[j] += __float_as_uint(fmaxf(w + kWeightScale, kWeightScale)) - 0x4B000000u;
        }
    }
    // the state back, in place
    if (full) {
        if (ITEMS == 4) {
            __stcs(reinterpret_cast<uint4*>(A.cells() + first), make_uint4(cl[0], cl[1], cl[2 % ITEMS], cl[3 % ITEMS]));
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (a < DIM)
                    __stcs(reinterpret_cast<float4*>(A.offs(a) + first),
                           make_float4(fo[0][a], fo[1][a], fo[2 % ITEMS][a], fo[3 % ITEMS][a]));
                __stcs(reinterpret_cast<float4*>(A.vels(a) + first),
                       make_float4(vv[0][a], vv[1][a], vv[2 % ITEMS][a], vv[3 % ITEMS][a]));
            }
        } else {
            __stcs(reinterpret_cast<uint2*>(A.cells() + first), make_uint2(cl[0], cl[1 % ITEMS]));
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (a < DIM)
                    __stcs(reinterpret_cast<float2*>(A.offs(a) + first), make_float2(fo[0][a], fo[1 % ITEMS][a]));
                __stcs(reinterpret_cast<float2*>(A.vels(a) + first), make_float2(vv[0][a], vv[1 % ITEMS][a]));
            }
        }
    } else {
#pragma unroll
        for (int k = 0; k < ITEMS; ++k) {
            const unsigned i = first + k;
            if (i >= S.n) continue;
            A.cells()[i] = cl[k];
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                if (a < DIM) A.offs(a)[i] = fo[k][a];
                A.vels(a)[i] = vv[k][a];
            }
        }
    }
    // each lane's last run: summed over the lanes that end in the same cell
    // segments of at most 4 lanes in 3D (a cell's run spans about 4 lanes at 8
    // particles per cell) and 8 in 2D: two or three shuffle steps instead of
    // five per node, for a few more commits; measured 5.89 -> 5.69 ms per
    // 256^3 step and 0.371 -> 0.368 ms per 512^2 step
    constexpr int RSEG = DIM == 3 ? 4 : 8;
    const unsigned key = rcell;
    const unsigned prev = __shfl_up_sync(0xffffffffu, key, 1);
    const bool head = (lane & (RSEG - 1)) == 0 || prev != key;
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const int start = 31 - __clz(heads & (0xFFFFFFFFu >> (31 - lane)));
    const bool tail = lane == 31 || ((heads >> (lane + 1)) & 1u);
#pragma unroll
    for (int j = 0; j < NN; ++j) {
        unsigned q = racc[j];
#pragma unroll
        for (int d = 1; d < RSEG; d <<= 1) {
            const unsigned t = __shfl_up_sync(0xffffffffu, q, d);
            if (lane - d >= start) q += t;
        }
        racc[j] = q;
    }
    if (tail && key != kNoCell) commit(key, racc);
}

// (3D states no CTAs per SM: 4 spilled, 128^3 with 4 particles a thread 272 -> 394 us a step)
template <int DIM, bool BORIS, int ITEMS, bool PROF>
__global__ void __launch_bounds__(kThreads, DIM == 2 ? 4 : 0)
    k_push32_run(ParamsND p, SpeciesND S, State32 A, int buf, unsigned long long* acc) {
    if constexpr (DIM == 2) {
        __shared__ unsigned s_sum[kDBoxNodes];
        const int nx = p.n[0], ny = p.n[1];
        // the box around the CTA's middle particle, read by every thread before the
        // barrier in push_run (no particle is stored before it)
        const unsigned mid = min(blockIdx.x * kThreads * ITEMS + (unsigned)(kThreads * ITEMS / 2), S.n - 1u);
        int ix, iy, iz;
        unpack_cell(A.cell[mid], ix, iy, iz);
        for (int q = threadIdx.x; q < kDBoxNodes; q += kThreads) s_sum[q] = 0u;
        const DepositBox box{s_sum, (ix - kDBoxX / 2) & (nx - 1), (iy - 1) & (ny - 1)};
        push_run<DIM, BORIS, ITEMS, PROF>(p, S, A, acc, box);
        __syncthreads();
        for (int q = threadIdx.x; q < kDBoxNodes; q += kThreads) {
            const unsigned long long v = s_sum[q];
            if (!v) continue;
            const int qx = q % (kDBoxX + 1), qy = q / (kDBoxX + 1);
            atomicAdd(acc + (size_t)((box.y0 + qy) & (ny - 1)) * nx + ((box.x0 + qx) & (nx - 1)), v);
        }
    } else {
        push_run<DIM, BORIS, ITEMS, PROF>(p, S, Buffer32{S, buf}, acc, DepositBox{nullptr, 0, 0});
    }
}

// After a tiled sort: the work items of the push, one per tile and more for
// tiles of many particles (about `target` each; nothing depends on their
// order).  cursor[last cell of a tile] is one past the tile's last particle.
__global__ void k_tile_items(const unsigned* __restrict__ cursor, unsigned ntiles, unsigned target, SpeciesND S) {
    const unsigned t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntiles) return;
    const unsigned first = t ? cursor[(size_t)t * kTileVolume - 1] : 0u;
    const unsigned last = cursor[(size_t)(t + 1) * kTileVolume - 1];
    const unsigned n = last - first, items = max(1u, (n + target / 2) / target);
    const unsigned extra = items > 1 ? atomicAdd(S.extra, items - 1) : 0u;
    for (unsigned k = 0; k < items; ++k) {
        const unsigned a = first + (unsigned)((unsigned long long)n * k / items);
        const unsigned b = first + (unsigned)((unsigned long long)n * (k + 1) / items);
        S.chunk[k == 0 ? t : ntiles + extra + k - 1] = make_uint4(t, a, b, 0u);
    }
}

// The FP32 step push of a tiled 3D species: one CTA per work item.  The field
// at the nodes of the tile and MARGIN cells around it is staged in shared
// memory, and the deposit is summed there, so the gathers and the deposit of a particle cost shared
// accesses whatever the order inside the tile, and one global atomic per touched node
// remains of the eight per particle.  Particles that drifted out of the box take the
// global path.  Each node's sum is one 32-bit word; an add that wraps carries 2^32
// into the global sum at once, so the charge is exact and the same as the
// other kernels'.  Push of 2 x 134 M particles on 256^3: 5.7 -> 4.06 ms a step (the
// untiled kernel was bound by the wavefronts of its global gathers and atomics; this
// one issues half of all cycles, at 0.57 of the measured HBM rate).
template <int MARGIN>
constexpr int kBoxSide = kTileCells + 2 * MARGIN + 1;
template <int MARGIN>
constexpr int kBoxNodes = kBoxSide<MARGIN> * kBoxSide<MARGIN> * kBoxSide<MARGIN>;
template <int MARGIN>
constexpr size_t tile32_smem() { return kBoxNodes<MARGIN> * (sizeof(float4) + sizeof(unsigned)); }

// G consecutive 32-bit values as one vector (2 or 4, aligned), streamed
template <int G, class V>
__device__ __forceinline__ void load_group(const V* p, V (&v)[G]) {
    static_assert(sizeof(V) == 4 && (G == 2 || G == 4), "8- or 16-byte groups");
    if constexpr (G == 4) {
        const uint4 q = __ldcs(reinterpret_cast<const uint4*>(p));
        v[0] = __builtin_bit_cast(V, q.x); v[1] = __builtin_bit_cast(V, q.y);
        v[2] = __builtin_bit_cast(V, q.z); v[3] = __builtin_bit_cast(V, q.w);
    } else {
        const uint2 q = __ldcs(reinterpret_cast<const uint2*>(p));
        v[0] = __builtin_bit_cast(V, q.x); v[1] = __builtin_bit_cast(V, q.y);
    }
}
template <int G, class V>
__device__ __forceinline__ void store_group(V* p, const V (&v)[G]) {
    if constexpr (G == 4)
        __stcs(reinterpret_cast<uint4*>(p), make_uint4(__builtin_bit_cast(unsigned, v[0]), __builtin_bit_cast(unsigned, v[1]),
                                                       __builtin_bit_cast(unsigned, v[2]), __builtin_bit_cast(unsigned, v[3])));
    else
        __stcs(reinterpret_cast<uint2*>(p), make_uint2(__builtin_bit_cast(unsigned, v[0]), __builtin_bit_cast(unsigned, v[1])));
}

// Groups of 4 and 3 CTAs per SM (256^3, both species, per step): 4.06 ms; groups
// of 2: 4.19 with 3 CTAs, 4.59 with 4; of 4: 5.67 with 4 (spills), 4.74 with 2.
constexpr int kTileGroup = 4;
constexpr int kTileBlocks = 3;  // per SM

template <bool BORIS, bool PROF, int MARGIN>
__global__ void __launch_bounds__(kThreads, kTileBlocks) k_push32_tile(ParamsND p, SpeciesND S, State32 A,
                                                                       unsigned long long* acc, unsigned ntiles) {
    constexpr int B = kBoxSide<MARGIN>, NB = kBoxNodes<MARGIN>;
    extern __shared__ __align__(16) unsigned char tile_raw[];
    float4* sE = reinterpret_cast<float4*>(tile_raw);
    unsigned* sQ = reinterpret_cast<unsigned*>(sE + NB);
    if (blockIdx.x >= ntiles + *S.extra) return;
    const uint4 item = S.chunk[blockIdx.x];
    const unsigned first = item.y, last = item.z;
    if (first >= last) return;
    const int nx = p.n[0], ny = p.n[1], nz = p.n[2];
    const int ntx = nx >> kTileLog, nty = ny >> kTileLog;
    const int x0 = (int)(item.x % ntx) * kTileCells - MARGIN, y0 = (int)(item.x / ntx % nty) * kTileCells - MARGIN,
              z0 = (int)(item.x / (ntx * nty)) * kTileCells - MARGIN;
    auto node_of = [&](int q) {  // box node -> mesh node
        const int qx = q % B, qy = q / B % B, qz = q / (B * B);
        return ((unsigned)((z0 + qz) & (nz - 1)) * ny + ((y0 + qy) & (ny - 1))) * nx + ((x0 + qx) & (nx - 1));
    };
    // node of the box at the lower corner of cell (ix, iy, iz), or -1 outside the box
    auto place = [&](int ix, int iy, int iz) {
        const int lx = (ix - x0) & (nx - 1), ly = (iy - y0) & (ny - 1), lz = (iz - z0) & (nz - 1);
        return lx < B - 1 && ly < B - 1 && lz < B - 1 ? (lz * B + ly) * B + lx : -1;
    };
    for (int q = threadIdx.x; q < NB; q += kThreads) {
        sE[q] = __ldg(reinterpret_cast<const float4*>(p.E32) + node_of(q));
        sQ[q] = 0u;
    }
    __syncthreads();
    // the summed weights of a run of particles in one cell
    auto commit = [&](unsigned cell, int b, const unsigned* w) {
        if (b >= 0) {
            unsigned old[8], high = 0u;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                old[j] = atomicAdd(sQ + b + (j & 1) + ((j >> 1) & 1) * B + (j >> 2) * (B * B), w[j]);
#pragma unroll
            for (int j = 0; j < 8; ++j) high |= old[j];
            if (high >> 31)  // an add (at most 2^25) can only wrap a word that is past its half
                for (int j = 0; j < 8; ++j) {
                    const int q = b + (j & 1) + ((j >> 1) & 1) * B + (j >> 2) * (B * B);
                    if (old[j] + w[j] < old[j]) atomicAdd(acc + node_of(q), 1ull << 32);
                }
            return;
        }
        int ix, iy, iz;
        unpack_cell(cell, ix, iy, iz);
        const int ix1 = (ix + 1) & (nx - 1), iy1 = (iy + 1) & (ny - 1), iz1 = (iz + 1) & (nz - 1);
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (w[j])
                atomicAdd(acc + ((size_t)((j & 4) ? iz1 : iz) * ny + ((j & 2) ? iy1 : iy)) * nx + ((j & 1) ? ix1 : ix),
                          (unsigned long long)w[j]);
    };
    // rows of 32 groups of G consecutive particles per warp, one group per lane;
    // the groups at the item's ends may hold another item's particles
    constexpr int G = kTileGroup;
    for (unsigned row = (first & ~(G - 1u)) + G * (threadIdx.x & ~31u); row < last; row += G * kThreads) {
        const unsigned i = row + G * (threadIdx.x & 31);
        if (i >= last) continue;
        unsigned cl[G];
        float fo[G][3], vv[G][3];
        const bool full = i >= first && i + G <= last;
        if (full) {
            load_group<G>(A.cell + i, cl);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                float f[G], v[G];
                load_group<G>(A.off[a] + i, f);
                load_group<G>(A.vel[a] + i, v);
#pragma unroll
                for (int k = 0; k < G; ++k) { fo[k][a] = f[k]; vv[k][a] = v[k]; }
            }
        } else {
#pragma unroll
            for (int k = 0; k < G; ++k) {
                const bool ok = i + k >= first && i + k < last;
                cl[k] = ok ? A.cell[i + k] : 0u;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    fo[k][a] = ok ? A.off[a][i + k] : 0.0f;
                    vv[k][a] = ok ? A.vel[a][i + k] : 0.0f;
                }
            }
        }
        unsigned w[8];
        unsigned rcell = 0xFFFFFFFFu;  // cell of the current run, and its place in the box
        int rplace = -1;
#pragma unroll
        for (int k = 0; k < G; ++k) {
            if (!full && (i + k < first || i + k >= last)) continue;
            int ix, iy, iz;
            unpack_cell(cl[k], ix, iy, iz);
            float* f = fo[k];
            float* v = vv[k];
            float e[3] = {0.0f, 0.0f, 0.0f};
            const int g = place(ix, iy, iz);
            if (g >= 0) {
                // trilinear gather, src/FieldSolver.cpp:978-1038 (the arithmetic of gather32)
                const float4* E = sE + g;
                const float wx[2] = {1.0f - f[0], f[0]}, wy[2] = {1.0f - f[1], f[1]}, wz[2] = {1.0f - f[2], f[2]};
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const float s = wx[j & 1] * (wy[(j >> 1) & 1] * wz[j >> 2]);
                    const float4 q = E[(j & 1) + ((j >> 1) & 1) * B + (j >> 2) * (B * B)];
                    e[0] = fmaf(q.x, s, e[0]);
                    e[1] = fmaf(q.y, s, e[1]);
                    e[2] = fmaf(q.z, s, e[2]);
                }
            } else {
                gather32<3>(p, ix, iy, iz, f, e);
            }
            // kick + drift, src/Pusher.cpp:109-128, :162-174
            if (BORIS && PROF) {
                float tp[3], sp[3];
                boris_ts32(p, S, ix, iy, iz, f, tp, sp);
                boris32(v, e, S.hqmdt, tp, sp);
            } else if (BORIS) {
                boris32(v, e, S.hqmdt, S.tb, S.sb);
            } else {
#pragma unroll
                for (int a = 0; a < 3; ++a) v[a] = fmaf(S.qmdt, e[a], v[a]);
            }
            advance(f[0], ix, v[0] * S.drift[0], nx);
            advance(f[1], iy, v[1] * S.drift[1], ny);
            advance(f[2], iz, v[2] * S.drift[2], nz);
            cl[k] = pack_cell(ix, iy, iz);
            // deposit at the pushed position into the run of its cell
            if (cl[k] != rcell) {
                if (rcell != 0xFFFFFFFFu) commit(rcell, rplace, w);
                rcell = cl[k];
                rplace = place(ix, iy, iz);
#pragma unroll
                for (int j = 0; j < 8; ++j) w[j] = 0u;
            }
            // the weights in units of 2^-23, to nearest even: adding 2^23 leaves the
            // integer in the low bits of the float (a weight is at most 2^23 units);
            // the scale, a power of two, is exact on any factor
            const float ux[2] = {(1.0f - f[0]) * kWeightScale, f[0] * kWeightScale};
            const float uy[2] = {1.0f - f[1], f[1]}, uz[2] = {1.0f - f[2], f[2]};
            // a NaN offset (see push_run) deposits nothing: tested on the last weight, which
            // is formed anyway (256^3: 4.05 ms a step, with a sum of the offsets 4.08)
            if (!(ux[1] * uy[1] * uz[1] >= 0.0f)) continue;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                w[j] += __float_as_uint(ux[j & 1] * uy[(j >> 1) & 1] * uz[j >> 2] + kWeightScale) - 0x4B000000u;
        }
        if (full) {
            store_group<G>(A.cell + i, cl);
#pragma unroll
            for (int a = 0; a < 3; ++a) {
                float f[G], v[G];
#pragma unroll
                for (int k = 0; k < G; ++k) { f[k] = fo[k][a]; v[k] = vv[k][a]; }
                store_group<G>(A.off[a] + i, f);
                store_group<G>(A.vel[a] + i, v);
            }
        } else {
#pragma unroll
            for (int k = 0; k < G; ++k) {
                if (i + k < first || i + k >= last) continue;
                A.cell[i + k] = cl[k];
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    A.off[a][i + k] = fo[k][a];
                    A.vel[a][i + k] = vv[k][a];
                }
            }
        }
        if (rcell != 0xFFFFFFFFu) commit(rcell, rplace, w);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < NB; q += kThreads) {
        const unsigned v = sQ[q];
        if (v) atomicAdd(acc + node_of(q), (unsigned long long)v);
    }
}

// FP64 staging <-> FP32 state.  The cell/offset split follows the periodic CIC
// index of the reference (wrap, divide by the cell size, floor).
template <int DIM>
__global__ void k_to_fp32(ParamsND p, SpeciesND S, int buf) {
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= S.n) return;
    int ii[3] = {0, 0, 0};
    for (int a = 0; a < DIM; ++a) {
        const Axis ax = axis(S.pos[buf][a][i], p.L[a], p.d[a], p.rd[a], p.n[a]);
        float f = (float)ax.f;
        int k = ax.i0;
        if (f >= 1.0f) { f = 0.0f; k = ax.i1; }
        ii[a] = k;
        S.off[buf][a][i] = f;
    }
    S.cell[buf][i] = pack_cell(ii[0], ii[1], ii[2]);
    for (int a = 0; a < 3; ++a) S.vel[buf][a][i] = (float)S.vh[buf][a][i];
}

template <int DIM>
__global__ void k_to_fp64(ParamsND p, SpeciesND S, int buf) {
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= S.n) return;
    int ii[3];
    unpack_cell(S.cell[buf][i], ii[0], ii[1], ii[2]);
    for (int a = 0; a < DIM; ++a) S.pos[buf][a][i] = ((double)ii[a] + (double)S.off[buf][a][i]) * p.d[a];
    for (int a = 0; a < 3; ++a) S.vh[buf][a][i] = (double)S.vel[buf][a][i];
}

// Sorting key of cell (x, y, z): tile by tile, x fastest among the tiles and inside one.
__device__ __forceinline__ unsigned tile_key(int ncx, int ncy, int x, int y, int z) {
    constexpr int k = kTileCells - 1;
    const unsigned tile = ((unsigned)(z >> kTileLog) * (ncy >> kTileLog) + (y >> kTileLog)) * (ncx >> kTileLog) + (x >> kTileLog);
    return tile * kTileVolume + (((z & k) << kTileLog | (y & k)) << kTileLog | (x & k));
}

__device__ __forceinline__ unsigned linear_cell(const ParamsND& p, const SpeciesND& S, unsigned c) {
    int x, y, z;
    unpack_cell(c, x, y, z);
    if (S.tiled) return tile_key(p.n[0], p.n[1], x, y, z);
    return ((unsigned)z * p.n[1] + y) * p.n[0] + x;
}

// Lanes of a warp that share a cell (particles are nearly sorted, so a warp
// spans few cells) take one atomic per cell: the group's leader adds the
// group's size and the lanes take consecutive slots in lane order.
__global__ void k_cell_hist32(ParamsND p, SpeciesND S, int buf, unsigned* count) {
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    const bool valid = i < S.n;
    const unsigned key = valid ? linear_cell(p, S, S.cell[buf][i]) : 0xFFFFFFFFu;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    if (valid && (int)(threadIdx.x & 31) == __ffs(peers) - 1) atomicAdd(count + key, (unsigned)__popc(peers));
}

// Counting-sort placement of the FP32 form in two passes.  k_cell_rank32 gives
// each particle its slot (lanes of a warp that share a cell take one atomic per
// cell: the group's leader adds the group's size and the lanes take
// consecutive slots in lane order) and records the particle's index there, in
// the id array of the target buffer; k_cell_gather32 then fills every slot
// from that index.  The stores of the second pass are coalesced, and the
// scattered accesses are reads, served mostly from L2 (a particle moves a few
// cells between sorts); a direct scatter instead writes a partial sector per
// field for every particle that changed its row or plane.
__global__ void k_cell_rank32(ParamsND p, SpeciesND S, int from, unsigned* cursor) {
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    const bool valid = i < S.n;
    const unsigned key = valid ? linear_cell(p, S, __ldcs(S.cell[from] + i)) : 0xFFFFFFFFu;
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int lane = threadIdx.x & 31, leader = __ffs(peers) - 1;
    unsigned base = 0;
    if (valid && lane == leader) base = atomicAdd(cursor + key, (unsigned)__popc(peers));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (!valid) return;
    S.id[from ^ 1][base + (unsigned)__popc(peers & ((1u << lane) - 1u))] = i;
}

// Histogram and ranks of a species that is already in tiles: one CTA per work
// item of the push, the cells of the tile and one around it counted in shared
// memory.  The kernels above group a warp's particles by match_any, whose cost
// grows with the cells a warp spans; here a particle is one shared add, and a
// cell one global add per item.  256^3 deck, 134 M electrons sorted every 3 steps: sorts
// 1.25 -> 0.98 ms a step.
constexpr int kBinSide = kTileCells + 2, kBins = kBinSide * kBinSide * kBinSide;

template <bool RANK>
__global__ void __launch_bounds__(kThreads) k_tile_count(ParamsND p, SpeciesND S, int from, unsigned* cursor,
                                                         unsigned ntiles) {
    __shared__ unsigned s_count[kBins], s_base[RANK ? kBins : 1];
    if (blockIdx.x >= ntiles + *S.extra) return;
    const uint4 item = S.chunk[blockIdx.x];
    const unsigned first = item.y, last = item.z;
    if (first >= last) return;
    const int nx = p.n[0], ny = p.n[1], nz = p.n[2];
    const int ntx = nx >> kTileLog, nty = ny >> kTileLog;
    const int x0 = (int)(item.x % ntx) * kTileCells - 1, y0 = (int)(item.x / ntx % nty) * kTileCells - 1,
              z0 = (int)(item.x / (ntx * nty)) * kTileCells - 1;
    for (int q = threadIdx.x; q < kBins; q += kThreads) s_count[q] = 0u;
    __syncthreads();
    auto bin_at = [&](unsigned c) {  // bin of packed cell c, or -1
        int x, y, z;
        unpack_cell(c, x, y, z);
        const int lx = (x - x0) & (nx - 1), ly = (y - y0) & (ny - 1), lz = (z - z0) & (nz - 1);
        return lx < kBinSide && ly < kBinSide && lz < kBinSide ? (lz * kBinSide + ly) * kBinSide + lx : -1;
    };
    for (unsigned i = first + threadIdx.x; i < last; i += kThreads) {
        const unsigned c = S.cell[from][i];
        const int b = bin_at(c);
        if (b >= 0) atomicAdd(s_count + b, 1u);
        else if (!RANK) atomicAdd(cursor + linear_cell(p, S, c), 1u);
    }
    __syncthreads();
    for (int q = threadIdx.x; q < kBins; q += kThreads) {
        const unsigned n = s_count[q];
        if (!n) continue;
        const unsigned key = tile_key(nx, ny, (x0 + q % kBinSide) & (nx - 1), (y0 + q / kBinSide % kBinSide) & (ny - 1),
                                      (z0 + q / (kBinSide * kBinSide)) & (nz - 1));
        const unsigned at = atomicAdd(cursor + key, n);
        if (RANK) {
            s_base[q] = at;
            s_count[q] = 0u;
        }
    }
    if (!RANK) return;
    __syncthreads();
    for (unsigned i = first + threadIdx.x; i < last; i += kThreads) {
        const unsigned c = S.cell[from][i];
        const int b = bin_at(c);
        const unsigned slot = b >= 0 ? s_base[RANK ? b : 0] + atomicAdd(s_count + b, 1u) : atomicAdd(cursor + linear_cell(p, S, c), 1u);
        S.id[from ^ 1][slot] = i;
    }
}

template <int DIM>
__global__ void k_cell_gather32(SpeciesND S, int from) {
    const unsigned d = blockIdx.x * kThreads + threadIdx.x;
    if (d >= S.n) return;
    const int to = from ^ 1;
    const unsigned i = S.id[to][d];
    const unsigned c = S.cell[from][i], id = S.id[from][i];
    float off[3], vel[3];
#pragma unroll
    for (int a = 0; a < DIM; ++a) off[a] = S.off[from][a][i];
#pragma unroll
    for (int a = 0; a < 3; ++a) vel[a] = S.vel[from][a][i];
    __stcs(S.cell[to] + d, c);
#pragma unroll
    for (int a = 0; a < DIM; ++a) __stcs(S.off[to][a] + d, off[a]);
#pragma unroll
    for (int a = 0; a < 3; ++a) __stcs(S.vel[to][a] + d, vel[a]);
    __stcs(S.id[to] + d, id);
}

// ---- particle sort by cell -------------------------------------------------------

template <int DIM, bool WALLS>
__device__ __forceinline__ unsigned cell_of(const ParamsND& p, const double pos[3]) {
    const Axis ax = axis2<WALLS>(p, 0, pos[0]);
    const Axis ay = axis2<WALLS>(p, 1, pos[1]);
    unsigned c = (unsigned)ay.i0 * p.n[0] + ax.i0;
    if (DIM == 3) {
        const Axis az = axis2<WALLS>(p, 2, pos[2]);
        c += (unsigned)az.i0 * p.n[0] * p.n[1];
    }
    return c;
}

// Runs with walls keep their absorbed particles (their positions can be read
// back) in one bin after the last cell, so the push meets them in whole warps.
template <int DIM, bool WALLS>
__device__ __forceinline__ unsigned bin_of(const ParamsND& p, const SpeciesND& S, int buf, unsigned i,
                                           const double pos[3]) {
    if (WALLS && S.alive[buf] && !S.alive[buf][i]) return (unsigned)(p.n[0] * p.n[1] * (DIM == 3 ? p.n[2] : 1));
    return cell_of<DIM, WALLS>(p, pos);
}

// One atomic for all lanes of a warp with the same bin: after the first sort a
// warp holds one or two cells, and the absorbed of a run with walls are one bin,
// whose count would otherwise take one atomic after another.
template <int DIM, bool WALLS>
__global__ void k_cell_hist(ParamsND p, SpeciesND S, int buf, unsigned* count) {
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    unsigned bin = ~0u;  // no particle
    if (i < S.n) {
        const double pos[3] = {S.pos[buf][0][i], S.pos[buf][1][i], DIM == 3 ? S.pos[buf][2][i] : 0.0};
        bin = bin_of<DIM, WALLS>(p, S, buf, i, pos);
    }
    const unsigned same = __match_any_sync(0xFFFFFFFFu, bin);
    if (bin != ~0u && (threadIdx.x & 31) == (unsigned)__ffs(same) - 1) atomicAdd(count + bin, (unsigned)__popc(same));
}

// exclusive scan of `count` (n entries) into `offset`, three launches
constexpr int kScanItems = 8;
constexpr int kScanBlock = kThreads * kScanItems;
__global__ void k_scan_local(const unsigned* count, unsigned* offset, unsigned* block_sums, unsigned n) {
    __shared__ unsigned s[kThreads];
    const unsigned base = blockIdx.x * kScanBlock + threadIdx.x * kScanItems;
    unsigned v[kScanItems], sum = 0;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        v[k] = base + k < n ? count[base + k] : 0u;
        sum += v[k];
    }
    s[threadIdx.x] = sum;
    __syncthreads();
    for (int o = 1; o < kThreads; o <<= 1) {
        const unsigned y = threadIdx.x >= (unsigned)o ? s[threadIdx.x - o] : 0u;
        __syncthreads();
        s[threadIdx.x] += y;
        __syncthreads();
    }
    unsigned run = s[threadIdx.x] - sum;
#pragma unroll
    for (int k = 0; k < kScanItems; ++k) {
        if (base + k < n) offset[base + k] = run;
        run += v[k];
    }
    if (threadIdx.x == kThreads - 1) block_sums[blockIdx.x] = s[threadIdx.x];
}

__global__ void k_scan_blocks(unsigned* block_sums, unsigned nblocks) {
    // one CTA: exclusive scan in place (nblocks <= kThreads * kScanItems * kThreads handled by a loop)
    __shared__ unsigned s[kThreads];
    __shared__ unsigned carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (unsigned b0 = 0; b0 < nblocks; b0 += kThreads) {
        const unsigned i = b0 + threadIdx.x;
        const unsigned v = i < nblocks ? block_sums[i] : 0u;
        s[threadIdx.x] = v;
        __syncthreads();
        for (int o = 1; o < kThreads; o <<= 1) {
            const unsigned y = threadIdx.x >= (unsigned)o ? s[threadIdx.x - o] : 0u;
            __syncthreads();
            s[threadIdx.x] += y;
            __syncthreads();
        }
        const unsigned c = carry;
        if (i < nblocks) block_sums[i] = c + s[threadIdx.x] - v;
        __syncthreads();
        if (threadIdx.x == kThreads - 1) carry = c + s[threadIdx.x];
        __syncthreads();
    }
}

// (last, when given, receives the offset of the last bin)
__global__ void k_scan_add(unsigned* offset, const unsigned* block_sums, unsigned n, unsigned* last) {
    const unsigned base = blockIdx.x * kScanBlock;
    const unsigned add = block_sums[blockIdx.x];
    for (unsigned k = threadIdx.x; k < (unsigned)kScanBlock; k += kThreads)
        if (base + k < n) {
            const unsigned v = offset[base + k] + add;
            offset[base + k] = v;
            if (last && base + k + 1 == n) *last = v;
        }
}

template <int DIM, bool WALLS>
__global__ void k_cell_scatter(ParamsND p, SpeciesND S, int from, unsigned* cursor) {
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    const int to = from ^ 1;
    const bool valid = i < S.n;
    const unsigned j = valid ? i : 0;
    // loads first, stores after: the buffers may alias as far as the compiler
    // knows, so loads placed after stores would each wait for the previous store
    const double pos[3] = {S.pos[from][0][j], S.pos[from][1][j], DIM == 3 ? S.pos[from][2][j] : 0.0};
    const double vh[3] = {S.vh[from][0][j], S.vh[from][1][j], S.vh[from][2][j]};
    const unsigned id = S.id[from][j];
    const uint8_t alive = WALLS && S.alive[from] ? S.alive[from][j] : 1;
    const unsigned bin = valid ? bin_of<DIM, WALLS>(p, S, from, i, pos) : ~0u;
    const unsigned same = __match_any_sync(0xFFFFFFFFu, bin);
    const int lane = threadIdx.x & 31, leader = __ffs(same) - 1;
    unsigned o = valid && lane == leader ? atomicAdd(cursor + bin, (unsigned)__popc(same)) : 0u;
    o = __shfl_sync(0xFFFFFFFFu, o, leader) + __popc(same & ((1u << lane) - 1u));
    if (!valid) return;
    for (int a = 0; a < DIM; ++a) S.pos[to][a][o] = pos[a];
    for (int a = 0; a < 3; ++a) S.vh[to][a][o] = vh[a];
    S.id[to][o] = id;
    if (WALLS && S.alive[to]) S.alive[to][o] = alive;
}

// Device-side loading for large runs: uniform positions displaced by
// amp/k sin(k x) along `mode_axis` (amp = 0: none) and Maxwellian velocities
// with thermal speed vt and x drift, from a Philox stream per particle
// (Box-Muller on 53-bit uniforms).
__global__ void k_load_maxwellian(SpeciesND S, int buf, int dims, unsigned n, uint64_t seed, double L0, double L1,
                                  double L2, double vt, double drift, int mode_axis, double amp) {
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    if (i >= n) return;
    uint32_t r[4], r2[4];
    philox4x32_10(i, 0x5eedu, 0u, 0u, (uint32_t)seed, (uint32_t)(seed >> 32), r);
    philox4x32_10(i, 0x5eedu, 1u, 0u, (uint32_t)seed, (uint32_t)(seed >> 32), r2);
    auto u53 = [](uint32_t a, uint32_t b) {
        return ((double)(((uint64_t)a << 21) ^ (uint64_t)b & 0x1FFFFFull) + 0.5) * 0x1.0p-53;
    };
    const double L[3] = {L0, L1, L2};
    const double u[3] = {u53(r[0], r[1]), u53(r[2], r[3]), u53(r2[0], r2[1])};
    for (int a = 0; a < dims; ++a) {
        double x = u[a] * L[a];
        if (amp != 0.0 && (mode_axis < 0 || a == mode_axis)) {
            const double k = 2.0 * 3.141592653589793 / L[a];
            x = x + amp / k * sin(k * x);
            x = fmod(fmod(x, L[a]) + L[a], L[a]);
        }
        S.pos[buf][a][i] = x;
    }
    uint32_t g1[4], g2[4];
    philox4x32_10(i, 0x5eedu, 2u, 0u, (uint32_t)seed, (uint32_t)(seed >> 32), g1);
    philox4x32_10(i, 0x5eedu, 3u, 0u, (uint32_t)seed, (uint32_t)(seed >> 32), g2);
    const double a1 = u53(g1[0], g1[1]), b1 = u53(g1[2], g1[3]), a2 = u53(g2[0], g2[1]), b2 = u53(g2[2], g2[3]);
    const double r1 = sqrt(-2.0 * log(a1)), r2v = sqrt(-2.0 * log(a2));
    const double twopi = 2.0 * 3.141592653589793;
    const double nv[3] = {r1 * cos(twopi * b1), r1 * sin(twopi * b1), r2v * cos(twopi * b2)};
    for (int a = 0; a < 3; ++a) {
        const double v = vt * nv[a] + (a == 0 ? drift : 0.0);
        S.v[a][i] = v;
        S.vh[buf][a][i] = v;
    }
    S.id[buf][i] = i;
}

// Read-back in load order: dst[id[i]] = src[i].
template <class T>
__global__ void k_unpermute(const unsigned* id, const T* src, T* dst, unsigned n) {
    const unsigned i = blockIdx.x * kThreads + threadIdx.x;
    if (i < n) dst[id[i]] = src[i];
}

// ---- spectral Poisson solve: line FFTs in shared memory -----------------------------

enum : int { kFwdFromRho = 0, kFwdInPlace = 1, kFwdMulInv = 2, kInvInPlace = 3, kInvToFields = 4 };
constexpr int kFftThreads = 256;             // threads per FFT tile
constexpr size_t kFftTileBytes = 100 * 1024;  // shared-memory budget of one tile (lines per tile follow)
// Largest dynamic shared memory of an FFT tile: four line buffers plus the
// twiddles fit the tile budget whenever a tile holds more than one line, and a
// single 1024-point line takes 4 x 16 KB + 16 KB.
constexpr size_t kFftSmemMax = kFftTileBytes > 5 * 1024 * 16 ? kFftTileBytes : 5 * 1024 * 16;

struct FftPass {
    int n, log2n;
    int log2T;              // log2 of T (every extent and T are powers of two)
    long long es, ls;       // element stride, stride between the tile's lines
    int T;                  // lines per tile
    long long tiles_inner;  // tiles per outer slab
    long long outer_stride;
    const Cplx* tw;         // exp(-2 pi i k / n), k < n/2
    int axis;               // axis of the lines (0, 1, 2)
};

struct FieldsND {
    int dims, nx, ny, nz;
    int lnx, lny;  // log2 nx, log2 ny (power-of-two extents)
    double L[3], eps, inv_scale, pack;  // pack: power of two that balances phi and E in one complex array
    unsigned long long* rho_acc;
    const double* rho_in;  // when set, the forward pass reads FP64 rho instead of the accumulator
    double* rho;
    Cplx* W;
    Cplx* A;
    Cplx* B;
    double* phi;
    double* E;
    float* E32;  // FP32 form: interleaved float copy of E (2 or 4 floats per node)
    const double* kvec[3];  // wavenumbers 2 pi m / L per axis and index (m the signed mode), or null
    int nacc;    // FP32 form: per-species weight accumulators
    unsigned long long* acc[APIC_MAX_SPECIES];
    double acc_scale[APIC_MAX_SPECIES];  // charge density per accumulator unit
};

__device__ __forceinline__ unsigned bitrev(unsigned x, int bits) { return __brev(x) >> (32 - bits); }

// W16^k = exp(-2 pi i k / 16): cos and sin of 2 pi k / 16, k < 16.
__device__ __forceinline__ double c16(int k) {
    constexpr double a = 0.92387953251128675613, b = 0.70710678118654752440, c = 0.38268343236508977173;
    switch (k & 15) {
        case 0: return 1.0;  case 1: return a;   case 2: return b;   case 3: return c;
        case 4: return 0.0;  case 5: return -c;  case 6: return -b;  case 7: return -a;
        case 8: return -1.0; case 9: return -a;  case 10: return -b; case 11: return -c;
        case 12: return 0.0; case 13: return c;  case 14: return b;  default: return a;
    }
}
__device__ __forceinline__ double s16(int k) { return c16(k + 12); }  // sin x = cos(x - pi/2)

__device__ __forceinline__ Cplx cadd(Cplx x, Cplx y) { return {x.re + y.re, x.im + y.im}; }
__device__ __forceinline__ Cplx csub(Cplx x, Cplx y) { return {x.re - y.re, x.im - y.im}; }
// x * W16^k (forward) or x * conj(W16^k) (inverse)
__device__ __forceinline__ Cplx cw16(Cplx x, int k, bool inv) {
    const double wr = c16(k), wi = inv ? s16(k) : -s16(k);
    return {x.re * wr - x.im * wi, x.re * wi + x.im * wr};
}

template <int R>
__device__ __forceinline__ void dft_small(Cplx* a, bool inv);

template <>
__device__ __forceinline__ void dft_small<2>(Cplx* a, bool) {
    const Cplx t = a[0];
    a[0] = cadd(t, a[1]);
    a[1] = csub(t, a[1]);
}

template <>
__device__ __forceinline__ void dft_small<4>(Cplx* a, bool inv) {
    const Cplx t0 = cadd(a[0], a[2]), t1 = csub(a[0], a[2]), t2 = cadd(a[1], a[3]);
    const Cplx d = csub(a[1], a[3]);
    const Cplx t3 = inv ? Cplx{-d.im, d.re} : Cplx{d.im, -d.re};  // (+i) d or (-i) d
    a[0] = cadd(t0, t2);
    a[2] = csub(t0, t2);
    a[1] = cadd(t1, t3);
    a[3] = csub(t1, t3);
}

// R = R1 R2 point DFT from two smaller ones (index m = R2 m1 + m2 in, p = p1 + R1 p2 out).
template <int R1, int R2>
__device__ __forceinline__ void dft_split(Cplx* a, bool inv) {
    constexpr int R = R1 * R2;
    Cplx b[R2][R1];
#pragma unroll
    for (int m2 = 0; m2 < R2; ++m2) {
        Cplx t[R1];
#pragma unroll
        for (int m1 = 0; m1 < R1; ++m1) t[m1] = a[R2 * m1 + m2];
        dft_small<R1>(t, inv);
#pragma unroll
        for (int p1 = 0; p1 < R1; ++p1) b[m2][p1] = (p1 * m2 == 0) ? t[p1] : cw16(t[p1], p1 * m2 * (16 / R), inv);
    }
#pragma unroll
    for (int p1 = 0; p1 < R1; ++p1) {
        Cplx t[R2];
#pragma unroll
        for (int m2 = 0; m2 < R2; ++m2) t[m2] = b[m2][p1];
        dft_small<R2>(t, inv);
#pragma unroll
        for (int p2 = 0; p2 < R2; ++p2) a[p1 + R1 * p2] = t[p2];
    }
}

template <>
__device__ __forceinline__ void dft_small<8>(Cplx* a, bool inv) { dft_split<4, 2>(a, inv); }
template <>
__device__ __forceinline__ void dft_small<16>(Cplx* a, bool inv) { dft_split<4, 4>(a, inv); }

template <int R>
__device__ __forceinline__ void dft_reg(Cplx (&a)[R], bool inv) { dft_small<R>(a, inv); }

// One Stockham radix-R stage over `lines` lines of n points (src -> dst):
// butterfly j reads src[j + m n/R], twiddles by w^(k m) with k = j mod L and
// w = exp(-2 pi i / (L R)), and writes dst[(j - k) R + k + p L].
template <int R>
__device__ void stockham_stage(const Cplx* __restrict__ src, Cplx* __restrict__ dst, int lines, int n, int ld, int L,
                               const Cplx* tw, bool inv) {
    const int nb = n / R;  // a power of two
    const int lnb = __ffs(nb) - 1;
    const int tstep = n / (L * R);
    for (int b = threadIdx.x; b < lines * nb; b += blockDim.x) {
        const int l = b >> lnb, j = b & (nb - 1);
        const int k = j & (L - 1);
        const Cplx* s = src + l * ld;
        Cplx a[R];
#pragma unroll
        for (int m = 0; m < R; ++m) a[m] = s[j + m * nb];
        if (L > 1) {
#pragma unroll
            for (int m = 1; m < R; ++m) {
                Cplx w = tw[k * m * tstep];
                if (inv) w.im = -w.im;
                const Cplx x = a[m];
                a[m] = {x.re * w.re - x.im * w.im, x.re * w.im + x.im * w.re};
            }
        }
        dft_reg<R>(a, inv);
        Cplx* d = dst + l * ld;
        const int o = (j - k) * R + k;
#pragma unroll
        for (int p = 0; p < R; ++p) d[o + p * L] = a[p];
    }
    __syncthreads();
}

// Transforms `lines` lines held in buf0 (buf1 is scratch of the same size);
// returns the buffer that holds the result.  Forward uses exp(-2 pi i k/n),
// inverse the conjugate and a 1/n scale per line, as fft_radix2 does
// (src/FieldSolver.cpp:171-201); the twiddles are exact table values.  Lines
// start ld >= n elements apart.
__device__ Cplx* fft_lines(Cplx* buf0, Cplx* buf1, int lines, int n, int ld, const Cplx* tw, bool inv) {
    Cplx* src = buf0;
    Cplx* dst = buf1;
    int L = 1, rem = n;
    while (rem > 1) {
        if (rem % 16 == 0) { stockham_stage<16>(src, dst, lines, n, ld, L, tw, inv); L *= 16; rem /= 16; }
        else if (rem % 8 == 0) { stockham_stage<8>(src, dst, lines, n, ld, L, tw, inv); L *= 8; rem /= 8; }
        else if (rem % 4 == 0) { stockham_stage<4>(src, dst, lines, n, ld, L, tw, inv); L *= 4; rem /= 4; }
        else { stockham_stage<2>(src, dst, lines, n, ld, L, tw, inv); L *= 2; rem /= 2; }
        Cplx* t = src; src = dst; dst = t;
    }
    if (inv) {
        const double sc = 1.0 / (double)n;
        for (int b = threadIdx.x; b < lines * n; b += blockDim.x) {
            Cplx& v = src[(b / n) * ld + (b & (n - 1))];
            v.re *= sc;
            v.im *= sc;
        }
        __syncthreads();
    }
    return src;
}

__device__ __forceinline__ long long tile_base(const FftPass& f, long long tile) {
    return (tile % f.tiles_inner) * f.T * f.ls + (tile / f.tiles_inner) * f.outer_stride;
}

// element b of the tile: (line l, element e) so that consecutive b are consecutive in memory
__device__ __forceinline__ void tile_elem(const FftPass& f, int b, int& l, int& e) {
    if (f.es == 1) { l = b >> f.log2n; e = b & (f.n - 1); }
    else { e = b >> f.log2T; l = b & (f.T - 1); }
}

// Forward input at node g: the species' fixed-point densities summed (or the
// FP64 rho of a stand-alone solve); the accumulators are cleared and rho kept.
__device__ __forceinline__ double density_at(const FieldsND& F, long long g) {
    double r;
    if (F.rho_in) {
        r = F.rho_in[g];
    } else if (F.nacc) {
        unsigned long long q[APIC_MAX_SPECIES] = {0, 0, 0, 0};
#pragma unroll
        for (int k = 0; k < APIC_MAX_SPECIES; ++k)
            if (k < F.nacc) q[k] = F.acc[k][g];
        r = 0.0;
#pragma unroll
        for (int k = 0; k < APIC_MAX_SPECIES; ++k)
            if (k < F.nacc) {
                r += (double)(long long)q[k] * F.acc_scale[k];
                F.acc[k][g] = 0ull;
            }
    } else {
        r = (double)(long long)F.rho_acc[g] * F.inv_scale;
        F.rho_acc[g] = 0ull;
    }
    F.rho[g] = r;
    return r;
}

// k-space multiply at node g (src/FieldSolver.cpp:470-488, :687-712) into two
// packed spectra A = phi_k + i Ex_k / pack, B = Ey_k / pack + i Ez_k / pack,
// each E component restricted to its Hermitian part (zero on its own Nyquist
// plane) so that both inverse transforms are real pairs
__device__ __forceinline__ void kspace_at(const FieldsND& F, long long g, Cplx r, Cplx& a, Cplx& bb) {
    const double twopi = 2.0 * 3.141592653589793;
    const double ip = 1.0 / F.pack;
    const int ix = (int)(g & (F.nx - 1));
    const int iy = (int)((g >> F.lnx) & (F.ny - 1));
    const int iz = F.dims == 3 ? (int)(g >> (F.lnx + F.lny)) : 0;
    a = {0.0, 0.0};
    bb = {0.0, 0.0};
    if (ix != 0 || iy != 0 || iz != 0) {
        const double mx = ix <= F.nx / 2 ? (double)ix : -(double)(F.nx - ix);
        const double my = iy <= F.ny / 2 ? (double)iy : -(double)(F.ny - iy);
        const double kx = twopi * mx / F.L[0];
        const double ky = twopi * my / F.L[1];
        double kz = 0.0, k2;
        if (F.dims == 3) {
            const double mz = iz <= F.nz / 2 ? (double)iz : -(double)(F.nz - iz);
            kz = twopi * mz / F.L[2];
            k2 = kx * kx + ky * ky + kz * kz;
        } else {
            k2 = kx * kx + ky * ky;
        }
        const double den = F.eps * k2;
        const double pr = r.re / den, pi = r.im / den;
        // -(0,1) k phik = (k pi, -(k pr))
        const bool nyx = (F.nx % 2 == 0) && ix == F.nx / 2;
        const bool nyy = (F.ny % 2 == 0) && iy == F.ny / 2;
        const bool nyz = F.dims == 3 && (F.nz % 2 == 0) && iz == F.nz / 2;
        const double exr = nyx ? 0.0 : kx * pi, exi = nyx ? 0.0 : -(kx * pr);
        const double eyr = nyy ? 0.0 : ky * pi, eyi = nyy ? 0.0 : -(ky * pr);
        const double ezr = nyz ? 0.0 : kz * pi, ezi = nyz ? 0.0 : -(kz * pr);
        a = {pr - exi * ip, pi + exr * ip};
        bb = {eyr * ip - ezi * ip, eyi * ip + ezr * ip};
    }
}

// kspace_at with the wavenumbers read from the per-axis tables (the same
// values, computed on the host) and one correctly rounded reciprocal of
// eps k^2 in place of two divisions
__device__ __forceinline__ void kspace_tab(const FieldsND& F, long long g, Cplx r, Cplx& a, Cplx& bb) {
    const double ip = 1.0 / F.pack;
    const int ix = (int)(g & (F.nx - 1));
    const int iy = (int)((g >> F.lnx) & (F.ny - 1));
    const int iz = F.dims == 3 ? (int)(g >> (F.lnx + F.lny)) : 0;
    a = {0.0, 0.0};
    bb = {0.0, 0.0};
    if (ix != 0 || iy != 0 || iz != 0) {
        const double kx = __ldg(F.kvec[0] + ix), ky = __ldg(F.kvec[1] + iy);
        const double kz = F.dims == 3 ? __ldg(F.kvec[2] + iz) : 0.0;
        const double k2 = F.dims == 3 ? kx * kx + ky * ky + kz * kz : kx * kx + ky * ky;
        const double inv = __drcp_rn(F.eps * k2);
        const double pr = r.re * inv, pi = r.im * inv;
        const bool nyx = ix == F.nx / 2, nyy = iy == F.ny / 2, nyz = F.dims == 3 && iz == F.nz / 2;
        const double exr = nyx ? 0.0 : kx * pi, exi = nyx ? 0.0 : -(kx * pr);
        const double eyr = nyy ? 0.0 : ky * pi, eyi = nyy ? 0.0 : -(ky * pr);
        const double ezr = nyz ? 0.0 : kz * pi, ezi = nyz ? 0.0 : -(kz * pr);
        a = {pr - exi * ip, pi + exr * ip};
        bb = {eyr * ip - ezi * ip, eyi * ip + ezr * ip};
    }
}

// phi and E at node g from the inverse transforms of the packed spectra
__device__ __forceinline__ void store_fields(const FieldsND& F, long long g, Cplx a, Cplx bb) {
    F.phi[g] = a.re;
    if (F.dims == 2) {
        reinterpret_cast<double2*>(F.E)[g] = make_double2(a.im * F.pack, bb.re * F.pack);
        if (F.E32) reinterpret_cast<float2*>(F.E32)[g] = make_float2((float)(a.im * F.pack), (float)(bb.re * F.pack));
    } else {
        reinterpret_cast<double4*>(F.E)[g] = make_double4(a.im * F.pack, bb.re * F.pack, bb.im * F.pack, 0.0);
        if (F.E32)
            reinterpret_cast<float4*>(F.E32)[g] =
                make_float4((float)(a.im * F.pack), (float)(bb.re * F.pack), (float)(bb.im * F.pack), 0.0f);
    }
}

template <int MODE>
__global__ void __launch_bounds__(kFftThreads) k_fft(FieldsND F, FftPass f) {
    extern __shared__ __align__(16) unsigned char fsm[];
    // shared memory: region0 (2 T lines) and region1 (2 T lines), then the
    // n twiddles; a single array ping-pongs inside region0, an (A, B) pair
    // occupies 2 T lines and ping-pongs between the two regions
    const int ld = f.n;
    Cplx* R0 = reinterpret_cast<Cplx*>(fsm);
    Cplx* R1 = R0 + 2 * f.T * ld;
    Cplx* tws = R1 + ((MODE == kFwdFromRho || MODE == kFwdInPlace) ? 0 : 2 * f.T * ld);
    for (int k = threadIdx.x; k < f.n; k += blockDim.x) tws[k] = f.tw[k];
    Cplx* X = R0;
    Cplx* Y = R0 + f.T * ld;  // B lines of a pair, right after the A lines
    const long long base = tile_base(f, blockIdx.x);
    const int total = f.T * f.n;
    // ---- load (bit-reversed within each line) ----
    for (int b = threadIdx.x; b < total; b += blockDim.x) {
        int l, e;
        tile_elem(f, b, l, e);
        const long long g = base + l * f.ls + e * f.es;
        const int s = l * ld + e;
        if (MODE == kFwdFromRho) {
            X[s] = {density_at(F, g), 0.0};
        } else if (MODE == kFwdInPlace || MODE == kFwdMulInv) {
            X[s] = F.W[g];
        } else {
            X[s] = F.A[g];
            Y[s] = F.B[g];
        }
    }
    __syncthreads();
    const bool inverse_first = (MODE == kInvInPlace || MODE == kInvToFields);
    Cplx* res;
    if (inverse_first) res = fft_lines(R0, R1, 2 * f.T, f.n, f.n, tws, true);           // A and B together
    else res = fft_lines(X, X + f.T * ld, f.T, f.n, f.n, tws, false);                    // ping-pong inside region0
    X = res;
    Y = res + f.T * ld;
    if (MODE == kFwdMulInv) {
        for (int b = threadIdx.x; b < total; b += blockDim.x) {
            int l, e;
            tile_elem(f, b, l, e);
            const long long g = base + l * f.ls + e * f.es;
            Cplx a, bb;
            kspace_at(F, g, X[l * ld + e], a, bb);
            const int s = l * ld + e;
            R1[s] = a;
            R1[f.T * ld + s] = bb;
        }
        __syncthreads();
        Cplx* pair = fft_lines(R1, R0, 2 * f.T, f.n, f.n, tws, true);
        X = pair;
        Y = pair + f.T * ld;
    }
    // ---- store ----
    for (int b = threadIdx.x; b < total; b += blockDim.x) {
        int l, e;
        tile_elem(f, b, l, e);
        const long long g = base + l * f.ls + e * f.es;
        const int s = l * ld + e;
        if (MODE == kFwdFromRho || MODE == kFwdInPlace) {
            F.W[g] = X[s];
        } else if (MODE == kFwdMulInv) {
            F.A[g] = X[s];
            F.B[g] = Y[s];
        } else if (MODE == kInvInPlace) {
            F.A[g] = X[s];
            F.B[g] = Y[s];
        } else {
            store_fields(F, g, X[s], Y[s]);
        }
    }
}

// ---- lines of 32 .. 256 points: a four-step FFT in registers -----------------------
//
// Lines of R1 x R2 points (R1 >= R2, both powers of two), eight lines per CTA
// and R2 threads per line.  Thread slot s of a line holds the points s + R2 j
// (j < R1) in registers: an R1-point DFT over j, the twiddles w^(s k1), one exchange
// through shared memory (thread s then holds the rows k1 = s + R2 q), R2-point
// DFTs, and the thread holds the transform at s + R2 j again, the same positions
// it loaded, so a pass reads and writes each element once and in place.  Lanes run
// along the line on the x pass (R2 consecutive points) and across the
// tile's lines on the strided y / z passes (8 consecutive lines, 128 B), so
// global accesses move whole segments; the registers hold the
// loads in flight (R1 or 2 R1 per thread) instead of a shared-memory tile.
// Against the shared-memory tiles of k_fft: 256^3 solve 2.77 -> 1.15 ms; 64^3
// 78 -> 39 us, 256 x 128 (few lines) 31.7 -> 29.8 us.
constexpr int kRegLines = 8;

template <int R2, bool XP>
__device__ __forceinline__ void reg_map(int tid, int& l, int& s) {
    if (XP) { s = tid & (R2 - 1); l = tid / R2; }
    else { l = tid & (kRegLines - 1); s = tid / kRegLines; }
}

// exchange slot of (line l, row r, column c): written by slot c as row r,
// read by column; spread over the banks for both lane layouts
template <int R1, int R2, bool XP>
__device__ __forceinline__ int reg_xi(int l, int r, int c) {
    return XP ? (l * R1 + r) * (R2 + 1) + c : (r * R2 + c) * kRegLines + l;
}
template <int R1, int R2, bool XP>
constexpr int reg_xsize() { return XP ? kRegLines * R1 * (R2 + 1) : kRegLines * R1 * R2; }

// forward (inv = false) or inverse transforms of NA lines held as a[k][R1]
template <int R1, int R2, bool XP, int NA>
__device__ __forceinline__ void fft_reg(Cplx (&a)[NA][R1], Cplx* xb, const Cplx* tws, int l, int s, bool inv) {
    constexpr int N = R1 * R2, Q = R1 / R2;
#pragma unroll
    for (int k = 0; k < NA; ++k) {
        dft_small<R1>(a[k], inv);
#pragma unroll
        for (int k1 = 1; k1 < R1; ++k1) {
            Cplx w = tws[(s * k1) & (N - 1)];
            if (inv) w.im = -w.im;
            const Cplx x = a[k][k1];
            a[k][k1] = {x.re * w.re - x.im * w.im, x.re * w.im + x.im * w.re};
        }
    }
    __syncthreads();  // earlier readers of the exchange buffers are done
#pragma unroll
    for (int k = 0; k < NA; ++k)
#pragma unroll
        for (int k1 = 0; k1 < R1; ++k1) xb[k * reg_xsize<R1, R2, XP>() + reg_xi<R1, R2, XP>(l, k1, s)] = a[k][k1];
    __syncthreads();
#pragma unroll
    for (int k = 0; k < NA; ++k)
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            Cplx t[R2];
#pragma unroll
            for (int c = 0; c < R2; ++c) t[c] = xb[k * reg_xsize<R1, R2, XP>() + reg_xi<R1, R2, XP>(l, s + R2 * q, c)];
            dft_small<R2>(t, inv);
#pragma unroll
            for (int c = 0; c < R2; ++c) {
                if (inv) {
                    t[c].re *= 1.0 / N;
                    t[c].im *= 1.0 / N;
                }
                a[k][q + Q * c] = t[c];
            }
        }
}

template <int MODE, bool XP, int R1, int R2>
__global__ void __launch_bounds__(kRegLines * R2, 48 / R2) k_fft_reg(FieldsND F, FftPass f) {
    extern __shared__ __align__(16) unsigned char reg_sm[];
    Cplx* tws = reinterpret_cast<Cplx*>(reg_sm);
    Cplx* xb = tws + R1 * R2;
    for (int k = threadIdx.x; k < R1 * R2; k += blockDim.x) tws[k] = f.tw[k];
    int l, s;
    reg_map<R2, XP>(threadIdx.x, l, s);
    const long long base = tile_base(f, blockIdx.x) + l * f.ls + s * f.es;
    const long long step = R2 * f.es;  // between a thread's points
    constexpr bool PAIR = MODE == kInvInPlace || MODE == kInvToFields;
    Cplx a[PAIR ? 2 : 1][R1];
    // ---- load ----
    if constexpr (MODE == kFwdFromRho) {
        // density_at with every load issued before the stores (the arrays may
        // alias as far as the compiler knows); the same sums in species order
        double r[R1];
        if (F.rho_in) {
#pragma unroll
            for (int j = 0; j < R1; ++j) r[j] = F.rho_in[base + j * step];
        } else if (F.nacc) {
#pragma unroll
            for (int j = 0; j < R1; ++j) r[j] = 0.0;
            for (int k = 0; k < F.nacc; ++k) {
                unsigned long long q[R1];
#pragma unroll
                for (int j = 0; j < R1; ++j) q[j] = F.acc[k][base + j * step];
#pragma unroll
                for (int j = 0; j < R1; ++j) r[j] += (double)(long long)q[j] * F.acc_scale[k];
            }
            for (int k = 0; k < F.nacc; ++k)
#pragma unroll
                for (int j = 0; j < R1; ++j) F.acc[k][base + j * step] = 0ull;
        } else {
            unsigned long long q[R1];
#pragma unroll
            for (int j = 0; j < R1; ++j) q[j] = F.rho_acc[base + j * step];
#pragma unroll
            for (int j = 0; j < R1; ++j) {
                r[j] = (double)(long long)q[j] * F.inv_scale;
                F.rho_acc[base + j * step] = 0ull;
            }
        }
#pragma unroll
        for (int j = 0; j < R1; ++j) {
            F.rho[base + j * step] = r[j];
            a[0][j] = {r[j], 0.0};
        }
    } else {
#pragma unroll
        for (int j = 0; j < R1; ++j) {
            const long long g = base + j * step;
            if (MODE == kFwdInPlace || MODE == kFwdMulInv) a[0][j] = F.W[g];
            else {
                a[0][j] = F.A[g];
                a[PAIR ? 1 : 0][j] = F.B[g];
            }
        }
    }
    __syncthreads();  // the twiddles are staged
    if constexpr (MODE == kFwdMulInv) {
        fft_reg<R1, R2, XP, 1>(a, xb, tws, l, s, false);
        Cplx ab[2][R1];
#pragma unroll
        for (int j = 0; j < R1; ++j) kspace_tab(F, base + j * step, a[0][j], ab[0][j], ab[1][j]);
        fft_reg<R1, R2, XP, 2>(ab, xb, tws, l, s, true);
#pragma unroll
        for (int j = 0; j < R1; ++j) {
            const long long g = base + j * step;
            F.A[g] = ab[0][j];
            F.B[g] = ab[1][j];
        }
    } else {
        fft_reg<R1, R2, XP, PAIR ? 2 : 1>(a, xb, tws, l, s, PAIR);
    // ---- store ----
#pragma unroll
    for (int j = 0; j < R1; ++j) {
        const long long g = base + j * step;
        if (MODE == kFwdFromRho || MODE == kFwdInPlace) F.W[g] = a[0][j];
        else if (MODE == kInvInPlace) {
            F.A[g] = a[0][j];
            F.B[g] = a[PAIR ? 1 : 0][j];
        } else {
            store_fields(F, g, a[0][j], a[PAIR ? 1 : 0][j]);
        }
    }
    }
}

// shared memory of a register pass: the twiddles and one exchange buffer per line set
template <int R1, int R2, bool XP>
constexpr size_t reg_smem(int mode) {
    return (R1 * R2 + (size_t)((mode == kFwdMulInv || mode == kInvInPlace || mode == kInvToFields) ? 2 : 1) *
                          reg_xsize<R1, R2, XP>()) * sizeof(Cplx);
}

// Simulation2D/3D sample reductions (src/Diagnostics.cpp:111-137, :205-232):
// kinetic energy of v per species and field energy / charge_l1 of the grid;
// per-block partials, the last block adds them in block order.
constexpr int kSampleBlocks = 148;
__global__ void __launch_bounds__(256) k_sample_nd(SpeciesND S, const uint8_t* alive, const unsigned* id, int dims,
                                                   double* partial, unsigned* done, double* out, const double* E, const double* rho,
                                                   long long N, double half_eps_vol, double vol, int species,
                                                   int last_species, int wall_x, int wall_y, int wall_z, int nx,
                                                   int ny, int nz) {
    __shared__ double red[8], red2[8], red3[8];
    __shared__ bool last;
    const int tid = threadIdx.x;
    double ke = 0.0, fe = 0.0, l1 = 0.0;
    for (unsigned i = blockIdx.x * 256 + tid; i < S.n; i += gridDim.x * 256)
        if (!alive || alive[i]) {
            const unsigned k = id ? id[i] : i;
            ke += S.hmw * (S.v[0][k] * S.v[0][k] + S.v[1][k] * S.v[1][k] + S.v[2][k] * S.v[2][k]);
        }
    if (last_species) {
        for (long long g = blockIdx.x * 256 + tid; g < N; g += gridDim.x * 256) {
            double e2;
            if (dims == 2) {
                const double2 e = reinterpret_cast<const double2*>(E)[g];
                e2 = e.x * e.x + e.y * e.y;
            } else {
                const double4 e = reinterpret_cast<const double4*>(E)[g];
                e2 = e.x * e.x + e.y * e.y + e.z * e.z;
            }
            // Mesh2D::node_area / Mesh3D::node_volume: half cells on the wall
            // nodes, src/Mesh2D.cpp:77-88, src/Mesh3D.cpp:52-60
            const int gi = (int)(g % nx), gj = (int)((g / nx) % ny), gk = (int)(g / ((long long)nx * ny));
            const double f = ((wall_x && (gi == 0 || gi == nx - 1)) ? 0.5 : 1.0) *
                             ((wall_y && (gj == 0 || gj == ny - 1)) ? 0.5 : 1.0) *
                             ((wall_z && (gk == 0 || gk == nz - 1)) ? 0.5 : 1.0);
            fe += half_eps_vol * e2 * f;
            l1 += fabs(rho[g]) * vol * f;
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        ke += __shfl_down_sync(0xffffffffu, ke, o);
        fe += __shfl_down_sync(0xffffffffu, fe, o);
        l1 += __shfl_down_sync(0xffffffffu, l1, o);
    }
    if ((tid & 31) == 0) { red[tid >> 5] = ke; red2[tid >> 5] = fe; red3[tid >> 5] = l1; }
    __syncthreads();
    if (tid == 0) {
        double a = 0, b = 0, c = 0;
        for (int w = 0; w < 8; ++w) { a += red[w]; b += red2[w]; c += red3[w]; }
        partial[3 * blockIdx.x] = a;
        partial[3 * blockIdx.x + 1] = b;
        partial[3 * blockIdx.x + 2] = c;
        __threadfence();
        last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || tid != 0) return;
    __threadfence();
    double a = 0, b = 0, c = 0;
    for (unsigned k = 0; k < gridDim.x; ++k) {
        a += ((volatile double*)partial)[3 * k];
        b += ((volatile double*)partial)[3 * k + 1];
        c += ((volatile double*)partial)[3 * k + 2];
    }
    out[species] = a;
    if (last_species) { out[4] = b; out[5] = c; }
    *done = 0;
}

// ---- host ----------------------------------------------------------------------------

static bool pow2(size_t v) { return v >= 2 && (v & (v - 1)) == 0; }
static int ilog2(size_t v) { int k = 0; while ((size_t(1) << k) < v) ++k; return k; }

// Raises the dynamic shared-memory limit of every FFT / wall-solve kernel, once
// per device, to a fixed bound that covers every tile any mesh here uses.  The
// limit is a property of the kernel function shared by every simulation and
// solve in the process, so it is never lowered to one mesh's need (a later
// small mesh would otherwise make an earlier large mesh's launches fail).
// Raises a kernel's limit of dynamic shared memory, once per device.  Called where a run is set
// up, for the kernels it will launch and no others: the call loads the kernel, and all of
// the field solves' together took 11 ms of a process's first run.
static void allow_smem(const void* kernel, size_t bytes) {
    static std::mutex mu;
    static std::set<std::pair<int, const void*>> done;
    int dev = 0;
    APIC_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if (done.count({dev, kernel})) return;
    APIC_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes));
    done.insert({dev, kernel});
}
template <class... Args>
static void allow_smem(void (*kernel)(Args...), size_t bytes) {
    allow_smem(reinterpret_cast<const void*>(kernel), bytes);
}

struct Solver {
    FieldsND F{};
    FftPass px{}, py{}, pz{};    // paired passes (four line buffers)
    FftPass pxs{}, pys{};        // single-array forward passes (two line buffers)
    bool in_regs[3] = {false, false, false};  // axis a runs the register kernels
    FftPass reg[3]{};
    size_t smem_fwd = 0, smem_pair = 0;
    std::vector<void*>* allocs = nullptr;
    cudaStream_t stream = nullptr;

    template <class T>
    T* alloc(size_t count) {
        void* p = nullptr;
        APIC_CUDA(cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T)));
        allocs->push_back(p);
        APIC_CUDA(cudaMemsetAsync(p, 0, std::max<size_t>(count, 1) * sizeof(T), stream));
        return static_cast<T*>(p);
    }

    Cplx* twiddles(int n) {
        std::vector<Cplx> h(n);
        const double twopi = 2.0 * 3.141592653589793;
        for (int k = 0; k < n; ++k) h[k] = {std::cos(twopi * k / n), -std::sin(twopi * k / n)};
        Cplx* d = alloc<Cplx>(h.size());
        APIC_CUDA(cudaMemcpyAsync(d, h.data(), h.size() * sizeof(Cplx), cudaMemcpyHostToDevice, stream));
        APIC_CUDA(cudaStreamSynchronize(stream));
        return d;
    }

    FftPass pass(int ax, int T) const {
        FftPass f{};
        const long long nx = F.nx, ny = F.ny, nz = F.dims == 3 ? F.nz : 1;
        f.axis = ax;
        f.T = T;
        if (ax == 0) {
            f.n = F.nx; f.es = 1; f.ls = nx;
            f.tiles_inner = ny * nz / T; f.outer_stride = 0;
        } else if (ax == 1) {
            f.n = F.ny; f.es = nx; f.ls = 1;
            f.tiles_inner = nx / T; f.outer_stride = nx * ny;
        } else {
            f.n = F.nz; f.es = nx * ny; f.ls = 1;
            f.tiles_inner = nx / T; f.outer_stride = nx;
        }
        f.log2n = ilog2(f.n);
        f.log2T = ilog2(T);
        return f;
    }

    long long tiles(const FftPass& f) const {
        const long long N = (long long)F.nx * F.ny * (F.dims == 3 ? F.nz : 1);
        return N / ((long long)f.T * f.n);
    }

    void setup(int dims, const size_t* n, const double* L, double eps, double inv_scale) {
        F.dims = dims;
        F.nx = (int)n[0]; F.ny = (int)n[1]; F.nz = dims == 3 ? (int)n[2] : 1;
        F.lnx = ilog2(F.nx);
        F.lny = ilog2(F.ny);
        for (int a = 0; a < 3; ++a) F.L[a] = a < dims ? L[a] : 1.0;
        F.eps = eps;
        F.inv_scale = inv_scale;
        double kmax = 0;
        for (int a = 0; a < dims; ++a) kmax = std::max(kmax, 3.141592653589793 * (double)n[a] / L[a]);
        F.pack = std::ldexp(1.0, (int)std::lround(std::log2(kmax)));
        const size_t N = (size_t)F.nx * F.ny * F.nz;
        F.rho_acc = alloc<unsigned long long>(N);
        F.rho = alloc<double>(N);
        F.W = alloc<Cplx>(N);
        F.A = alloc<Cplx>(N);
        F.B = alloc<Cplx>(N);
        F.phi = alloc<double>(N);
        F.E = alloc<double>(N * (dims == 2 ? 2 : 4));
        // lines per tile: up to 8 (128 B rows in the strided passes), bounded
        // so that the paired passes (three line buffers) fit in shared memory
        // lines per tile: up to 8 (128 B rows in the strided passes), bounded
        // so that two CTAs fit on an SM (about 100 KB of shared memory each)
        auto lines = [](int n, long long available, int buffers) {
            int T = 8;
            while (T > 1 && (size_t)buffers * T * n * sizeof(Cplx) + n * sizeof(Cplx) > kFftTileBytes) T >>= 1;
            while (T > 1 && available % T) T >>= 1;
            return T;
        };
        px = pass(0, lines(F.nx, (long long)F.ny * F.nz, 4));
        pxs = pass(0, lines(F.nx, (long long)F.ny * F.nz, 2));
        py = pass(1, lines(F.ny, F.nx, 4));
        pys = pass(1, lines(F.ny, F.nx, 2));
        if (dims == 3) pz = pass(2, lines(F.nz, F.nx, 4));
        px.tw = pxs.tw = twiddles(F.nx);
        py.tw = pys.tw = F.ny == F.nx ? px.tw : twiddles(F.ny);
        if (dims == 3) pz.tw = F.nz == F.nx ? px.tw : (F.nz == F.ny ? py.tw : twiddles(F.nz));
        for (int a = 0; a < dims; ++a) {  // kspace_at's wavenumbers, src/FieldSolver.cpp:687-712
            const int na = a == 0 ? F.nx : (a == 1 ? F.ny : F.nz);
            std::vector<double> kv(na);
            const double twopi = 2.0 * 3.141592653589793;
            for (int i = 0; i < na; ++i) {
                const double m = i <= na / 2 ? (double)i : -(double)(na - i);
                kv[i] = twopi * m / F.L[a];
            }
            double* d = alloc<double>(na);
            APIC_CUDA(cudaMemcpyAsync(d, kv.data(), na * sizeof(double), cudaMemcpyHostToDevice, stream));
            APIC_CUDA(cudaStreamSynchronize(stream));
            F.kvec[a] = d;
        }
        for (int a = 0; a < dims; ++a) {
            const long long lines = a == 0 ? (long long)F.ny * F.nz : F.nx;
            in_regs[a] = n[a] >= 32 && n[a] <= 256 && lines % kRegLines == 0;
            if (in_regs[a]) {
                reg[a] = pass(a, kRegLines);
                reg[a].tw = a == 0 ? px.tw : (a == 1 ? py.tw : pz.tw);
            }
        }
        smem_pair = std::max(smem_of(px, kFwdMulInv), smem_of(py, kFwdMulInv));
        if (dims == 3) smem_pair = std::max(smem_pair, smem_of(pz, kFwdMulInv));
        require(smem_pair <= kFftSmemMax, "FFT tile exceeds the shared-memory bound", APIC_ERR_UNSUPPORTED);
        allow_passes();
    }

    // the shared memory of the passes of solve()
    void allow_passes() {
        if (F.dims == 2) {
            allow_pass<kFwdFromRho>(0);
            allow_pass<kFwdMulInv>(1);
        } else {
            allow_pass<kFwdFromRho>(0);
            allow_pass<kFwdInPlace>(1);
            allow_pass<kFwdMulInv>(2);
            allow_pass<kInvInPlace>(1);
        }
        allow_pass<kInvToFields>(0);
    }
    template <int MODE, int R1, int R2>
    static void allow_reg(int axis) {
        if (axis == 0) allow_smem(k_fft_reg<MODE, true, R1, R2>, reg_smem<R1, R2, true>(MODE));
        else allow_smem(k_fft_reg<MODE, false, R1, R2>, reg_smem<R1, R2, false>(MODE));
    }
    template <int MODE>
    void allow_pass(int axis) {
        if (!in_regs[axis]) allow_smem(k_fft<MODE>, kFftSmemMax);
        else if (reg[axis].n == 256) allow_reg<MODE, 16, 16>(axis);
        else if (reg[axis].n == 128) allow_reg<MODE, 16, 8>(axis);
        else if (reg[axis].n == 64) allow_reg<MODE, 8, 8>(axis);
        else allow_reg<MODE, 8, 4>(axis);
    }

    size_t smem_of(const FftPass& f, int mode) const {
        const size_t line = (size_t)f.T * f.n * sizeof(Cplx);
        const size_t tw = (size_t)f.n * sizeof(Cplx);
        return (mode == kFwdFromRho || mode == kFwdInPlace) ? 2 * line + tw : 4 * line + tw;
    }

    // one pass along `axis`: the register kernel where the extent
    // allows it, else the shared-memory tile kernel with pass `tile`
    template <int MODE, int R1, int R2>
    void reg_pass(int axis) {
        const FftPass& q = reg[axis];
        const unsigned g = (unsigned)tiles(q);
        if (axis == 0)
            k_fft_reg<MODE, true, R1, R2><<<g, kRegLines * R2, reg_smem<R1, R2, true>(MODE), stream>>>(F, q);
        else
            k_fft_reg<MODE, false, R1, R2><<<g, kRegLines * R2, reg_smem<R1, R2, false>(MODE), stream>>>(F, q);
    }
    template <int MODE>
    void fft_pass(int axis, const FftPass& tile) {
        if (!in_regs[axis]) k_fft<MODE><<<(unsigned)tiles(tile), kFftThreads, smem_of(tile, MODE), stream>>>(F, tile);
        else if (reg[axis].n == 256) reg_pass<MODE, 16, 16>(axis);
        else if (reg[axis].n == 128) reg_pass<MODE, 16, 8>(axis);
        else if (reg[axis].n == 64) reg_pass<MODE, 8, 8>(axis);
        else reg_pass<MODE, 8, 4>(axis);
    }

    // rho_acc -> rho, phi, E (the fixed-point accumulator is cleared)
    void solve() {
        if (F.dims == 2) {
            fft_pass<kFwdFromRho>(0, pxs);
            fft_pass<kFwdMulInv>(1, py);
            fft_pass<kInvToFields>(0, px);
        } else {
            fft_pass<kFwdFromRho>(0, pxs);
            fft_pass<kFwdInPlace>(1, pys);
            fft_pass<kFwdMulInv>(2, pz);
            fft_pass<kInvInPlace>(1, py);
            fft_pass<kInvToFields>(0, px);
        }
        APIC_CUDA(cudaGetLastError());
    }
};

// ---- field solves with walls --------------------------------------------------------
//
// One periodic axis (2D): solve_mixed_spectral_tridiagonal and
// compute_electric_field, src/FieldSolver.cpp:501-657, :298-346: the rows are
// transformed along the periodic axis, each mode solves a tridiagonal system
// across the walls (eigenvalue 4 sin^2(pi m / N) / h^2 of the periodic second
// difference, wall potentials on mode 0 scaled by N) and is transformed back.
// The density is real, so two rows share one complex transform and only the
// modes m <= N / 2 are kept, mode by mode: hat[m][row].
//
// Walls on every side (2D, and 3D grounded): the reference iterates SOR to a
// 1e-11 update (solve_dirichlet_iterative, src/FieldSolver.cpp:761-907); the same
// discrete system is solved directly.  The discrete sine transform (DST-I)
// diagonalises the second difference of each axis (eigenvalues
// 4 sin^2(pi m / (2 (M + 1))) / h^2 over the M interior nodes): DST passes, a
// division and DST passes again, a DST-I being an odd-extended FFT of length
// 2 (M + 1), two real lines in one complex transform.  Wall potentials (2D
// sides, corners the mean of their two sides) enter the right-hand side of the
// nodes next to the walls.
//
// Solve per step on the B200, before (one real line per CTA and transform, a
// serial sweep per mode, separate passes for every elementwise stage) -> now:
// 512 x 513 (mixed) 87 -> 39 us, 129^3 949 -> 304 us, with the register transforms 133 us.
constexpr size_t kWallTileBytes = 72 * 1024;  // shared memory of a tile: three CTAs per SM
constexpr size_t kWallSmemMax = (2 * ((size_t)kMaxLine + 1) + kMaxLine) * sizeof(Cplx) > kWallTileBytes
                                    ? (2 * ((size_t)kMaxLine + 1) + kMaxLine) * sizeof(Cplx) : kWallTileBytes;

// line pairs per tile for transforms of length n over `lines` real lines: as
// many as the tile's shared memory holds, while two waves of CTAs remain
inline int wall_pairs(int n, long long lines) {
    int T = 8;
    while (T > 1 && ((2 * (size_t)T * (n + 1) + n) * sizeof(Cplx) > kWallTileBytes || lines / (2 * T) < 2 * 148)) T >>= 1;
    return T;
}
inline size_t wall_smem(int n, int T) { return (2 * (size_t)T * (n + 1) + n) * sizeof(Cplx); }

enum : int { kDstFromRho = 0, kDstInPlace = 1, kDstSolve = 2, kDstToPhi = 3 };

struct DstPass {
    int M, log2N;                  // interior nodes of the axis; N = 2 (M + 1)
    int T;                         // line pairs per CTA
    int lines, lines_a;            // real lines; lines of the faster of the two other axes
    long long stride, stride_a, stride_b;  // in the compact interior array
    int axis;
    const Cplx* tw;                // exp(-2 pi i k / N)
    const double* eig[3];          // eigenvalues per axis and interior index
    double scale;                  // inverse normalisation (kDstSolve)
    bool in_regs;                  // k_dst_reg
};
// Lines from which the register passes are taken: a CTA holds 16 of them and each thread a chain of
// 16-point transforms, so few lines are few CTAs of long latency, where k_dst_pass spreads a line pair
// over a CTA.  Step of runs with 2 particles a node, registers against tiles, us: 63 lines
// (65^2) 35 / 28, 225 (129 x 17 x 17) 60 / 58, 511 (513 x 65) 41.2 / 39.5, 961 (33^3) 50 / 60.
constexpr int kDstRegLines = 512;

struct WallMesh {
    int dims, n[3];
    double d[3], eps;
    double side[4];                // 2D potentials: left, right, bottom, top
    int wall[3];
    double rd[2][3], reps;         // reciprocals of d and of 2 d, and of eps
    double ih2[2];                 // 1 / d^2 of x and y
};

// Lines of M values in place (or from rho, or into phi): X_m = sum_k x_k
// sin(pi k m / (M + 1)).  With two odd-extended lines as real and imaginary
// parts, the transform is 2 X2 - 2 i X1.  kDstSolve transforms, divides by the
// eigenvalues of minus the Laplacian and transforms again.
template <int MODE>
__global__ void __launch_bounds__(kFftThreads) k_dst_pass(double* __restrict__ u, WallMesh w, DstPass f,
                                                          const double* __restrict__ rho, double* __restrict__ phi) {
    extern __shared__ __align__(16) unsigned char dsm[];
    const int M = f.M, N = 2 * (M + 1), ld = N + 1, n2 = 2 * f.T;
    Cplx* a = reinterpret_cast<Cplx*>(dsm);
    Cplx* b = a + f.T * ld;
    Cplx* tws = b + f.T * ld;
    for (int k = threadIdx.x; k < N; k += blockDim.x) tws[k] = f.tw[k];
    const int first = blockIdx.x * n2;
    const int lt = 31 - __clz(n2), total = n2 << (f.log2N - 1);
    // place t of the tile: line l (of n2) and element e in [0, M]; consecutive
    // t are consecutive in memory (e = M is the unused last slot of a line)
    auto place = [&](int t, int& l, int& e) {
        if (f.axis == 0) { l = t >> (f.log2N - 1); e = t & M; }
        else { e = t >> lt; l = t & (n2 - 1); }
    };
    auto put = [&](Cplx* z, int l, int e, double v) {  // interior value e of line l, odd extension
        double* r = reinterpret_cast<double*>(z + (l >> 1) * ld) + (l & 1);
        r[2 * (e + 1)] = v;
        r[2 * (N - 1 - e)] = -v;
    };
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int l, e;
        place(t, l, e);
        const int line = first + l;
        if (e == M) {  // the two zeros of the extension
            double* r = reinterpret_cast<double*>(a + (l >> 1) * ld) + (l & 1);
            r[0] = 0.0;
            r[2 * (M + 1)] = 0.0;
            continue;
        }
        double v = 0.0;
        if (line < f.lines) {
            const int la = line % f.lines_a, lb = line / f.lines_a;
            if (MODE == kDstFromRho) {  // axis 0: line (j, k) = (la, lb), right-hand side at node e
                const size_t node = ((size_t)(w.dims == 3 ? lb + 1 : 0) * w.n[1] + (la + 1)) * w.n[0] + (e + 1);
                v = cells_of(rho[node], w.eps, w.reps);
                if (w.dims == 2) {  // 2D walls at their potentials; 3D walls are grounded
                    if (e == 0) v += w.side[0] * w.ih2[0];
                    if (e == M - 1) v += w.side[1] * w.ih2[0];
                    if (la == 0) v += w.side[2] * w.ih2[1];
                    if (la == w.n[1] - 3) v += w.side[3] * w.ih2[1];
                }
            } else {
                v = u[la * f.stride_a + lb * f.stride_b + e * f.stride];
            }
        }
        put(a, l, e, v);
    }
    __syncthreads();
    Cplx* r = fft_lines(a, b, f.T, N, ld, tws, false);
    auto value = [&](const Cplx* z, int l, int e) {
        const Cplx c = z[(l >> 1) * ld + e + 1];
        return l & 1 ? 0.5 * c.re : -0.5 * c.im;
    };
    if (MODE == kDstSolve) {
        Cplx* o = r == a ? b : a;
        for (int t = threadIdx.x; t < total; t += blockDim.x) {
            int l, e;
            place(t, l, e);
            if (e == M) {
                double* q = reinterpret_cast<double*>(o + (l >> 1) * ld) + (l & 1);
                q[0] = 0.0;
                q[2 * (M + 1)] = 0.0;
                continue;
            }
            const int line = first + l;
            const int la = line % f.lines_a, lb = line / f.lines_a;
            // (the last axis: la is the x index, lb the y index in 3D)
            double lam = f.eig[0][la] + (w.dims == 3 ? f.eig[1][min(lb, w.n[1] - 3)] + f.eig[2][e] : f.eig[1][e]);
            put(o, l, e, value(r, l, e) * (f.scale / lam));
        }
        __syncthreads();
        r = fft_lines(o, r, f.T, N, ld, tws, false);
    }
    for (int t = threadIdx.x; t < total; t += blockDim.x) {
        int l, e;
        place(t, l, e);
        const int line = first + l;
        if (e == M || line >= f.lines) continue;
        const int la = line % f.lines_a, lb = line / f.lines_a;
        const double v = value(r, l, e);
        if (MODE == kDstToPhi)
            phi[((size_t)(w.dims == 3 ? lb + 1 : 0) * w.n[1] + (la + 1)) * w.n[0] + (e + 1)] = v;
        else
            u[la * f.stride_a + lb * f.stride_b + e * f.stride] = v;
    }
}

// The same passes for N = R1 R2 = 64 .. 256 (33 to 129 nodes) in registers, for the many
// lines of a 3D mesh (kDstRegLines; 2D meshes have at most 511): eight
// line pairs per CTA, laid out as in k_fft_reg.  Both halves of the odd extension are read
// from the interior values, and the transform of an odd sequence is odd, so
// the second transform of kDstSolve starts from the first one's own positions.
template <int MODE, bool XP, int R1, int R2>
__global__ void __launch_bounds__(kRegLines * R2, 48 / R2) k_dst_reg(double* __restrict__ u, WallMesh w, DstPass f,
                                                                      const double* __restrict__ rho,
                                                                      double* __restrict__ phi) {
    extern __shared__ __align__(16) unsigned char reg_sm[];
    constexpr int N = R1 * R2, M = N / 2 - 1;
    Cplx* tws = reinterpret_cast<Cplx*>(reg_sm);
    Cplx* xb = tws + N;
    for (int k = threadIdx.x; k < N; k += blockDim.x) tws[k] = f.tw[k];
    int l, s;
    reg_map<R2, XP>(threadIdx.x, l, s);
    int la[2], lb[2];  // the pair's two real lines
    bool in[2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        // strided passes: lane l takes lines l and l + 8 of the tile, so both loads are contiguous
        const int line = blockIdx.x * (2 * kRegLines) + (XP ? 2 * l + c : l + kRegLines * c);
        in[c] = line < f.lines;
        la[c] = in[c] ? line % f.lines_a : 0;
        lb[c] = in[c] ? line / f.lines_a : 0;
    }
    // every load first (no branch between them), then the right-hand side and the extension
    const double* src[2];
    long long stride = 1;
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        if (MODE == kDstFromRho) {
            src[c] = rho + ((size_t)(lb[c] + 1) * w.n[1] + (la[c] + 1)) * w.n[0] + 1;
        } else {
            src[c] = u + la[c] * f.stride_a + lb[c] * f.stride_b;
            stride = f.stride;
        }
    }
    Cplx a[1][R1];
#pragma unroll
    for (int j = 0; j < R1; ++j) {
        const int k = s + R2 * j;
        // (k = 0 and k = M + 1, the extension's zeros, load a neighbour)
        const int e = k <= M ? max(k - 1, 0) : min(N - k - 1, M - 1);
        a[0][j] = {src[0][e * stride], src[1][e * stride]};
    }
#pragma unroll
    for (int j = 0; j < R1; ++j) {
        const int k = s + R2 * j;
        const bool zero = k == 0 || k == M + 1;
        double x[2] = {a[0][j].re, a[0][j].im};
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            if (MODE == kDstFromRho) x[c] = cells_of(x[c], w.eps, w.reps);  // (3D walls are grounded)
            x[c] = zero || !in[c] ? 0.0 : (k <= M ? x[c] : -x[c]);
        }
        a[0][j] = {x[0], x[1]};
    }
    __syncthreads();  // the twiddles are staged
    fft_reg<R1, R2, XP, 1>(a, xb, tws, l, s, false);
    if (MODE == kDstSolve) {
#pragma unroll
        for (int j = 0; j < R1; ++j) {
            const int k = s + R2 * j;
            const bool zero = k == 0 || k == M + 1;
            const int e = zero ? 0 : (k <= M ? k - 1 : N - k - 1);
            double g[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                // (the last axis: la is the x index, lb the y index)
                const double lam = __ldg(f.eig[0] + la[c]) + (__ldg(f.eig[1] + lb[c]) + __ldg(f.eig[2] + e));
                g[c] = zero ? 0.0 : f.scale * __drcp_rn(lam);
            }
            a[0][j] = {-0.5 * a[0][j].im * g[0], 0.5 * a[0][j].re * g[1]};
        }
        fft_reg<R1, R2, XP, 1>(a, xb, tws, l, s, false);
    }
#pragma unroll
    for (int j = 0; j < R1; ++j) {
        const int k = s + R2 * j;
        if (k == 0 || k > M) continue;
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            if (!in[c]) continue;
            const double v = c ? 0.5 * a[0][j].re : -0.5 * a[0][j].im;
            if (MODE == kDstToPhi)
                phi[((size_t)(lb[c] + 1) * w.n[1] + (la[c] + 1)) * w.n[0] + k] = v;
            else
                u[la[c] * f.stride_a + lb[c] * f.stride_b + (k - 1) * f.stride] = v;
        }
    }
}

// The mixed solve's rows: element q of wall row d at rho[d * sd + q * sq].
// Rows 1 .. nd - 2 in pairs, T pairs per CTA; hat[m * ni + row - 1], m <= np / 2.
__global__ void __launch_bounds__(kFftThreads) k_mixed_forward(const double* __restrict__ rho, Cplx* __restrict__ hat,
                                                               int ni, int np, int T, long long sd, long long sq,
                                                               const Cplx* tw) {
    extern __shared__ __align__(16) unsigned char msm[];
    const int ld = np + 1, n2 = 2 * T, first = blockIdx.x * n2;
    Cplx* a = reinterpret_cast<Cplx*>(msm);
    Cplx* b = a + T * ld;
    Cplx* tws = b + T * ld;
    for (int q = threadIdx.x; q < np; q += blockDim.x) tws[q] = tw[q];
    for (int t = threadIdx.x; t < n2 * np; t += blockDim.x) {
        const int l = sq == 1 ? t / np : t & (n2 - 1), q = sq == 1 ? t & (np - 1) : t / n2;
        const double v = first + l < ni ? rho[(first + l + 1) * sd + q * sq] : 0.0;
        reinterpret_cast<double*>(a + (l >> 1) * ld + q)[l & 1] = v;
    }
    __syncthreads();
    const Cplx* z = fft_lines(a, b, T, np, ld, tws, false);
    for (int t = threadIdx.x; t < n2 * (np / 2 + 1); t += blockDim.x) {
        const int l = t & (n2 - 1), m = t / n2;
        if (first + l >= ni) continue;
        const Cplx p = z[(l >> 1) * ld + m], q = z[(l >> 1) * ld + ((np - m) & (np - 1))];
        // p + conj(q) = 2 H_even, p - conj(q) = 2 i H_odd
        hat[(size_t)m * ni + first + l] = l & 1 ? Cplx{0.5 * (p.im + q.im), 0.5 * (q.re - p.re)}
                                                : Cplx{0.5 * (p.re + q.re), 0.5 * (p.im - q.im)};
    }
}

__global__ void __launch_bounds__(kFftThreads) k_mixed_inverse(const Cplx* __restrict__ hat, double* __restrict__ phi,
                                                               int ni, int np, int T, long long sd, long long sq,
                                                               const Cplx* tw) {
    extern __shared__ __align__(16) unsigned char msm[];
    const int ld = np + 1, n2 = 2 * T, first = blockIdx.x * n2;
    Cplx* a = reinterpret_cast<Cplx*>(msm);
    Cplx* b = a + T * ld;
    Cplx* tws = b + T * ld;
    for (int q = threadIdx.x; q < np; q += blockDim.x) tws[q] = tw[q];
    for (int t = threadIdx.x; t < T * (np / 2 + 1); t += blockDim.x) {
        const int l = t & (T - 1), m = t / T, row = first + 2 * l;
        const Cplx h0 = row < ni ? hat[(size_t)m * ni + row] : Cplx{0.0, 0.0};
        const Cplx h1 = row + 1 < ni ? hat[(size_t)m * ni + row + 1] : Cplx{0.0, 0.0};
        a[l * ld + m] = {h0.re - h1.im, h0.im + h1.re};                       // h0 + i h1
        if (m && 2 * m < np) a[l * ld + np - m] = {h0.re + h1.im, h1.re - h0.im};  // conj(h0) + i conj(h1)
    }
    __syncthreads();
    const Cplx* z = fft_lines(a, b, T, np, ld, tws, true);
    for (int t = threadIdx.x; t < n2 * np; t += blockDim.x) {
        const int l = sq == 1 ? t / np : t & (n2 - 1), q = sq == 1 ? t & (np - 1) : t / n2;
        if (first + l < ni) phi[(first + l + 1) * sd + q * sq] = reinterpret_cast<const double*>(z + (l >> 1) * ld + q)[l & 1];
    }
}

// The elimination coefficients of every mode's system depend on the mode
// only: modified_upper mu[m * ni + k] and the reciprocal of the pivot
// inv[m * ni + k], computed once per mesh with the reference's arithmetic.
__global__ void k_mixed_coeffs(double* __restrict__ mu, double* __restrict__ inv, int nd, int np, double inv_dsq,
                               double inv_psq) {
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m > np / 2) return;
    const int ni = nd - 2;
    const double angle = 3.141592653589793 * (double)m / (double)np;
    const double eig = 4.0 * sin(angle) * sin(angle) * inv_psq;
    const double diag = 2.0 * inv_dsq + eig;
    const double off = -inv_dsq;
    double pu = 0.0;
    for (int k = 0; k < ni; ++k) {
        const double den = k == 0 ? diag : diag - off * pu;
        const double u = k == 0 ? off / diag : (k + 1 == ni ? 0.0 : off / den);
        mu[(size_t)m * ni + k] = u;
        inv[(size_t)m * ni + k] = 1.0 / den;
        pu = u;
    }
}

// One warp per mode.  The elimination x_k = (r_k - off x_{k-1}) / pivot and the
// back substitution x_k -= mu_k x_{k+1} are affine recurrences: each lane
// composes its run of consecutive rows, a shuffle scan composes the lanes, and
// each lane runs its rows again from the value that reaches it: 4 ni / 32 steps
// in place of 2 ni.  STAGED: the mode's column and coefficients in shared
// memory (each lane's run one element further apart than its length, so the
// lanes' accesses spread over the banks); longer wall axes read them in place.
constexpr int kMixedSweepMaxRows = 4000;
constexpr size_t mixed_sweep_smem(int ni) { return (size_t)(ni + 32) * (sizeof(Cplx) + 2 * sizeof(double)); }

template <bool STAGED>
__global__ void __launch_bounds__(32) k_mixed_sweep(Cplx* __restrict__ hat, const double* __restrict__ mu,
                                                    const double* __restrict__ inv, int ni, int np, double inv_dsq,
                                                    double eps, double lower, double upper) {
    extern __shared__ __align__(16) unsigned char ssm[];
    const int m = blockIdx.x, lane = threadIdx.x;
    const int run = (ni + 31) / 32;
    Cplx* const col = hat + (size_t)m * ni;
    const double* const cu = mu + (size_t)m * ni;
    const double* const cv = inv + (size_t)m * ni;
    Cplx* R = STAGED ? reinterpret_cast<Cplx*>(ssm) : col;
    double* U = STAGED ? reinterpret_cast<double*>(R + ni + 32) : const_cast<double*>(cu);
    double* V = STAGED ? U + ni + 32 : const_cast<double*>(cv);
    if (STAGED) {
        for (int k = lane; k < ni; k += 32) {
            const int s = k + k / run;
            R[s] = col[k];
            U[s] = cu[k];
            V[s] = cv[k];
        }
        __syncwarp();
    }
    const double ieps = 1.0 / eps, scale = (double)np;
    const double lb = m == 0 ? lower * scale : 0.0, ub = m == 0 ? upper * scale : 0.0;
    const int k0 = min(lane * run, ni), k1 = min(k0 + run, ni), shift = STAGED ? lane : 0;
    // x -> a x + (br, bi): this lane's rows composed, then the lanes before it
    auto scan = [&](double a, double br, double bi, bool up, double& xr, double& xi) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double pa = up ? __shfl_up_sync(0xffffffffu, a, o) : __shfl_down_sync(0xffffffffu, a, o);
            const double pr = up ? __shfl_up_sync(0xffffffffu, br, o) : __shfl_down_sync(0xffffffffu, br, o);
            const double pi = up ? __shfl_up_sync(0xffffffffu, bi, o) : __shfl_down_sync(0xffffffffu, bi, o);
            if (up ? lane >= o : lane + o < 32) {
                br += a * pr;
                bi += a * pi;
                a *= pa;
            }
        }
        const double qr = up ? __shfl_up_sync(0xffffffffu, br, 1) : __shfl_down_sync(0xffffffffu, br, 1);
        const double qi = up ? __shfl_up_sync(0xffffffffu, bi, 1) : __shfl_down_sync(0xffffffffu, bi, 1);
        const bool first = up ? lane == 0 : lane == 31;
        xr = first ? 0.0 : qr;
        xi = first ? 0.0 : qi;
    };
    auto row = [&](int k, double& rr, double& ri) {
        const Cplx h = R[k + shift];
        rr = h.re * ieps;
        ri = h.im * ieps;
        if (k == 0) rr += inv_dsq * lb;  // the boundary terms are real
        if (k + 1 == ni) rr += inv_dsq * ub;
    };
    double a = 1.0, br = 0.0, bi = 0.0, xr, xi;
    for (int k = k0; k < k1; ++k) {  // x_k = (r_k + inv_dsq x_{k-1}) V_k
        double rr, ri;
        row(k, rr, ri);
        const double v = V[k + shift], c = k == 0 ? 0.0 : inv_dsq * v;
        br = c * br + rr * v;
        bi = c * bi + ri * v;
        a *= c;
    }
    scan(a, br, bi, true, xr, xi);
    for (int k = k0; k < k1; ++k) {
        double rr, ri;
        row(k, rr, ri);
        const double v = V[k + shift];
        xr = (k == 0 ? rr : rr + inv_dsq * xr) * v;
        xi = (k == 0 ? ri : ri + inv_dsq * xi) * v;
        R[k + shift] = {xr, xi};
    }
    a = 1.0, br = 0.0, bi = 0.0;
    for (int k = k1 - 1; k >= k0; --k) {  // x_k -= mu_k x_{k+1} (mu of the last row is zero)
        const Cplx h = R[k + shift];
        const double u = U[k + shift];
        br = h.re - u * br;
        bi = h.im - u * bi;
        a *= -u;
    }
    scan(a, br, bi, false, xr, xi);
    for (int k = k1 - 1; k >= k0; --k) {
        const Cplx h = R[k + shift];
        const double u = U[k + shift];
        xr = h.re - u * xr;
        xi = h.im - u * xi;
        R[k + shift] = {xr, xi};
    }
    if (STAGED) {
        __syncwarp();
        for (int k = lane; k < ni; k += 32) col[k] = R[k + k / run];
    }
}

// The wall nodes' potentials (apply_dirichlet_boundary_potentials,
// src/FieldSolver.cpp:267-296; grounded in 3D), which no solve changes.
__global__ void k_wall_sides(double* __restrict__ phi, WallMesh w) {
    const size_t N = (size_t)w.n[0] * w.n[1] * w.n[2];
    for (size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x; q < N; q += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(q % w.n[0]), j = (int)((q / w.n[0]) % w.n[1]), k = (int)(q / ((size_t)w.n[0] * w.n[1]));
        const bool wi = w.wall[0] && (i == 0 || i == w.n[0] - 1), wj = w.wall[1] && (j == 0 || j == w.n[1] - 1);
        const bool wk = w.wall[2] && (k == 0 || k == w.n[2] - 1);
        if (!wi && !wj && !wk) continue;
        const double si = i == 0 ? w.side[0] : w.side[1], sj = j == 0 ? w.side[2] : w.side[3];
        phi[q] = w.dims == 3 ? 0.0 : (wi && wj ? 0.5 * (si + sj) : (wj ? sj : si));
    }
}

// compute_electric_field(Mesh2D&) and the 3D differences, src/FieldSolver.cpp:298-346,
// :872-904: central, one-sided at the walls, into the push's interleaved
// layout or into planes (Ex | Ey (| Ez)).  The differences are divided through
// reciprocals (cells_of); rd holds 1 / d, then 1 / (2 d).
template <int DIM>
__global__ void __launch_bounds__(256) k_wall_efield(const double* __restrict__ phi, double* __restrict__ E,
                                                     double* __restrict__ planes, WallMesh w) {
    const unsigned nx = w.n[0], ny = w.n[1], nz = DIM == 3 ? w.n[2] : 1, N = nx * ny * nz;
    for (unsigned q = blockIdx.x * blockDim.x + threadIdx.x; q < N; q += gridDim.x * blockDim.x) {
        const unsigned row = q / nx;
        const unsigned c[3] = {q - row * nx, DIM == 3 ? row % ny : row, DIM == 3 ? row / ny : 0u};
        const unsigned n[3] = {nx, ny, nz}, stride[3] = {1u, nx, nx * ny};
        double e[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int a = 0; a < DIM; ++a) {
            const bool low = c[a] == 0u, high = c[a] + 1u == n[a];
            // the neighbours: wrapped on a periodic axis, the node itself past a wall
            const unsigned up = high ? (w.wall[a] ? q : q - c[a] * stride[a]) : q + stride[a];
            const unsigned dn = low ? (w.wall[a] ? q : q + (n[a] - 1u) * stride[a]) : q - stride[a];
            const bool one = w.wall[a] && (low || high);
            const double d = one ? w.d[a] : 2.0 * w.d[a];
            e[a] = -cells_of(__ldg(phi + up) - __ldg(phi + dn), d, one ? w.rd[0][a] : w.rd[1][a]);
        }
        if (planes) {
#pragma unroll
            for (int a = 0; a < DIM; ++a) planes[a * (size_t)N + q] = e[a];
        } else if (DIM == 3) {
            reinterpret_cast<double4*>(E)[q] = make_double4(e[0], e[1], e[2], 0.0);
        } else {
            reinterpret_cast<double2*>(E)[q] = make_double2(e[0], e[1]);
        }
    }
}

struct WallSolver {
    cudaStream_t stream = nullptr;
    std::function<void*(size_t)> alloc;  // device memory that outlives the solver
    WallMesh w{};
    bool mixed = false;
    // one wall axis
    int pa = 0, ni = 0, np = 0;  // periodic axis, interior wall rows, periodic extent
    double hd = 1.0;
    double *mu = nullptr, *inv = nullptr;
    Cplx *hat = nullptr, *tw = nullptr;
    // walls on every side
    double* u = nullptr;
    DstPass pass[3]{};

    template <class V>
    V* upload(const std::vector<V>& h) {
        V* d = static_cast<V*>(alloc(h.size() * sizeof(V)));
        APIC_CUDA(cudaMemcpyAsync(d, h.data(), h.size() * sizeof(V), cudaMemcpyHostToDevice, stream));
        APIC_CUDA(cudaStreamSynchronize(stream));
        return d;
    }
    Cplx* twiddles(int n) {
        std::vector<Cplx> t(n);
        const double twopi = 2.0 * 3.141592653589793;
        for (int k = 0; k < n; ++k) t[k] = {std::cos(twopi * k / n), -std::sin(twopi * k / n)};
        return upload(t);
    }

    void setup(int dims, const int* n, const double* d, const int* wall, double eps, const double* pot) {
        w.dims = dims;
        w.eps = eps;
        w.reps = reciprocal_spacing(eps);
        for (int a = 0; a < 2; ++a) w.ih2[a] = 1.0 / (d[a] * d[a]);
        for (int a = 0; a < 3; ++a) {
            w.n[a] = a < dims ? n[a] : 1;
            w.d[a] = a < dims ? d[a] : 1.0;
            w.wall[a] = a < dims ? wall[a] : 0;
            w.rd[0][a] = reciprocal_spacing(w.d[a]);
            w.rd[1][a] = reciprocal_spacing(2.0 * w.d[a]);
        }
        for (int k = 0; k < 4; ++k) w.side[k] = dims == 2 ? pot[k] : 0.0;
        mixed = dims == 2 && !(wall[0] && wall[1]);
        if (mixed) {
            pa = wall[0] ? 1 : 0;
            np = w.n[pa];
            ni = w.n[1 - pa] - 2;
            hd = w.d[1 - pa];
            const double hp = w.d[pa];
            const size_t modes = (size_t)np / 2 + 1;
            mu = static_cast<double*>(alloc(modes * ni * sizeof(double)));
            inv = static_cast<double*>(alloc(modes * ni * sizeof(double)));
            hat = static_cast<Cplx*>(alloc(modes * ni * sizeof(Cplx)));
            tw = twiddles(np);
            allow_smem(k_mixed_forward, kWallSmemMax);
            allow_smem(k_mixed_inverse, kWallSmemMax);
            if (ni <= kMixedSweepMaxRows) allow_smem(k_mixed_sweep<true>, mixed_sweep_smem(kMixedSweepMaxRows));
            k_mixed_coeffs<<<(unsigned)((modes + 127) / 128), 128, 0, stream>>>(mu, inv, ni + 2, np, 1.0 / (hd * hd),
                                                                                1.0 / (hp * hp));
            APIC_CUDA(cudaGetLastError());
            return;
        }
        const int M[3] = {w.n[0] - 2, w.n[1] - 2, dims == 3 ? w.n[2] - 2 : 1};
        u = static_cast<double*>(alloc((size_t)M[0] * M[1] * M[2] * sizeof(double)));
        const double* eig[3] = {nullptr, nullptr, nullptr};
        double scale = 1.0;
        for (int a = 0; a < dims; ++a) {
            std::vector<double> lam(M[a]);
            const double ih2 = 1.0 / (w.d[a] * w.d[a]);
            for (int m = 0; m < M[a]; ++m) {
                const double sn = std::sin(3.141592653589793 * (m + 1) / (2.0 * (M[a] + 1)));
                lam[m] = 4.0 * sn * sn * ih2;
            }
            eig[a] = upload(lam);
            scale *= 2.0 / (double)(M[a] + 1);
        }
        const long long s[3] = {1, M[0], (long long)M[0] * M[1]};
        for (int a = 0; a < dims; ++a) {
            DstPass& f = pass[a];
            f.M = M[a];
            f.log2N = ilog2(2 * (M[a] + 1));
            f.axis = a;
            f.stride = s[a];
            const int fast = a == 0 ? 1 : 0, slow = a == 2 ? 1 : 2;
            f.lines_a = M[fast];
            f.lines = M[fast] * M[slow];
            f.stride_a = s[fast];
            f.stride_b = s[slow];
            f.T = wall_pairs(2 * (M[a] + 1), f.lines);
            f.tw = twiddles(2 * (M[a] + 1));
            f.scale = scale;
            for (int b = 0; b < 3; ++b) f.eig[b] = eig[b];
            f.in_regs = dims == 3 && f.log2N >= 6 && f.log2N <= 8 && f.lines >= kDstRegLines;
            if (f.in_regs) continue;  // within the default limit
            if (a == 0) {
                allow_smem(k_dst_pass<kDstFromRho>, kWallSmemMax);
                allow_smem(k_dst_pass<kDstToPhi>, kWallSmemMax);
            } else if (a == dims - 1) {
                allow_smem(k_dst_pass<kDstSolve>, kWallSmemMax);
            } else {
                allow_smem(k_dst_pass<kDstInPlace>, kWallSmemMax);
            }
        }
    }

    void set_sides(double* phi) {
        const size_t N = (size_t)w.n[0] * w.n[1] * w.n[2];
        k_wall_sides<<<(unsigned)std::min<size_t>((N + 255) / 256, 4096), 256, 0, stream>>>(phi, w);
        APIC_CUDA(cudaGetLastError());
    }

    template <int MODE>
    void dst(int a, const double* rho, double* phi) {
        const DstPass& f = pass[a];
        auto in_regs = [&](auto r1, auto r2) {
            constexpr int R1 = decltype(r1)::value, R2 = decltype(r2)::value;
            const unsigned g = (unsigned)((f.lines + 2 * kRegLines - 1) / (2 * kRegLines));
            if (a == 0)
                k_dst_reg<MODE, true, R1, R2><<<g, kRegLines * R2, reg_smem<R1, R2, true>(kFwdInPlace), stream>>>(u, w, f, rho, phi);
            else
                k_dst_reg<MODE, false, R1, R2><<<g, kRegLines * R2, reg_smem<R1, R2, false>(kFwdInPlace), stream>>>(u, w, f, rho, phi);
        };
        using I8 = std::integral_constant<int, 8>;
        using I16 = std::integral_constant<int, 16>;
        if (f.in_regs) {
            if (f.log2N == 6) in_regs(I8{}, I8{});
            else if (f.log2N == 7) in_regs(I16{}, I8{});
            else in_regs(I16{}, I16{});
            return;
        }
        const unsigned g = (unsigned)((f.lines + 2 * f.T - 1) / (2 * f.T));
        k_dst_pass<MODE><<<g, kFftThreads, wall_smem(2 * (f.M + 1), f.T), stream>>>(u, w, f, rho, phi);
    }

    // rho -> phi (wall nodes set by set_sides) and E, interleaved or as planes
    void solve(const double* rho, double* phi, double* E, double* planes) {
        if (mixed) {
            const long long sd = pa == 1 ? 1 : w.n[0], sq = pa == 1 ? w.n[0] : 1;
            const double lo = pa == 1 ? w.side[0] : w.side[2], hi = pa == 1 ? w.side[1] : w.side[3];
            const int T = wall_pairs(np, ni);
            const unsigned g = (unsigned)((ni + 2 * T - 1) / (2 * T));
            k_mixed_forward<<<g, kFftThreads, wall_smem(np, T), stream>>>(rho, hat, ni, np, T, sd, sq, tw);
            if (ni <= kMixedSweepMaxRows)
                k_mixed_sweep<true><<<np / 2 + 1, 32, mixed_sweep_smem(ni), stream>>>(hat, mu, inv, ni, np,
                                                                                     1.0 / (hd * hd), w.eps, lo, hi);
            else
                k_mixed_sweep<false><<<np / 2 + 1, 32, 0, stream>>>(hat, mu, inv, ni, np, 1.0 / (hd * hd), w.eps, lo, hi);
            k_mixed_inverse<<<g, kFftThreads, wall_smem(np, T), stream>>>(hat, phi, ni, np, T, sd, sq, tw);
        } else if (w.dims == 2) {
            dst<kDstFromRho>(0, rho, phi);
            dst<kDstSolve>(1, rho, phi);
            dst<kDstToPhi>(0, rho, phi);
        } else {
            dst<kDstFromRho>(0, rho, phi);
            dst<kDstInPlace>(1, rho, phi);
            dst<kDstSolve>(2, rho, phi);
            dst<kDstInPlace>(1, rho, phi);
            dst<kDstToPhi>(0, rho, phi);
        }
        const unsigned grid = (unsigned)(((size_t)w.n[0] * w.n[1] * w.n[2] + 255) / 256);
        if (w.dims == 2) k_wall_efield<2><<<grid, 256, 0, stream>>>(phi, E, planes, w);
        else k_wall_efield<3><<<grid, 256, 0, stream>>>(phi, E, planes, w);
        APIC_CUDA(cudaGetLastError());
    }
};

// the interleaved field as planes
template <int DIM>
__global__ void k_split_field(const double* __restrict__ E, double* __restrict__ ex, double* __restrict__ ey,
                              double* __restrict__ ez, size_t N) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < N; i += (size_t)gridDim.x * blockDim.x) {
        if (DIM == 2) {
            const double2 e = reinterpret_cast<const double2*>(E)[i];
            ex[i] = e.x;
            ey[i] = e.y;
        } else {
            const double4 e = reinterpret_cast<const double4*>(E)[i];
            ex[i] = e.x;
            ey[i] = e.y;
            ez[i] = e.z;
        }
    }
}

// Device to pageable host copies of a few hundred megabytes: kWorkers threads
// take 1 MB pieces in turn, each with two pinned buffers and a stream of its own, so
// the transfers overlap the host copies and the page faults of fresh
// destinations, which one thread would take one after another.  Small reads take the driver's
// own path, and so do page-locked destinations, which the GPU writes itself (256^3, one
// array: 2.4 ms, through the pieces 3.8).  The buffers (16 MB pinned) and streams belong
// to the run.  They take 10 to 20 ms to make, as long as the driver's path takes for 100 MB of
// fresh destinations, so a read makes them from kHuge bytes on or, with the field, when the
// run has read its field before (rho and phi of 128^3, read once: 1.8 ms, with the set-up 13;
// a one-off 1024 x 1024 solve: 20, with the set-up 28).
struct HostCopier {
    static constexpr int kWorkers = 8;
    static constexpr size_t kPiece = 1 << 20, kLarge = 16 << 20, kHuge = 256 << 20;
    struct Job {
        double* dst;
        const double* src;
        size_t bytes;
    };
    unsigned char* pinned = nullptr;
    cudaStream_t streams[kWorkers] = {};
    bool field_read = false;

    ~HostCopier() {
        for (auto& s : streams)
            if (s) cudaStreamDestroy(s);
        if (pinned) cudaFreeHost(pinned);
    }

    static bool page_locked(const void* p) {
        cudaPointerAttributes a{};
        APIC_CUDA(cudaPointerGetAttributes(&a, p));
        return a.type != cudaMemoryTypeUnregistered;
    }

    // the sources must be complete: the workers' streams do not wait for `stream`.
    void run(std::vector<Job> jobs, cudaStream_t stream, bool field) {
        const auto direct = std::partition(jobs.begin(), jobs.end(), [](const Job& j) { return !page_locked(j.dst); });
        size_t total = 0;
        for (auto j = jobs.begin(); j != direct; ++j) total += j->bytes;
        const bool plain = total < kLarge || !(pinned || total >= kHuge || (field && field_read));
        field_read = field_read || field;
        for (auto j = plain ? jobs.begin() : direct; j != jobs.end(); ++j)
            APIC_CUDA(cudaMemcpyAsync(j->dst, j->src, j->bytes, cudaMemcpyDeviceToHost, stream));
        APIC_CUDA(cudaStreamSynchronize(stream));
        if (plain) return;
        jobs.erase(direct, jobs.end());
        if (!pinned) APIC_CUDA(cudaHostAlloc(&pinned, 2 * kWorkers * kPiece, cudaHostAllocDefault));
        for (auto& s : streams)
            if (!s) APIC_CUDA(cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking));
        struct Piece {
            unsigned char* dst;
            const unsigned char* src;
            size_t bytes;
        };
        std::vector<Piece> pieces;
        for (const Job& j : jobs)
            for (size_t o = 0; o < j.bytes; o += kPiece)
                pieces.push_back({reinterpret_cast<unsigned char*>(j.dst) + o,
                                  reinterpret_cast<const unsigned char*>(j.src) + o, std::min(kPiece, j.bytes - o)});
        int device = 0;
        APIC_CUDA(cudaGetDevice(&device));
        std::atomic<size_t> next{0};
        std::atomic<int> failed{0};
        auto work = [&](int t) {
            unsigned char* buf[2] = {pinned + 2 * t * kPiece, pinned + (2 * t + 1) * kPiece};
            cudaError_t e = cudaSetDevice(device);
            const Piece* held = nullptr;  // copied into buf[which ^ 1], not yet handed over
            int which = 0;
            while (e == cudaSuccess) {
                const size_t k = next.fetch_add(1);
                const Piece* p = k < pieces.size() ? &pieces[k] : nullptr;
                if (held) e = cudaStreamSynchronize(streams[t]);
                if (e == cudaSuccess && p)
                    e = cudaMemcpyAsync(buf[which], p->src, p->bytes, cudaMemcpyDeviceToHost, streams[t]);
                if (e != cudaSuccess) break;
                if (held) std::memcpy(held->dst, buf[which ^ 1], held->bytes);
                held = p;
                which ^= 1;
                if (!p) break;
            }
            if (e != cudaSuccess) failed.store((int)e);
        };
        std::vector<std::thread> threads;
        threads.reserve(kWorkers);
        for (int t = 1; t < kWorkers; ++t) {
            try {
                threads.emplace_back(work, t);
            } catch (...) {  // no thread, or no memory for one (a joinable thread must not be unwound)
                break;       // fewer workers: those that run take every piece
            }
        }
        work(0);
        for (auto& t : threads) t.join();
        // (a worker that failed leaves with its copy possibly in flight)
        if (failed.load()) {
            for (auto& s : streams) cudaStreamSynchronize(s);
            APIC_CUDA((cudaError_t)failed.load());
        }
    }
};

struct SimND {
    apic_config_nd cfg{};
    std::string last_error;
    cudaStream_t stream = nullptr;
    std::vector<void*> allocations;
    ParamsND p{};
    SpeciesND sp[APIC_MAX_SPECIES]{};
    int buf[APIC_MAX_SPECIES] = {0, 0, 0, 0};
    Solver solver;
    bool boris = false;
    bool fp32 = false;
    bool initialized = false;
    double time = 0.0;
    uint64_t step_count = 0;
    size_t sort_interval = 16;
    uint64_t launches = 0;  // kernels launched by step()
    size_t steps_since_sort = 0;                   // of the most frequently sorted species
    size_t since_sort[APIC_MAX_SPECIES] = {0, 0, 0, 0};
    size_t species_interval[APIC_MAX_SPECIES] = {16, 16, 16, 16};
    unsigned* cell_count = nullptr;
    unsigned* cell_offset = nullptr;
    unsigned* block_sums = nullptr;
    size_t ncells = 0;
    double* sample_partial = nullptr;
    unsigned* sample_done = nullptr;
    double* sample_out = nullptr;
    bool timing = false;
    double push_ms = 0, solve_ms = 0, sort_ms = 0;
    uint64_t timed_steps = 0;
    struct Ev { cudaEvent_t a, b, c, d; bool sorted; };
    std::vector<Ev> events;

    template <class T>
    T* dalloc(size_t count) {
        void* ptr = nullptr;
        APIC_CUDA(cudaMalloc(&ptr, std::max<size_t>(count, 1) * sizeof(T)));
        allocations.push_back(ptr);
        APIC_CUDA(cudaMemsetAsync(ptr, 0, std::max<size_t>(count, 1) * sizeof(T), stream));
        return static_cast<T*>(ptr);
    }

    ~SimND() {
        if (stream) cudaStreamSynchronize(stream);
        drop_graphs();
        for (auto& e : events) { cudaEventDestroy(e.a); cudaEventDestroy(e.b); cudaEventDestroy(e.c); cudaEventDestroy(e.d); }
        for (void* a : allocations) cudaFree(a);
        if (stream) cudaStreamDestroy(stream);
    }

    void create(const apic_config_nd& c) {
        cfg = c;
        require(c.dims == 2 || c.dims == 3, "dims must be 2 or 3");
        require(c.precision == APIC_FP64 || c.precision == APIC_FP32, "unknown precision");
        fp32 = c.precision == APIC_FP32;
        walls = c.wall_axis[0] != 0 || c.wall_axis[1] != 0 || (c.dims == 3 && c.wall_axis_z != 0);
        if (walls) {
            require(!fp32, "runs with walls use the FP64 particle form", APIC_ERR_UNSUPPORTED);
            for (int k = 0; k < 4; ++k) {
                require(c.particle_boundary[k] >= 0 && c.particle_boundary[k] <= 3, "unknown particle boundary");
                require(std::isfinite(c.wall_potential[k]), "wall potentials must be finite");
            }
            if (c.dims == 3) {
                // Simulation3DConfig has one field boundary for the mesh (src/Mesh3D.cpp:37-48)
                require(c.wall_axis[0] && c.wall_axis[1] && c.wall_axis_z,
                        "3D meshes are periodic or Dirichlet on every axis", APIC_ERR_UNSUPPORTED);
                require(c.wall_potential[0] == 0.0 && c.wall_potential[1] == 0.0 && c.wall_potential[2] == 0.0 &&
                            c.wall_potential[3] == 0.0,
                        "3D Dirichlet walls are grounded");
                for (int k = 0; k < 2; ++k)
                    require(c.particle_boundary_z[k] >= 0 && c.particle_boundary_z[k] <= 3,
                            "unknown particle boundary");
            }
        }
        for (int a = 0; a < c.dims; ++a) {
            require(c.n[a] >= 3, "mesh extents must be at least 3");
            const bool wall = walls && (a < 2 ? c.wall_axis[a] != 0 : c.wall_axis_z != 0);
            if (!wall)
                require(pow2(c.n[a]) && c.n[a] <= (size_t)kMaxLine,
                        "periodic device meshes need power-of-two extents up to 1024", APIC_ERR_UNSUPPORTED);
            else if (c.wall_axis[0] && c.wall_axis[1])
                require(pow2(c.n[a] - 1) && 2 * (c.n[a] - 1) <= (size_t)kMaxLine,
                        "walls on every side need extents of 2^k + 1 nodes up to 513", APIC_ERR_UNSUPPORTED);
            else
                require(c.n[a] <= 65536, "the wall axis allows up to 65536 nodes", APIC_ERR_UNSUPPORTED);
            require(std::isfinite(c.length[a]) && c.length[a] > 0, "domain lengths must be positive and finite");
        }
        require(std::isfinite(c.dt) && c.dt > 0, "simulation dt must be positive and finite");
        require(c.nspecies >= 1 && c.nspecies <= APIC_MAX_SPECIES, "species count out of range");
        require(c.push_items == 0 || c.push_items == 1 || c.push_items == 2 || c.push_items == 4 ||
                    c.push_items == 8,
                "push_items must be 0, 1, 2, 4 or 8");
        const double rel = c.relative_permittivity == 0.0 ? 1.0 : c.relative_permittivity;
        require(std::isfinite(rel) && rel > 0, "relative_permittivity must be positive and finite");
        const double depth = c.out_of_plane_depth == 0.0 ? 1.0 : c.out_of_plane_depth;
        require(std::isfinite(depth) && depth > 0, "2D deposition depth must be positive and finite");
        int ndev = 0;
        if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
            throw Error(APIC_ERR_NO_DEVICE, "no CUDA device is visible");
        APIC_CUDA(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking));
        sort_interval = c.sort_interval ? c.sort_interval : 16;
        for (int k = 0; k < APIC_MAX_SPECIES; ++k)
            species_interval[k] = c.species_sort_interval[k] ? c.species_sort_interval[k] : sort_interval;

        p.dims = c.dims;
        size_t N = 1;
        double cellvol = 1.0;
        for (int a = 0; a < 3; ++a) {
            p.n[a] = a < c.dims ? (int)c.n[a] : 1;
            p.L[a] = a < c.dims ? c.length[a] : 1.0;
            // Mesh2D/Mesh3D dx: L / n periodic, L / (n - 1) on a wall axis,
            // src/Mesh2D.cpp:57-62, src/Mesh3D.cpp:43-45
            const bool wall_a = walls && a < c.dims && (a < 2 ? c.wall_axis[a] != 0 : c.wall_axis_z != 0);
            p.d[a] = p.L[a] / (double)(wall_a ? p.n[a] - 1 : p.n[a]);
            p.rd[a] = reciprocal_spacing(p.d[a]);
            p.B[a] = c.magnetic_field[a];
            N *= (size_t)p.n[a];
            if (a < c.dims) cellvol *= p.d[a];
        }
        ncells = N;
        boris = c.magnetic_field[0] != 0.0 || c.magnetic_field[1] != 0.0 || c.magnetic_field[2] != 0.0;
        if (c.profile_rows) {
            // Simulation2D / Simulation3D constructor checks, src/Simulation3D.cpp:184-196
            require(!boris, std::string(c.dims == 2 ? "2D" : "3D") +
                                " uniform magnetic_field components and magnetic_field_profile are mutually exclusive");
            require(c.profile_axis >= 0 && c.profile_axis <= 2, "coordinate axis must be x, y, or z");
            require(c.profile_rows >= 2, "tabulated vector field requires at least two rows");
            require(c.profile_coordinates && c.profile_values, "tabulated vector field arrays are required");
            for (size_t k = 0; k < c.profile_rows; ++k) {
                require(std::isfinite(c.profile_coordinates[k]) && std::isfinite(c.profile_values[3 * k]) &&
                            std::isfinite(c.profile_values[3 * k + 1]) && std::isfinite(c.profile_values[3 * k + 2]),
                        "tabulated vector field values must be finite");
                require(k == 0 || c.profile_coordinates[k] > c.profile_coordinates[k - 1],
                        "tabulated vector field coordinates must be strictly increasing");
            }
            const double hi = c.profile_axis < c.dims ? c.length[c.profile_axis] : 0.0;
            require(c.profile_coordinates[0] <= 0.0 && c.profile_coordinates[c.profile_rows - 1] >= hi,
                    "tabulated magnetic field does not cover the simulation domain");
            require(c.profile_rows < (1u << 30), "tabulated vector field too long");
            boris = true;
        }
        p.dt = c.dt;
        p.eps = (c.units == APIC_SI ? 8.8541878128e-12 : 1.0) * rel;
        double bound = 0.0;
        for (int s = 0; s < c.nspecies; ++s) {
            const auto& S = c.species[s];
            require(std::isfinite(S.mass) && S.mass > 0, "species mass must be positive and finite");
            require(S.capacity > 0 && S.capacity < (1ull << 31), "species capacity out of range");
            const double w = c.dims == 2 ? S.weight / depth : S.weight;  // Species2D::deposit_charge
            // a wall node's half cells (a corner's eighth) raise its density by up to 2^dims
            bound += (double)S.capacity * std::fabs(S.charge * w) / cellvol * (walls ? (double)(1 << c.dims) : 1.0);
        }
        const int bits = bound > 0 ? (int)std::floor(61.0 - std::log2(bound)) : 0;
        p.rho_scale = std::ldexp(1.0, bits);
        p.inv_rho_scale = std::ldexp(1.0, -bits);
        for (int s = 0; s < c.nspecies; ++s) {
            const auto& S = c.species[s];
            SpeciesND& D = sp[s];
            D.qm = S.charge / S.mass;
            const double w = c.dims == 2 ? S.weight / depth : S.weight;
            D.dep = S.charge * w / cellvol;
            D.hmw = 0.5 * S.mass * S.weight;
            D.n = 0;
            for (int b = 0; b < 2; ++b) {
                for (int a = 0; a < c.dims; ++a) D.pos[b][a] = dalloc<double>(S.capacity);
                for (int a = 0; a < 3; ++a) D.vh[b][a] = dalloc<double>(S.capacity);
                D.id[b] = dalloc<unsigned>(S.capacity);
            }
            for (int a = 0; a < 3; ++a) D.v[a] = dalloc<double>(S.capacity);
            if (fp32) {
                for (int b = 0; b < 2; ++b) {
                    D.cell[b] = dalloc<unsigned>(S.capacity);
                    for (int a = 0; a < c.dims; ++a) D.off[b][a] = dalloc<float>(S.capacity);
                    for (int a = 0; a < 3; ++a) D.vel[b][a] = dalloc<float>(S.capacity);
                }
            }
            const double hq = 0.5 * D.qm * c.dt;
            D.hqmdt = (float)hq;
            D.qmdt = (float)(D.qm * c.dt);
            double t2 = 0.0;
            for (int a = 0; a < 3; ++a) { D.tb[a] = (float)(hq * c.magnetic_field[a]); t2 += (hq * c.magnetic_field[a]) * (hq * c.magnetic_field[a]); }
            for (int a = 0; a < 3; ++a) D.sb[a] = (float)(2.0 * hq * c.magnetic_field[a] / (1.0 + t2));
            for (int a = 0; a < 3; ++a) D.drift[a] = a < c.dims ? (float)(c.dt / p.d[a]) : 0.0f;
            D.dep_fixed = (float)(D.dep * p.rho_scale);
            D.bh = hq;  // t and s of boris(), in its own order of operations
            double bt2 = 0.0;
            for (int a = 0; a < 3; ++a) { D.bt[a] = hq * c.magnetic_field[a]; bt2 += D.bt[a] * D.bt[a]; }
            const double sf = 2.0 / (1.0 + bt2);
            for (int a = 0; a < 3; ++a) D.bs[a] = sf * D.bt[a];
            D.index = s;
        }
        solver.allocs = &allocations;
        solver.stream = stream;
        if (walls) {
            setup_walls(c);
        } else {
            solver.setup(c.dims, c.n, c.length, p.eps, p.inv_rho_scale);
        }
        p.E = solver.F.E;
        p.rho_acc = solver.F.rho_acc;
        if (c.profile_rows) {  // copied: the caller's arrays may go away after create
            double* pc = dalloc<double>(c.profile_rows);
            double* pv = dalloc<double>(3 * c.profile_rows);
            APIC_CUDA(cudaMemcpyAsync(pc, c.profile_coordinates, c.profile_rows * sizeof(double),
                                      cudaMemcpyHostToDevice, stream));
            APIC_CUDA(cudaMemcpyAsync(pv, c.profile_values, 3 * c.profile_rows * sizeof(double),
                                      cudaMemcpyHostToDevice, stream));
            p.prof_axis = c.profile_axis;
            p.prof_rows = (int)c.profile_rows;
            p.prof_c = pc;
            p.prof_v = pv;
            cfg.profile_coordinates = nullptr;  // not kept
            cfg.profile_values = nullptr;
        }
        if (fp32) {
            solver.F.E32 = dalloc<float>(N * (c.dims == 2 ? 2 : 4));
            p.E32 = solver.F.E32;
            solver.F.nacc = c.nspecies;
            for (int s = 0; s < c.nspecies; ++s) {
                solver.F.acc[s] = dalloc<unsigned long long>(N);
                solver.F.acc_scale[s] = sp[s].dep / (double)kWeightScale;
            }
        }
        cell_count = dalloc<unsigned>(N + 1);
        cell_offset = dalloc<unsigned>(N + 1);
        block_sums = dalloc<unsigned>((N + kScanBlock) / kScanBlock + 1);
        tileable = fp32 && c.dims == 3;
        for (int a = 0; a < c.dims; ++a) tileable = tileable && p.n[a] % kTileCells == 0;
        if (tileable) {
            ntiles = (unsigned)(N / kTileVolume);
            for (int s = 0; s < c.nspecies; ++s) {
                // at most 2 n / target + 1 items past the first of every tile
                sp[s].chunk = dalloc<uint4>(ntiles + 2 * (c.species[s].capacity / kTileMinTarget) + 1);
                sp[s].extra = dalloc<unsigned>(1);
            }
            const auto allow = [](auto one, auto two) {
                allow_smem(one, tile32_smem<1>());
                allow_smem(two, tile32_smem<2>());
            };
            if (boris && p.prof_rows) allow(k_push32_tile<true, true, 1>, k_push32_tile<true, true, 2>);
            else if (boris) allow(k_push32_tile<true, false, 1>, k_push32_tile<true, false, 2>);
            else allow(k_push32_tile<false, false, 1>, k_push32_tile<false, false, 2>);
        }
        sample_partial = dalloc<double>(3 * kSampleBlocks);
        sample_done = dalloc<unsigned>(1);
        sample_out = dalloc<double>(8);
        APIC_CUDA(cudaStreamSynchronize(stream));
    }

    SpeciesND view(int s) const { return sp[s]; }

    // Tiles: 3D meshes whose every extent holds a tile, from kTileMinPpc particles a
    // cell on average (below, filling and flushing a tile's box costs more than its
    // particles save) and enough work items.
    unsigned ntiles = 0;
    bool tileable = false;
    bool tiles_ready[APIC_MAX_SPECIES] = {};  // sorted in tiles since its particles were loaded
    unsigned tile_target(int s) const {  // particles per work item: enough items for four waves of CTAs
        return (unsigned)std::min<size_t>(8192, std::max<size_t>(kTileMinTarget, sp[s].n / (148 * 16)));
    }
    unsigned tile_extra_max(int s) const { return 2 * (sp[s].n / tile_target(s)) + 1; }
    void choose_tiles(int s) {
        SpeciesND& S = sp[s];
        const double ppc = (double)S.n / (double)ncells;
        const size_t items = std::max<size_t>(ntiles, S.n / kTileMinTarget);
        S.tiled = tileable && ppc >= kTileMinPpc && (items >= kTileMinItems || ppc >= kTileCrowdedPpc);
        tiles_ready[s] = false;
    }

    static State32 state32(const SpeciesND& S, int b) {
        State32 A{S.cell[b], {}, {}};
        for (int a = 0; a < 3; ++a) { A.off[a] = S.off[b][a]; A.vel[a] = S.vel[b][a]; }
        return A;
    }

    template <int DIM, bool BORIS>
    void launch_step32(int items, const SpeciesND& S, int b, int s) {
        const unsigned g = (unsigned)((S.n + (unsigned)items * kThreads - 1) / ((unsigned)items * kThreads));
        unsigned long long* acc = solver.F.acc[s];
        if (BORIS && p.prof_rows) {
            switch (items) {
                case 1: k_push32_step<DIM, BORIS, 1, true><<<g, kThreads, 0, stream>>>(p, S, b, acc); break;
                case 2: k_push32_step<DIM, BORIS, 2, true><<<g, kThreads, 0, stream>>>(p, S, b, acc); break;
                case 4: k_push32_step<DIM, BORIS, 4, true><<<g, kThreads, 0, stream>>>(p, S, b, acc); break;
                default: k_push32_step<DIM, BORIS, 8, true><<<g, kThreads, 0, stream>>>(p, S, b, acc); break;
            }
            return;
        }
        switch (items) {
            case 1: k_push32_step<DIM, BORIS, 1, false><<<g, kThreads, 0, stream>>>(p, S, b, acc); break;
            case 2: k_push32_run<DIM, BORIS, 2, false><<<g, kThreads, 0, stream>>>(p, S, state32(S, b), b, acc); break;
            case 4: k_push32_run<DIM, BORIS, 4, false><<<g, kThreads, 0, stream>>>(p, S, state32(S, b), b, acc); break;
            default: k_push32_step<DIM, BORIS, 8, false><<<g, kThreads, 0, stream>>>(p, S, b, acc); break;
        }
    }

    template <int MODE>
    void launch_push(int s) {
        const SpeciesND& S = sp[s];
        if (S.n == 0) return;
        const unsigned blocks = (S.n + kThreads - 1) / kThreads;
        const int b = buf[s];
        if (fp32 && MODE == kPushStep && S.tiled) {
            const unsigned g = ntiles + tile_extra_max(s);
            const State32 A = state32(S, b);
            // one cell around the tile when few particles leave it between sorts, else two
            // (a thermal electron moves about 0.1 cell a step, a heavier species at the same
            // temperature less; push of 256^3, one against two cells, electrons sorted every 3
            // steps 4.06 / 4.27 ms, 4: 4.10 / 4.30, 6: 4.24 / 4.36, 8: 4.53 / 4.40, 16: 5.23 / 4.94)
            double lightest = cfg.species[0].mass;
            for (int k = 1; k < cfg.nspecies; ++k) lightest = std::min(lightest, cfg.species[k].mass);
            const double reach = (double)species_interval[s] * std::sqrt(lightest / cfg.species[s].mass);
            auto run = [&](auto margin) {
                constexpr int M = decltype(margin)::value;
                constexpr size_t smem = tile32_smem<M>();
                unsigned long long* acc = solver.F.acc[s];
                if (boris && p.prof_rows) k_push32_tile<true, true, M><<<g, kThreads, smem, stream>>>(p, S, A, acc, ntiles);
                else if (boris) k_push32_tile<true, false, M><<<g, kThreads, smem, stream>>>(p, S, A, acc, ntiles);
                else k_push32_tile<false, false, M><<<g, kThreads, smem, stream>>>(p, S, A, acc, ntiles);
            };
            if (reach <= 4.0) run(std::integral_constant<int, 1>{});
            else run(std::integral_constant<int, 2>{});
            APIC_CUDA(cudaGetLastError());
            return;
        }
        if (fp32 && MODE == kPushStep) {
            // particles per thread: configured, else the measured best (4 in 2D, 2 in 3D)
            const int items = cfg.push_items ? cfg.push_items : (cfg.dims == 2 ? 4 : 2);
            if (cfg.dims == 2) {
                if (boris) launch_step32<2, true>(items, S, b, s);
                else launch_step32<2, false>(items, S, b, s);
            } else {
                if (boris) launch_step32<3, true>(items, S, b, s);
                else launch_step32<3, false>(items, S, b, s);
            }
            APIC_CUDA(cudaGetLastError());
            return;
        }
        if (fp32) {
            if (cfg.dims == 2) {
                if (boris) k_push32<2, true, MODE><<<blocks, kThreads, 0, stream>>>(p, S, b, solver.F.acc[s]);
                else k_push32<2, false, MODE><<<blocks, kThreads, 0, stream>>>(p, S, b, solver.F.acc[s]);
            } else {
                if (boris) k_push32<3, true, MODE><<<blocks, kThreads, 0, stream>>>(p, S, b, solver.F.acc[s]);
                else k_push32<3, false, MODE><<<blocks, kThreads, 0, stream>>>(p, S, b, solver.F.acc[s]);
            }
            APIC_CUDA(cudaGetLastError());
            return;
        }
        if (MODE == kPushStep) {
            const int items = S.n <= kOneItemMax ? 1 : kRunItems;
            const unsigned g = (S.n + items * kThreads - 1) / (items * kThreads);
            const int kind = !boris ? kNoField : (p.prof_rows ? kProfileField : kUniformField);
            State64 A{{}, {}, S.alive[b], S.live_end};
            for (int a = 0; a < 3; ++a) { A.pos[a] = S.pos[b][a]; A.vh[a] = S.vh[b][a]; }
            auto launch = [&](auto dim, auto wall, auto per) {
                constexpr int D = decltype(dim)::value, I = decltype(per)::value;
                constexpr bool Wl = decltype(wall)::value;
                if (kind == kNoField) k_push_run<D, kNoField, Wl, I><<<g, kThreads, 0, stream>>>(p, S, A);
                else if (kind == kUniformField) k_push_run<D, kUniformField, Wl, I><<<g, kThreads, 0, stream>>>(p, S, A);
                else k_push_run<D, kProfileField, Wl, I><<<g, kThreads, 0, stream>>>(p, S, A);
            };
            auto run = [&](auto dim, auto wall) {
                if (items == 1) launch(dim, wall, std::integral_constant<int, 1>{});
                else launch(dim, wall, std::integral_constant<int, kRunItems>{});
            };
            using D2 = std::integral_constant<int, 2>;
            using D3 = std::integral_constant<int, 3>;
            if (cfg.dims == 2) walls ? run(D2{}, std::true_type{}) : run(D2{}, std::false_type{});
            else walls ? run(D3{}, std::true_type{}) : run(D3{}, std::false_type{});
            APIC_CUDA(cudaGetLastError());
            return;
        }
        if constexpr (MODE != kPushStep) {
        if (cfg.dims == 2 && walls) {
            if (boris) k_push<2, true, MODE, true><<<blocks, kThreads, 0, stream>>>(p, S, b);
            else k_push<2, false, MODE, true><<<blocks, kThreads, 0, stream>>>(p, S, b);
        } else if (walls) {
            if (boris) k_push<3, true, MODE, true><<<blocks, kThreads, 0, stream>>>(p, S, b);
            else k_push<3, false, MODE, true><<<blocks, kThreads, 0, stream>>>(p, S, b);
        } else if (cfg.dims == 2) {
            if (boris) k_push<2, true, MODE><<<blocks, kThreads, 0, stream>>>(p, S, b);
            else k_push<2, false, MODE><<<blocks, kThreads, 0, stream>>>(p, S, b);
        } else {
            if (boris) k_push<3, true, MODE><<<blocks, kThreads, 0, stream>>>(p, S, b);
            else k_push<3, false, MODE><<<blocks, kThreads, 0, stream>>>(p, S, b);
        }
        APIC_CUDA(cudaGetLastError());
        }
    }

    void sort_species(int s) {
        SpeciesND& S = sp[s];
        if (S.n == 0) return;
        const unsigned blocks = (S.n + kThreads - 1) / kThreads;
        const unsigned nbins = (unsigned)ncells + (walls ? 1u : 0u);  // with walls: one bin for the absorbed
        const unsigned nb = (nbins + kScanBlock - 1) / kScanBlock;
        APIC_CUDA(cudaMemsetAsync(cell_count, 0, nbins * sizeof(unsigned), stream));
        const bool in_tiles = S.tiled && tiles_ready[s];
        const unsigned items = ntiles + tile_extra_max(s);
        if (fp32 && in_tiles) k_tile_count<false><<<items, kThreads, 0, stream>>>(p, S, buf[s], cell_count, ntiles);
        else if (fp32) k_cell_hist32<<<blocks, kThreads, 0, stream>>>(p, S, buf[s], cell_count);
        else if (walls && cfg.dims == 2) k_cell_hist<2, true><<<blocks, kThreads, 0, stream>>>(p, S, buf[s], cell_count);
        else if (walls) k_cell_hist<3, true><<<blocks, kThreads, 0, stream>>>(p, S, buf[s], cell_count);
        else if (cfg.dims == 2) k_cell_hist<2, false><<<blocks, kThreads, 0, stream>>>(p, S, buf[s], cell_count);
        else k_cell_hist<3, false><<<blocks, kThreads, 0, stream>>>(p, S, buf[s], cell_count);
        k_scan_local<<<nb, kThreads, 0, stream>>>(cell_count, cell_offset, block_sums, nbins);
        k_scan_blocks<<<1, kThreads, 0, stream>>>(block_sums, nb);
        k_scan_add<<<nb, kThreads, 0, stream>>>(cell_offset, block_sums, nbins, walls ? S.live_end : nullptr);
        if (fp32) {
            if (in_tiles) k_tile_count<true><<<items, kThreads, 0, stream>>>(p, S, buf[s], cell_offset, ntiles);
            else k_cell_rank32<<<blocks, kThreads, 0, stream>>>(p, S, buf[s], cell_offset);
            if (cfg.dims == 2) k_cell_gather32<2><<<blocks, kThreads, 0, stream>>>(S, buf[s]);
            else k_cell_gather32<3><<<blocks, kThreads, 0, stream>>>(S, buf[s]);
            if (S.tiled) {
                APIC_CUDA(cudaMemsetAsync(S.extra, 0, sizeof(unsigned), stream));
                k_tile_items<<<(ntiles + 255) / 256, 256, 0, stream>>>(cell_offset, ntiles, tile_target(s), S);
            }
        } else if (walls) {
            if (cfg.dims == 2) k_cell_scatter<2, true><<<blocks, kThreads, 0, stream>>>(p, S, buf[s], cell_offset);
            else k_cell_scatter<3, true><<<blocks, kThreads, 0, stream>>>(p, S, buf[s], cell_offset);
        } else if (cfg.dims == 2) {
            k_cell_scatter<2, false><<<blocks, kThreads, 0, stream>>>(p, S, buf[s], cell_offset);
        } else {
            k_cell_scatter<3, false><<<blocks, kThreads, 0, stream>>>(p, S, buf[s], cell_offset);
        }
        APIC_CUDA(cudaGetLastError());
        buf[s] ^= 1;
    }

    void to_fp32(int s) {
        const SpeciesND& S = sp[s];
        if (!fp32 || S.n == 0) return;
        const unsigned blocks = (S.n + kThreads - 1) / kThreads;
        if (cfg.dims == 2) k_to_fp32<2><<<blocks, kThreads, 0, stream>>>(p, S, buf[s]);
        else k_to_fp32<3><<<blocks, kThreads, 0, stream>>>(p, S, buf[s]);
        APIC_CUDA(cudaGetLastError());
    }

    void to_fp64(int s) {
        const SpeciesND& S = sp[s];
        if (!fp32 || S.n == 0) return;
        const unsigned blocks = (S.n + kThreads - 1) / kThreads;
        if (cfg.dims == 2) k_to_fp64<2><<<blocks, kThreads, 0, stream>>>(p, S, buf[s]);
        else k_to_fp64<3><<<blocks, kThreads, 0, stream>>>(p, S, buf[s]);
        APIC_CUDA(cudaGetLastError());
    }

    // a species' n particles are about to be loaded: none absorbed, not sorted yet
    void all_alive(int s, size_t n) {
        const SpeciesND& S = sp[s];
        if (S.alive[buf[s]] && n) APIC_CUDA(cudaMemsetAsync(S.alive[buf[s]], 1, n, stream));
        if (S.live_end) APIC_CUDA(cudaMemsetAsync(S.live_end, 0xFF, sizeof(unsigned), stream));
    }

    void load(int s, size_t n, const double* pos, const double* v, const double* vh) {
        require(s >= 0 && s < cfg.nspecies, "species index out of range");
        require(pos && v, "positions and velocities are required");
        require(n <= cfg.species[s].capacity, "initial particle count exceeds max_particles_per_species",
                APIC_ERR_CAPACITY);
        SpeciesND& S = sp[s];
        const int b = buf[s];
        all_alive(s, n);
        const size_t bytes = n * sizeof(double);
        for (int a = 0; a < cfg.dims; ++a)
            APIC_CUDA(cudaMemcpyAsync(S.pos[b][a], pos + a * n, bytes, cudaMemcpyHostToDevice, stream));
        for (int a = 0; a < 3; ++a) {
            APIC_CUDA(cudaMemcpyAsync(S.v[a], v + a * n, bytes, cudaMemcpyHostToDevice, stream));
            APIC_CUDA(cudaMemcpyAsync(S.vh[b][a], (vh ? vh : v) + a * n, bytes, cudaMemcpyHostToDevice, stream));
        }
        std::vector<unsigned> ids(n);
        for (size_t i = 0; i < n; ++i) ids[i] = (unsigned)i;
        APIC_CUDA(cudaMemcpyAsync(S.id[b], ids.data(), n * sizeof(unsigned), cudaMemcpyHostToDevice, stream));
        APIC_CUDA(cudaStreamSynchronize(stream));
        if (S.n != (unsigned)n) drop_graphs();  // captured launches carry the particle count
        S.n = (unsigned)n;
        choose_tiles(s);
        to_fp32(s);
        initialized = false;
    }

    void load_maxwellian(int s, size_t n, uint64_t seed, double vt, double drift, int axis, double amp) {
        require(s >= 0 && s < cfg.nspecies, "species index out of range");
        require(n <= cfg.species[s].capacity, "initial particle count exceeds max_particles_per_species",
                APIC_ERR_CAPACITY);
        require(std::isfinite(vt) && vt >= 0 && std::isfinite(drift) && std::isfinite(amp), "invalid loading parameters");
        SpeciesND& S = sp[s];
        const unsigned blocks = (unsigned)((n + kThreads - 1) / kThreads);
        all_alive(s, n);
        if (n) k_load_maxwellian<<<blocks, kThreads, 0, stream>>>(S, buf[s], cfg.dims, (unsigned)n, seed, p.L[0],
                                                                   p.L[1], p.L[2], vt, drift, axis, amp);
        APIC_CUDA(cudaGetLastError());
        if (S.n != (unsigned)n) drop_graphs();  // captured launches carry the particle count
        S.n = (unsigned)n;
        choose_tiles(s);
        to_fp32(s);
        initialized = false;
    }

    // ---- walls: persistent solve scratch on the run's stream ----
    bool walls = false;
    WallSolver wall_solver;
    double* wall_planes = nullptr;  // read_fields: Ex | Ey (| Ez)
    HostCopier copier;

    void setup_walls(const apic_config_nd& c) {
        const int dims = c.dims;
        const size_t N = c.n[0] * c.n[1] * (dims == 3 ? c.n[2] : 1);
        for (int k = 0; k < 2 * dims; ++k) {
            const int kind = k < 4 ? c.particle_boundary[k] : c.particle_boundary_z[k - 4];
            const bool wall = k < 4 ? c.wall_axis[k >> 1] != 0 : c.wall_axis_z != 0;
            // resolve_particle_boundary, src/Simulation2D.cpp:38-41, src/Simulation3D.cpp:25-28
            // (Auto follows the field boundary)
            p.pbc[k] = kind == 0 ? (wall ? 1 : 0) : (kind == 1 ? 1 : (kind == 2 ? 2 : 0));
        }
        p.wall[0] = c.wall_axis[0] != 0;
        p.wall[1] = c.wall_axis[1] != 0;
        p.wall[2] = dims == 3 && c.wall_axis_z != 0;
        p.losses = dalloc<unsigned long long>(6 * APIC_MAX_SPECIES);
        bool absorbing = false;
        for (int k = 0; k < 2 * dims; ++k) absorbing = absorbing || p.pbc[k] == 1;
        for (int s = 0; s < c.nspecies; ++s)
            for (int b = 0; b < 2; ++b) sp[s].alive[b] = absorbing ? dalloc<uint8_t>(c.species[s].capacity) : nullptr;
        for (int s = 0; s < c.nspecies; ++s) {
            sp[s].live_end = absorbing ? dalloc<unsigned>(1) : nullptr;
            if (absorbing) APIC_CUDA(cudaMemsetAsync(sp[s].live_end, 0xFF, sizeof(unsigned), stream));
        }
        solver.F.dims = dims;
        solver.F.rho_acc = dalloc<unsigned long long>(N);
        solver.F.rho = dalloc<double>(N);
        solver.F.phi = dalloc<double>(N);
        solver.F.E = dalloc<double>((dims == 3 ? 4 : 2) * N);
        wall_solver.stream = stream;
        wall_solver.alloc = [this](size_t bytes) -> void* { return dalloc<unsigned char>(bytes); };
        wall_solver.setup(dims, p.n, p.d, p.wall, p.eps, c.wall_potential);
        wall_solver.set_sides(solver.F.phi);
        wall_planes = dalloc<double>(dims * N);
        APIC_CUDA(cudaStreamSynchronize(stream));
    }

    // FieldSolver::solve(Mesh2D&) / solve(Mesh3D&) with walls, src/FieldSolver.cpp:389-405
    void solve_walls() {
        const size_t N = (size_t)p.n[0] * p.n[1] * p.n[2];
        const unsigned g = (unsigned)std::min<size_t>((N + 255) / 256, 4096);
        k_walls_rho<<<g, 256, 0, stream>>>(solver.F.rho_acc, solver.F.rho, N, p.inv_rho_scale);
        wall_solver.solve(solver.F.rho, solver.F.phi, solver.F.E, nullptr);
    }

    void solve_fields() {
        if (walls) solve_walls();
        else solver.solve();
    }

    void deposit_and_solve() {
        for (int s = 0; s < cfg.nspecies; ++s) launch_push<kPushDepositOnly>(s);
        solve_fields();
    }

    void initialize() {
        time = 0.0;
        step_count = 0;
        deposit_and_solve();
        for (int s = 0; s < cfg.nspecies; ++s) launch_push<kPushInitHalf>(s);
        initialized = true;
        steps_since_sort = sort_interval;  // sort before the first step
        for (int k = 0; k < APIC_MAX_SPECIES; ++k) since_sort[k] = species_interval[k];
    }

    void resume(double t, uint64_t k) {
        time = t;
        step_count = k;
        deposit_and_solve();
        initialized = true;
        steps_since_sort = sort_interval;
        for (int k = 0; k < APIC_MAX_SPECIES; ++k) since_sort[k] = species_interval[k];
    }

    // One step as a CUDA graph: its kernel parameters depend only on which
    // species are sorted this step and on each species' buffer parity, so the
    // graphs are cached under that key (at most a few per run).
    struct StepGraph {
        unsigned key;
        cudaGraphExec_t exec;
    };
    std::vector<StepGraph> step_graphs;

    void drop_graphs() {
        for (auto& g : step_graphs) cudaGraphExecDestroy(g.exec);
        step_graphs.clear();
    }

    void enqueue_step(unsigned sort_mask) {
        for (int s = 0; s < cfg.nspecies; ++s)
            if (sort_mask >> s & 1u) sort_species(s);
        for (int s = 0; s < cfg.nspecies; ++s) launch_push<kPushStep>(s);
        solve_fields();
    }

    void launch_step_graph(unsigned sort_mask) {
        unsigned key = sort_mask;
        for (int s = 0; s < cfg.nspecies; ++s)
            key |= (unsigned)buf[s] << (APIC_MAX_SPECIES + s) | (unsigned)tiles_ready[s] << (2 * APIC_MAX_SPECIES + s);
        cudaGraphExec_t exec = nullptr;
        for (const auto& g : step_graphs)
            if (g.key == key) exec = g.exec;
        if (!exec) {
            int saved[APIC_MAX_SPECIES];
            for (int s = 0; s < APIC_MAX_SPECIES; ++s) saved[s] = buf[s];
            cudaGraph_t g = nullptr;
            APIC_CUDA(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
            enqueue_step(sort_mask);
            const cudaError_t ce = cudaStreamEndCapture(stream, &g);
            for (int s = 0; s < APIC_MAX_SPECIES; ++s) buf[s] = saved[s];
            APIC_CUDA(ce);
            const cudaError_t ie = cudaGraphInstantiate(&exec, g, 0);
            cudaGraphDestroy(g);
            APIC_CUDA(ie);
            step_graphs.push_back({key, exec});
        }
        APIC_CUDA(cudaGraphLaunch(exec, stream));
        for (int s = 0; s < cfg.nspecies; ++s)
            if (sort_mask >> s & 1u) {
                buf[s] ^= 1;
                tiles_ready[s] = true;
            }
    }

    // 2D runs with walls of this many particles a node stay in load order: a sorted warp's
    // particles, and its neighbours', commit to the same few nodes, and the more of them share a
    // node the longer its atomics queue, while particles in load order spread over the mesh,
    // which L2 holds.  us a step, load order against sorted every 16 steps, both species: 260 a
    // node on 100 x 128 nodes 341 / 430, 129 x 129 406 / 529, 250 x 256 1225 / 1660, 500 x 512
    // 4649 / 5608; 520 a node on 60 x 64 407 / 445, 250 x 256 2383 / 4152.  Sorted is faster on
    // 60 x 64 at 260 a node (214 / 174) and at 104 (74 / 64).
    bool crowded(int s) const { return walls && cfg.dims == 2 && sp[s].n / ncells >= (size_t)kCrowdedPpc; }
    static constexpr int kCrowdedPpc = 256;

    void do_steps(size_t nsteps) {
        require(initialized, "initialize() or resume() must precede step()", APIC_ERR_STATE);
        for (size_t it = 0; it < nsteps; ++it) {
            unsigned sort_mask = 0;
            for (int s = 0; s < cfg.nspecies; ++s)
                if (since_sort[s] >= species_interval[s] && sp[s].n && !crowded(s)) sort_mask |= 1u << s;
            for (int s = 0; s < cfg.nspecies; ++s) {
                if (since_sort[s] >= species_interval[s]) since_sort[s] = 0;
                // histogram, three scan passes, scatter (FP32: rank + gather; tiles: their items)
                if (sort_mask >> s & 1u) launches += (fp32 ? 6 : 5) + (sp[s].tiled ? 1 : 0);
            }
            if (sort_mask) steps_since_sort = 0;
            for (int s = 0; s < cfg.nspecies; ++s)
                if (sp[s].n) ++launches;
            launches += (cfg.dims == 2 ? 3 : 5) + (walls ? 2 : 0);  // transform passes (walls: density and field too)
            if (!timing) {
                launch_step_graph(sort_mask);
            } else {
                // kernel by kernel, with events between the phases
                Ev ev{};
                APIC_CUDA(cudaEventCreate(&ev.a)); APIC_CUDA(cudaEventCreate(&ev.b));
                APIC_CUDA(cudaEventCreate(&ev.c)); APIC_CUDA(cudaEventCreate(&ev.d));
                APIC_CUDA(cudaEventRecord(ev.a, stream));
                for (int s = 0; s < cfg.nspecies; ++s)
                    if (sort_mask >> s & 1u) {
                        sort_species(s);
                        tiles_ready[s] = true;
                    }
                APIC_CUDA(cudaEventRecord(ev.b, stream));
                for (int s = 0; s < cfg.nspecies; ++s) launch_push<kPushStep>(s);
                APIC_CUDA(cudaEventRecord(ev.c, stream));
                solve_fields();
                APIC_CUDA(cudaEventRecord(ev.d, stream));
                ev.sorted = sort_mask != 0;
                events.push_back(ev);
            }
            ++steps_since_sort;
            for (int s = 0; s < cfg.nspecies; ++s) ++since_sort[s];
            time += cfg.dt;
            ++step_count;
        }
    }

    void collect_timing() {
        for (auto& e : events) {
            float t_sort = 0, t_push = 0, t_solve = 0;
            APIC_CUDA(cudaEventElapsedTime(&t_sort, e.a, e.b));
            APIC_CUDA(cudaEventElapsedTime(&t_push, e.b, e.c));
            APIC_CUDA(cudaEventElapsedTime(&t_solve, e.c, e.d));
            sort_ms += t_sort;
            push_ms += t_push;
            solve_ms += t_solve;
            ++timed_steps;
            cudaEventDestroy(e.a); cudaEventDestroy(e.b); cudaEventDestroy(e.c); cudaEventDestroy(e.d);
        }
        events.clear();
    }

    void sync() {
        const cudaError_t e = bounded_wait(stream, 600.0);
        if (e == cudaErrorNotReady) throw Error(APIC_ERR_TIMEOUT, "device work did not complete in time");
        APIC_CUDA(e);
    }

    size_t read_particles(int s, size_t cap, double* pos, double* v, double* vh) {
        require(s >= 0 && s < cfg.nspecies, "species index out of range");
        const SpeciesND& S = sp[s];
        const size_t n = S.n;
        require(cap >= n, "output capacity below the particle count", APIC_ERR_CAPACITY);
        if (fp32) to_fp64(s);
        if (initialized) launch_push<kPushSync>(s);  // time-centred v of the current state
        const int b = buf[s];
        const int o = b ^ 1;
        // un-permute into the other buffer's arrays (free outside a sort)
        double* scratch[7];
        int k = 0;
        for (int a = 0; a < cfg.dims; ++a) scratch[k++] = S.pos[o][a];
        for (int a = 0; a < 3; ++a) scratch[k++] = S.vh[o][a];
        const unsigned blocks = (unsigned)((n + kThreads - 1) / kThreads);
        auto fetch = [&](const double* src, double* host, double* tmp) {
            if (!host || n == 0) return;
            k_unpermute<<<blocks, kThreads, 0, stream>>>(S.id[b], src, tmp, (unsigned)n);
            APIC_CUDA(cudaGetLastError());
            APIC_CUDA(cudaMemcpyAsync(host, tmp, n * sizeof(double), cudaMemcpyDeviceToHost, stream));
            APIC_CUDA(cudaStreamSynchronize(stream));
        };
        for (int a = 0; a < cfg.dims; ++a) fetch(S.pos[b][a], pos ? pos + a * n : nullptr, scratch[0]);
        if (pos && cfg.dims == 2) std::memset(pos + 2 * n, 0, n * sizeof(double));
        for (int a = 0; a < 3; ++a) fetch(S.vh[b][a], vh ? vh + a * n : nullptr, scratch[0]);
        if (walls && v) {  // in load order already
            for (int a = 0; a < 3 && n; ++a)
                APIC_CUDA(cudaMemcpyAsync(v + a * n, S.v[a], n * sizeof(double), cudaMemcpyDeviceToHost, stream));
        } else {
            for (int a = 0; a < 3; ++a) fetch(S.v[a], v ? v + a * n : nullptr, scratch[0]);
        }
        sync();
        return n;
    }

    void read_alive(int s, size_t cap, uint8_t* alive) {
        require(s >= 0 && s < cfg.nspecies, "species index out of range");
        const size_t n = sp[s].n;
        require(cap >= n, "output capacity below the particle count", APIC_ERR_CAPACITY);
        sync();
        if (sp[s].alive[0] && n) {  // in load order, through the other buffer (free outside a sort)
            const int b = buf[s];
            k_unpermute<<<(unsigned)((n + kThreads - 1) / kThreads), kThreads, 0, stream>>>(
                sp[s].id[b], sp[s].alive[b], sp[s].alive[b ^ 1], (unsigned)n);
            APIC_CUDA(cudaGetLastError());
            APIC_CUDA(cudaMemcpyAsync(alive, sp[s].alive[b ^ 1], n, cudaMemcpyDeviceToHost, stream));
        } else {
            std::memset(alive, 1, n);
        }
        APIC_CUDA(cudaStreamSynchronize(stream));
    }

    // absorbed counts of species s per side: 4 in 2D, 6 in 3D
    void read_losses(int s, uint64_t* out) {
        require(s >= 0 && s < cfg.nspecies, "species index out of range");
        sync();
        unsigned long long h[6] = {0, 0, 0, 0, 0, 0};
        if (p.losses) APIC_CUDA(cudaMemcpyAsync(h, p.losses + 6 * s, sizeof h, cudaMemcpyDeviceToHost, stream));
        APIC_CUDA(cudaStreamSynchronize(stream));
        for (int k = 0; k < 2 * cfg.dims; ++k) out[k] = h[k];
    }

    // The components are separated on the device (a strided loop over the interleaved
    // field on the host took longer than 48 steps of the 256^3 deck) into
    // the work arrays of the solve, which are free between steps.  A small field is read in one
    // piece and separated here: a kernel and more copies take longer (all fields of 16^2 48 against
    // 66 us, 64^2 83 / 100, 16^3 96 / 115, 32 x 16^2 140 / 150, 128^2 the same).
    static constexpr size_t kSmallField = 256 << 10;
    void read_fields(double* rho, double* phi, double* E) {
        const size_t N = ncells;
        const size_t st = cfg.dims == 2 ? 2 : 4;  // doubles of E per node on the device
        if (E && N * st * sizeof(double) <= kSmallField) {
            sync();
            std::vector<double> h(N * st);
            if (rho) APIC_CUDA(cudaMemcpyAsync(rho, solver.F.rho, N * sizeof(double), cudaMemcpyDeviceToHost, stream));
            if (phi) APIC_CUDA(cudaMemcpyAsync(phi, solver.F.phi, N * sizeof(double), cudaMemcpyDeviceToHost, stream));
            APIC_CUDA(cudaMemcpyAsync(h.data(), solver.F.E, N * st * sizeof(double), cudaMemcpyDeviceToHost, stream));
            APIC_CUDA(cudaStreamSynchronize(stream));
            for (int c = 0; c < cfg.dims; ++c)
                for (size_t g = 0; g < N; ++g) E[c * N + g] = h[g * st + c];
            return;
        }
        std::vector<HostCopier::Job> jobs;
        if (rho) jobs.push_back({rho, solver.F.rho, N * sizeof(double)});
        if (phi) jobs.push_back({phi, solver.F.phi, N * sizeof(double)});
        if (E) {
            double* plane[3];
            for (int c = 0; c < cfg.dims; ++c)
                plane[c] = walls ? wall_planes + c * N
                                 : reinterpret_cast<double*>(c < 2 ? solver.F.A : solver.F.B) + (c & 1) * N;
            const unsigned g = (unsigned)std::min<size_t>((N + 255) / 256, 4096);
            if (cfg.dims == 2) k_split_field<2><<<g, 256, 0, stream>>>(solver.F.E, plane[0], plane[1], nullptr, N);
            else k_split_field<3><<<g, 256, 0, stream>>>(solver.F.E, plane[0], plane[1], plane[2], N);
            APIC_CUDA(cudaGetLastError());
            for (int c = 0; c < cfg.dims; ++c) jobs.push_back({E + c * N, plane[c], N * sizeof(double)});
        }
        sync();
        copier.run(jobs, stream, E != nullptr);
    }

    void sample(apic_sample_nd* out) {
        std::memset(out, 0, sizeof *out);
        double vol = 1.0;
        for (int a = 0; a < cfg.dims; ++a) vol *= p.d[a];
        if (cfg.dims == 2) vol *= (cfg.out_of_plane_depth == 0.0 ? 1.0 : cfg.out_of_plane_depth);
        for (int s = 0; s < cfg.nspecies; ++s) {
            if (initialized) launch_push<kPushSync>(s);
            k_sample_nd<<<kSampleBlocks, 256, 0, stream>>>(sp[s], sp[s].alive[buf[s]], walls ? sp[s].id[buf[s]] : nullptr,
                                                           cfg.dims, sample_partial, sample_done, sample_out, solver.F.E, solver.F.rho, (long long)ncells,
                                                           0.5 * p.eps * vol, vol, s, s == cfg.nspecies - 1,
                                                           p.wall[0], p.wall[1], p.wall[2], p.n[0], p.n[1], p.n[2]);
            APIC_CUDA(cudaGetLastError());
        }
        double h[8];
        unsigned long long lost[6 * APIC_MAX_SPECIES] = {};
        APIC_CUDA(cudaMemcpyAsync(h, sample_out, sizeof h, cudaMemcpyDeviceToHost, stream));
        if (p.losses) APIC_CUDA(cudaMemcpyAsync(lost, p.losses, sizeof lost, cudaMemcpyDeviceToHost, stream));
        sync();
        for (int s = 0; s < cfg.nspecies; ++s) {
            out->kinetic_by_species[s] = h[s];
            out->kinetic_energy += h[s];
            // live_count: absorbed particles stay in place, flagged dead, each counted once in the ledger
            uint64_t dead = 0;
            for (int k = 0; k < 6; ++k) dead += lost[6 * s + k];
            out->live_particles += sp[s].n - dead;
        }
        out->field_energy = h[4];
        out->charge_l1 = h[5];
        out->total_energy = out->kinetic_energy + out->field_energy;
        out->step = step_count;
        out->time = time;
    }
};

}  // namespace nd
}  // namespace apic

// ---- stand-alone solves with walls -----------------------------------------------------

namespace apic {
namespace nd {

// device arrays and stream of one call, released on every exit path
struct MixedScratch {
    cudaStream_t s = nullptr;
    std::vector<void*> a;
    ~MixedScratch() {
        if (s) cudaStreamSynchronize(s);
        for (void* p : a) cudaFree(p);
        if (s) cudaStreamDestroy(s);
    }
    template <class T>
    T* get(size_t count) {
        void* p = nullptr;
        APIC_CUDA(cudaMalloc(&p, std::max<size_t>(count, 1) * sizeof(T)));
        a.push_back(p);
        return static_cast<T*>(p);
    }
};

static void solve_mixed_2d(const size_t* n, const double* length, int periodic_axis, double permittivity,
                           double lower, double upper, const double* rho, double* phi, double* electric) {
    require(n && length && rho && phi && electric, "null argument");
    require(periodic_axis == 0 || periodic_axis == 1, "periodic_axis must be 0 (x) or 1 (y)");
    require(std::isfinite(permittivity) && permittivity > 0, "field-solver permittivity must be positive and finite");
    require(std::isfinite(lower) && std::isfinite(upper), "wall potentials must be finite");
    const int periodic_y = periodic_axis == 1;
    const size_t nx = n[0], ny = n[1];
    const size_t nd = periodic_y ? nx : ny, np = periodic_y ? ny : nx;
    require(nd >= 3, "the wall axis needs at least 3 nodes");
    require(pow2(np) && np <= (size_t)kMaxLine, "the periodic extent must be a power of two up to 1024",
            APIC_ERR_UNSUPPORTED);
    for (int a = 0; a < 2; ++a)
        require(std::isfinite(length[a]) && length[a] > 0, "domain lengths must be positive and finite");
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
        throw Error(APIC_ERR_NO_DEVICE, "no CUDA device is visible");
    // Mesh2D spacings, src/Mesh2D.cpp:57-60
    const double dx = length[0] / (double)(periodic_y ? nx - 1 : nx);
    const double dy = length[1] / (double)(periodic_y ? ny : ny - 1);
    const size_t N = nx * ny;
    MixedScratch S;
    APIC_CUDA(cudaStreamCreateWithFlags(&S.s, cudaStreamNonBlocking));
    double* d_rho = S.get<double>(N);
    double* d_phi = S.get<double>(N);
    double* d_E = S.get<double>(2 * N);
    APIC_CUDA(cudaMemcpyAsync(d_rho, rho, N * sizeof(double), cudaMemcpyHostToDevice, S.s));
    WallSolver W;
    W.stream = S.s;
    W.alloc = [&](size_t bytes) -> void* { return S.get<unsigned char>(bytes); };
    const int nn[3] = {(int)nx, (int)ny, 1}, wall[3] = {periodic_y, !periodic_y, 0};
    const double d[3] = {dx, dy, 1.0};
    const double pot[4] = {lower, upper, lower, upper};  // (those of the periodic axis are not read)
    W.setup(2, nn, d, wall, permittivity, pot);
    W.set_sides(d_phi);
    W.solve(d_rho, d_phi, nullptr, d_E);
    APIC_CUDA(cudaMemcpyAsync(phi, d_phi, N * sizeof(double), cudaMemcpyDeviceToHost, S.s));
    APIC_CUDA(cudaMemcpyAsync(electric, d_E, 2 * N * sizeof(double), cudaMemcpyDeviceToHost, S.s));
    const cudaError_t e = bounded_wait(S.s, 600.0);
    if (e == cudaErrorNotReady) throw Error(APIC_ERR_TIMEOUT, "device work did not complete in time");
    APIC_CUDA(e);
}

static void solve_dirichlet_nd(int dims, const size_t* n, const double* length, double permittivity,
                               const double* pot, const double* rho, double* phi, double* electric) {
    require(dims == 2 || dims == 3, "dims must be 2 or 3");
    require(n && length && rho && phi && electric, "null argument");
    require(std::isfinite(permittivity) && permittivity > 0, "field-solver permittivity must be positive and finite");
    double side[4] = {0.0, 0.0, 0.0, 0.0};
    if (pot) {
        for (int a = 0; a < 4; ++a) {
            require(std::isfinite(pot[a]), "wall potentials must be finite");
            side[a] = pot[a];
        }
        require(dims == 2 || (side[0] == 0.0 && side[1] == 0.0 && side[2] == 0.0 && side[3] == 0.0),
                "3D Dirichlet walls are grounded");
    }
    size_t N = 1;
    for (int a = 0; a < dims; ++a) {
        require(n[a] >= 3 && pow2(n[a] - 1) && 2 * (n[a] - 1) <= (size_t)kMaxLine,
                "each extent must be 2^k + 1 nodes, 3 to 513", APIC_ERR_UNSUPPORTED);
        require(std::isfinite(length[a]) && length[a] > 0, "domain lengths must be positive and finite");
        N *= n[a];
    }
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0)
        throw Error(APIC_ERR_NO_DEVICE, "no CUDA device is visible");
    const int nx = (int)n[0], ny = (int)n[1], nz3 = dims == 3 ? (int)n[2] : 1;
    // Mesh2D / Mesh3D Dirichlet spacing L / (n - 1)
    const double d[3] = {length[0] / (double)(nx - 1), length[1] / (double)(ny - 1),
                         dims == 3 ? length[2] / (double)(nz3 - 1) : 1.0};
    MixedScratch S;
    APIC_CUDA(cudaStreamCreateWithFlags(&S.s, cudaStreamNonBlocking));
    double* d_rho = S.get<double>(N);
    double* d_phi = S.get<double>(N);
    double* d_E = S.get<double>((size_t)dims * N);
    APIC_CUDA(cudaMemcpyAsync(d_rho, rho, N * sizeof(double), cudaMemcpyHostToDevice, S.s));
    WallSolver W;
    W.stream = S.s;
    W.alloc = [&](size_t bytes) -> void* { return S.get<unsigned char>(bytes); };
    const int nn[3] = {nx, ny, nz3}, wall[3] = {1, 1, dims == 3};
    W.setup(dims, nn, d, wall, permittivity, side);
    W.set_sides(d_phi);
    W.solve(d_rho, d_phi, nullptr, d_E);
    APIC_CUDA(cudaMemcpyAsync(phi, d_phi, N * sizeof(double), cudaMemcpyDeviceToHost, S.s));
    APIC_CUDA(cudaMemcpyAsync(electric, d_E, (size_t)dims * N * sizeof(double), cudaMemcpyDeviceToHost, S.s));
    const cudaError_t e = bounded_wait(S.s, 600.0);
    if (e == cudaErrorNotReady) throw Error(APIC_ERR_TIMEOUT, "device work did not complete in time");
    APIC_CUDA(e);
}

}  // namespace nd
}  // namespace apic

// ---- C ABI ---------------------------------------------------------------------------

struct apic_sim_nd {
    apic::nd::SimND impl;
};

namespace {
thread_local std::string g_nd_error;

template <class F>
int guarded_nd(apic_sim_nd* h, F&& f) {
    try {
        f();
        return APIC_OK;
    } catch (const apic::Error& e) {
        if (h) h->impl.last_error = e.what();
        g_nd_error = e.what();
        return e.status;
    } catch (const std::exception& e) {
        if (h) h->impl.last_error = e.what();
        g_nd_error = e.what();
        return APIC_ERR_INVALID;
    }
}
}  // namespace

extern "C" {

int apic_simnd_create(const apic_config_nd* cfg, apic_sim_nd** out) {
    if (!cfg || !out) return APIC_ERR_INVALID;
    *out = nullptr;
    auto h = std::make_unique<apic_sim_nd>();
    const int rc = guarded_nd(h.get(), [&] { h->impl.create(*cfg); });
    if (rc == APIC_OK) *out = h.release();
    return rc;
}

void apic_simnd_destroy(apic_sim_nd* sim) { delete sim; }

const char* apic_simnd_last_error(const apic_sim_nd* sim) {
    return sim ? sim->impl.last_error.c_str() : g_nd_error.c_str();
}

int apic_simnd_load_particles(apic_sim_nd* sim, int species, size_t n, const double* pos, const double* v,
                              const double* v_half) {
    if (!sim) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] { sim->impl.load(species, n, pos, v, v_half); });
}

int apic_simnd_load_maxwellian(apic_sim_nd* sim, int species, size_t n, uint64_t seed, double thermal_speed,
                               double drift_x, int perturb_axis, double perturb_amplitude) {
    if (!sim) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] {
        sim->impl.load_maxwellian(species, n, seed, thermal_speed, drift_x, perturb_axis, perturb_amplitude);
    });
}

int apic_simnd_initialize(apic_sim_nd* sim) {
    if (!sim) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] { sim->impl.initialize(); });
}

int apic_simnd_resume(apic_sim_nd* sim, double time, uint64_t step) {
    if (!sim) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] { sim->impl.resume(time, step); });
}

int apic_simnd_step(apic_sim_nd* sim, size_t nsteps) {
    if (!sim) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] { sim->impl.do_steps(nsteps); });
}

int apic_simnd_synchronize(apic_sim_nd* sim) {
    if (!sim) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] { sim->impl.sync(); });
}

int apic_simnd_count(apic_sim_nd* sim, int species, size_t* n) {
    if (!sim || !n || species < 0 || species >= sim->impl.cfg.nspecies) return APIC_ERR_INVALID;
    *n = sim->impl.sp[species].n;
    return APIC_OK;
}

int apic_simnd_read_particles(apic_sim_nd* sim, int species, size_t capacity, double* pos, double* v, double* v_half,
                              size_t* n) {
    if (!sim) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] {
        const size_t got = sim->impl.read_particles(species, capacity, pos, v, v_half);
        if (n) *n = got;
    });
}

int apic_simnd_read_fields(apic_sim_nd* sim, double* rho, double* phi, double* electric) {
    if (!sim) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] { sim->impl.read_fields(rho, phi, electric); });
}
int apic_simnd_read_alive(apic_sim_nd* sim, int species, size_t capacity, uint8_t* alive) {
    if (!sim || !alive) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] { sim->impl.read_alive(species, capacity, alive); });
}
int apic_simnd_boundary_losses(apic_sim_nd* sim, int species, uint64_t* absorbed) {
    if (!sim || !absorbed) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] { sim->impl.read_losses(species, absorbed); });
}

int apic_simnd_sample(apic_sim_nd* sim, apic_sample_nd* out) {
    if (!sim || !out) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] { sim->impl.sample(out); });
}

int apic_simnd_cuda_stream(apic_sim_nd* sim, void** stream) {
    if (!sim || !stream) return APIC_ERR_INVALID;
    *stream = (void*)sim->impl.stream;
    return APIC_OK;
}

int apic_simnd_set_kernel_timing(apic_sim_nd* sim, int enable) {
    if (!sim) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] {
        sim->impl.sync();
        sim->impl.collect_timing();
        sim->impl.timing = enable != 0;
        sim->impl.push_ms = sim->impl.solve_ms = sim->impl.sort_ms = 0;
        sim->impl.timed_steps = 0;
    });
}

int apic_simnd_kernel_times(apic_sim_nd* sim, double* push_ms, double* solve_ms, double* sort_ms, uint64_t* steps) {
    if (!sim) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] {
        sim->impl.sync();
        sim->impl.collect_timing();
        if (push_ms) *push_ms = sim->impl.push_ms;
        if (solve_ms) *solve_ms = sim->impl.solve_ms;
        if (sort_ms) *sort_ms = sim->impl.sort_ms;
        if (steps) *steps = sim->impl.timed_steps;
    });
}

int apic_simnd_launch_count(apic_sim_nd* sim, uint64_t* launches) {
    if (!sim || !launches) return APIC_ERR_INVALID;
    return guarded_nd(sim, [&] { *launches = sim->impl.launches; });
}

int apic_field_solve_periodic_nd(int dims, const size_t* n, const double* length, double permittivity,
                                 const double* rho, double* phi, double* electric) {
    return guarded_nd(nullptr, [&] {
        apic::require(dims == 2 || dims == 3, "dims must be 2 or 3");
        apic::require(std::isfinite(permittivity) && permittivity > 0,
                      "field-solver permittivity must be positive and finite");
        apic_config_nd c{};
        c.dims = dims;
        for (int a = 0; a < dims; ++a) { c.n[a] = n[a]; c.length[a] = length[a]; }
        c.dt = 1.0;
        c.units = APIC_NORMALIZED;
        c.relative_permittivity = permittivity;
        c.nspecies = 1;
        c.species[0] = {1.0, 1.0, 1.0, 1};
        apic::nd::SimND S;
        S.create(c);
        size_t N = 1;
        for (int a = 0; a < dims; ++a) N *= n[a];
        double* d_rho = S.dalloc<double>(N);
        APIC_CUDA(cudaMemcpyAsync(d_rho, rho, N * 8, cudaMemcpyHostToDevice, S.stream));
        S.solver.F.rho_in = d_rho;
        S.solver.solve();
        S.read_fields(nullptr, phi, electric);
    });
}

int apic_field_solve_dirichlet_nd(int dims, const size_t* n, const double* length, double permittivity,
                                  const double* side_potentials, const double* rho, double* phi, double* electric) {
    return guarded_nd(nullptr, [&] {
        apic::nd::solve_dirichlet_nd(dims, n, length, permittivity, side_potentials, rho, phi, electric);
    });
}

int apic_field_solve_mixed_2d(const size_t* n, const double* length, int periodic_axis, double permittivity,
                              double lower_potential, double upper_potential, const double* rho, double* phi,
                              double* electric) {
    return guarded_nd(nullptr, [&] { apic::nd::solve_mixed_2d(n, length, periodic_axis, permittivity,
                                                              lower_potential, upper_potential, rho, phi, electric); });
}

}  // extern "C"

// ---- allocation-free periodic field solve --------------------------------------
//
// Some callers cannot call cudaMalloc: hosts that own every byte of device
// memory through their own pool or arena, and time-stepping loops that must not
// hit cudaMalloc's implicit device synchronisation (or run where allocation is
// not allowed).  apic_field_solve_periodic_nd_noalloc serves them: the caller
// passes device buffers for rho, phi and E, and the FFT work arrays live in the
// file-scope device array below, which every GPU that loads this library keeps
// until the process exits.

namespace apic {
namespace nd {

constexpr size_t kNoAllocMaxPoints = 65536;  // largest mesh (nx * ny * nz) the array serves
constexpr size_t kNoAllocMaxLine = 1024;     // largest extent per axis
// W, A, B (complex), interleaved E (4 doubles), rho copy, and three twiddle tables
constexpr size_t kNoAllocScratchBytes =
    3 * kNoAllocMaxPoints * sizeof(Cplx) + 4 * kNoAllocMaxPoints * sizeof(double) +
    kNoAllocMaxPoints * sizeof(double) + 3 * kNoAllocMaxLine * sizeof(Cplx);

static __device__ __align__(256) unsigned char g_solve_scratch[kNoAllocScratchBytes];

// exp(-2 pi i k / n), k < n
__global__ void k_noalloc_twiddles(Cplx* tw, int n) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    double s, c;
    sincospi(2.0 * (double)k / (double)n, &s, &c);
    tw[k] = {c, -s};
}

// interleaved E (2 or 4 doubles per node) -> [dims][N]
__global__ void k_noalloc_deinterleave(const double* E, int dims, long long N, double* out) {
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= N) return;
    const int st = dims == 2 ? 2 : 4;
    for (int c = 0; c < dims; ++c) out[c * N + g] = E[g * st + c];
}

}  // namespace nd
}  // namespace apic

namespace {
// A caller buffer of the allocation-free solve must be device (or managed)
// memory of the current device: a host pointer would make the kernels fault.
void require_device_buffer(const void* ptr, const char* name) {
    cudaPointerAttributes a{};
    const cudaError_t e = cudaPointerGetAttributes(&a, ptr);
    if (e != cudaSuccess) {
        cudaGetLastError();
        throw apic::Error(APIC_ERR_INVALID, std::string(name) + " is not a device pointer");
    }
    apic::require(a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged,
                  std::string(name) + " must be device or managed memory (got a host pointer)");
    if (a.type == cudaMemoryTypeDevice) {
        int dev = 0;
        APIC_CUDA(cudaGetDevice(&dev));
        apic::require(a.device == dev, std::string(name) + " belongs to another device than the current one");
    }
}
}  // namespace

extern "C" int apic_field_solve_periodic_nd_noalloc(int dims, const size_t* n, const double* length,
                                                     double permittivity, const double* d_rho, double* d_phi,
                                                     double* d_electric, void* stream) {
    using namespace apic::nd;
    return guarded_nd(nullptr, [&] {
        apic::require(dims == 2 || dims == 3, "dims must be 2 or 3");
        apic::require(n && length && d_rho && d_phi && d_electric, "null argument");
        apic::require(std::isfinite(permittivity) && permittivity > 0,
                      "field-solver permittivity must be positive and finite");
        size_t N = 1;
        for (int a = 0; a < dims; ++a) {
            apic::require(pow2(n[a]) && n[a] <= kNoAllocMaxLine,
                          "allocation-free solve: extents must be powers of two up to 1024", APIC_ERR_UNSUPPORTED);
            apic::require(std::isfinite(length[a]) && length[a] > 0, "domain lengths must be positive and finite");
            N *= n[a];
        }
        apic::require(N <= kNoAllocMaxPoints,
                      "allocation-free solve: mesh has " + std::to_string(N) + " points, the scratch array holds " +
                          std::to_string(kNoAllocMaxPoints),
                      APIC_ERR_CAPACITY);
        require_device_buffer(d_rho, "d_rho");
        require_device_buffer(d_phi, "d_phi");
        require_device_buffer(d_electric, "d_electric");
        // the scratch array's address in the current device's context, looked
        // up on every call (cheap), so it stays valid after a device reset
        void* base = nullptr;
        APIC_CUDA(cudaGetSymbolAddress(&base, g_solve_scratch));
        unsigned char* bytes = static_cast<unsigned char*>(base);
        Cplx* W = reinterpret_cast<Cplx*>(bytes);
        Cplx* A = W + kNoAllocMaxPoints;
        Cplx* B = A + kNoAllocMaxPoints;
        double* E = reinterpret_cast<double*>(B + kNoAllocMaxPoints);
        double* rho = E + 4 * kNoAllocMaxPoints;
        Cplx* tw = reinterpret_cast<Cplx*>(rho + kNoAllocMaxPoints);
        cudaStream_t s = static_cast<cudaStream_t>(stream);

        Solver S;
        S.stream = s;
        FieldsND& F = S.F;
        F.dims = dims;
        F.nx = (int)n[0];
        F.ny = (int)n[1];
        F.nz = dims == 3 ? (int)n[2] : 1;
        F.lnx = ilog2(F.nx);
        F.lny = ilog2(F.ny);
        for (int a = 0; a < 3; ++a) F.L[a] = a < dims ? length[a] : 1.0;
        F.eps = permittivity;
        F.inv_scale = 1.0;
        double kmax = 0;
        for (int a = 0; a < dims; ++a) kmax = std::max(kmax, 3.141592653589793 * (double)n[a] / length[a]);
        F.pack = std::ldexp(1.0, (int)std::lround(std::log2(kmax)));
        F.rho_in = d_rho;  // every scratch element below is written before it is read
        F.rho = rho;
        F.W = W;
        F.A = A;
        F.B = B;
        F.phi = d_phi;
        F.E = E;
        auto lines = [](int len, long long available, int buffers) {
            int T = 8;
            while (T > 1 && (size_t)buffers * T * len * sizeof(Cplx) + len * sizeof(Cplx) > kFftTileBytes) T >>= 1;
            while (T > 1 && available % T) T >>= 1;
            return T;
        };
        S.px = S.pass(0, lines(F.nx, (long long)F.ny * F.nz, 4));
        S.pxs = S.pass(0, lines(F.nx, (long long)F.ny * F.nz, 2));
        S.py = S.pass(1, lines(F.ny, F.nx, 4));
        S.pys = S.pass(1, lines(F.ny, F.nx, 2));
        if (dims == 3) S.pz = S.pass(2, lines(F.nz, F.nx, 4));
        const int len[3] = {F.nx, F.ny, F.nz};
        for (int a = 0; a < dims; ++a) {
            k_noalloc_twiddles<<<(len[a] + 255) / 256, 256, 0, s>>>(tw + a * kNoAllocMaxLine, len[a]);
        }
        S.px.tw = S.pxs.tw = tw;
        S.py.tw = S.pys.tw = tw + kNoAllocMaxLine;
        if (dims == 3) S.pz.tw = tw + 2 * kNoAllocMaxLine;
        APIC_CUDA(cudaGetLastError());
        S.allow_passes();  // the FFT kernels' fixed shared-memory limit (set once per device)
        S.solve();
        k_noalloc_deinterleave<<<(unsigned)((N + 255) / 256), 256, 0, s>>>(E, dims, (long long)N, d_electric);
        APIC_CUDA(cudaGetLastError());
    });
}
