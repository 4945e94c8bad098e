// records.cuh — the per-record and per-lane work of a pass, shared by the
// fused passes (pass.cu) and the resident minimizer loop (cg_loop_kernel.cuh): one
// lane of a chain warp tile, one generic record, one branch point. Pos maps a
// coordinate offset to a position; each kernel brings its own (read-only
// loads where a kernel's positions do not change, plain loads where they do).
// Target takes the forces (target_add): a ForceTarget, or a target whose sums
// are fixed at compile time.
#pragma once

#include "internal.h"
#include "potentials.cuh"

namespace mb {
namespace {

constexpr int kWarpOut = 30;  // forces written per chain warp tile: lanes 1..30 of 32 centres
constexpr unsigned char kLink = 1, kBend = 2;
constexpr unsigned kFull = 0xffffffffu;

__device__ __forceinline__ V3 shfl_up3(const V3& v) {
    return V3{__shfl_up_sync(kFull, v.x, 1), __shfl_up_sync(kFull, v.y, 1), __shfl_up_sync(kFull, v.z, 1)};
}
__device__ __forceinline__ V3 shfl_down3(const V3& v) {
    return V3{__shfl_down_sync(kFull, v.x, 1), __shfl_down_sync(kFull, v.y, 1), __shfl_down_sync(kFull, v.z, 1)};
}
template <class R>
__device__ __forceinline__ T3<R> shfl_up3(const T3<R>& v) {
    return T3<R>{__shfl_up_sync(kFull, v.x, 1), __shfl_up_sync(kFull, v.y, 1), __shfl_up_sync(kFull, v.z, 1)};
}
template <class R>
__device__ __forceinline__ T3<R> shfl_down3(const T3<R>& v) {
    return T3<R>{__shfl_down_sync(kFull, v.x, 1), __shfl_down_sync(kFull, v.y, 1), __shfl_down_sync(kFull, v.z, 1)};
}

// One lane's share of a chain warp tile: the link (q, q+1) and the bend centred
// at q are evaluated once; lanes that own their position (own: not lane 0) add the five
// terms acting on it to f and the link's and bend's energy to es and eb.
template <class R, bool E, bool F, class Target>
__device__ __forceinline__ void chain_lane(const V3& cprev, const V3& c, const V3& cnext, unsigned fl, const double2& lp,
                                           const double2& bp, bool own, int q, const Target& t, double* __restrict__ f,
                                           double& es, double& eb) {
    if constexpr (F) {
        T3<R> Fl{0, 0, 0}, A{0, 0, 0}, B{0, 0, 0};
        if (fl & kLink) Fl = stretch_force<R>(c, cnext, lp.x, lp.y);
        if (fl & kBend) bend_force<R>(diff<R>(cprev, c), diff<R>(c, cnext), bp.x, bp.y, A, B);
        const T3<R> Fp = shfl_up3(Fl), Bp = shfl_up3(B), An = shfl_down3(A);
        if (own) {
            // link (q-1, q) acts on q; link (q, q+1) reacts on q; bends centred
            // at q-1 (third bead), q (middle), q+1 (first bead); summed in double
            const double fx = double(Fp.x) - double(Fl.x) + double(Bp.x) + (double(A.x) - double(B.x)) - double(An.x);
            const double fy = double(Fp.y) - double(Fl.y) + double(Bp.y) + (double(A.y) - double(B.y)) - double(An.y);
            const double fz = double(Fp.z) - double(Fl.z) + double(Bp.z) + (double(A.z) - double(B.z)) - double(An.z);
            target_add(t, f, 3 * q, fx, fy, fz);
        }
    }
    if constexpr (E) {
        // a bond's length serves its link and both its bends: one square root
        // per lane, the previous bond's from the lane before
        const T3<double> r = diff<double>(c, cnext);
        const double len = sqrt(dot(r, r)), before = __shfl_up_sync(kFull, len, 1);
        if (own) {
            if (fl & kLink) es += stretch_energy_of(len, lp.x, lp.y);
            if (fl & kBend) eb += bend_energy_of<double>(diff<double>(cprev, c), r, before, len, bp.x, bp.y);
        }
    }
}

// Record i of bonded segment s (0 leftover stretch, 1 leftover bend, 2
// linker, 3 motor, 5 boundary): energy into acc[0], forces added to f.
template <class R, bool E, bool F, class Target, class Pos>
__device__ __forceinline__ void bonded_record(const DeviceFF& ff, const Target& t, const Pos& P,
                                              double* __restrict__ f, int s, int i, double (&acc)[4]) {
    switch (s) {
        case 0:
            if (i < ff.n_stretch) {
                const int2 q = ff.stretch_bs[i];
                const double2 p = ff.stretch_p[i];
                const V3 c1 = P(q.x), c2 = P(q.y);
                if constexpr (E) acc[0] += stretch_energy<double>(c1, c2, p.x, p.y);
                if constexpr (F) {
                    const T3<R> Fs = stretch_force<R>(c1, c2, p.x, p.y);
                    target_add(t, f, q.y, Fs.x, Fs.y, Fs.z);
                    target_add(t, f, q.x, -Fs.x, -Fs.y, -Fs.z);
                }
            }
            break;
        case 1:
            if (i < ff.n_bend) {
                const int4 q = ff.bend_bs[i];
                const double2 p = ff.bend_p[i];
                const V3 c1 = P(q.x), c2 = P(q.y), c3 = P(q.z);
                if constexpr (E) acc[0] += bend_energy<double>(diff<double>(c1, c2), diff<double>(c2, c3), p.x, p.y);
                if constexpr (F) {
                    T3<R> Fr1, Fr2;
                    bend_force<R>(diff<R>(c1, c2), diff<R>(c2, c3), p.x, p.y, Fr1, Fr2);
                    target_add(t, f, q.x, -Fr1.x, -Fr1.y, -Fr1.z);
                    target_add(t, f, q.y, Fr1.x - Fr2.x, Fr1.y - Fr2.y, Fr1.z - Fr2.z);
                    target_add(t, f, q.z, Fr2.x, Fr2.y, Fr2.z);
                }
            }
            break;
        case 2:
        case 3: {
            const int n = s == 2 ? ff.n_linker : ff.n_motor;
            if (i < n) {
                const int4 q = s == 2 ? ff.linker_bs[i] : ff.motor_bs[i];
                const double4 p = s == 2 ? ff.linker_p[i] : ff.motor_p[i];
                const V3 c1 = P(q.x), c2 = P(q.y), c3 = P(q.z), c4 = P(q.w);
                if constexpr (E) acc[0] += spring_energy<double>(c1, c2, c3, c4, p.x, p.y, p.z, p.w);
                if constexpr (F) {
                    const T3<R> Fl = spring_force<R>(c1, c2, c3, c4, p.x, p.y, p.z, p.w);
                    const R a1 = R(1) - R(p.z), a2 = R(p.z), b1 = R(1) - R(p.w), b2 = R(p.w);
                    target_add(t, f, q.x, -Fl.x * a1, -Fl.y * a1, -Fl.z * a1);
                    target_add(t, f, q.y, -Fl.x * a2, -Fl.y * a2, -Fl.z * a2);
                    target_add(t, f, q.z, Fl.x * b1, Fl.y * b1, Fl.z * b1);
                    target_add(t, f, q.w, Fl.x * b2, Fl.y * b2, Fl.z * b2);
                }
            }
            break;
        }
        default:
            if (i < ff.n_boundary) {
                const int o = ff.boundary_bs[i];
                const double2 p = ff.boundary_p[i];
                const double4 pl = ff.planes[ff.boundary_plane[i]];
                const V3 c = P(o);
                if constexpr (E) acc[0] += boundary_energy<double>(pl, c, p.x, p.y);
                if constexpr (F) {
                    const R f0 = boundary_force_mag<R>(pl, c, p.x, p.y);
                    target_add(t, f, o, f0 * R(pl.x), f0 * R(pl.y), f0 * R(pl.z));
                }
            }
            break;
    }
}

// Branch point i: energies of its four potentials into acc, forces added to f.
template <class R, bool E, bool F, class Target, class Pos>
__device__ __forceinline__ void branch_record(const DeviceFF& ff, const Target& t, const Pos& P, double* __restrict__ f, int i,
                                              double (&acc)[4]) {
    const int4 q = ff.branch_bs[i];
    const double4 pa = ff.branch_pa[i], pb = ff.branch_pb[i];
    const V3 c1 = P(q.x), c2 = P(q.y), c3 = P(q.z), c4 = P(q.w);
    const int m = ff.branch_mask;
    if constexpr (E) {
        if (m & 1) acc[0] += branch_stretch_energy<double>(c1, c2, c3, pa.y, pa.z, pa.x);
        if (m & 2) acc[1] += bend_energy<double>(diff<double>(c1, c2), diff<double>(c3, c4), pa.w, pb.x);
        if (m & 4) acc[2] += branch_dihedral_energy<double>(c1, c2, c3, c4, pb.y, pa.x);
        if (m & 8) acc[3] += branch_position_energy<double>(c1, c2, c3, pb.z, pa.x);
    }
    if constexpr (F) {
        T3<R> F1{0, 0, 0}, F2{0, 0, 0}, F3{0, 0, 0}, F4{0, 0, 0};
        if (m & 1) {
            const T3<R> g = branch_stretch_force<R>(c1, c2, c3, pa.y, pa.z, pa.x);
            const R pm1 = R(pa.x) - R(1), pp = R(pa.x);
            F1.x += -g.x * pm1; F1.y += -g.y * pm1; F1.z += -g.z * pm1;
            F2.x += g.x * pp; F2.y += g.y * pp; F2.z += g.z * pp;
            F3.x += -g.x; F3.y += -g.y; F3.z += -g.z;
        }
        if (m & 2) {
            T3<R> Fr1, Fr2;
            bend_force<R>(diff<R>(c1, c2), diff<R>(c3, c4), pa.w, pb.x, Fr1, Fr2);
            F1.x += -Fr1.x; F1.y += -Fr1.y; F1.z += -Fr1.z;
            F2.x += Fr1.x; F2.y += Fr1.y; F2.z += Fr1.z;
            F3.x += -Fr2.x; F3.y += -Fr2.y; F3.z += -Fr2.z;
            F4.x += Fr2.x; F4.y += Fr2.y; F4.z += Fr2.z;
        }
        if (m & 4) {
            T3<R> L1, L2, L3, L4;
            branch_dihedral_force<R>(c1, c2, c3, c4, pb.y, pa.x, L1, L2, L3, L4);
            F1.x += L1.x; F1.y += L1.y; F1.z += L1.z;
            F2.x += L2.x; F2.y += L2.y; F2.z += L2.z;
            F3.x += L3.x; F3.y += L3.y; F3.z += L3.z;
            F4.x += L4.x; F4.y += L4.y; F4.z += L4.z;
        }
        if (m & 8) {
            T3<R> P1, P2, P3;
            branch_position_force<R>(c1, c2, c3, pb.z, pa.x, P1, P2, P3);
            F1.x += P1.x; F1.y += P1.y; F1.z += P1.z;
            F2.x += P2.x; F2.y += P2.y; F2.z += P2.z;
            F3.x += P3.x; F3.y += P3.y; F3.z += P3.z;
        }
        target_add(t, f, q.x, F1.x, F1.y, F1.z);
        target_add(t, f, q.y, F2.x, F2.y, F2.z);
        target_add(t, f, q.z, F3.x, F3.y, F3.z);
        target_add(t, f, q.w, F4.x, F4.y, F4.z);
    }
}

}  // namespace
}  // namespace mb
