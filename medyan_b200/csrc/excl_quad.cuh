// excl_quad.cuh — a cylinder pair's excluded volume on four lanes.
//
// The analytic integral (excl.cuh) is a sum over four arctangent blocks that
// share their formula: block j of a pair has the root
// Q = sqrt((P + gam)(P - gam)), P = sqrt(alpha beta), two arctangents of u/Q
// and a numerator N. A thread that evaluates the whole pair runs them one
// after another, about 10 us of dependent FP64 work and of instructions
// executed once; here lane j of four consecutive lanes takes block j, so the
// work of a pair is a quarter as deep, the code a quarter as long and the
// registers fit twice the threads. The geometry and the final forces are split
// the same way (lane j returns the force on bead j).
//
// Every value is the one of excl.cuh bit for bit: the same expressions in the
// same order, the sums over the blocks taken in block order from lane to lane.
// All 32 lanes of the warp must call; lanes of one pair pass the same pair.
#pragma once

#include "excl.cuh"

namespace mb {

struct ExclQuad {
    double a, b, c, d, e, F;      // dot products of the pair (excl_scalars)
    double JJ;                    // minus the square of the triple product
    T3<double> r12, r34, r31;
    double Q, N, u1, u2;          // this lane's block: A, E, B, F for j = 0 .. 3
};

__device__ __forceinline__ double quad_pick(int j, double v0, double v1, double v2, double v3) {
    return j < 2 ? (j == 0 ? v0 : v1) : (j == 2 ? v2 : v3);
}
__device__ __forceinline__ double quad_lane(double v, int j) { return __shfl_sync(0xffffffffu, v, j, 4); }
__device__ __forceinline__ V3 quad_lane3(const V3& v, int j) {
    return V3{quad_lane(v.x, j), quad_lane(v.y, j), quad_lane(v.z, j)};
}
// v of the four lanes added in lane order.
__device__ __forceinline__ double quad_sum(double v) {
    return quad_lane(v, 0) + quad_lane(v, 1) + quad_lane(v, 2) + quad_lane(v, 3);
}

__device__ __forceinline__ ExclQuad excl_quad(int j, const V3& c1, const V3& c2, const V3& c3, const V3& c4) {
    ExclQuad s;
    s.r12 = diff<double>(c1, c2);
    s.r34 = diff<double>(c3, c4);
    s.r31 = diff<double>(c3, c1);
    const T3<double> r14 = diff<double>(c1, c4), r32 = diff<double>(c3, c2);
    s.a = dot(s.r12, s.r12);
    s.b = dot(s.r34, s.r34);
    s.c = dot(s.r31, s.r31);
    s.d = dot(s.r12, s.r34);
    s.e = dot(s.r12, s.r31);
    s.F = dot(s.r34, s.r31);
    const double a = s.a, b = s.b, d = s.d, e = s.e, F = s.F;
    const double g = dot(s.r12, r14), h = dot(s.r34, r32), I = dot(s.r34, r14);
    const double CC = d * e - a * F, DD = b * e - d * F, GG = d * g - a * I, HH = CC + GG - DD;
    const double alpha = j < 2 ? a : b, gam = quad_pick(j, e, g, F, h);
    const T3<double>& rb = j == 1 ? r14 : (j == 3 ? r32 : s.r31);
    const double P = sqrt(alpha * dot(rb, rb));
    s.Q = sqrt(stdmax<double>(0.0, (P + gam) * (P - gam)));
    s.N = quad_pick(j, CC, GG, DD, HH);
    s.u1 = quad_pick(j, a + e, a + e - d, F, d + F);
    s.u2 = quad_pick(j, e, e - d, F - b, d + F - b);
    const double cx = s.r12.y * s.r34.z - s.r12.z * s.r34.y, cy = s.r12.z * s.r34.x - s.r12.x * s.r34.z,
                 cz = s.r12.x * s.r34.y - s.r12.y * s.r34.x;
    const double jj = cx * s.r31.x + cy * s.r31.y + cz * s.r31.z;
    s.JJ = -jj * jj;
    return s;
}

// excl_energy of the pair, in all four lanes.
__device__ __forceinline__ double excl_energy_quad(int j, const V3& c1, const V3& c2, const V3& c3, const V3& c4,
                                                   double kRS) {
    const ExclQuad s = excl_quad(j, c1, c2, c3, c4);
    const double rQ = __drcp_rn(s.Q);
    const double ATG = atan(div_by(s.u1, s.Q, rQ)) - atan(div_by(s.u2, s.Q, rQ));
    return 0.5 * kRS / s.JJ * quad_sum(div_by(s.N, s.Q, rQ) * ATG);
}

// excl_force<EXACT> of the pair: the force on bead j (false in all four lanes
// when the analytic forces are rejected).
template <bool EXACT>
__device__ __forceinline__ bool excl_force_quad(int j, const V3& c1, V3 c2, const V3& c3, const V3& c4, double kRS,
                                                T3<double>& fo) {
    {
        // in_plane and move_bead2_out_of_plane: lane k < 3 normalizes component k
        const T3<double> v1 = diff<double>(c1, c2), v2 = diff<double>(c1, c3), v3 = diff<double>(c1, c4);
        const double cx = v1.y * v2.z - v1.z * v2.y, cy = v1.z * v2.x - v1.x * v2.z, cz = v1.x * v2.y - v1.y * v2.x;
        const double n = quad_pick(j, cx, cy, cz, cz) / sqrt(cx * cx + cy * cy + cz * cz);
        const double p = quad_pick(j, v3.x, v3.y, v3.z, v3.z) / sqrt(dot(v3, v3)) * n;
        const double along = quad_lane(p, 0) + quad_lane(p, 1) + quad_lane(p, 2);
        const double nx = quad_lane(n, 0), ny = quad_lane(n, 1), nz = quad_lane(n, 2);
        if (fabs(along) < 1e-1) c2 = V3{c2.x + nx * 0.01, c2.y + ny * 0.01, c2.z + nz * 0.01};
    }
    const ExclQuad s = excl_quad(j, c1, c2, c3, c4);
    const double a = s.a, b = s.b, c = s.c, d = s.d, e = s.e, F = s.F, Q = s.Q, N = s.N, u1 = s.u1, u2 = s.u2;
    const double iQ = EXACT ? __drcp_rn(Q) : 1.0 / Q;
    double bN, bQ, bd, b1, T;  // derivatives of block j (excl_force_exact), its share of the sum
    if constexpr (EXACT) {
        const double Q2 = Q * Q, iQ2 = __drcp_rn(Q2);
        const double ATG = atan(div_by(u1, Q, iQ)) - atan(div_by(u2, Q, iQ));
        const double W1 = Q2 / (Q2 + u1 * u1), W2 = Q2 / (Q2 + u2 * u2);
        bN = div_by(ATG, Q, iQ);
        bQ = div_by(-(ATG * N), Q2, iQ2) + (-W1 * u1 + W2 * u2) * N / (Q2 * Q);
        bd = div_by((W1 - W2) * N, Q2, iQ2);
        b1 = div_by(W1 * N, Q2, iQ2);
        T = div_by(N, Q, iQ) * ATG;
    } else {
        const double ATG = atan(u1 * iQ) - atan(u2 * iQ);
        const double Q2 = Q * Q, iQ2 = iQ * iQ;
        const double W1 = Q2 / (Q2 + u1 * u1), W2 = Q2 / (Q2 + u2 * u2), NiQ2 = N * iQ2;
        bN = ATG * iQ;
        bQ = -(ATG * NiQ2) + (-W1 * u1 + W2 * u2) * NiQ2 * iQ;
        bd = (W1 - W2) * NiQ2;
        b1 = W1 * NiQ2;
        T = N * iQ * ATG;
    }
    const double sumBlock = quad_sum(T);
    // block j's terms of b_ij: bN cn + bQ (cq / Q) + bd cd + b1 c1, added to
    // the sum of the blocks before it; a term a block does not have adds zero
    double bij[6];
    {
        const double cn[6] = {quad_pick(j, -2 * F, 2 * (F - b), 0.0, -2 * b), quad_pick(j, e, 2 * d - e, -F, 2 * d + F),
                              quad_pick(j, d, -d, b, -b), quad_pick(j, 0.0, -2 * a, 2 * e, -2 * (a + e)),
                              quad_pick(j, -a, a, -d, d), 0.0};
        const double cq[6] = {quad_pick(j, c, b + c - 2 * F, 0.0, b), quad_pick(j, 0.0, e - d, 0.0, -(d + F)),
                              quad_pick(j, -e, -(e - d), 0.0, b), quad_pick(j, 0.0, a, c, a + c + 2 * e),
                              quad_pick(j, 0.0, -a, -F, -(d + F)), j < 2 ? a : b};
        constexpr int kHasQ[6] = {0b1011, 0b1010, 0b1011, 0b1110, 0b1110, 0b1111};  // bit j: block j has the term
        const double cd[6] = {0.0, quad_pick(j, 0.0, -1.0, 0.0, 1.0), j < 2 ? 1.0 : 0.0, j < 2 ? 0.0 : -2.0,
                              j < 2 ? 0.0 : 1.0, 0.0};
        const double c1f = j < 2 ? 2.0 : 0.0, c1b = j < 2 ? 0.0 : 2.0;  // b11's of A and E, b22's of B and F
#pragma unroll
        for (int i = 0; i < 6; ++i) {
            const double tn = i == 5 ? 0.0 : bN * cn[i];
            const bool has_q = (kHasQ[i] >> j) & 1;
            const double tq = !has_q ? 0.0 : (EXACT ? bQ * div_by(cq[i], Q, iQ) : bQ * (cq[i] * iQ));
            const double td = (i == 0 || i == 5) ? 0.0 : bd * cd[i];
            const double t1 = i == 0 ? (j == 3 ? 0.0 : b1 * c1f) : (i == 3 ? b1 * c1b : 0.0);
            double p = 0.0, got = 0.0;
#pragma unroll
            for (int step = 0; step < 4; ++step) {  // lane `step` extends the sum of lane step - 1
                p = got + tn;
                p = p + tq;
                if (!(i == 0 || i == 5)) p = p + td;
                if (i == 0 || i == 3) p = p + t1;
                got = quad_lane(p, step);
            }
            bij[i] = got;
        }
    }
    const double b11 = bij[0], b12 = bij[1], b13 = bij[2], b22 = bij[3], b23 = bij[4], b33 = bij[5];
    const double invJJ = 1.0 / s.JJ;
    const double enFactor = EXACT ? kRS * invJJ / 2.0 : kRS * invJJ * 0.5;
    const double J11 = 2 * (-b * c + F * F), J12 = 2 * (c * d - e * F), J13 = 2 * (b * e - d * F);
    const double J22 = 2 * (-a * c + e * e), J23 = 2 * (-d * e + a * F), J33 = 2 * (d * d - a * b);
    const double q = -invJJ * sumBlock;
    const double dv0 = enFactor * (q * quad_pick(j, J13 - J11, J11, -J13 - J12, J12) +
                                   quad_pick(j, b13 - b11, b11, -b13 - b12, b12));
    const double dv1 = enFactor * (q * quad_pick(j, J23 - J12, J12, -J23 - J22, J22) +
                                   quad_pick(j, b23 - b12, b12, -b23 - b22, b22));
    const double dv2 = enFactor * (q * quad_pick(j, J33 - J13, J13, -J33 - J23, J23) +
                                   quad_pick(j, b33 - b13, b13, -b33 - b23, b23));
    fo.x = -(dv0 * s.r12.x + dv1 * s.r34.x + dv2 * s.r31.x);
    fo.y = -(dv0 * s.r12.y + dv1 * s.r34.y + dv2 * s.r31.y);
    fo.z = -(dv0 * s.r12.z + dv1 * s.r34.z + dv2 * s.r31.z);
    const bool bad = bad_force(fo.x) | bad_force(fo.y) | bad_force(fo.z);
    return ((__ballot_sync(0xffffffffu, bad) >> ((threadIdx.x & 31) & ~3)) & 15u) == 0u;
}

}  // namespace mb
