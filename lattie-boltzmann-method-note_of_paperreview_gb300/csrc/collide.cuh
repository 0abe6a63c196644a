// Collision tail of C/evolution.h:597-652 (mass correction, moments, equilibrium, MRT relaxation with
// the operator of C/MRT_Process.h:4-179, optionally the Smagorinsky rate, body force) for one node
// (float, double) or one packed node pair (V2).
//
// The operator is worked out on the non-equilibrium parts of a few sums only. With the opposite pairs
// (1,2) (3,4) (5,6) (7,10) (8,9) (11,14) (12,13) (15,18) (16,17), pair sums S and differences A:
//   * the equilibrium of a pair sum is 2 w (rho - 1.5 rho u.u + 4.5 rho (e.u)^2), of a difference
//     6 w e.j; the sums over the two diagonals of a plane and their difference (= the shear stress)
//     need rho u_a u_b only, so no equilibrium of a single direction is formed;
//   * mass and momentum are conserved, so the axis-diagonal sum is -(d0 + AX) and the heat-flux
//     moment q_x is -5 (A_x - j_x/3): energy, its square and q come from d0, AX and the axis pairs;
//   * the relaxed moments are folded into the updates of the pairs (ev, od below), with the body
//     force in the odd part;
//   * Smagorinsky: tau* = tau + 3 C |S| with |S| = (sqrt(nu0^2 + 18 C sqrt(Q)) - nu0)/(6 C), that is
//     tau* = tau + (sqrt(nu0^2 + 18 C sqrt(Q)) - nu0)/2: two square roots and one reciprocal.
// FP64 uses it. FP32 arithmetic keeps the moment-by-moment forms (collide_node, collide_pairs,
// collide_x2): their rounding biases the flow by up to 2e-5 in the velocity over the runs compared
// (2.7e-6 with this one), and FP32 and 16-bit runs are to continue what earlier ones gave.
// About 180 operations per node (with the closure 195) against 270 of the moment-by-moment form.
#pragma once

#include "step_common.cuh"

namespace islbm {

// square roots and reciprocals by type: FP64 IEEE (the parity path), FP32 the hardware
// approximations (within 1 and 2 units in the last place)
__device__ __forceinline__ double c_sqrt(double v) { return sqrt(v); }
__device__ __forceinline__ double c_rcp(double v) { return 1.0/v; }
__device__ __forceinline__ float c_sqrt(float v) {
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}
__device__ __forceinline__ float c_rcp(float v) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
    return r;
}

// F: streamed populations on entry, post-collision ones on exit. R: the scalar type of T.
template <bool LES, class T, class R>
__device__ __forceinline__ void collide(T (&F)[19], R rho_modify, R f6, R f12, R tau, R lesC, T &rho, T &u1, T &v1, T &w1) {
    constexpr double se = 1.19, seps = 1.4, sq = 1.2, spi = 1.4, sm = 1.5;
    F[0] = F[0] + T(rho_modify);
    const T S0 = F[1] + F[2], S1 = F[3] + F[4], S2 = F[5] + F[6], S3 = F[7] + F[10], S4 = F[8] + F[9];
    const T S5 = F[11] + F[14], S6 = F[12] + F[13], S7 = F[15] + F[18], S8 = F[16] + F[17];
    const T A0 = F[1] - F[2], A1 = F[3] - F[4], A2 = F[5] - F[6], A3 = F[7] - F[10], A4 = F[8] - F[9];
    const T A5 = F[11] - F[14], A6 = F[12] - F[13], A7 = F[15] - F[18], A8 = F[16] - F[17];
    const T a = S3 + S4, b = S5 + S6, c = S7 + S8;             // diagonals of the xy, xz, yz planes
    const T d34 = A3 - A4, s34 = A3 + A4, d56 = A5 - A6, s56 = A5 + A6, d78 = A7 - A8, s78 = A7 + A8;
    rho = (F[0] + ((S0 + S1) + S2)) + ((a + b) + c);
    const T jx = (A0 + d34) + d56, jy = (A1 + s34) + d78, jz = (A2 + s56) + s78;
    const T inv = c_rcp(rho);
    u1 = T(jx*inv); v1 = T(jy*inv); w1 = T(jz*inv);
    // non-equilibrium parts
    const T xx = T(jx*u1), yy = T(jy*v1), zz = T(jz*w1);
    const T bp = T(R(1.0/9.0))*rho - T(R(1.0/6.0))*((xx + yy) + zz);
    const T X = T(R(0.5))*xx + bp, Y = T(R(0.5))*yy + bp, Z = T(R(0.5))*zz + bp;
    const T x = S0 - X, y = S1 - Y, z = S2 - Z, d0 = F[0] - T(R(3))*bp;
    const T cn = c - (T(R(0.5))*zz + Y);
    const T ab = (a - b) - (Y - Z);
    const T mxy = (S3 - S4) - jx*v1, mxz = (S5 - S6) - jx*w1, myz = (S7 - S8) - jy*w1;
    const T AX = (x + y) + z;
    const T d1 = x - cn, sd = y - z, pww = sd + ab;
    T nu;
    if constexpr (LES) {
        const T h = d0 + d1, p = d1 - (d0 + AX);   // -(Pi_yy + Pi_zz), Pi_xx
        T s1 = T(h*h), s2 = T(mxy*mxy), Q = T(p*p);
        s1 = pww*pww + s1;
        s2 = mxz*mxz + s2;
        s2 = myz*myz + s2;
        Q = T(R(0.5))*s1 + Q;
        Q = T(R(2))*s2 + Q;
        const R nu0 = (tau - R(0.5))*R(1.0/3.0);
        const T s = c_sqrt(T(T(R(18)*lesC)*c_sqrt(Q) + T(nu0*nu0)));
        nu = c_rcp(T(T(R(0.5))*s + T(tau - R(0.5)*nu0)));
    } else {
        nu = c_rcp(T(tau));
    }
    // relaxed moments, folded: energy and energy square in F0, the axes (e1) and the diagonals (e2)
    const T e1 = T(R(22.0/126*se - 44.0/252*seps))*d0 + T(R(11.0/126*se + 20.0/252*seps))*AX;
    const T e2 = T(R(-16.0/126*se + 11.0/252*seps))*d0 + T(R(-8.0/126*se - 5.0/252*seps))*AX;
    F[0] = F[0] - T(R(60.0/126*se + 132.0/252*seps))*d0;
    F[0] = F[0] - T(R(30.0/126*se - 60.0/252*seps))*AX;
    const T r9 = T(T(nu*T(R(1.0/36.0)))*(T(R(3))*d1 - (T(R(2))*AX + d0)));
    const T p10 = (AX - d0) - T(R(3))*(T(R(2))*x + cn);
    const T t = T(R(-2.0/72*spi))*p10 + r9, g = T(R(1.0/72*spi))*p10 + r9;
    const T r11 = T(T(nu*T(R(1.0/12.0)))*pww);
    const T piw = ab - T(R(2))*sd;
    const T q = T(R(-2.0/24*spi))*piw + r11, k = T(R(1.0/24*spi))*piw + r11;
    const T n4 = T(nu*T(R(0.25)));
    const T ex = T(R(2))*t + e1, eyz = e1 - t, ey = eyz + q, ez = eyz - q;
    const T eg = e2 + g, exy = eg + k, exz = eg - k, ed = e2 - T(R(2))*g;
    // odd part: q from the axis differences, the antisymmetric third-order moments, the force
    const T dx = A0 - T(R(1.0/3.0))*jx, dy = A1 - T(R(1.0/3.0))*jy, dz = A2 - T(R(1.0/3.0))*jz;
    const T r4 = T(T(R(-0.125*sq))*dx), r6 = T(T(R(-0.125*sq))*dy), r8 = T(T(R(-0.125*sq))*dz);
    const T m16 = d34 - d56, m17 = d78 - s34, m18 = s56 - s78;
    const T al = T(R(0.125*sm))*m16 + r4, al2 = r4 - T(R(0.125*sm))*m16;
    const T r6f = r6 - T(f12);
    const T be = r6f - T(R(0.125*sm))*m17, be2 = T(R(0.125*sm))*m17 + r6f;
    const T ga = T(R(0.125*sm))*m18 + r8, ga2 = r8 - T(R(0.125*sm))*m18;
    const T oy = T(R(0.5*sq))*dy - T(f6);
    F[1] -= T(R(0.5*sq))*dx + ex; F[2] -= ex - T(R(0.5*sq))*dx;
    F[3] -= ey + oy; F[4] -= ey - oy;
    F[5] -= T(R(0.5*sq))*dz + ez; F[6] -= ez - T(R(0.5*sq))*dz;
    {
        const T ev = n4*mxy + exy, od = be + al;
        F[7] -= ev + od; F[10] -= ev - od;
    }
    {
        const T ev = exy - n4*mxy, od = be - al;
        F[8] -= ev + od; F[9] -= ev - od;
    }
    {
        const T ev = n4*mxz + exz, od = ga + al2;
        F[11] -= ev + od; F[14] -= ev - od;
    }
    {
        const T ev = exz - n4*mxz, od = ga - al2;
        F[12] -= ev + od; F[13] -= ev - od;
    }
    {
        const T ev = n4*myz + ed, od = ga2 + be2;
        F[15] -= ev + od; F[18] -= ev - od;
    }
    {
        const T ev = ed - n4*myz, od = ga2 - be2;
        F[16] -= ev + od; F[17] -= ev - od;
    }
}

}  // namespace islbm
