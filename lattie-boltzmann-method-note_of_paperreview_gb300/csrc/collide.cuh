// Collision tail of C/evolution.h:597-652 (mass correction, moments, equilibrium, MRT relaxation with
// the operator of C/MRT_Process.h:4-179, optionally the Smagorinsky rate, body force) for one node
// in FP64.
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
// FP32 arithmetic keeps the moment-by-moment forms (collide_node, collide_node_pairs,
// collide_x2): their rounding biases the flow by up to 2e-5 in the velocity over the runs compared
// (2.7e-6 with this one), and FP32 and 16-bit runs are to continue what earlier ones gave.
// About 180 operations per node (with the closure 195), two thirds of the moment-by-moment forms.
#pragma once

#include "step_common.cuh"

namespace islbm {

// F: streamed populations on entry, post-collision ones on exit.
template <bool LES>
__device__ __forceinline__ void collide(double (&F)[19], double rho_modify, double f6, double f12, double tau, double lesC, double &rho,
                                        double &u1, double &v1, double &w1) {
    constexpr double se = 1.19, seps = 1.4, sq = 1.2, spi = 1.4, sm = 1.5;
    F[0] = F[0] + rho_modify;
    const double S0 = F[1] + F[2], S1 = F[3] + F[4], S2 = F[5] + F[6], S3 = F[7] + F[10], S4 = F[8] + F[9];
    const double S5 = F[11] + F[14], S6 = F[12] + F[13], S7 = F[15] + F[18], S8 = F[16] + F[17];
    const double A0 = F[1] - F[2], A1 = F[3] - F[4], A2 = F[5] - F[6], A3 = F[7] - F[10], A4 = F[8] - F[9];
    const double A5 = F[11] - F[14], A6 = F[12] - F[13], A7 = F[15] - F[18], A8 = F[16] - F[17];
    const double a = S3 + S4, b = S5 + S6, c = S7 + S8;             // diagonals of the xy, xz, yz planes
    const double d34 = A3 - A4, s34 = A3 + A4, d56 = A5 - A6, s56 = A5 + A6, d78 = A7 - A8, s78 = A7 + A8;
    rho = (F[0] + ((S0 + S1) + S2)) + ((a + b) + c);
    const double jx = (A0 + d34) + d56, jy = (A1 + s34) + d78, jz = (A2 + s56) + s78;
    const double inv = 1.0/rho;
    u1 = jx*inv; v1 = jy*inv; w1 = jz*inv;
    // non-equilibrium parts
    const double xx = jx*u1, yy = jy*v1, zz = jz*w1;
    const double bp = (1.0/9.0)*rho - (1.0/6.0)*((xx + yy) + zz);
    const double X = 0.5*xx + bp, Y = 0.5*yy + bp, Z = 0.5*zz + bp;
    const double x = S0 - X, y = S1 - Y, z = S2 - Z, d0 = F[0] - 3*bp;
    const double cn = c - (0.5*zz + Y);
    const double ab = (a - b) - (Y - Z);
    const double mxy = (S3 - S4) - jx*v1, mxz = (S5 - S6) - jx*w1, myz = (S7 - S8) - jy*w1;
    const double AX = (x + y) + z;
    const double d1 = x - cn, sd = y - z, pww = sd + ab;
    double nu;
    if constexpr (LES) {
        const double h = d0 + d1, p = d1 - (d0 + AX);   // -(Pi_yy + Pi_zz), Pi_xx
        double s1 = h*h, s2 = mxy*mxy, Q = p*p;
        s1 = pww*pww + s1;
        s2 = mxz*mxz + s2;
        s2 = myz*myz + s2;
        Q = 0.5*s1 + Q;
        Q = 2*s2 + Q;
        const double nu0 = (tau - 0.5)*(1.0/3.0);
        const double s = sqrt((18*lesC)*sqrt(Q) + (nu0*nu0));
        nu = 1.0/(0.5*s + (tau - 0.5*nu0));
    } else {
        nu = 1.0/tau;
    }
    // relaxed moments, folded: energy and energy square in F0, the axes (e1) and the diagonals (e2)
    const double e1 = (22.0/126*se - 44.0/252*seps)*d0 + (11.0/126*se + 20.0/252*seps)*AX;
    const double e2 = (-16.0/126*se + 11.0/252*seps)*d0 + (-8.0/126*se - 5.0/252*seps)*AX;
    F[0] = F[0] - (60.0/126*se + 132.0/252*seps)*d0;
    F[0] = F[0] - (30.0/126*se - 60.0/252*seps)*AX;
    const double r9 = (nu*(1.0/36.0))*(3*d1 - (2*AX + d0));
    const double p10 = (AX - d0) - 3*(2*x + cn);
    const double t = (-2.0/72*spi)*p10 + r9, g = (1.0/72*spi)*p10 + r9;
    const double r11 = (nu*(1.0/12.0))*pww;
    const double piw = ab - 2*sd;
    const double q = (-2.0/24*spi)*piw + r11, k = (1.0/24*spi)*piw + r11;
    const double n4 = nu*0.25;
    const double ex = 2*t + e1, eyz = e1 - t, ey = eyz + q, ez = eyz - q;
    const double eg = e2 + g, exy = eg + k, exz = eg - k, ed = e2 - 2*g;
    // odd part: q from the axis differences, the antisymmetric third-order moments, the force
    const double dx = A0 - (1.0/3.0)*jx, dy = A1 - (1.0/3.0)*jy, dz = A2 - (1.0/3.0)*jz;
    const double r4 = (-0.125*sq)*dx, r6 = (-0.125*sq)*dy, r8 = (-0.125*sq)*dz;
    const double m16 = d34 - d56, m17 = d78 - s34, m18 = s56 - s78;
    const double al = (0.125*sm)*m16 + r4, al2 = r4 - (0.125*sm)*m16;
    const double r6f = r6 - f12;
    const double be = r6f - (0.125*sm)*m17, be2 = (0.125*sm)*m17 + r6f;
    const double ga = (0.125*sm)*m18 + r8, ga2 = r8 - (0.125*sm)*m18;
    const double oy = (0.5*sq)*dy - f6;
    F[1] -= (0.5*sq)*dx + ex; F[2] -= ex - (0.5*sq)*dx;
    F[3] -= ey + oy; F[4] -= ey - oy;
    F[5] -= (0.5*sq)*dz + ez; F[6] -= ez - (0.5*sq)*dz;
    {
        const double ev = n4*mxy + exy, od = be + al;
        F[7] -= ev + od; F[10] -= ev - od;
    }
    {
        const double ev = exy - n4*mxy, od = be - al;
        F[8] -= ev + od; F[9] -= ev - od;
    }
    {
        const double ev = n4*mxz + exz, od = ga + al2;
        F[11] -= ev + od; F[14] -= ev - od;
    }
    {
        const double ev = exz - n4*mxz, od = ga - al2;
        F[12] -= ev + od; F[13] -= ev - od;
    }
    {
        const double ev = n4*myz + ed, od = ga2 + be2;
        F[15] -= ev + od; F[18] -= ev - od;
    }
    {
        const double ev = ed - n4*myz, od = ga2 - be2;
        F[16] -= ev + od; F[17] -= ev - od;
    }
}

}  // namespace islbm
