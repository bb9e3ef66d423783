// Device-side exchange-correlation functionals (FP64).
//
// Each functional is written in its open-shell form f(rhoA, rhoB, gAA, gAB, gBB)
// with first derivatives, following the reference's formulas; the closed-shell
// grid path evaluates it at rhoB = rhoA, gAB = gBB = gAA exactly as
// DfFunctional_{LDA,GGA}'s closed-shell overloads do
// (src/libpdf/DfFunctional.h:98-126, :182-233).
//   Slater       src/libpdf/DfFunctional_Slater.cpp:25-85
//   VWN5 / VWN3  src/libpdf/DfFunctional_VWN.cpp:19-340, DfFunctional_VWN3.cpp:21-54
//   Becke 88     src/libpdf/DfFunctional_Becke88.cpp:25-165 (+ _ExceptLDA.cpp:25-32)
//   LYP          src/libpdf/DfFunctional_LYP.cpp:25-675
//   composites   SVWN (DfFunctional_SVWN.cpp:25-41), B88LYP (DfFunctional_B88LYP.cpp),
//                B3LYP 0.80/0.72/0.19/0.81 (DfFunctional_B3LYP.cpp:25-150)
//   PBE          not in the reference: pbe.cuh (Perdew-Burke-Ernzerhof 1996, PW92 correlation)
// Transcendentals are CUDA's own cbrt/exp/log/atan/sqrt.
#pragma once

#include "pbe.cuh"

namespace pdfxc {

struct XcOut {
    double f, va, vb, vgaa, vgab, vgbb;
};

namespace fdetail {

// Cube roots: the fractional powers of the densities (4/3, 8/3, 11/3, 1/6, ...) are products of
// cbrt(rho) and whole powers, so a spin's cube root is taken once and shared by the parts of a
// functional. (The functional kernels are bound by the FP64 pipe; pow costs several times cbrt. B3LYP
// over 3.5 M points: 0.88 -> 0.25 ms.)
__device__ __forceinline__ void slater(double ra, double rb, double ca, double cb, double& f, double& va, double& vb) {
    const double coef = -0.93052573634910002500;   // -(3/2) (3 / (4 pi))^(1/3)
    const double dcoef = -1.24070098179880003333;  // 4/3 of it
    f = coef * (ra * ca + rb * cb);
    va = dcoef * ca;
    vb = dcoef * cb;
}

struct VwnPar {
    double A, b, c, x0;
};

__device__ __forceinline__ double vwn_eps(const VwnPar p, double x) {
    const double X = x * (x + p.b) + p.c;
    const double X0 = p.x0 * (p.x0 + p.b) + p.c;
    const double Q = sqrt(4 * p.c - p.b * p.b);
    const double at = atan(Q / (2.0 * x + p.b));
    const double xx0 = x - p.x0;
    return p.A * (log(x * x / X) + 2.0 * p.b / Q * at -
                  p.b * p.x0 / X0 * (log(xx0 * xx0 / X) + 2.0 * (2.0 * p.x0 + p.b) / Q * at));
}

__device__ __forceinline__ double vwn_eps_prime(const VwnPar p, double x) {
    const double X = x * (x + p.b) + p.c;
    const double X0 = p.x0 * (p.x0 + p.b) + p.c;
    const double Q = sqrt(4 * p.c - p.b * p.b);
    const double x2b = 2.0 * x + p.b;
    const double inv = 1.0 / (x2b * x2b + Q * Q);
    return p.A * (2.0 / x - x2b / X - 4.0 * p.b * inv -
                  p.b * p.x0 / X0 * (2.0 / (x - p.x0) - x2b / X - 4.0 * (2.0 * p.x0 + p.b) * inv));
}

// v3 = true: the VWN3 paramagnetic/ferromagnetic sets (B3LYP); false: VWN5.
__device__ __forceinline__ void vwn(bool v3, double ra, double rb, double& f, double& va, double& vb) {
    const VwnPar P = v3 ? VwnPar{0.0310907, 13.0720, 42.7198, -0.409286}
                        : VwnPar{0.0310907, 3.72744, 12.9352, -0.10498};
    const VwnPar F = v3 ? VwnPar{0.01554535, 20.1231, 101.578, -0.743294}
                        : VwnPar{0.01554535, 7.06042, 18.0578, -0.325};
    const VwnPar A = VwnPar{-1.0 / (6.0 * M_PI * M_PI), 1.13107, 13.0045, -0.0047584};
    const double ec_coef = 1.70992093416136561766;  // 4 / (9 (2^(1/3) - 1))
    const double rho = ra + rb;
    const double inv = 1.0 / rho;
    const double x = sqrt(cbrt(3.0 / (4.0 * M_PI) * inv));
    const double zeta = (ra - rb) * inv;
    const double ep = vwn_eps(P, x), epp = vwn_eps_prime(P, x);
    if (zeta == 0.0) {  // no polarisation: g = g' = 0, only the paramagnetic fit remains
        f = rho * ep;
        const double v = ep + rho * (-x / (6.0 * rho) * epp);
        va = (ra > 1.0e-20) ? v : 0.0;
        vb = (rb > 1.0e-20) ? v : 0.0;
        return;
    }
    const double ef = vwn_eps(F, x), ea = vwn_eps(A, x);
    const double zp13 = cbrt(1.0 + zeta), zm13 = cbrt(1.0 - zeta);
    const double g = 9.0 / 8.0 * ((1.0 + zeta) * zp13 + (1.0 - zeta) * zm13 - 2.0);
    const double z3 = zeta * zeta * zeta, z4 = z3 * zeta;
    const double EC = ep + ea * g * (1.0 + (ec_coef * (ef - ep) / ea - 1.0) * z4);
    f = rho * EC;
    const double efp = vwn_eps_prime(F, x), eap = vwn_eps_prime(A, x);
    const double gp = 1.5 * (zp13 - zm13);
    const double h = ec_coef * ((ef - ep) / ea) - 1.0;
    const double hp = ec_coef / ea * (efp - epp - (ef - ep) / ea * eap);
    const double t1 = -x / (6.0 * rho) * (epp + eap * g * (1.0 + h * z4) + ea * g * hp * z4);
    const double t2c = ea * (gp * (1.0 + h * z4) + 4.0 * g * h * z3);
    va = (ra > 1.0e-20) ? EC + rho * (t1 + t2c * (inv * (1.0 - zeta))) : 0.0;
    vb = (rb > 1.0e-20) ? EC + rho * (t1 + t2c * (-inv * (1.0 + zeta))) : 0.0;
}

// One spin of Becke 88 from its density r, cube root c and gamma g: energy, d/dr, d/dgamma (zero
// potential where the density or gamma is below 1e-16, as the reference).
__device__ __forceinline__ void b88_spin(bool full, double r, double c, double g, double& t, double& v, double& vg) {
    const double EPS = 1.0e-16;
    t = v = vg = 0.0;
    if (!(r > EPS)) return;
    const double beta = 0.0042;
    const double G = full ? -0.93052573634910002500 : 0.0;  // -(3/2) (3 / (4 pi))^(1/3)
    const double r43 = r * c, sg = sqrt(g), x = sg / r43;
    const double bx = beta * x, sq = sqrt(x * x + 1.0);
    const double as = log(x + sq);
    const double M = 1.0 + 6.0 * bx * as;
    const double gx = G - (bx * x) / M;
    t = r43 * gx;
    if (!(g > EPS)) return;
    const double gp = 6.0 * bx * bx * (as + x / sq) / (M * M) - 2.0 * bx / M;
    v = 4.0 / 3.0 * c * (gx - x * gp);
    vg = 0.5 / sg * gp;
}

__device__ __forceinline__ void b88(bool full, double ra, double rb, double ca, double cb, double gaa, double gbb,
                                    double& f, double& va, double& vb, double& vgaa, double& vgbb) {
    double tA, tB;
    b88_spin(full, ra, ca, gaa, tA, va, vgaa);
    if (rb == ra && gbb == gaa) tB = tA, vb = va, vgbb = vgaa;
    else b88_spin(full, rb, cb, gbb, tB, vb, vgbb);
    f = tA + tB;
}

constexpr double LA = 0.04918, LB = 0.132, LC = 0.2533, LD = 0.349;

constexpr double LCF = 36.462398978764778;  // 2^(11/3) 3/10 (3 pi^2)^(2/3)
// omega and delta from m13 = rho^(-1/3)
__device__ __forceinline__ double lyp_omega(double rho, double m13) {
    const double m113 = m13 * m13 / (rho * rho * rho);  // rho^(-11/3)
    return exp(-LC * m13) * m113 / (1.0 + LD * m13);
}
__device__ __forceinline__ double lyp_delta(double m13) { return LC * m13 + LD * m13 / (1.0 + LD * m13); }
__device__ __forceinline__ void lyp_dgamma(double rho, double ra, double rb, double om, double de,
                                           double& gaa, double& gab, double& gbb) {
    const double rab = ra * rb, abo = LA * LB * om;
    gaa = -abo * (1.0 / 9.0 * rab * (1.0 - 3.0 * de - (de - 11.0) * ra / rho) - rb * rb);
    gbb = -abo * (1.0 / 9.0 * rab * (1.0 - 3.0 * de - (de - 11.0) * rb / rho) - ra * ra);
    gab = -abo * (1.0 / 9.0 * rab * (47.0 - 7.0 * de) - 4.0 / 3.0 * rho * rho);
}

// energy (every density) and potential (both densities above 1e-20)
__device__ __forceinline__ void lyp(double ra, double rb, double ca, double cb, double gaa, double gab, double gbb,
                                    double& f, double& va, double& vb, double& vgaa, double& vgab, double& vgbb) {
    const double TOL = 1.0e-20;
    va = vb = vgaa = vgab = vgbb = 0.0;
    const double rho = ra + rb, rab = ra * rb, ir = 1.0 / rho;
    const double r13 = cbrt(rho), rm13 = 1.0 / r13, rm43 = ir * rm13;
    const double ra83 = ra * ra * ca * ca, rb83 = rb * rb * cb * cb;
    const double om = lyp_omega(rho, rm13), abo = LA * LB * om;
    const double de = lyp_delta(rm13);
    const double d1 = 1.0 + LD * rm13;
    double daa, dab, dbb;
    lyp_dgamma(rho, ra, rb, om, de, daa, dab, dbb);
    f = -4.0 * LA / d1 * rab / rho - LCF * abo * rab * (ra83 + rb83) + daa * gaa + dab * gab + dbb * gbb;
    if (!(fabs(ra) > TOL && fabs(rb) > TOL)) return;
    const double opo = -1.0 / 3.0 * rm43 * (11.0 * r13 - LC - LD / d1);  // omega' / omega
    const double omp = opo * om;
    const double dep = 1.0 / 3.0 * (LD * LD * rm43 * rm13 / (d1 * d1) - ir * de);
    const double ra_aa = opo * daa - abo * (1.0 / 9.0 * rb * (1.0 - 3.0 * de - (de - 11.0) * ra * ir) -
                                            1.0 / 9.0 * rab * ((3.0 + ra * ir) * dep + (de - 11.0) * rb * ir * ir));
    const double rb_bb = opo * dbb - abo * (1.0 / 9.0 * ra * (1.0 - 3.0 * de - (de - 11.0) * rb * ir) -
                                            1.0 / 9.0 * rab * ((3.0 + rb * ir) * dep + (de - 11.0) * ra * ir * ir));
    const double t21 = 1.0 / 9.0 * (47.0 - 7.0 * de), t22 = -7.0 / 9.0 * rab * dep - 8.0 / 3.0 * rho;
    const double ra_ab = opo * dab - abo * (t21 * rb + t22);
    const double rb_ab = opo * dab - abo * (t21 * ra + t22);
    const double ra_bb = opo * dbb - abo * (1.0 / 9.0 * rb * (1.0 - 3.0 * de - (de - 11.0) * rb * ir) -
                                            1.0 / 9.0 * rab * ((3.0 + rb * ir) * dep - (de - 11.0) * rb * ir * ir) -
                                            2.0 * ra);
    const double rb_aa = opo * daa - abo * (1.0 / 9.0 * ra * (1.0 - 3.0 * de - (de - 11.0) * ra * ir) -
                                            1.0 / 9.0 * rab * ((3.0 + ra * ir) * dep - (de - 11.0) * ra * ir * ir) -
                                            2.0 * rb);
    const double a1c = -4.0 * LA / d1 * rab / rho;
    const double a1A = a1c * (1.0 / 3.0 * LD * rm43 / d1 + 1.0 / ra - ir);
    const double a1B = a1c * (1.0 / 3.0 * LD * rm43 / d1 + 1.0 / rb - ir);
    const double a2A = -LCF * LA * LB * (omp * rab * (ra83 + rb83) + om * rb * (11.0 / 3.0 * ra83 + rb83));
    const double a2B = -LCF * LA * LB * (omp * rab * (rb83 + ra83) + om * ra * (11.0 / 3.0 * rb83 + ra83));
    if (ra > TOL) {
        va = a1A + a2A + ra_aa * gaa + ra_ab * gab + ra_bb * gbb;
        vgaa = daa;
    }
    if (rb > TOL) {
        vb = a1B + a2B + rb_aa * gaa + rb_ab * gab + rb_bb * gbb;
        vgbb = dbb;
    }
    if (ra > TOL && rb > TOL) vgab = dab;
}

}  // namespace fdetail

__host__ __device__ constexpr bool functional_is_gga(int fn) { return fn == 2 || fn == 3 || fn == 4 || fn == 5; }

__device__ __forceinline__ XcOut eval_functional(int fn, double ra, double rb, double gaa, double gab,
                                                 double gbb) {
    using namespace fdetail;
    XcOut o{0, 0, 0, 0, 0, 0};
    double f1, a1, b1, f2, a2, b2, g1, g2, g3, g4, g5;
    const double ca = fn == 5 ? 0.0 : cbrt(ra), cb = fn == 5 ? 0.0 : (rb == ra ? ca : cbrt(rb));
    switch (fn) {
        case 0:  // SVWN
            slater(ra, rb, ca, cb, f1, a1, b1);
            vwn(false, ra, rb, f2, a2, b2);
            o.f = f1 + f2, o.va = a1 + a2, o.vb = b1 + b2;
            break;
        case 1:  // HFS
            slater(ra, rb, ca, cb, o.f, o.va, o.vb);
            break;
        case 2:  // HFB
            b88(true, ra, rb, ca, cb, gaa, gbb, o.f, o.va, o.vb, o.vgaa, o.vgbb);
            break;
        case 3:  // BLYP
            b88(true, ra, rb, ca, cb, gaa, gbb, f1, a1, b1, g1, g3);
            lyp(ra, rb, ca, cb, gaa, gab, gbb, f2, a2, b2, g2, g4, g5);
            o.f = f1 + f2, o.va = a1 + a2, o.vb = b1 + b2;
            o.vgaa = g1 + g2, o.vgab = g4, o.vgbb = g3 + g5;
            break;
        case 5: {  // PBE: value and the five first derivatives through dual numbers
            const Dual5 f = pbe::pbe(dvar(ra, 0), dvar(rb, 1), dvar(gaa, 2), dvar(gab, 3), dvar(gbb, 4));
            o.f = f.v, o.va = f.d[0], o.vb = f.d[1], o.vgaa = f.d[2], o.vgab = f.d[3], o.vgbb = f.d[4];
            break;
        }
        default: {  // B3LYP
            double fs, as, bs, fv, av, bv, fb, ab, bb, gba, gbb2, fl, al, bl, gla, glab, glb;
            slater(ra, rb, ca, cb, fs, as, bs);
            vwn(true, ra, rb, fv, av, bv);
            b88(false, ra, rb, ca, cb, gaa, gbb, fb, ab, bb, gba, gbb2);
            lyp(ra, rb, ca, cb, gaa, gab, gbb, fl, al, bl, gla, glab, glb);
            o.f = 0.80 * fs + 0.72 * fb + 0.19 * fv + 0.81 * fl;
            o.va = 0.80 * as + 0.72 * ab + 0.19 * av + 0.81 * al;
            o.vb = 0.80 * bs + 0.72 * bb + 0.19 * bv + 0.81 * bl;
            o.vgaa = 0.72 * gba + 0.81 * gla;
            o.vgab = 0.81 * glab;
            o.vgbb = 0.72 * gbb2 + 0.81 * glb;
        }
    }
    return o;
}

}  // namespace pdfxc
