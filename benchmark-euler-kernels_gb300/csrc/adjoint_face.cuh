// Transposed HLLC flux of one face: the arithmetic of the reverse step
// (adjoint.cu), in a header that also compiles as plain host C++ so that the
// CPU tests can check it against the host tangent-linear model.
//
// The flux differentiated is hllc::operator() of euler_operators/hllc.hpp:50-105.
// At exact ties (equal min/max arguments, ustar == 0 in the subsonic case)
// the derivative is the mean of the two one-sided derivatives.
#pragma once

#include <cstring>

#include "halve.cuh"

#if defined(__CUDACC__)
#include "euler_device.cuh"
#define EULR_ADJ_FN __host__ __device__ __forceinline__
#else
#define EULR_ADJ_FN inline
#endif

namespace eulr {

// Reciprocal and product: on the GPU on the integer pipes (rcp_alu within
// 0.5001 ulp, mul_alu rounded to nearest), correctly rounded on the host.
EULR_ADJ_FN double adj_rcp(double x)
{
#if defined(__CUDA_ARCH__)
    return rcp_alu(x);
#else
    return 1.0 / x;
#endif
}

EULR_ADJ_FN double adj_mul(double a, double b)
{
#if defined(__CUDA_ARCH__)
    return mul_alu(a, b);
#else
    return a * b;
#endif
}

// x * 0.5: on the GPU from the bit pattern on the integer pipe (the same bits
// as the FP64 multiply, halve.cuh), which saves an FP64 slot.
EULR_ADJ_FN double adj_half(double x)
{
#if defined(__CUDA_ARCH__)
    unsigned long long b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
    return __longlong_as_double(static_cast<long long>(halve_bits(b)));
#else
    return x * 0.5;
#endif
}

// Decisions on the integer pipe: on GB300 an FP64 compare takes a full slot
// of the FP64 pipe, which bounds the reverse step; the same decisions taken
// on the bit patterns cost nothing there.
EULR_ADJ_FN long long adj_bits(double x)
{
#if defined(__CUDA_ARCH__)
    // an opaque move: the compiler would otherwise turn some bit tests back
    // into FP64 compares, which take FP64-pipe slots
    long long b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
    return b;
#else
    long long b;
    std::memcpy(&b, &x, sizeof b);
    return b;
#endif
}

// Integer key with the order of the doubles, -0 and +0 equal (ties must
// see them as one value).
EULR_ADJ_FN long long adj_key(double x)
{
    long long const b = adj_bits(x);
    return (b << 1) == 0 ? 0 : (b ^ ((b >> 63) & 0x7fffffffffffffffLL));
}

EULR_ADJ_FN bool adj_neg(double x) // x < 0
{
    long long const b = adj_bits(x);
    return b < 0 && (b << 1) != 0;
}

EULR_ADJ_FN bool adj_pos(double x) // x > 0 (for non-NaN x)
{
    return adj_bits(x) > 0;
}

EULR_ADJ_FN bool adj_zero(double x) // x == +0 or -0
{
    return (adj_bits(x) << 1) == 0;
}

// One side of a face in the face frame: normal velocity un, tangential t1, t2.
struct FaceSide {
    double r, p, un, t1, t2;
    double c, cp, cr; // sound speed, dc/dp, dc/drho
    double e, ke;     // total energy per volume, kinetic energy per mass
};

struct FaceBar {
    double r, p, un, t1, t2;
};

EULR_ADJ_FN void zero(FaceBar& b) { b.r = b.p = b.un = b.t1 = b.t2 = 0.0; }

// One side's share of d flux / d ustar at ustar == 0 (a = S - un of the side,
// iS = 1/S): there the flux's mass and energy terms are b d and b E with
// b = a ustar/(S - ustar) and E = e + p + S d w, w = ustar - un.
EULR_ADJ_FN double tie_side_bar(FaceSide const& q, double a, double S, double iS, double gd, double ge, double gt1,
                                double gt2)
{
    double const E = (q.e + q.p) - S * (q.r * q.un);
    double const gb = (gd + gt1 * q.t1 + gt2 * q.t2) * q.r + ge * E;
    return gb * (a * iS);
}

// Transposed HLLC flux of one face (hllc.hpp:50-105).  The cotangent of the
// face flux is ds * (dd, de, dn, dt1, dt2) in the face frame (mass, energy,
// normal and tangential momentum); with UNIT the caller has already folded
// ds into (dd, ..., dt2) and ds is not read.  SETS the cotangents of the two
// sides' primitive states, bL and bR.
//
// What is transposed is the flux in the forward step's form (hllc_upwind
// in euler_device.cuh), which is the reference's in exact arithmetic:
//   A = cmax + max(u_L - u_R, 0), G = A (d_L + d_R),
//   n = A (d_L u_L + d_R u_R) - (p_R - p_L), ustar = n/G,
//   and with the upwind side's S = u + a, a = -+A, w = ustar - u and
//   b = a ustar/(S - ustar):  mass d b, energy b (e + p + S d w), normal
//   momentum d b ustar + p + a d w, tangential d b t.
// One acoustic speed in place of two wave speeds and two impedances: about 83
// FP64 operations a face where the form with both took 103, and 18 of its
// products and the reciprocal run on the integer pipes (a reverse godunov of
// 128^3 1239 -> 1047 us, of 64^3 193 -> 165).  The pressure
// term is the upwind side's, p_q + rc_q (ustar - un_q): the reference's mean
// of the two sides' values is the same function wherever ustar = num/den.
//
// Written for SIMT: the upwind side q (L when ustar > 0) is selected field by
// field instead of branching on it, so a warp whose faces point both ways
// runs the star branch once, not twice; only the rare supersonic faces and
// the ustar == 0 ties take their own paths.
template <bool UNIT = false>
EULR_ADJ_FN void hllc_bar(FaceSide const& L, FaceSide const& R, double dd, double de, double dn, double dt1,
                          double dt2, double ds, double inv_gm1, FaceBar& bL, FaceBar& bR)
{
    long long const kuL = adj_key(L.un), kuR = adj_key(R.un);
    long long const kcL = adj_key(L.c), kcR = adj_key(R.c);
    bool const u_lt = kuL < kuR;
    bool const u_gt = kuR < kuL;
    bool const c_lt = kcL < kcR;
    bool const c_gt = kcR < kcL;
    double const cmax = c_lt ? R.c : L.c;
    double const du = L.un - R.un;
    double const A = cmax + (u_gt ? du : 0.0);
    double const D = L.r + R.r;
    double const G = adj_mul(A, D);
    double const mom = L.r * L.un + R.r * R.un;
    double const n = A * mom - (R.p - L.p); // G > 0, so ustar has the sign of n
    bool const left = adj_pos(n);
    bool const tie = adj_zero(n);
    double const gd = UNIT ? dd : ds * dd;
    double const ge = UNIT ? de : ds * de;
    double const gn = UNIT ? dn : ds * dn;
    double const gt1 = UNIT ? dt1 : ds * dt1;
    double const gt2 = UNIT ? dt2 : ds * dt2;

    FaceSide q; // the upwind side's fields the branches read
    q.r = left ? L.r : R.r;
    q.p = left ? L.p : R.p;
    q.un = left ? L.un : R.un;
    q.t1 = left ? L.t1 : R.t1;
    q.t2 = left ? L.t2 : R.t2;
    q.e = left ? L.e : R.e;
    q.ke = left ? L.ke : R.ke;
    double const a = left ? -A : A; // S - un
    double const S = q.un + a;

    FaceBar bq;
    if (left ? adj_pos(S) : adj_neg(S)) {
        // supersonic: the flux is the upwind side's physical flux
        double const m = q.r * q.un;
        double const gm = gd + gn * q.un + gt1 * q.t1 + gt2 * q.t2;
        double const gE = ge * q.un;
        double const gEd = gE * q.r;
        bq.un = gn * m + ge * (q.e + q.p) + gm * q.r + gE * m;
        bq.r = gm * q.un + gE * q.ke;
        bq.p = gn + gE + gE * inv_gm1;
        bq.t1 = gt1 * m + gEd * q.t1;
        bq.t2 = gt2 * m + gEd * q.t2;
        bL.r = left ? bq.r : 0.0;
        bL.p = left ? bq.p : 0.0;
        bL.un = left ? bq.un : 0.0;
        bL.t1 = left ? bq.t1 : 0.0;
        bL.t2 = left ? bq.t2 : 0.0;
        bR.r = left ? 0.0 : bq.r;
        bR.p = left ? 0.0 : bq.p;
        bR.un = left ? 0.0 : bq.un;
        bR.t1 = left ? 0.0 : bq.t1;
        bR.t2 = left ? 0.0 : bq.t2;
        return;
    }

    double iG, ustar, gus, ga;
    if (tie) {
        // ustar == 0: the mean of the two branches, each taking half of the
        // cotangent.  b and the mass flux vanish, so each side adds only its
        // b's derivative; the pressure term p + a d w (q's) is as elsewhere.
        // One reciprocal gives 1/G, 1/S_L and 1/S_R.
        double const SL = L.un - A;
        double const SR = R.un + A;
        double const P = SL * SR;
        double const Rr = adj_rcp(G * P);
        iG = P * Rr;
        ustar = 0.0;
        double const hd = adj_half(gd), he = adj_half(ge), ht1 = adj_half(gt1), ht2 = adj_half(gt2);
        double const gw = q.r * (gn * a);
        gus = tie_side_bar(L, -A, SL, (G * SR) * Rr, hd, he, ht1, ht2) +
              tie_side_bar(R, A, SR, (G * SL) * Rr, hd, he, ht1, ht2) + gw;
        ga = -gn * (q.r * q.un);
        bq.r = -(gn * a) * q.un;
        bq.p = gn;
        bq.un = -gw;
        bq.t1 = 0.0;
        bq.t2 = 0.0;
    } else {
        double const M = S * G - n; // G (S - ustar)
        double const Rr = adj_rcp(adj_mul(G, M));
        double const nR = adj_mul(n, Rr);
        iG = adj_mul(M, Rr);
        ustar = adj_mul(nR, M);
        double const iu = adj_mul(nR, G);              // ustar/(S - ustar)
        double const y = adj_mul(G, adj_mul(G, Rr));   // 1/(S - ustar)
        double const b = adj_mul(a, iu);
        double const w = ustar - q.un;
        double const dw = adj_mul(q.r, w);
        double const m = adj_mul(q.r, b);
        double const E = S * dw + (q.e + q.p);
        double const gm = gd + gn * ustar + gt1 * q.t1 + gt2 * q.t2; // d/d (d b)
        double const gb = gm * q.r + ge * E;                         // d/d b
        double const gE = adj_mul(ge, b);                            // d/d E
        double const K = gE * S + gn * a;                            // d/d (d w)
        double const gw = adj_mul(q.r, K);
        double const gby = adj_mul(gb, y);
        double const gS = gE * dw - gby * b; // db/dS = -b y
        ga = gn * dw + gb * iu + gS;         // S = un + a
        gus = gn * m + gw + gby * (a + b);   // db/dustar = (a + b) y
        double const gEd = adj_mul(gE, q.r);
        bq.r = gm * b + K * w + gE * q.ke;
        bq.p = gn + gE + gE * inv_gm1;
        bq.un = gS - gw + gEd * q.un;
        bq.t1 = gt1 * m + gEd * q.t1;
        bq.t2 = gt2 * m + gEd * q.t2;
    }

    // to the upwind side
    bL.r = left ? bq.r : 0.0;
    bL.p = left ? bq.p : 0.0;
    bL.un = left ? bq.un : 0.0;
    bL.t1 = left ? bq.t1 : 0.0;
    bL.t2 = left ? bq.t2 : 0.0;
    bR.r = left ? 0.0 : bq.r;
    bR.p = left ? 0.0 : bq.p;
    bR.un = left ? 0.0 : bq.un;
    bR.t1 = left ? 0.0 : bq.t1;
    bR.t2 = left ? 0.0 : bq.t2;
    // ustar = n / G
    double const gN = adj_mul(gus, iG);
    double const gG = adj_mul(-gN, ustar);
    bL.p += gN;
    bR.p -= gN;
    // n's momentum sum and G's density sum
    double const gmom = adj_mul(gN, A);
    double const gD = adj_mul(gG, A);
    bL.r += gmom * L.un + gD;
    bR.r += gmom * R.un + gD;
    bL.un += gmom * L.r;
    bR.un += gmom * R.r;
    double const gA = gN * mom + gG * D + (left ? -ga : ga);
    // A = cmax + max(u_L - u_R, 0) (equal: half to each side)
    double const half_gA = adj_half(gA);
    double const gdu = u_gt ? gA : (u_lt ? 0.0 : half_gA);
    bL.un += gdu;
    bR.un -= gdu;
    double const gcL = c_lt ? 0.0 : (c_gt ? gA : half_gA);
    double const gcR = gA - gcL;
    bL.p += gcL * L.cp;
    bL.r += gcL * L.cr;
    bR.p += gcR * R.cp;
    bR.r += gcR * R.cr;
}

} // namespace eulr
