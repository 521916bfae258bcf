// Device-side building blocks shared by the Euler kernels (sm_103a).
//
// Two arithmetic styles are used:
//  * "exact" helpers (mul_rn, add_rn, ...) issue one IEEE-rounded operation
//    each and never contract into FMA.  The pointwise operators use them so
//    that their results are bit-identical to the reference operators, which
//    are written as separately rounded products and sums.
//  * plain C++ arithmetic, which nvcc contracts into FMAs.  The flux kernels
//    use it: every face is solved once instead of twice, shared reciprocals
//    replace divisions, and the results agree with the reference to a few
//    units in the last place per step.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "halve.cuh"

namespace eulr {

template <class T>
struct Bundle {
    T* f[5];
};

template <class T>
struct CBundle {
    const T* f[5];
};

// Grid extents and strides of a layout_left block (i fastest).
struct Geom {
    int n0, n1, n2;
    long long s1; // n0
    long long s2; // n0 * n1
    __host__ __device__ long long ncell() const { return s2 * n2; }
    __host__ __device__ long long at(int i, int j, int k) const { return i + s1 * j + s2 * k; }
};

inline Geom make_geom(int n0, int n1, int n2)
{
    Geom g;
    g.n0 = n0;
    g.n1 = n1;
    g.n2 = n2;
    g.s1 = n0;
    g.s2 = static_cast<long long>(n0) * n1;
    return g;
}

// ------------------------------------------------ separately rounded ops
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double sub_rn(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float sub_rn(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ double fma_rn(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float fma_rn(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rcp_rn(double a) { return __drcp_rn(a); }
__device__ __forceinline__ float rcp_rn(float a) { return __frcp_rn(a); }
__device__ __forceinline__ double div_rn(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float div_rn(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double sqrt_rn(double a) { return __dsqrt_rn(a); }
__device__ __forceinline__ float sqrt_rn(float a) { return __fsqrt_rn(a); }
__device__ __forceinline__ double abs_(double a) { return fabs(a); }
// x * 0.5 with the bits of a DMUL by 0.5, on the integer pipe (halve.cuh);
// the asm move keeps the compiler from turning the bit arithmetic back into
// an FP64 multiply.
__device__ __forceinline__ double half_exact(double x)
{
    unsigned long long b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
    return __longlong_as_double(static_cast<long long>(halve_bits(b)));
}
__device__ __forceinline__ float half_exact(float x) { return __fmul_rn(x, 0.5f); }
__device__ __forceinline__ float abs_(float a) { return fabsf(a); }

// Faithful FP64 reciprocal and square root (within one ulp of the correctly
// rounded result, not always equal to it) for kernels whose parity bar is a
// relative tolerance: for the operands that rcp_alu and sqrt_alu below leave to
// the FP64 unit, and the adjoint's cell conversion.  Each refines the PTX hardware approximation
// (rcp.approx.ftz.f64, rsqrt.approx.ftz.f64; both measured at most 2^-19.9
// relative error on sm_103a) by one Newton-Raphson step carried to third
// order, from the series 1/(1-e) = 1 + e + e^2 + ... and
// 1/sqrt(1-e) = 1 + e/2 + 3e^2/8 + ...:
//   1/x:      r0 ~ 1/x,       e = 1 - x r0,       1/x     ~ r0 (1 + e + e^2)
//   sqrt(x):  y0 ~ 1/sqrt(x), t = x y0, e = 1 - t y0, sqrt(x) ~ t (1 + e/2 + 3e^2/8)
// The truncation error is O(e^3) <= 2^-59, so the result is within one ulp
// of the correctly rounded value (measured: at most 1 ulp over 4M arguments
// spanning 2^+-100); three (five) FP64 instructions in place of the
// correctly rounded sequences.  Zero, infinite and subnormal
// arguments give NaN or zero instead of the IEEE results (the approximations
// flush subnormals): physical Euler states never reach them, and a
// non-physical state is reported as non-finite either way.
__device__ __forceinline__ double rcp_faithful(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    double e = __fma_rn(-x, r, 1.0);
    e = __fma_rn(e, e, e);
    return __fma_rn(r, e, r);
}

__device__ __forceinline__ double sqrt_faithful(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double const t = x * y;
    double const e = __fma_rn(-t, y, 1.0);
    double const q = __fma_rn(0.375, e, 0.5);
    return __fma_rn(t, e * q, t);
}

// The hardware's FP32 approximations themselves (one MUFU instruction each,
// relative error below 2^-22): the FP32 steps' error is set by the state's
// own rounding.  Inputs are normal positive numbers there; ftz maps a
// subnormal input to zero (1/x = +inf) and a result below 2^-126 to zero,
// which no physical state reaches.
__device__ __forceinline__ float rcp_approx(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rsqrt_approx(float x)
{
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// sqrt(x / d) for x, d > 0 without a reciprocal: x * rsqrt(x d), the PTX
// approximation of 1/sqrt refined by the third-order step of sqrt_faithful
// (y (1 + e/2 + 3e^2/8), e = 1 - z y^2).  Seven FP64 instructions and one
// seed where rcp_faithful + sqrt_faithful take ten and two; within two ulps
// of the correctly rounded sqrt(x/d) (checked against it on 4M argument
// pairs).  (Sound speeds are formed by sqrt_alu and rcp_alu now; only its test
// uses this one.)
__device__ __forceinline__ double sqrt_quotient_faithful(double x, double d)
{
    double const z = x * d;
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(z));
    double const e = __fma_rn(-(z * y), y, 1.0);
    double const q = __fma_rn(0.375, e, 0.5);
    return x * __fma_rn(y, e * q, y);
}

// Non-negative values ordered as their bit patterns; NaN maps to 0 so that it
// never wins a max (the reference's Kokkos::min over 1/invdt skips NaN).
__device__ __forceinline__ unsigned long long order_bits(double v)
{
    return (v >= 0.0) ? static_cast<unsigned long long>(__double_as_longlong(v)) : 0ull;
}
__device__ __forceinline__ unsigned long long order_bits(float v)
{
    return order_bits(static_cast<double>(v));
}

template <class T>
__device__ __forceinline__ T warp_max(T v)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        T const w = __shfl_xor_sync(0xffffffffu, v, o);
        v = (w > v) ? w : v;
    }
    return v;
}

// ------------------------------------------------- integer-pipe predicates
// On GB300 an FP64 compare, min or max takes a full slot of the FP64 pipe
// (1/64 of the FP32 rate); the same decisions taken on the bit patterns run
// on the integer pipe, which the flux kernels leave almost idle.
// The bit pattern through an opaque move: tests written on the bits must stay
// on the integer pipe.  With a plain reinterpretation the compiler rewrote
// (bits << 1) != 0 into the equivalent FP64 compare x != 0, which takes an
// FP64 slot (four per HLLC face: 12.6 FP64 instructions per cell of the step).
__device__ __forceinline__ long long dbits(double x)
{
    long long b;
    asm("mov.b64 %0, %1;" : "=l"(b) : "d"(x));
    return b;
}

// x is neither +0 nor -0.
__device__ __forceinline__ bool nonzero_(double x) { return (dbits(x) << 1) != 0; }

// a*b > 0 for non-NaN a, b, decided from signs: both non-zero and of one sign.
// (Only its test uses it: hllc_upwind needs the sign of one number.)
__device__ __forceinline__ bool product_positive(double a, double b)
{
    return nonzero_(a) && nonzero_(b) && ((dbits(a) ^ dbits(b)) >= 0);
}

// a < b with IEEE semantics (false when either is NaN; -0 and +0 equal),
// decided on the integer pipe: the bit patterns mapped to ordered keys with
// both zeros at 0.  The same answer as the FP64 compare, which would take an
// FP64 slot.
__device__ __forceinline__ bool is_nan_bits(long long b) { return (b & 0x7fffffffffffffffLL) > 0x7ff0000000000000LL; }
__device__ __forceinline__ bool less_ieee(double a, double b)
{
    long long const x = dbits(a), y = dbits(b);
    long long const kx = (x << 1) == 0 ? 0 : (x ^ ((x >> 63) & 0x7fffffffffffffffLL));
    long long const ky = (y << 1) == 0 ? 0 : (y ^ ((y >> 63) & 0x7fffffffffffffffLL));
    return !is_nan_bits(x) && !is_nan_bits(y) && kx < ky;
}
__device__ __forceinline__ bool less_ieee(float a, float b) { return a < b; }

// ------------------------------------------- FP64 work on the integer pipes
// The FP64 unit's product, for the operands mul_alu does not take, zeros aside.
// Out of line: inlined, it was predicated instead of branched around, and a
// predicated-off FP64 instruction takes its slot of the pipe all the same.
static __device__ __noinline__ double mul_rare(double a, double b)
{
    long long const ab = dbits(a), bb = dbits(b);
    long long const inf = 0x7ff0000000000000LL;
    if ((ab & inf) != inf && (bb & inf) != inf && ((ab << 1) == 0 || (bb << 1) == 0)) {
        return __longlong_as_double((ab ^ bb) & static_cast<long long>(0x8000000000000000ull));
    }
    return mul_rn(a, b);
}

// a*b on the integer pipes: the 53 x 53-bit product of the significands in
// four 32-bit multiplies, rounded to nearest.  A tie goes to the even
// neighbour (EVEN: the bits of the FP64 multiply, for the kernels that owe
// the reference's bits) or away from zero (the same error bound for three
// instructions less: 3.5 % of a 512^3 step).  FP64 kernels leave 85 % of the
// issue slots idle while the FP64 pipe is full, and one FP64 instruction
// holds that pipe as long as about 60 issue slots last; this takes about 30.
// A step of 512^3 went from 31.2 ms to 27.4 with 22 of 127 FP64 instructions a
// cell replaced by it, to 24.2 with rcp_alu and ten more products, to 23.9
// with sqrt_alu and add_alu, and to 20.6 with the FP64 unit's forms out of
// line.
// Operands with a magnitude outside [2^-255, 2^257) take the FP64 multiply,
// except zeros.
template <bool EVEN>
__device__ __forceinline__ double mul_int(double a, double b)
{
    long long const ab = dbits(a), bb = dbits(b);
    unsigned const a0 = static_cast<unsigned>(ab), a1 = static_cast<unsigned>(ab >> 32);
    unsigned const b0 = static_cast<unsigned>(bb), b1 = static_cast<unsigned>(bb >> 32);
    if (((2u * a1 - 0x60000000u) | (2u * b1 - 0x60000000u)) >= 0x40000000u) {
        return mul_rare(a, b);
    }
    unsigned const am = (a1 & 0xfffffu) | 0x100000u, bm = (b1 & 0xfffffu) | 0x100000u;
    unsigned long long const t = static_cast<unsigned long long>(a0) * b0;
    unsigned long long const u = static_cast<unsigned long long>(a0) * bm + (t >> 32);
    unsigned long long const v = static_cast<unsigned long long>(am) * b0 + static_cast<unsigned>(u);
    unsigned long long w = static_cast<unsigned long long>(am) * bm + (u >> 32) + (v >> 32);
    // the product w : low word of v : low word of t has 106 bits (c = 1) or 105
    unsigned const c = static_cast<unsigned>(w >> 41);
    unsigned const x = static_cast<unsigned>(v);
    unsigned const y = x + (0x80000u << c);
    w += y < x ? 1u : 0u;
    unsigned lo = __funnelshift_r(y, static_cast<unsigned>(w), 20u + c);
    if (EVEN) {
        bool const tie = (x << (12u - c)) == 0x80000000u && static_cast<unsigned>(t) == 0u;
        lo &= tie ? ~1u : ~0u;
    }
    unsigned const hi = __funnelshift_r(static_cast<unsigned>(w), static_cast<unsigned>(w >> 32), 20u + c) +
                        (a1 & 0xfff00000u) + (b1 & 0xfff00000u) - 0x40000000u + (c << 20);
    return __hiloint2double(static_cast<int>(hi), static_cast<int>(lo));
}

static __device__ __noinline__ double rcp_rare(double x) { return rcp_faithful(x); }
static __device__ __noinline__ double rcp_rn_rare(double x) { return rcp_rn(x); }
static __device__ __noinline__ double sqrt_rare(double x) { return sqrt_faithful(x); }
static __device__ __noinline__ double add_rare(double a, double b) { return add_rn(a, b); }

// 2^53 / f, f the significand of x in [1, 2), rounded to nearest but for an
// error of up to 0.5001 units: an FP32 seed q of 1/f, its error E = 1 - f q
// exactly in 64-bit fixed point, and q (1 + E + E^2), for a seed within two
// FP32 ulps.
__device__ __forceinline__ unsigned long long rcp_significand(unsigned x0, unsigned x1)
{
    // f to 24 bits; q / 2^24 in [1/2, 1)
    unsigned const f24 = (((__funnelshift_l(x0, x1, 4) & 0xffffffu) + 1u) >> 1) + 0x3f800000u;
    unsigned const seed = min(max(__float_as_uint(rcp_approx(__uint_as_float(f24))), 0x3f000000u), 0x3f7fffffu);
    unsigned const q = (seed & 0x7fffffu) | 0x800000u;
    // E in units of 2^-76, from f q modulo 2^64
    unsigned long long const t = static_cast<unsigned long long>(x0) * q;
    unsigned const u = ((x1 & 0xfffffu) | 0x100000u) * q + static_cast<unsigned>(t >> 32);
    long long const e = -static_cast<long long>((static_cast<unsigned long long>(u) << 32) | static_cast<unsigned>(t));
    int const eh = static_cast<int>(e >> 24);
    long long const e2 = e + ((static_cast<long long>(eh) * eh) >> 28);
    // q (1 + E + E^2) in units of 2^-53
    unsigned long long const p = static_cast<unsigned long long>(q) * static_cast<unsigned>(e2);
    long long const c = static_cast<long long>(static_cast<int>(q)) * static_cast<int>(e2 >> 32) + static_cast<long long>(p >> 32);
    return (static_cast<unsigned long long>(q) << 29) + static_cast<unsigned long long>((c + 0x4000) >> 15);
}

// g 2^-53 / 2^n for x = f 2^n, with the sign of x.
__device__ __forceinline__ double rcp_pack(unsigned long long g, unsigned x1)
{
    unsigned const hi = static_cast<unsigned>(g >> 32) + 0x7fc00000u - (x1 & 0xfff00000u);
    return __hiloint2double(static_cast<int>(hi), static_cast<int>(static_cast<unsigned>(g)));
}

// 1/x on the integer pipes, within 0.5001 ulp.  Magnitudes outside
// [2^-255, 2^257) take rcp_faithful.
__device__ __forceinline__ double rcp_alu(double x)
{
    long long const xb = dbits(x);
    unsigned const x0 = static_cast<unsigned>(xb), x1 = static_cast<unsigned>(xb >> 32);
    if (2u * x1 - 0x60000000u >= 0x40000000u) {
        return rcp_rare(x);
    }
    return rcp_pack(rcp_significand(x0, x1), x1);
}

// 1/x correctly rounded, on the integer pipes: the remainder 2^105 - f 2^52 g
// is exact modulo 2^64, and g moves by one where it exceeds half of f 2^52
// (equality cannot occur).
__device__ __forceinline__ double rcp_rn_alu(double x)
{
    long long const xb = dbits(x);
    unsigned const x0 = static_cast<unsigned>(xb), x1 = static_cast<unsigned>(xb >> 32);
    if (2u * x1 - 0x60000000u >= 0x40000000u) {
        return rcp_rn_rare(x);
    }
    unsigned long long const m = (static_cast<unsigned long long>((x1 & 0xfffffu) | 0x100000u) << 32) | x0;
    unsigned long long g = rcp_significand(x0, x1);
    long long const rem2 = -static_cast<long long>((m * g) << 1);
    if (rem2 > static_cast<long long>(m)) {
        ++g;
    } else if (rem2 < -static_cast<long long>(m)) {
        --g;
    }
    return rcp_pack(g, x1);
}

// sqrt(x) on the integer pipes: s = f y from an FP32 seed y of 1/sqrt(f), cut
// to 32 bits, the exact residual R = f - s^2 in 64-bit fixed point and
// s + R y/2 (1 + (3/2 d - cut) y), d = R y/2: within 0.52 ulp for a seed
// within two FP32 ulps.  Magnitudes outside [2^-255, 2^257), zeros and
// negative values take sqrt_faithful.
__device__ __forceinline__ double sqrt_alu(double x)
{
    long long const xb = dbits(x);
    unsigned const x0 = static_cast<unsigned>(xb), x1 = static_cast<unsigned>(xb >> 32);
    if (x1 - 0x30000000u >= 0x20000000u) {
        return sqrt_rare(x);
    }
    // x = f 4^n with f in [1, 4), m = f 2^52; q / 2^24 in [1/2, 1)
    unsigned const odd = (~x1 >> 20) & 1u;
    unsigned long long const m = ((static_cast<unsigned long long>((x1 & 0xfffffu) | 0x100000u) << 32) | x0) << odd;
    unsigned const f24 = (((__funnelshift_l(x0, x1, 4) & 0xffffffu) + 1u) >> 1) + 0x3f800000u + (odd << 23);
    unsigned const seed = min(max(__float_as_uint(rsqrt_approx(__uint_as_float(f24))), 0x3f000000u), 0x3f7fffffu);
    unsigned const q = (seed & 0x7fffffu) | 0x800000u;
    unsigned long long const t = static_cast<unsigned long long>(static_cast<unsigned>(m)) * q;
    unsigned long long const s = static_cast<unsigned long long>(static_cast<unsigned>(m >> 32)) * q + (t >> 32); // 2^-44
    unsigned const sh = (s >> 45) != 0 ? 0xffffffffu : static_cast<unsigned>(s >> 13);                            // 2^-31
    long long const res = static_cast<long long>((m << 10) - static_cast<unsigned long long>(sh) * sh);           // 2^-62
    long long const d = (res >> 5) * static_cast<long long>(q);                                                   // 2^-82
    int const dh = static_cast<int>(d >> 32);                                                                     // 2^-50
    int const cut = static_cast<int>((static_cast<unsigned>(s) - (sh << 13)) << 6);                               // 2^-50
    int const z = static_cast<int>((static_cast<long long>(dh) * (dh + (dh >> 1) - cut)) >> 40);                  // 2^-60
    long long const z2 = static_cast<long long>(z) * static_cast<int>(q);                                         // 2^-84
    unsigned long long const g = ((static_cast<unsigned long long>(sh) << 31) + static_cast<unsigned long long>(d >> 20) +
                                  static_cast<unsigned long long>(z2 >> 22) + 512u) >> 10;                        // 2^-52
    unsigned const hi = static_cast<unsigned>(g >> 32) + (((x1 >> 1) + 0x1ff80000u - (odd << 19)) & 0xfff00000u) - 0x100000u;
    return __hiloint2double(static_cast<int>(hi), static_cast<int>(static_cast<unsigned>(g)));
}

// a + b on the integer pipes for a, b >= 0, rounded to nearest even as the
// FP64 add.  Exponents 32 or more apart, and operands or sums out of the
// normal range, take the FP64 add.
__device__ __forceinline__ double add_alu(double a, double b)
{
    unsigned long long const x = static_cast<unsigned long long>(dbits(a)), y = static_cast<unsigned long long>(dbits(b));
    unsigned long long const g = x > y ? x : y, l = x > y ? y : x;
    unsigned const g1 = static_cast<unsigned>(g >> 32), l1 = static_cast<unsigned>(l >> 32), l0 = static_cast<unsigned>(l);
    unsigned const d = (g1 >> 20) - (l1 >> 20);
    if (d >= 32u || g1 >= 0x7fe00000u || l1 < 0x00100000u) {
        return add_rare(a, b);
    }
    unsigned const lm = (l1 & 0xfffffu) | 0x100000u;
    unsigned const rest = __funnelshift_r(0u, l0, d); // what the alignment shifts out
    unsigned long long t = (g & 0xfffffffffffffull) + 0x10000000000000ull +
                           ((static_cast<unsigned long long>(lm >> d) << 32) | __funnelshift_r(l0, lm, d));
    unsigned const c = static_cast<unsigned>(t >> 53);
    bool const tie = c != 0 ? (rest == 0u && (t & 1u) != 0) : rest == 0x80000000u;
    t += c != 0 ? 1u : rest >> 31;
    t >>= c;
    t -= tie ? (t & 1u) : 0u;
    return __longlong_as_double(static_cast<long long>(t + (static_cast<unsigned long long>((g1 >> 20) - 1u + c) << 52)));
}

__device__ __forceinline__ double mul_alu(double a, double b) { return mul_int<false>(a, b); }
__device__ __forceinline__ double mul_rn_alu(double a, double b) { return mul_int<true>(a, b); }

// The same names for the kernels that are templates of the type.
__device__ __forceinline__ float mul_rn_alu(float a, float b) { return mul_rn(a, b); }
__device__ __forceinline__ float rcp_rn_alu(float x) { return rcp_rn(x); }

// Correctly rounded x / y given r = RN(1/y): q0 = RN(x r) is within one ulp
// of x/y, the remainder x - q0 y is exact through one FMA, and
// RN(q0 + rem r) is the correctly rounded quotient (Markstein's correction
// step; P. Markstein, "Computation of elementary functions on the IBM RISC
// System/6000 processor", IBM J. Res. Dev. 34(1), 1990).  Valid away from
// overflow and underflow, which the Euler states here never approach.
template <class T>
__device__ __forceinline__ T div_by_rcp(T x, T y, T r)
{
    T const q0 = mul_rn_alu(x, r);
    T const rem = fma_rn(-q0, y, x);
    return fma_rn(rem, r, q0);
}

// cons_to_prim of one cell, bit-identical to cons_to_prim.hpp:20-32 with
// kinetic_energy(cons) (euler_arrays.hpp:44-48), PerfectGas::pressure
// (perfect_gas.hpp:25-28) and to_prim (euler_arrays.hpp:66-75):
//   ke = ((m.m)/d)/2, p = (gamma-1)*(e-ke), u_i = m_i * (1/d).
// Both quotients come from one reciprocal of d (div_by_rcp).
template <class T>
__device__ __forceinline__ void cons_to_prim_exact(T d, T e, T m0, T m1, T m2, T gm1, T& p, T& u0, T& u1, T& u2)
{
    T const r = rcp_rn_alu(d);
    T const mm = add_rn(add_rn(mul_rn_alu(m0, m0), mul_rn_alu(m1, m1)), mul_rn_alu(m2, m2));
    T const ke = half_exact(div_by_rcp(mm, d, r));
    p = mul_rn_alu(gm1, sub_rn(e, ke));
    u0 = mul_rn_alu(m0, r);
    u1 = mul_rn_alu(m1, r);
    u2 = mul_rn_alu(m2, r);
}

// (c + |u0|)/dx0 + (c + |u1|)/dx1 + (c + |u2|)/dx2 of one cell with
// c = sqrt((gamma p)/d), bit-identical to time_step.hpp:28-33 and
// perfect_gas.hpp:15-18 (ix_d = 1/dx_d computed by the caller in T).
template <class T>
__device__ __forceinline__ T cell_invdt_exact(T d, T p, T u0, T u1, T u2, T gamma, T ix0, T ix1, T ix2)
{
    T const cs = sqrt_rn(div_rn(mul_rn(gamma, p), d));
    T const c0 = add_rn(cs, abs_(u0));
    T const c1 = add_rn(cs, abs_(u1));
    T const c2 = add_rn(cs, abs_(u2));
    return add_rn(add_rn(mul_rn(c0, ix0), mul_rn(c1, ix1)), mul_rn(c2, ix2));
}

// ------------------------------------------- FP32 cons_to_prim with FP64 rescue
// Below this fraction of e the FP32 internal-energy subtraction
// e - |m|^2/(2 rho) has lost more than 8 of its 24 bits.
constexpr float kLowPressure = 1.0f / 256.0f;

// The FP64 internal energy of a low-pressure cell, (gamma-1) (e - |m|^2/(2 rho))
// from the FP32 words (hi, plus the low words when the state stores them).
// 1/rho is the FP32 reciprocal r refined by one Newton step in FP64
// (relative error about 2^-44): no FP64 division routine.  Out of line: the
// path is rare, and inlined its FP64 registers weigh on every cell's code.
static __device__ __noinline__ float pressure_f64_rescue(float d, float e, float m0, float m1, float m2, float r, float gm1,
                                                  const float* lo)
{
    double const dd = static_cast<double>(d) + (lo ? static_cast<double>(lo[0]) : 0.0);
    double const ed = static_cast<double>(e) + (lo ? static_cast<double>(lo[1]) : 0.0);
    double const a0 = static_cast<double>(m0) + (lo ? static_cast<double>(lo[2]) : 0.0);
    double const a1 = static_cast<double>(m1) + (lo ? static_cast<double>(lo[3]) : 0.0);
    double const a2 = static_cast<double>(m2) + (lo ? static_cast<double>(lo[4]) : 0.0);
    double rd = static_cast<double>(r);
    rd = rd * __fma_rn(-dd, rd, 2.0);
    double const ke = 0.5 * (a0 * a0 + a1 * a1 + a2 * a2) * rd;
    return static_cast<float>(static_cast<double>(gm1) * (ed - ke));
}

// Pressure of an FP32 conservative state: the subtraction runs in FP32
// unless the cell's internal energy is below kLowPressure of its total
// energy, where it is redone in FP64 (pressure_f64_rescue).
__device__ __forceinline__ float pressure_f32c(float d, float e, float m0, float m1, float m2, float r, float gm1,
                                               const float* lo)
{
    float const mm = m0 * m0 + m1 * m1 + m2 * m2;
    float const eint = e - (0.5f * r) * mm;
    if (eint > kLowPressure * e) {
        return gm1 * eint;
    }
    return pressure_f64_rescue(d, e, m0, m1, m2, r, gm1, lo);
}

// invdt of one cell of a cons-only FP32 state, with the pressure the fused
// FP32 step uses (compensated states rescue low-pressure cells in FP64).
__device__ __forceinline__ float cons_invdt_f32(float d, float e, float m0, float m1, float m2, float gamma, float gm1,
                                                float ix0, float ix1, float ix2, bool compensated)
{
    float const r = 1.0f / d;
    float const pr = compensated ? pressure_f32c(d, e, m0, m1, m2, r, gm1, nullptr)
                                 : gm1 * (e - (0.5f * r) * (m0 * m0 + m1 * m1 + m2 * m2));
    return cell_invdt_exact(d, pr, m0 * r, m1 * r, m2 * r, gamma, ix0, ix1, ix2);
}

// ------------------------------------------------------------------ HLLC
// One side of a face in the face's frame: normal velocity un, tangential
// velocities ut1/ut2 (in the cyclic order of the axes after the normal), sound
// speed c and, in `e`, the sum e + p of total energy density and pressure:
// the HLLC needs only that sum, which the staging forms once per cell.
template <class T>
struct Side {
    T d, p, un, ut1, ut2, c, e;
};

template <class T>
struct Flux {
    T d, e, n, t1, t2;
};

// One side of a face of the FP64 kernels: what decides the face's flux, with
// the normal momentum mn = d un and h = e + p; the tangential momenta are
// read where the flux is used.
struct StagedSide {
    double d, p, un, mn, c, h;
};

// Finite and > 0.
__device__ __forceinline__ bool finite_positive(double x)
{
    long long const b = dbits(x);
    return b > 0 && b < 0x7ff0000000000000LL;
}

// HLLC flux of hllc::operator() (euler_operators/hllc.hpp:50-105) in the face
// frame: wave speeds (:64-68), acoustic star state (:70-76), upwind side by
// the sign of ustar (:78-79), supersonic test S_L*S_R > 0 (:84-85), star
// density and energy (:86-88) and the flux (:90-102).  Reformulated to spend
// as few FP64 instructions as possible; in exact arithmetic it is the same
// function:
//  * one acoustic speed.  S_L = min(u) - cmax and S_R = max(u) + cmax give
//    S_L - u_L = -A and S_R - u_R = A with the same
//    A = cmax + max(u_L - u_R, 0), so with D = d_L + d_R, G = A D and the
//    momenta m = d u
//      ustar = n / G,  n = A (m_L + m_R) - (p_R - p_L),
//    and only the upwind side's wave speed S = u -+ A is formed: the face is
//    supersonic exactly when S has the sign of ustar.
//  * ustar and 1/(S - ustar) = G/M, M = S G - n, come from ONE reciprocal
//    R = 1/(G M): ustar = (n R) M, and ustar/(S - ustar) = (n R) G, which is
//    all the flux needs of 1/(S - ustar).  The side (sign of ustar) is the
//    sign of n, read before any division.
//  * pstar: the reference averages p_L + rc_L (ustar-u_L) and
//    p_R + rc_R (ustar-u_R), which are equal by the definition of ustar; the
//    upwind one is used.
//  * with a = S - u = -+A, w = ustar - u and b = a ustar/(S - ustar) the
//    flux is
//      mass                d_star ustar    = b d,
//      tangential momentum mass u_t        = b m_t,
//      energy  (e_star + pstar) ustar      = b ((e + p) + S d w),
//      normal momentum                     = b d ustar + p + a d w,
//    because e_star + pstar = [a e + pstar ustar - p u + pstar (S - ustar)]/(S - ustar)
//                           = [a (e + p) + S (pstar - p)]/(S - ustar)
//    and pstar - p = a d w, with d w = d ustar - m.
//  * in the supersonic case the reference's ratio (S-u)/(S-u) is exactly 1
//    and its energy correction exactly 0: ustar := u and b := u (so w = 0)
//    give the upwind state's own flux with two selects.
//  * max and the sign tests run on the integer pipe, on the bit patterns.
// So four of the five fluxes are b times a value of the upwind side, and the
// FP64 kernels never form them: the face keeps b, h = (e + p) + S d w and the
// normal momentum's flux, the side is the sign of b, and each cell adds b d,
// b m_t and b h to its update with one fma each.
// Every sum of products is written as the fma it becomes, so that all kernels
// that inline this give a face the same bits whatever the compiler contracts.
// 22 FP64 operations and a reciprocal seed a face, against 27 and a seed with
// all five fluxes formed from velocities; the seven products, the
// reciprocal and the sum of the densities run on the integer pipes (mul_alu,
// rcp_alu, add_alu), which leaves 11.  (A's sum there too measured 4 % slower
// in the operator godunov and 1-2 % faster in the batch.)
struct UpwindFlux {
    double b;  // carries d, m_t and h of its upwind side: the left one where b > 0
    double h;  // e + p of that side plus S d w
    double fn; // flux of the normal momentum
};

__device__ __forceinline__ UpwindFlux hllc_upwind(StagedSide const& L, StagedSide const& R)
{
    double const cmax = (dbits(L.c) > dbits(R.c)) ? L.c : R.c; // sound speeds are >= 0
    double const du = L.un - R.un;
    double const A = cmax + (dbits(du) < 0 ? 0.0 : du);
    double const G = mul_alu(A, add_alu(L.d, R.d));
    double const n = fma_rn(A, L.mn + R.mn, sub_rn(L.p, R.p));

    bool const left = dbits(n) > 0; // ustar > 0 (G > 0)
    double const qd = left ? L.d : R.d;
    double const qp = left ? L.p : R.p;
    double const qun = left ? L.un : R.un;
    double const qmn = left ? L.mn : R.mn;
    double const qh = left ? L.h : R.h;
    // a = -A on the left, A on the right: the sign bit, on the integer pipe
    double const a = __longlong_as_double(dbits(A) ^ (left ? static_cast<long long>(0x8000000000000000ull) : 0LL));

    double const S = qun + a;
    double const M = fma_rn(S, G, -n); // G (S - ustar)
    double const nR = mul_alu(n, rcp_alu(mul_alu(G, M)));
    // S = -0 cannot occur (a is not zero), so the sign bit decides
    bool const supersonic = left ? dbits(S) > 0 : dbits(S) < 0;
    double const ustar = supersonic ? qun : mul_alu(nR, M);
    double const dus = mul_alu(qd, ustar);
    double const dw = fma_rn(qd, ustar, -qmn);

    UpwindFlux f;
    f.b = supersonic ? qun : mul_alu(a, mul_alu(nR, G));
    f.h = fma_rn(S, dw, qh);
    f.fn = fma_rn(f.b, dus, fma_rn(a, dw, qp));
    return f;
}

// FP32 version: the same algebra with all five fluxes formed, FP32 min/max and
// the hardware reciprocal.
__device__ __forceinline__ Flux<float> hllc_flux(Side<float> const& L, Side<float> const& R)
{
    float const A = fmaxf(L.c, R.c) + fmaxf(L.un - R.un, 0.0f);
    float const G = A * (L.d + R.d);
    float const n = fma_rn(A, fma_rn(L.d, L.un, mul_rn(R.d, R.un)), sub_rn(L.p, R.p));
    bool const left = n > 0.0f;
    float const qd = left ? L.d : R.d;
    float const qp = left ? L.p : R.p;
    float const qun = left ? L.un : R.un;
    float const qut1 = left ? L.ut1 : R.ut1;
    float const qut2 = left ? L.ut2 : R.ut2;
    float const qh = left ? L.e : R.e; // e + p of the upwind side
    float const a = left ? -A : A;
    float const S = qun + a;
    float const M = fma_rn(S, G, -n);
    float const nR = n * rcp_approx(G * M); // |G M| is far from the ends of the float range for any physical state
    bool const supersonic = left ? S > 0.0f : S < 0.0f;
    float const ustar = supersonic ? qun : nR * M;
    float const b = supersonic ? qun : a * (nR * G);
    float const dw = mul_rn(qd, sub_rn(ustar, qun));
    Flux<float> f;
    f.d = qd * b;
    f.e = b * fma_rn(S, dw, qh);
    f.n = fma_rn(f.d, ustar, fma_rn(a, dw, qp));
    f.t1 = f.d * qut1;
    f.t2 = f.d * qut2;
    return f;
}

} // namespace eulr
