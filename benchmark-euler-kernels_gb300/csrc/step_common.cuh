// Device helpers shared by the FP64 tile engine (flux.cu) and the FP32
// column engine (flux_f32.cu).  Internal to the library.
#pragma once

#include "euler_device.cuh"
#include "kernels.h"

#include <cfloat>

namespace eulr {
namespace {

constexpr int kFields = 10; // staged values of a cell: d, p, u0, u1, u2, c, e + p, m0, m1, m2
constexpr long long kInfBits = 0x7ff0000000000000LL;

// g / D for 0 <= g < 2^12 and a compile-time 0 < D < 256, as one product and
// a shift: floor(g (floor(2^20/D) + 1) / 2^20) exceeds g/D by less than
// g/2^20 < 2^-8, which stays below the gap 1/D to the next integer.  (The
// kernels use the run-time form below; this one only its test does.)
template <int D>
__device__ __forceinline__ int div_small(int g)
{
    static_assert(D > 0 && D < 256, "divisor range");
    constexpr unsigned kM = (1u << 20) / D + 1u;
    return static_cast<int>((static_cast<unsigned>(g) * kM) >> 20);
}

// The same with a divisor known at run time (an FP64 tile's extents are its
// grid's): the magic once per work item, a product and a shift per use.
__device__ __forceinline__ unsigned div_magic20(int d) { return (1u << 20) / static_cast<unsigned>(d) + 1u; }
__device__ __forceinline__ int div_runtime(int g, unsigned magic)
{
    return static_cast<int>((static_cast<unsigned>(g) * magic) >> 20);
}

__device__ __forceinline__ unsigned smem_u32(const void* p)
{
    return static_cast<unsigned>(__cvta_generic_to_shared(p));
}

// Pressure of an FP32 conservative state: compensated states rescue the
// low-pressure cells in FP64 (pressure_f32c), plain FP32 does not.
template <int COMP>
__device__ __forceinline__ float cons_pressure(float d, float e, float m0, float m1, float m2, float r, float gm1,
                                               const float* lo)
{
    if (COMP != kCompNone) {
        return pressure_f32c(d, e, m0, m1, m2, r, gm1, lo);
    }
    return gm1 * (e - (0.5f * r) * (m0 * m0 + m1 * m1 + m2 * m2));
}
template <int COMP>
__device__ __forceinline__ double cons_pressure(double, double, double, double, double, double, double, const double*)
{
    return 0.0; // FP64 states store prim: no caller reads this
}

// Sound speed sqrt(gamma p / rho), faithful: fewer FP64 instructions than a
// correctly rounded sqrt, within one ulp of it.
__device__ __forceinline__ double fast_sound_speed(double c2) { return sqrt_faithful(c2); }
__device__ __forceinline__ float fast_sound_speed(float c2) { return c2 * rsqrt_approx(c2); }

__device__ __forceinline__ long long wave_key(double v)
{
    long long const b = dbits(v);
    return b <= kInfBits ? b : 0LL; // NaN never wins (the reference skips it)
}
__device__ __forceinline__ long long wave_key(float v) { return wave_key(static_cast<double>(v)); }

__device__ __forceinline__ bool cell_ok(float d, float pr, float invdt)
{
    return d > 0.0f && pr > 0.0f && invdt <= 3.0e38f;
}

// dt/dv, from the device dt when there is one (godunov.hpp:37 with the
// cfl * dt of euler_simulation.cpp:65), evaluated in double.
template <class T>
__device__ __forceinline__ T dt_over_dv(FluxParams<T> const& p)
{
    if (p.dt_seq != nullptr) {
        return static_cast<T>(p.dt_seq[*p.step_dev] / p.dv);
    }
    if (p.dt_dev != nullptr) {
        return static_cast<T>((p.cfl * *p.dt_dev) / p.dv);
    }
    return p.dtodv;
}

// Turns the max-wavespeed accumulator into the next step's dt
// (time_step.hpp:34-39: min over cells of 1/invdt == 1/max invdt), adds the
// step just taken to the simulated time and clears the accumulator.  The
// accumulator is read with a volatile load: other CTAs of the same launch
// raised it by atomics, and a cached copy must not answer.
template <class T>
__device__ __forceinline__ void finalize_one(SimScalars* s, T cfl, int add_time, const double* dt_seq = nullptr,
                                             double* dt_log = nullptr)
{
    if (add_time) {
        // the step just taken, cfl*dt (or the fixed dt), added with separate
        // roundings (no FMA) so every kernel that inlines this agrees bit for bit
        double const step = dt_seq != nullptr ? dt_seq[s->steps]
                                              : (sizeof(T) == 8 ? __dmul_rn(static_cast<double>(cfl), s->dt)
                                                                : static_cast<double>(cfl * static_cast<T>(s->dt)));
        s->t = __dadd_rn(s->t, step);
        if (dt_log != nullptr) {
            dt_log[s->steps] = step;
        }
        s->steps += 1;
    }
    unsigned long long const w = *reinterpret_cast<volatile unsigned long long*>(&s->wmax);
    unsigned long long const wk = w > s->ghost_wmax ? w : s->ghost_wmax;
    T const m = static_cast<T>(__longlong_as_double(static_cast<long long>(wk)));
    T const dt = (m > T(0)) ? rcp_rn(m) : (sizeof(T) == 8 ? T(DBL_MAX) : T(FLT_MAX));
    s->dt = static_cast<double>(dt);
    s->wmax = 0ull;
}

// The step's own finalize, so that a step is one launch.  Called by thread 0
// of every CTA of a single-grid step launch after its wavespeed flush (the
// atomicMax precedes it in the same thread): the fence orders that flush
// before the count, and the CTA that counts last -- every other CTA has
// flushed and read this step's dt by then -- finalizes the step and rewinds
// the counter for the next launch.
template <class T>
__device__ __forceinline__ void step_done(FluxParams<T> const& p)
{
    if (p.fin == nullptr || threadIdx.x != 0) {
        return;
    }
    __threadfence();
    if (atomicAdd(&p.fin->done, 1u) == gridDim.x - 1) {
        __threadfence();
        finalize_one(p.fin, static_cast<T>(p.cfl), 1, p.dt_seq, p.dt_log);
        p.fin->done = 0u;
    }
}

// The same for one work item of a batch launch: the grid's last item to
// finish finalizes that grid (its items were all taken from the queue before,
// so no CTA reads the grid's dt afterwards in this launch).  Thread 0, after
// the item's flush.
template <class T>
__device__ __forceinline__ void item_done(FluxParams<T> const& gp)
{
    if (gp.fin == nullptr || threadIdx.x != 0) {
        return;
    }
    __threadfence();
    if (atomicAdd(&gp.fin->done, 1u) == static_cast<unsigned>(gp.grid_items) - 1u) {
        __threadfence();
        finalize_one(gp.fin, static_cast<T>(gp.cfl), 1, gp.dt_seq);
        gp.fin->done = 0u;
    }
}

// A batch CTA leaving (the queue is empty for it).  Thread 0.  The last CTA
// to leave rewinds the queue head for the next launch -- every CTA has made
// its last pop by then -- and finalizes the grids that have no work item.
template <class T>
__device__ __forceinline__ void batch_cta_done(BatchParams<T> const& b)
{
    if (b.exited == nullptr || threadIdx.x != 0) {
        return;
    }
    __threadfence();
    if (atomicAdd(b.exited, 1u) == gridDim.x - 1) {
        __threadfence();
        for (int i = 0; i < b.nidle; ++i) {
            FluxParams<T> const& g = b.grids[b.idle[i]];
            if (g.fin != nullptr) {
                finalize_one(g.fin, static_cast<T>(g.cfl), 1, g.dt_seq);
            }
        }
        *b.head = 0u;
        *b.exited = 0u;
    }
}

// ------------------------------------------ exact max wavespeed, screened
// The CFL step needs the max over cells of the reference's wavespeed
// (time_step.hpp:28-33; cell_invdt_exact: a correctly rounded FP64 division
// and square root per cell, about 25 FP64 issue slots), exactly.  But the
// exact value is needed only where it can be the max, so an FP32 estimate
// screens the cells, with no FP64 instruction at all: its inputs are built
// from the doubles' high words on the integer pipe (the mantissa truncated to
// 20 bits, a relative error in (-2^-20, 0]) and the rest runs on the FP32
// pipe.  Where rho, p and gamma p/rho lie in [1e-30, 1e30] and the estimate
// is at most 1e30, its relative error is below 2^-20 + 2^-21 + 5 * 2^-24 to
// first order: p/rho carries under 2^-20 (both truncations go toward zero),
// the square root halves it, |u| carries under 2^-20, the hardware's
// approximations of the reciprocal and the reciprocal square root under 2^-22
// each, and gamma, 1/dx and eight FP32 operations add 2^-24 each along any
// path.  Two estimates can thus misorder cells by at most 3.7 * 2^-20
// relative, 59 FP32 ulps; a cell is
// evaluated exactly when its estimate is within 128 ulps of the running max of
// estimates (a thread's own and then its block's, CflRecord; a warp's in the
// fused step).  Every other cell -- NaN, infinite or out-of-range values -- is
// always evaluated exactly.  So the cell holding the exact max is always
// evaluated, and the max of the exact values over the evaluated cells is the
// exact max.
struct WaveScreen {
    float g, ix0, ix1, ix2;
    bool on;        // gamma and 1/dx in FP32's safe range: screening is sound
    unsigned run;   // the warp's running max of the estimates' bit patterns

    __device__ __forceinline__ static bool in_range(float x) { return x >= 1e-30f && x <= 1e30f; }

    // x with its mantissa truncated to 20 bits, from the high word alone: 0
    // below FP32's normal range, infinity above it (and for NaN).
    __device__ __forceinline__ static float high_word_float(double x)
    {
        unsigned const hi = static_cast<unsigned>(static_cast<unsigned long long>(__double_as_longlong(x)) >> 32);
        int const e = static_cast<int>((hi >> 20) & 0x7ffu) - (1023 - 127);
        unsigned const mag = e <= 0 ? 0u : (e >= 255 ? 0x7f800000u : (static_cast<unsigned>(e) << 23) | ((hi & 0xfffffu) << 3));
        return __uint_as_float((hi & 0x80000000u) | mag);
    }

    __device__ __forceinline__ WaveScreen(float gamma, float x0, float x1, float x2)
        : g(gamma), ix0(x0), ix1(x1), ix2(x2), run(0u)
    {
        on = in_range(g) && in_range(ix0) && in_range(ix1) && in_range(ix2);
    }
    __device__ __forceinline__ WaveScreen(double gamma, double x0, double x1, double x2)
        : WaveScreen(static_cast<float>(gamma), static_cast<float>(x0), static_cast<float>(x1), static_cast<float>(x2))
    {
    }

    // Bit pattern of a cell's estimate, and whether the estimate's bound
    // holds for it.
    __device__ __forceinline__ unsigned estimate(double d, double p, double u0, double u1, double u2, bool& sure) const
    {
        float const d32 = high_word_float(d);
        float const p32 = high_word_float(p);
        float const x32 = g * p32 * rcp_approx(d32);
        float const c32 = x32 * rsqrt_approx(x32);
        float const v32 = (c32 + fabsf(high_word_float(u0))) * ix0 + (c32 + fabsf(high_word_float(u1))) * ix1 +
                          (c32 + fabsf(high_word_float(u2))) * ix2;
        sure = on && in_range(d32) && in_range(p32) && in_range(x32) && v32 <= 1e30f;
        return __float_as_uint(v32);
    }

    // The same for FP32 cells, whose wavespeed takes a correctly rounded
    // quotient and square root: the hardware's approximations, each within
    // 2^-22, put the estimate within 2^-21 + 6 * 2^-24 of the true value and
    // the exact expression's own roundings add 6 * 2^-24, so two estimates
    // misorder exact values by at most 28 ulps.
    __device__ __forceinline__ unsigned estimate(float d, float p, float u0, float u1, float u2, bool& sure) const
    {
        float const x = g * p * rcp_approx(d);
        float const c = x * rsqrt_approx(x);
        float const v = (c + fabsf(u0)) * ix0 + (c + fabsf(u1)) * ix1 + (c + fabsf(u2)) * ix2;
        sure = on && in_range(d) && in_range(p) && in_range(x) && v <= 1e30f;
        return __float_as_uint(v);
    }

    // The fused FP64 step's form (warp-collective: all 32 lanes call it
    // together): true when this lane's cell, if valid, needs its exact
    // wavespeed.  The step has the
    // new state's faithful sound speed cs and its velocities, and its
    // wavespeed is (3 cs + |v0| + |v1| + |v2|) / dx on cubic cells, else
    // sum_d (cs + |v_d|) / dx_d.  The estimate truncates cs and |v_d| (each
    // under 2^-20) and adds at most six FP32 roundings and 1/dx's own, so
    // its relative error is below 2^-20 + 6 * 2^-24, and two estimates
    // misorder by at most 44 ulps: the 128-ulp band holds here too.
    // Velocities below FP32's normal range read as zero: an error under
    // 2^-26 relative to cs >= 1e-30, far inside the band.
    __device__ __forceinline__ bool step_exact_needed(bool valid, double cs, double v0, double v1, double v2, bool cubic)
    {
        float const c32 = high_word_float(cs);
        float const a0 = fabsf(high_word_float(v0));
        float const a1 = fabsf(high_word_float(v1));
        float const a2 = fabsf(high_word_float(v2));
        float const v32 = cubic ? (3.0f * c32 + a0 + a1 + a2) * ix0
                                : (c32 + a0) * ix0 + (c32 + a1) * ix1 + (c32 + a2) * ix2;
        bool const sure = on && in_range(c32) && v32 <= 1e30f;
        unsigned const key = (valid && sure) ? __float_as_uint(v32) : 0u;
        unsigned const m = __reduce_max_sync(0xffffffffu, key);
        run = m > run ? m : run;
        return valid && (!sure || key + 128u >= run);
    }
};

// gamma and 1/dx in FP32, converted on the host: four conversions a thread
// would go through the FP64 pipe.
struct ScreenArgs {
    float gamma, ix0, ix1, ix2;
};

// Block max of non-negative values, in thread 0; on the integer pipe.
__device__ __forceinline__ double block_max(double v)
{
    __shared__ long long best[32];
    long long b = dbits(v);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        long long const w = __shfl_xor_sync(0xffffffffu, b, o);
        b = w > b ? w : b;
    }
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        best[threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w) {
            b = best[w] > b ? best[w] : b;
        }
    }
    return __longlong_as_double(b);
}
__device__ __forceinline__ float block_max(float v)
{
    __shared__ unsigned best[32];
    unsigned b = __reduce_max_sync(0xffffffffu, __float_as_uint(v));
    __syncthreads();
    if ((threadIdx.x & 31) == 0) {
        best[threadIdx.x >> 5] = b;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w) {
            b = best[w] > b ? best[w] : b;
        }
    }
    return __uint_as_float(b);
}

__device__ __forceinline__ bool same_bits(double a, double b) { return dbits(a) == dbits(b); }
__device__ __forceinline__ bool same_bits(float a, float b) { return __float_as_uint(a) == __float_as_uint(b); }

// A thread's cells offered one by one: keeps the one with the largest
// estimate and drops those that it outranks by more than the band, so that a
// pass over the grid evaluates the exact wavespeed about once per block (the
// warps' own running maxima, as the fused step takes them, cost a pass at
// 129 x 96 x 73 more than its memory traffic: 46 us, 17 this way).  Cells within
// the band of the kept one are evaluated at once, bit-equal ones skipped.
template <class T>
struct CflRecord {
    unsigned best = 0u; // the kept cell's estimate; 0: none
    T d = T(1), p = T(1), u0 = T(0), u1 = T(0), u2 = T(0);
    T local = T(0); // max over the cells evaluated

    __device__ __forceinline__ void take(T v) { local = v > local ? v : local; } // NaN never wins

    // ix: 1/dx in T, as the exact expression takes them
    __device__ __forceinline__ void offer(WaveScreen const& screen, T cd, T cp, T c0, T c1, T c2, T gamma, T ix0, T ix1,
                                          T ix2)
    {
        bool sure;
        unsigned const key = screen.estimate(cd, cp, c0, c1, c2, sure);
        if (!sure || key <= 256u) { // out of the estimate's range, or too small for a band in ulps
            take(cell_invdt_exact(cd, cp, c0, c1, c2, gamma, ix0, ix1, ix2));
            return;
        }
        if (key + 128u < best) {
            return;
        }
        if (best + 128u >= key) {
            if (same_bits(cd, d) && same_bits(cp, p) && same_bits(c0, u0) && same_bits(c1, u1) && same_bits(c2, u2)) {
                return;
            }
            take(cell_invdt_exact(d, p, u0, u1, u2, gamma, ix0, ix1, ix2)); // the kept cell; the new one is kept
        }
        best = key;
        d = cd;
        p = cp;
        u0 = c0;
        u1 = c1;
        u2 = c2;
    }

    // Block-collective: the exact wavespeed of the kept cells within the band
    // of the block's largest estimate.
    __device__ __forceinline__ void finish(T gamma, T ix0, T ix1, T ix2)
    {
        __shared__ unsigned top;
        if (threadIdx.x == 0) {
            top = 0u;
        }
        __syncthreads();
        unsigned const w = __reduce_max_sync(0xffffffffu, best);
        if ((threadIdx.x & 31) == 0) {
            atomicMax(&top, w);
        }
        __syncthreads();
        if (best != 0u && best + 128u >= top) {
            take(cell_invdt_exact(d, p, u0, u1, u2, gamma, ix0, ix1, ix2));
        }
    }
};

} // namespace
} // namespace eulr
