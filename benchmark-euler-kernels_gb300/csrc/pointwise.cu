// Pointwise Euler operators and the CFL reduction (sm_103a).
//
// Each kernel restates one reference operator with separately rounded
// operations in the reference's operand order, so the results are
// bit-identical to euler_operators/*.hpp compiled without FMA contraction.
// time_step and the FP32 passes are bound by HBM.  prim_to_cons and
// cons_to_prim in FP64 were bound by the FP64 pipe (1/64 of the FP32 rate):
// divisions by the loop-invariant gamma-1 use a precomputed reciprocal plus
// one Markstein correction, cons_to_prim derives both of its quotients from
// one reciprocal of rho, and the products and that reciprocal run on the
// integer pipes, correctly rounded (mul_rn_alu, rcp_rn_alu).  At 256^3 that
// took prim_to_cons from 440 to 277 us and cons_to_prim from 576 to 324 (at
// rest, whose zero products leave the fast path, to 397 and 400); HBM alone
// would take 203.
#include "euler_device.cuh"
#include "kernels.h"
#include "step_common.cuh"

#include <cfloat>

namespace eulr {

// Cells whose loads a thread of a memory-bound pass has in flight.
template <class T>
constexpr int kCellsInFlight = sizeof(T) == 8 ? 2 : 4;

// ------------------------------------------------------------ init_implode
// init_implode.hpp:24-44.  Cell centres are computed in double (the literal 0.5
// promotes (i-1) to double) and rounded to T, as in the reference's float
// instantiation.
template <class T>
__global__ void __launch_bounds__(256) init_implode_kernel(Bundle<T> prim, Geom g, double dx0, double dx1, double dx2)
{
    long long const n = g.ncell();
    T const radius2 = static_cast<T>(0.25 * 0.25);
    for (long long c = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; c < n;
         c += static_cast<long long>(gridDim.x) * blockDim.x) {
        int const i = static_cast<int>(c % g.n0);
        long long const jk = c / g.n0;
        int const j = static_cast<int>(jk % g.n1);
        int const k = static_cast<int>(jk / g.n1);
        T const x0 = static_cast<T>(__dsub_rn(__dmul_rn(__dadd_rn(static_cast<double>(i - 1), 0.5), dx0), 0.5));
        T const x1 = static_cast<T>(__dsub_rn(__dmul_rn(__dadd_rn(static_cast<double>(j - 1), 0.5), dx1), 0.5));
        T const x2 = static_cast<T>(__dsub_rn(__dmul_rn(__dadd_rn(static_cast<double>(k - 1), 0.5), dx2), 0.5));
        T const r2 = add_rn(add_rn(mul_rn(x0, x0), mul_rn(x1, x1)), mul_rn(x2, x2));
        bool const inside = r2 < radius2;
        prim.f[0][c] = inside ? T(1) : T(0.125);
        prim.f[1][c] = inside ? T(1) : T(0.14);
        prim.f[2][c] = T(0);
        prim.f[3][c] = T(0);
        prim.f[4][c] = T(0);
    }
}

// One pass over n cells from five fields to five others.  FP32 is bound by
// HBM: a thread has four cells' loads in flight (256^3: 125 -> 115 us, 6.0 TB/s).
// FP64 is bound by its arithmetic and takes one cell at a time.
template <class T, class Cell>
__device__ __forceinline__ void pointwise_pass(CBundle<T> const& in, Bundle<T> const& out, long long n, Cell cell)
{
    constexpr int kCells = sizeof(T) == 8 ? 1 : kCellsInFlight<T>;
    long long const stride = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long base = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; base < n; base += kCells * stride) {
        T a[kCells][5];
#pragma unroll
        for (int u = 0; u < kCells; ++u) {
            long long const c = base + u * stride;
            if (c < n) {
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    a[u][f] = in.f[f][c];
                }
            }
        }
#pragma unroll
        for (int u = 0; u < kCells; ++u) {
            long long const c = base + u * stride;
            if (c < n) {
                T b[5];
                cell(a[u], b);
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    out.f[f][c] = b[f];
                }
            }
        }
    }
}

// ------------------------------------------------------------ prim_to_cons
// prim_to_cons.hpp:20-32 with to_cons (euler_arrays.hpp:56-64):
//   e = d*((u0*u0 + u1*u1) + u2*u2)/2 + p/(gamma-1),  m_i = d*u_i.
template <class T>
__global__ void __launch_bounds__(256) prim_to_cons_kernel(CBundle<T> prim, Bundle<T> cons, long long n, T gm1, T rgm1)
{
    pointwise_pass(prim, cons, n, [=](T const* q, T* u) {
        T const int_e = div_by_rcp(q[1], gm1, rgm1);
        T const ke = half_exact(mul_rn_alu(q[0], add_rn(add_rn(mul_rn_alu(q[2], q[2]), mul_rn_alu(q[3], q[3])), mul_rn_alu(q[4], q[4]))));
        u[0] = q[0];
        u[1] = add_rn(ke, int_e);
        u[2] = mul_rn_alu(q[0], q[2]);
        u[3] = mul_rn_alu(q[0], q[3]);
        u[4] = mul_rn_alu(q[0], q[4]);
    });
}

// ------------------------------------------------------------ cons_to_prim
// cons_to_prim.hpp:20-32 with kinetic_energy(cons) (euler_arrays.hpp:44-48),
// PerfectGas::pressure and to_prim (euler_arrays.hpp:66-75):
//   ke = ((m.m)/d)/2, p = (gamma-1)*(e-ke), u_i = m_i * (1/d).
template <class T>
__global__ void __launch_bounds__(256) cons_to_prim_kernel(CBundle<T> cons, Bundle<T> prim, long long n, T gm1)
{
    pointwise_pass(cons, prim, n, [=](T const* u, T* q) {
        q[0] = u[0];
        cons_to_prim_exact(u[0], u[1], u[2], u[3], u[4], gm1, q[1], q[2], q[3], q[4]);
    });
}

// --------------------------------------------------------------- time_step
// time_step.hpp:22-39.  The reference takes min over cells of 1/invdt; since
// correctly rounded division is monotonic, min_c RN(1/x_c) = RN(1/max_c x_c),
// so the kernel reduces max(invdt) (exact, order-free) and divides once.
// The max is screened (WaveScreen, CflRecord), so the kernel reads each cell
// and evaluates its exact wavespeed only where it can be the max; the dt is
// still the reference's bit for bit.  Bound by HBM (256^3: FP64 167 -> 114 us,
// 6.1 TB/s; FP32, which took every exact wavespeed, 90 -> 62).  NaN never wins (the reference's Kokkos::min
// skips it) and an all-zero grid returns the reduction identity T's max, as
// the reference's Min reducer does.
template <class T>
__global__ void __launch_bounds__(256) time_step_kernel(CBundle<T> prim, long long n, T gamma, T ix0, T ix1, T ix2,
                                                        ScreenArgs a, T* partials, unsigned int* counter, T* dt_out)
{
    WaveScreen const screen(a.gamma, a.ix0, a.ix1, a.ix2);
    CflRecord<T> record;
    // several cells' loads in flight at a time
    constexpr int kCells = kCellsInFlight<T>;
    long long const stride = static_cast<long long>(gridDim.x) * blockDim.x;
    for (long long base = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; base < n; base += kCells * stride) {
        T q[kCells][5];
#pragma unroll
        for (int u = 0; u < kCells; ++u) {
            long long const c = base + u * stride < n ? base + u * stride : base; // loaded without a branch
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                q[u][f] = prim.f[f][c];
            }
        }
#pragma unroll
        for (int u = 0; u < kCells; ++u) {
            if (base + u * stride < n) {
                record.offer(screen, q[u][0], q[u][1], q[u][2], q[u][3], q[u][4], gamma, ix0, ix1, ix2);
            }
        }
    }
    record.finish(gamma, ix0, ix1, ix2);
    __shared__ bool is_last;
    T const mine = block_max(record.local);
    if (threadIdx.x == 0) {
        partials[blockIdx.x] = mine;
        __threadfence();
        unsigned int const done = atomicAdd(counter, 1u);
        is_last = (done == gridDim.x - 1);
    }
    __syncthreads();
    if (is_last) {
        // Last block to finish: fold the per-block maxima and publish dt.
        __threadfence();
        T b = T(0);
        for (unsigned int w = threadIdx.x; w < gridDim.x; w += blockDim.x) {
            T const v = __ldcg(&partials[w]);
            b = (v > b) ? v : b;
        }
        T const m = block_max(b);
        if (threadIdx.x == 0) {
            *dt_out = (m > T(0)) ? rcp_rn(m) : (sizeof(T) == 8 ? T(DBL_MAX) : T(FLT_MAX));
            *counter = 0u;
        }
    }
}

// Max invdt over all cells of a cons-only FP32 state.
__global__ void __launch_bounds__(256) invdt_max_cons_kernel(CBundle<float> cons, long long n, float gamma, float ix0,
                                                             float ix1, float ix2, int comp, unsigned long long* wmax)
{
    float local = 0.0f;
    float const gm1 = gamma - 1.0f;
    for (long long c = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; c < n;
         c += static_cast<long long>(gridDim.x) * blockDim.x) {
        float const v = cons_invdt_f32(cons.f[0][c], cons.f[1][c], cons.f[2][c], cons.f[3][c], cons.f[4][c], gamma, gm1, ix0,
                                       ix1, ix2, comp);
        local = (v > local) ? v : local;
    }
    __shared__ float warp_best[8];
    local = warp_max(local);
    if ((threadIdx.x & 31) == 0) {
        warp_best[threadIdx.x >> 5] = local;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        float b = warp_best[0];
        for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w) {
            b = (warp_best[w] > b) ? warp_best[w] : b;
        }
        atomicMax(wmax, order_bits(b));
    }
}

// Loading a primitive state into an FP64 simulation or batch grid, in one
// pass (bound by the FP64 pipe, so what it also moves is nearly free):
//  * prim itself when copy is set -- the caller's device arrays are read in
//    place, not copied first (10.9 GB of traffic less at 514^3);
//  * cons = prim_to_cons(prim) when cons is set, bit-identical to
//    prim_to_cons_kernel;
//  * the stored sound speed as the fused step computes it, within two ulps (a
//    reciprocal of rho and a square root; the step multiplies gamma and 1/rho
//    first, this gamma and p, so the two may differ by an ulp), and e + p;
//  * the EXACT max wavespeed of time_step.hpp:28-33 for the first dt, with
//    the exact per-cell value evaluated only where WaveScreen says it can be
//    the max.
__global__ void __launch_bounds__(256) load_prim_kernel(CBundle<double> prim, Bundle<double> cons, Bundle<double> copy,
                                                        double* cs, double* h, const double* e_in, long long n,
                                                        double gamma, double gm1, double rgm1, double ix0, double ix1,
                                                        double ix2, ScreenArgs a, unsigned long long* wmax)
{
    WaveScreen const screen(a.gamma, a.ix0, a.ix1, a.ix2);
    CflRecord<double> record;
    for (long long c = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; c < n;
         c += static_cast<long long>(gridDim.x) * blockDim.x) {
        double const d = prim.f[0][c];
        double const p = prim.f[1][c];
        double const u0 = prim.f[2][c];
        double const u1 = prim.f[3][c];
        double const u2 = prim.f[4][c];
        if (copy.f[0] != nullptr) {
            copy.f[0][c] = d;
            copy.f[1][c] = p;
            copy.f[2][c] = u0;
            copy.f[3][c] = u1;
            copy.f[4][c] = u2;
        }
        if (cons.f[0] != nullptr) {
            double const int_e = div_by_rcp(p, gm1, rgm1);
            double const ke = half_exact(mul_rn_alu(d, add_rn(add_rn(mul_rn_alu(u0, u0), mul_rn_alu(u1, u1)), mul_rn_alu(u2, u2))));
            double const e = add_rn(ke, int_e);
            cons.f[0][c] = d;
            cons.f[1][c] = e;
            cons.f[2][c] = mul_rn_alu(d, u0);
            cons.f[3][c] = mul_rn_alu(d, u1);
            cons.f[4][c] = mul_rn_alu(d, u2);
            h[c] = add_rn(e, p);
        } else {
            h[c] = add_rn(e_in[c], p);
        }
        cs[c] = sqrt_alu(mul_alu(mul_alu(gamma, p), rcp_alu(d)));
        record.offer(screen, d, p, u0, u1, u2, gamma, ix0, ix1, ix2);
    }
    record.finish(gamma, ix0, ix1, ix2);
    double const mine = block_max(record.local);
    if (threadIdx.x == 0) {
        atomicMax(wmax, static_cast<unsigned long long>(dbits(mine)));
    }
}

// ----------------------------------------------------------- init_step
// Step discontinuity on x + y + z < c, the initial condition of the batched
// workload (it has no counterpart in the reference): cell centres
// ((i-1)+0.5) dx in double as in init_implode.hpp:33-36 but on [0,1]^3,
// (rho_in, p_in) below the plane, (rho_out, p_out) above it, u = 0.
template <class T>
__global__ void __launch_bounds__(256) init_step_kernel(Bundle<T> prim, Geom g, double dx0, double dx1, double dx2,
                                                        double c, double rho_in, double p_in, double rho_out,
                                                        double p_out)
{
    long long const n = g.ncell();
    for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < n;
         idx += static_cast<long long>(gridDim.x) * blockDim.x) {
        int const i = static_cast<int>(idx % g.n0);
        long long const jk = idx / g.n0;
        int const j = static_cast<int>(jk % g.n1);
        int const k = static_cast<int>(jk / g.n1);
        double const x0 = __dmul_rn(__dadd_rn(static_cast<double>(i - 1), 0.5), dx0);
        double const x1 = __dmul_rn(__dadd_rn(static_cast<double>(j - 1), 0.5), dx1);
        double const x2 = __dmul_rn(__dadd_rn(static_cast<double>(k - 1), 0.5), dx2);
        bool const inside = __dadd_rn(__dadd_rn(x0, x1), x2) < c;
        prim.f[0][idx] = static_cast<T>(inside ? rho_in : rho_out);
        prim.f[1][idx] = static_cast<T>(inside ? p_in : p_out);
        prim.f[2][idx] = T(0);
        prim.f[3][idx] = T(0);
        prim.f[4][idx] = T(0);
    }
}

// ------------------------------------------------------------------ launch
static int grid_for(long long n, int sms)
{
    long long const blocks = (n + 255) / 256;
    long long const cap = static_cast<long long>(sms) * 8;
    return static_cast<int>(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
}

template <class T>
static ScreenArgs screen_args(T gamma, T ix0, T ix1, T ix2)
{
    return ScreenArgs{static_cast<float>(gamma), static_cast<float>(ix0), static_cast<float>(ix1), static_cast<float>(ix2)};
}

template <class T>
cudaError_t launch_init_implode(Bundle<T> prim, Geom g, double dx0, double dx1, double dx2, int sms, cudaStream_t s)
{
    init_implode_kernel<T><<<grid_for(g.ncell(), sms), 256, 0, s>>>(prim, g, dx0, dx1, dx2);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_prim_to_cons(CBundle<T> prim, Bundle<T> cons, long long n, T gm1, T rgm1, int sms, cudaStream_t s)
{
    prim_to_cons_kernel<T><<<grid_for(n, sms), 256, 0, s>>>(prim, cons, n, gm1, rgm1);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_cons_to_prim(CBundle<T> cons, Bundle<T> prim, long long n, T gm1, int sms, cudaStream_t s)
{
    cons_to_prim_kernel<T><<<grid_for(n, sms), 256, 0, s>>>(cons, prim, n, gm1);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_time_step(CBundle<T> prim, long long n, T gamma, T ix0, T ix1, T ix2, T* partials,
                             int max_partials, unsigned int* counter, T* dt_out, int sms, cudaStream_t s)
{
    int grid = grid_for((n + kCellsInFlight<T> - 1) / kCellsInFlight<T>, sms);
    if (grid > max_partials) {
        grid = max_partials;
    }
    time_step_kernel<T><<<grid, 256, 0, s>>>(prim, n, gamma, ix0, ix1, ix2, screen_args(gamma, ix0, ix1, ix2), partials,
                                             counter, dt_out);
    return cudaGetLastError();
}

cudaError_t launch_load_prim(CBundle<double> prim, Bundle<double> cons, Bundle<double> copy, double* cs, double* h,
                             const double* e_in, long long n, double gamma, double ix0, double ix1, double ix2,
                             unsigned long long* wmax, int sms, cudaStream_t s)
{
    double const gm1 = gamma - 1.0;
    load_prim_kernel<<<grid_for(n, sms), 256, 0, s>>>(prim, cons, copy, cs, h, e_in, n, gamma, gm1, 1.0 / gm1, ix0, ix1,
                                                      ix2, screen_args(gamma, ix0, ix1, ix2), wmax);
    return cudaGetLastError();
}

// Bound by HBM: 16-byte accesses, each thread's loads of every field in
// flight before its stores.  A state's 11 fields in one launch instead of a
// copy each (64^3: 11 launches of about 2.5 us for 8 us of traffic).
__global__ void __launch_bounds__(256) copy_fields_kernel(const __grid_constant__ CopyFieldsParams p)
{
    if (p.sc != nullptr && blockIdx.x == 0 && threadIdx.x == 0) {
        SimScalars v{};
        v.steps = p.step;
        *p.sc = v;
    }
    long long const pairs = (p.n + 1) / 2; // fields are padded to 256 bytes
    for (long long c = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; c < pairs;
         c += static_cast<long long>(gridDim.x) * blockDim.x) {
        double2 v[11];
#pragma unroll
        for (int f = 0; f < 11; ++f) {
            if (f < p.count) {
                v[f] = reinterpret_cast<const double2*>(p.src[f])[c];
            }
        }
#pragma unroll
        for (int f = 0; f < 11; ++f) {
            if (f < p.count) {
                reinterpret_cast<double2*>(p.dst[f])[c] = v[f];
            }
        }
        if (p.h != nullptr) {
            reinterpret_cast<double2*>(p.h)[c] = make_double2(__dadd_rn(v[6].x, v[1].x), __dadd_rn(v[6].y, v[1].y));
        }
    }
}

cudaError_t launch_copy_fields(CopyFieldsParams const& p, int sms, cudaStream_t s)
{
    copy_fields_kernel<<<grid_for((p.n + 1) / 2, sms), 256, 0, s>>>(p);
    return cudaGetLastError();
}

cudaError_t launch_init_step(Bundle<double> prim, Geom g, double dx0, double dx1, double dx2, double c,
                             double rho_in, double p_in, double rho_out, double p_out, int sms, cudaStream_t s)
{
    init_step_kernel<double><<<grid_for(g.ncell(), sms), 256, 0, s>>>(prim, g, dx0, dx1, dx2, c, rho_in, p_in, rho_out,
                                                                       p_out);
    return cudaGetLastError();
}

cudaError_t launch_invdt_max_cons(CBundle<float> cons, long long n, float gamma, float ix0, float ix1, float ix2,
                                  int comp, unsigned long long* wmax, int sms, cudaStream_t s)
{
    invdt_max_cons_kernel<<<grid_for(n, sms), 256, 0, s>>>(cons, n, gamma, ix0, ix1, ix2, comp, wmax);
    return cudaGetLastError();
}

#define EULR_INSTANTIATE_POINTWISE(T)                                                                        \
    template cudaError_t launch_init_implode<T>(Bundle<T>, Geom, double, double, double, int, cudaStream_t); \
    template cudaError_t launch_prim_to_cons<T>(CBundle<T>, Bundle<T>, long long, T, T, int, cudaStream_t);  \
    template cudaError_t launch_cons_to_prim<T>(CBundle<T>, Bundle<T>, long long, T, int, cudaStream_t);     \
    template cudaError_t launch_time_step<T>(CBundle<T>, long long, T, T, T, T, T*, int, unsigned int*, T*,  \
                                             int, cudaStream_t);

EULR_INSTANTIATE_POINTWISE(double)
EULR_INSTANTIATE_POINTWISE(float)

} // namespace eulr
