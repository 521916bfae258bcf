// The reference's godunov, bit for bit (eulr_godunov_exact_{f64,f32}).
//
// The default godunov (flux.cu) solves each face once with a reformulated
// HLLC -- one shared reciprocal, FMA contraction, selects for the
// supersonic case -- and agrees with the reference to a few ulps per face.
// This kernel is the opt-in alternative for callers who need the
// reference's numbers exactly: it follows godunov.hpp:15-92 and
// hllc.hpp:50-105 operation by operation, every product, quotient, sum and
// square root rounded separately (__dmul_rn, __ddiv_rn, ...; no FMA) in the
// reference's evaluation order, with the reference's divisions and its
// two-sided pstar.
//
// The reference solves each interior face twice, once from each of its
// cells, and recomputes a cell's sound speed and total energy for every
// face it touches.  Both are the same function on the same arguments, so
// their bits do not depend on which cell asks: here each face is solved
// once and each cell's sound speed and total energy computed once, and the
// results are still the reference's.  A CTA owns a tile of at most 16 x 16
// columns, cut evenly out of the interior, and marches up a run of planes
// (the tile engine's work split, choose_tiles in flux.cu):
//   * two plane buffers in shared memory hold d, p, u0..u2, the sound speed
//     and the total energy of a plane (the tile and its x/y halo);
//   * per plane, the x-faces and y-faces (one index space, 544 for a whole
//     tile) are solved into shared memory, and each thread solves the z-face
//     above its cell into registers (the one below is the previous plane's);
//   * each cell then sums ds_a (F_R - F_L) over a = 0, 1, 2 from zero and
//     subtracts dtodv times the sum from cons, as godunov.hpp:82-90 does.
//
// It is FP64-bound.  The two quotients by S - ustar share one correctly
// rounded reciprocal; against whole 16 x 8 tiles in chunks of planes and three
// full divisions a face: 256^3 9.96 -> 8.10 ms, 129 x 96 x 73 653 -> 480 us,
// 16^3 136 -> 24 us.  Products and reciprocals run on the integer pipes with
// the FP64 unit's bits (mul_rn_alu, rcp_rn_alu): 256^3 8.12 -> 5.93 ms,
// 128 x 95 x 72 472 -> 358 us, 64^3 165 -> 129 us.
#include "euler_device.cuh"
#include "kernels.h"
#include "step_common.cuh"

namespace eulr {

namespace {

constexpr int kExTX = 16;                          // most tile cells along i
template <class T>
constexpr int kExTY = sizeof(T) == 8 ? 16 : 8;     // and along j
template <class T>
constexpr int kExNT = kExTX * kExTY<T>;            // threads per CTA
constexpr int kExPW = kExTX + 2;                   // plane buffer row (tile + x halo)
template <class T>
constexpr int kExPC = kExPW * (kExTY<T> + 2);      // plane buffer cells
template <class T>
constexpr int kExNF = (kExTX + 1) * kExTY<T> + kExTX * (kExTY<T> + 1); // x- and y-faces of a whole tile's plane

// Shared memory of a CTA.
template <class T>
struct ExactShared {
    T planes[2][7][kExPC<T>];
    T faces[5][kExNF<T>];
};

// Fields of a plane buffer: the prim fields in the global order, then the
// sound speed and the total energy of each cell.
constexpr int kFieldC = 5;
constexpr int kFieldE = 6;

// Kokkos::min / Kokkos::max on two values (the reference's helpers): the
// first argument unless the second is strictly smaller / larger.  The
// comparisons run on the integer pipe with the FP64 compare's answer
// (less_ieee), so each saves an FP64 slot.
template <class T>
__device__ __forceinline__ T kmin(T a, T b)
{
    return less_ieee(b, a) ? b : a;
}
template <class T>
__device__ __forceinline__ T kmax(T a, T b)
{
    return less_ieee(a, b) ? b : a;
}

// ratio = x1/y1 and gain = x2/y, correctly rounded.  In the subsonic case y1
// is y, and both quotients come from one correctly rounded reciprocal
// (div_by_rcp: 11 FP64 instructions instead of two full divisions' 17); in
// the supersonic case y1 is x1 and the first is exactly 1.  That holds where
// the operands lie in 2^+-400 (FP32: 2^+-40), so that no step leaves the
// normal range, or x2 is zero, whose quotient is a zero with the product of
// the signs; anything else takes the divisions.
__device__ __forceinline__ bool mid_range(double x)
{
    unsigned const e = static_cast<unsigned>(static_cast<unsigned long long>(dbits(x)) >> 52) & 0x7ffu;
    return e - (1023u - 400u) <= 800u;
}
__device__ __forceinline__ void star_quotients(bool supersonic, double x1, double y1, double x2, double y, double& ratio,
                                               double& gain)
{
    bool const zero = !nonzero_(x2);
    if (mid_range(x1) && mid_range(y) && (zero || mid_range(x2))) {
        double const r = rcp_rn_alu(y);
        double const q1 = div_by_rcp(x1, y, r);
        double const q2 = div_by_rcp(x2, y, r);
        ratio = supersonic ? 1.0 : q1;
        gain = zero ? __longlong_as_double((dbits(x2) ^ dbits(y)) & static_cast<long long>(0x8000000000000000ull)) : q2;
    } else {
        ratio = div_rn(x1, y1);
        gain = div_rn(x2, y);
    }
}
__device__ __forceinline__ bool mid_range(float x)
{
    unsigned const e = (__float_as_uint(x) >> 23) & 0xffu;
    return e - (127u - 40u) <= 80u;
}
__device__ __forceinline__ void star_quotients(bool supersonic, float x1, float y1, float x2, float y, float& ratio,
                                               float& gain)
{
    bool const zero = x2 == 0.0f;
    if (mid_range(x1) && mid_range(y) && (zero || mid_range(x2))) {
        float const r = rcp_rn(y);
        float const q1 = div_by_rcp(x1, y, r);
        float const q2 = div_by_rcp(x2, y, r);
        ratio = supersonic ? 1.0f : q1;
        gain = zero ? __uint_as_float((__float_as_uint(x2) ^ __float_as_uint(y)) & 0x80000000u) : q2;
    } else {
        ratio = div_rn(x1, y1);
        gain = div_rn(x2, y);
    }
}

// x/y, correctly rounded; the ranges as above.
static __device__ __noinline__ double quotient_rare(double x, double y) { return div_rn(x, y); }
__device__ __forceinline__ double quotient(double x, double y)
{
    if (mid_range(x) && mid_range(y)) {
        return div_by_rcp(x, y, rcp_rn_alu(y));
    }
    return quotient_rare(x, y);
}
__device__ __forceinline__ float quotient(float x, float y) { return div_rn(x, y); }

// 0 + x: x, but +0 for -0 (the sum over axes starts from zero), in FP64 on the
// integer pipe.
__device__ __forceinline__ double from_zero(double x) { return nonzero_(x) ? x : 0.0; }
__device__ __forceinline__ float from_zero(float x) { return add_rn(0.0f, x); }

// hllc::operator() (hllc.hpp:50-105) across the face between cell ca of
// plane A (left) and cell cb of plane B (right), normal direction dir.
// The flux comes back as (d, e, normal momentum, tangential momenta along
// t1 < t2).  PerfectGas::speed_of_sound (perfect_gas.hpp:15-18) and the
// total energy (euler_arrays.hpp:38-42) come from the plane buffers, where
// each was computed once per cell with the reference's operations.
template <class T>
__device__ __forceinline__ void solve_face_exact(T const (*A)[kExPC<T>], int ca, T const (*B)[kExPC<T>], int cb, int dir,
                                                 T f[5])
{
    int const t1 = dir == 0 ? 1 : 0;
    int const t2 = dir == 2 ? 1 : 2;
    T const d_L = A[0][ca], p_L = A[1][ca], un_L = A[2 + dir][ca], c_L = A[kFieldC][ca];
    T const d_R = B[0][cb], p_R = B[1][cb], un_R = B[2 + dir][cb], c_R = B[kFieldC][cb];
    T const S_L = sub_rn(kmin(un_L, un_R), kmax(c_L, c_R));
    T const S_R = add_rn(kmax(un_L, un_R), kmax(c_L, c_R));
    T const rc_L = mul_rn_alu(d_L, sub_rn(S_L, un_L));
    T const rc_R = mul_rn_alu(d_R, sub_rn(S_R, un_R));
    // acoustic star state: q_R.p - q_L.p + rc_L * un_L - rc_R * un_R, left to right
    T const ustar = quotient(sub_rn(add_rn(sub_rn(p_R, p_L), mul_rn_alu(rc_L, un_L)), mul_rn_alu(rc_R, un_R)), sub_rn(rc_L, rc_R));
    T const pstar = half_exact(add_rn(add_rn(add_rn(p_L, p_R), mul_rn_alu(rc_L, sub_rn(ustar, un_L))),
                                          mul_rn_alu(rc_R, sub_rn(ustar, un_R))));
    bool const left = less_ieee(T(0), ustar);
    T const (*Q)[kExPC<T>] = left ? A : B;
    int const cq = left ? ca : cb;
    T const S = left ? S_L : S_R;
    T const d = left ? d_L : d_R;
    T const p = left ? p_L : p_R;
    T const un = left ? un_L : un_R;
    T const etot = Q[kFieldE][cq];
    bool const supersonic = less_ieee(T(0), mul_rn_alu(S_L, S_R));
    T const un_o = supersonic ? un : ustar;
    T const ptot_o = supersonic ? p : pstar;
    T ratio, gain; // (S - un)/(S - un_o), (ptot_o un_o - p un)/(S - ustar)
    star_quotients(supersonic, sub_rn(S, un), sub_rn(S, un_o), sub_rn(mul_rn_alu(ptot_o, un_o), mul_rn_alu(p, un)),
                   sub_rn(S, ustar), ratio, gain);
    T const d_o = mul_rn_alu(ratio, d);
    T const etot_o = add_rn(mul_rn_alu(ratio, etot), gain);
    T const m = mul_rn_alu(d_o, un_o);
    f[0] = m;
    f[1] = mul_rn_alu(add_rn(etot_o, ptot_o), un_o);
    f[2] = add_rn(mul_rn_alu(m, un_o), ptot_o);
    f[3] = mul_rn_alu(m, Q[2 + t1][cq]);
    f[4] = mul_rn_alu(m, Q[2 + t2][cq]);
}

// Loads plane k of the tile and its x/y halo with each cell's sound speed
// sqrt(gamma p / d) and total energy p / (gamma - 1) + d |u|^2 / 2.  The
// quotient by the constant gamma - 1 is the correctly rounded one formed
// from rgm1 = RN(1 / (gamma - 1)) (div_by_rcp), as prim_to_cons forms it.
template <class T, bool WHOLE>
__device__ __forceinline__ void load_plane_exact(T (*P)[kExPC<T>], CBundle<T> const& prim, Geom const& g, int i0, int j0,
                                                 int w, int h, unsigned magic, int k, T gamma, T gm1, T rgm1)
{
#pragma unroll 1
    for (int c = threadIdx.x; c < (w + 2) * (h + 2); c += kExNT<T>) {
        int const y = WHOLE ? c / (w + 2) : div_runtime(c, magic); // magic of w + 2
        int const x = c - y * (w + 2);
        int const t = y * kExPW + x;
        if (WHOLE && (i0 - 1 + x >= g.n0 || j0 - 1 + y >= g.n1)) {
            continue; // outside the array: no face reads it
        }
        long long const o = g.at(i0 - 1 + x, j0 - 1 + y, k);
        T const d = prim.f[0][o], p = prim.f[1][o];
        T const u0 = prim.f[2][o], u1 = prim.f[3][o], u2 = prim.f[4][o];
        P[0][t] = d;
        P[1][t] = p;
        P[2][t] = u0;
        P[3][t] = u1;
        P[4][t] = u2;
        P[kFieldC][t] = sqrt_rn(quotient(mul_rn_alu(gamma, p), d));
        // the reference's "/ 2" as "* 0.5": both are the correctly rounded
        // value of the same real number, so the bits are equal
        T const ke = half_exact(mul_rn_alu(d, add_rn(add_rn(mul_rn_alu(u0, u0), mul_rn_alu(u1, u1)), mul_rn_alu(u2, u2))));
        P[kFieldE][t] = add_rn(div_by_rcp(p, gm1, rgm1), ke);
    }
}

template <class T>
struct ExactParams {
    CBundle<T> prim;
    Bundle<T> cons;
    Geom g;
    T gamma, gm1, rgm1, ds0, ds1, ds2, dtodv;
    TileSplit sx, sy;
    int nwork; // planes of all tiles
};

// godunov.hpp:32-91 for the interior cells of tile (tx, ty) in planes [kb, ke).
// WHOLE: tiles of the full extent, a compile-time one, whose cells and faces
// past the grid are masked.
template <class T, bool WHOLE>
__device__ __forceinline__ void exact_run(ExactParams<T> const& p, ExactShared<T>& sh, int tx, int ty, int kb, int ke)
{
    Geom const& g = p.g;
    int const i0 = 1 + (WHOLE ? tx * kExTX : p.sx.start(tx)), w = WHOLE ? kExTX : 1 + p.sx.start(tx + 1) - i0;
    int const j0 = 1 + (WHOLE ? ty * kExTY<T> : p.sy.start(ty)), h = WHOLE ? kExTY<T> : 1 + p.sy.start(ty + 1) - j0;
    unsigned const mw = div_magic20(w), mw1 = div_magic20(w + 1), mw2 = div_magic20(w + 2);
    int const nfx = (w + 1) * h;
    int const nf = nfx + w * (h + 1);
    int const cy = WHOLE ? threadIdx.x / w : div_runtime(threadIdx.x, mw);
    int const cx = threadIdx.x - cy * w;
    // this thread has a column
    bool const mine = WHOLE ? i0 + cx <= g.n0 - 2 && j0 + cy <= g.n1 - 2 : cy < h;
    int const ccell = (cx + 1) + kExPW * (cy + 1);   // its cell in a plane buffer

    T zlo[5], zhi[5];
    __syncthreads(); // the previous run's readers are done
    load_plane_exact<T, WHOLE>(sh.planes[(kb - 1) & 1], p.prim, g, i0, j0, w, h, mw2, kb - 1, p.gamma, p.gm1, p.rgm1);
    load_plane_exact<T, WHOLE>(sh.planes[kb & 1], p.prim, g, i0, j0, w, h, mw2, kb, p.gamma, p.gm1, p.rgm1);
    __syncthreads();
    if (mine) {
        solve_face_exact(sh.planes[(kb - 1) & 1], ccell, sh.planes[kb & 1], ccell, 2, zlo);
    }
    __syncthreads(); // plane kb - 1 is overwritten next
    for (int k = kb; k < ke; ++k) {
        T const (*cur)[kExPC<T>] = sh.planes[k & 1];
        load_plane_exact<T, WHOLE>(sh.planes[(k + 1) & 1], p.prim, g, i0, j0, w, h, mw2, k + 1, p.gamma, p.gm1, p.rgm1);
        __syncthreads();
        // x-faces (i-1 | i) for the w + 1 of each row, then y-faces (j-1 | j)
#pragma unroll 1
        for (int t = threadIdx.x; t < nf; t += kExNT<T>) {
            bool const xf = t < nfx;
            int const u = xf ? t : t - nfx;
            int const b = WHOLE ? (xf ? u / (w + 1) : u / w) : div_runtime(u, xf ? mw1 : mw);
            int const a = u - b * (xf ? w + 1 : w);
            if (WHOLE && (xf ? i0 + a > g.n0 - 1 || j0 + b > g.n1 - 2 : i0 + a > g.n0 - 2 || j0 + b > g.n1 - 1)) {
                continue;
            }
            int const cl = xf ? a + kExPW * (b + 1) : (a + 1) + kExPW * b;
            int const cr = cl + (xf ? 1 : kExPW);
            int const dir = xf ? 0 : 1;
            T f[5];
            solve_face_exact(cur, cl, cur, cr, dir, f);
            sh.faces[0][t] = f[0];
            sh.faces[1][t] = f[1];
            sh.faces[2 + dir][t] = f[2];
            sh.faces[xf ? 3 : 2][t] = f[3];
            sh.faces[4][t] = f[4];
        }
        if (mine) {
            solve_face_exact(cur, ccell, sh.planes[(k + 1) & 1], ccell, 2, zhi);
        }
        __syncthreads();
        if (mine) {
            int const xl = cx + (w + 1) * cy;
            int const yl = nfx + cx + w * cy;
            long long const c = g.at(i0 + cx, j0 + cy, k);
            T const zl[5] = {zlo[0], zlo[1], zlo[3], zlo[4], zlo[2]}; // (d, e, m0, m1, m2)
            T const zh[5] = {zhi[0], zhi[1], zhi[3], zhi[4], zhi[2]};
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                T flux = from_zero(mul_rn_alu(p.ds0, sub_rn(sh.faces[f][xl + 1], sh.faces[f][xl])));
                flux = add_rn(flux, mul_rn_alu(p.ds1, sub_rn(sh.faces[f][yl + w], sh.faces[f][yl])));
                flux = add_rn(flux, mul_rn_alu(p.ds2, sub_rn(zh[f], zl[f])));
                p.cons.f[f][c] = sub_rn(p.cons.f[f][c], mul_rn_alu(p.dtodv, flux));
            }
        }
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            zlo[f] = zhi[f];
        }
    }
}

// CTA b takes an even share of all tiles' planes, as in the tile engine.
template <class T>
__global__ void __launch_bounds__(kExNT<T>) godunov_exact_kernel(const __grid_constant__ ExactParams<T> p)
{
    extern __shared__ __align__(16) unsigned char exact_smem[];
    ExactShared<T>& sh = *reinterpret_cast<ExactShared<T>*>(exact_smem);
    int const iz = p.g.n2 - 2;
    int w = static_cast<int>(static_cast<long long>(p.nwork) * blockIdx.x / gridDim.x);
    int const end = static_cast<int>(static_cast<long long>(p.nwork) * (blockIdx.x + 1) / gridDim.x);
    while (w < end) {
        int const tile = w / iz;
        int const k = w - tile * iz;
        int const run = min(end - w, iz - k);
        exact_run<T, false>(p, sh, tile % p.sx.parts, tile / p.sx.parts, 1 + k, 1 + k + run);
        w += run;
    }
}

// FP32 on a grid that fills the GPU many times over: whole tiles, a CTA for
// each (tile, chunk of planes), neighbouring tiles of one chunk at work at one
// time.  FP32 is bound by issue and memory, not by the FP64 pipe: runtime
// extents cost it 10 %, and CTAs at different heights lose the halos they
// share in L2 (256^3: 582 us this way, 712 on even runs).
__global__ void __launch_bounds__(kExNT<float>) godunov_exact_whole_kernel(const __grid_constant__ ExactParams<float> p)
{
    __shared__ ExactShared<float> sh;
    int const iz = p.g.n2 - 2;
    int const chunks = gridDim.y;
    exact_run<float, true>(p, sh, blockIdx.x % p.sx.parts,
                           blockIdx.x / p.sx.parts, 1 + static_cast<int>(static_cast<long long>(blockIdx.y) * iz / chunks),
                           1 + static_cast<int>(static_cast<long long>(blockIdx.y + 1) * iz / chunks));
}

} // namespace

template <class T>
cudaError_t launch_godunov_exact(CBundle<T> prim, Bundle<T> cons, Geom g, T gamma, T dx0, T dx1, T dx2, T dt,
                                 int sms, cudaStream_t s)
{
    if (g.n0 < 3 || g.n1 < 3 || g.n2 < 3) {
        return cudaSuccess; // no interior cell
    }
    // UniformMesh3d: ds0 = dx1 dx2, ds1 = dx2 dx0, ds2 = dx0 dx1, dv = dx0 dx1 dx2
    // (uniform_mesh.hpp:33-51), and dtodv = dt / dv (godunov.hpp:31), all in T
    ExactParams<T> p{};
    p.prim = prim;
    p.cons = cons;
    p.g = g;
    p.gamma = gamma;
    p.gm1 = gamma - T(1);
    p.rgm1 = T(1) / p.gm1;
    p.ds0 = dx1 * dx2;
    p.ds1 = dx2 * dx0;
    p.ds2 = dx0 * dx1;
    T const dv = (dx0 * dx1) * dx2;
    p.dtodv = dt / dv;
    constexpr int kBytes = static_cast<int>(sizeof(ExactShared<T>));
    int per_sm = 0;
    cudaError_t const e = resident_ctas<godunov_exact_kernel<T>>(kExNT<T>, kBytes, &per_sm);
    if (e != cudaSuccess) {
        return e;
    }
    // FP64 instructions: about 62 a face, 50 a cell's update, 27 a staged cell,
    // as before its products moved to the integer pipes (134 a cell are left)
    TilePlan plan = choose_tiles(g.n0 - 2, g.n1 - 2, g.n2 - 2, sms, per_sm, 62, 50, 27, 1);
    int const fewest = (g.n1 - 2 + kExTY<T> - 1) / kExTY<T>;
    plan.ny = plan.ny < fewest ? fewest : plan.ny;
    p.sx = split_tiles(g.n0 - 2, plan.nx, 1);
    p.sy = split_tiles(g.n1 - 2, plan.ny, 1);
    int const slots = sms * per_sm;
    p.nwork = plan.nx * plan.ny * (g.n2 - 2);
    if constexpr (sizeof(T) == 4) {
        int const nx = (g.n0 - 2 + kExTX - 1) / kExTX, ny = (g.n1 - 2 + kExTY<T> - 1) / kExTY<T>;
        // about 64 CTAs per SM, so that the last wave is a small part, in
        // chunks of at least 8 planes
        long long const tiles = static_cast<long long>(nx) * ny;
        long long chunks = (64LL * sms + tiles - 1) / tiles;
        chunks = chunks > (g.n2 - 2) / 8 ? (g.n2 - 2) / 8 : chunks;
        if (tiles * chunks >= 4LL * slots && chunks <= 65535) {
            p.sx.parts = nx;
            godunov_exact_whole_kernel<<<dim3(nx * ny, static_cast<unsigned>(chunks)), kExNT<T>, 0, s>>>(p);
            return cudaGetLastError();
        }
    }
    godunov_exact_kernel<T><<<slots < p.nwork ? slots : p.nwork, kExNT<T>, kBytes, s>>>(p);
    return cudaGetLastError();
}

template cudaError_t launch_godunov_exact<double>(CBundle<double>, Bundle<double>, Geom, double, double, double,
                                                  double, double, int, cudaStream_t);
template cudaError_t launch_godunov_exact<float>(CBundle<float>, Bundle<float>, Geom, float, float, float, float,
                                                 float, int, cudaStream_t);

} // namespace eulr
