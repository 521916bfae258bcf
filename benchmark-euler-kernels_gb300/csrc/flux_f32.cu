// The column engine: the FP32 states' fused step, single grid and batch, and
// the per-operator FP32 godunov.  (FP64 runs on the tile engine of flux.cu.)
#include "euler_device.cuh"
#include "kernels.h"
#include "step_common.cuh"

namespace eulr {

namespace {

// ------------------------------------------------- FP32 step, column engine
// The fused step of the FP32 states (cons only in HBM) with a regular
// face-per-thread mapping.  Thread (ti, tj) of a 256-column CTA (32 x 8,
// 16 x 16 or 8 x 32; in a batch 128 columns of 16 x 8 too: tiny and narrow
// grids leave fewer of its threads idle, and a double-float state has four CTAs
// on an SM instead of two) owns the column (i0 + ti, j0 + tj) and marches it up z,
// keeping its cell's primitive state of planes k and k+1 in registers.  Per
// plane it solves
//   x: the face on its cell's left  (the right one is lane+1's, by shuffle;
//      the tile's right boundary faces are solved by the first lanes of one
//      warp, a row each, and read by the rows' last lanes from shared memory:
//      solved in those lanes, each would cost its warp a whole extra HLLC of
//      issue),
//   y: the face below its cell      (the one above is the next row's, through
//      shared memory; the last row also solves the tile's top boundary faces),
//   z: the face above its cell      (both sides in registers; the face below
//      is the previous plane's).
// Shared memory holds two slots of primitive tiles with their halo rings
// (for the y and boundary neighbours): plane k's, read by the faces, and
// plane k+1's, whose halo ring (threads 0..NHALO-1) is staged meanwhile, so that
// no halo conversion stands between a plane's own staging and its barrier.
// The y fluxes and the right boundary fluxes go through shared memory too.
// Cons of plane k+2 (own cell) and k+2 (halo ring) are prefetched with
// cp.async a plane before they are converted; the own cell's stay in a ring
// of three planes for the update, which in registers cost spills.
//
// It is bound by instruction issue.  Measured (one step): compensated state
// 70 Gcell/s at 512^3 and 67 at 256^3, plain 73 and 72, double-float 37 (27
// on the shared-memory tile engine it had before), operator 72 (40 before).
//
// The state is plain FP32 (kCompNone), compensated (kCompSum), or
// double-float (kCompHiLo: a low word per field, which only the update reads;
// it arrives by cp.async while the faces are solved).  The per-operator
// godunov (kCompOperator) stages the caller's prim instead of cons, updates
// the caller's cons in place and computes no wavespeed.
//
// The compensated update rounds once at the scale of the state.  The state
// word is FP32, so its own rounding, 0.5 ulp of cons per step, is the floor
// of the error; what compensation removes is every other rounding at that
// scale.  Per field:
//   * the three flux differences F_low - F_high of the axes, each exact where
//     the two fluxes lie within a factor of two of each other (Sterbenz) and
//     otherwise rounded relative to the difference, not to the fluxes;
//   * their sum (cubic cells: k0 == k1 == k2) times k, with the product's
//     rounding error kept (TwoProduct through one FMA); other cells take
//     each axis's product k_d d_d with its error;
//   * cons + product by Knuth's TwoSum, and the rounding errors of the sum
//     and of the product added back before the one final rounding.
// The plain FP32 state instead subtracts the three axis terms from cons one
// after another: three roundings at the state's scale per step.  Summing the
// six fluxes exactly (TwoSum chains, 46 operations per field instead of 15)
// gave the same 1000-step implosion error (rho L1 1.61e-7 against 1.60e-7 at
// 256^3): the state's own rounding and the FP32 fluxes dominate it.
namespace f32col {

constexpr int kCompOperator = 3; // the per-operator godunov

// A tile of TX columns along x, one per thread of its CTA; a warp holds
// 32 / TX rows of it.
template <int TX_, int NT_ = 256>
struct Tile {
    static constexpr int NT = NT_;
    static constexpr int TX = TX_;
    static constexpr int TY = NT / TX;
    static constexpr int HX = TX + 2;
    static constexpr int HY = TY + 2;
    static constexpr int PLANE = HX * HY;
    static constexpr int NHALO = 2 * TY + 2 * TX; // left, right columns, bottom, top rows
    // The warp whose first TY lanes solve the tile's right boundary x faces:
    // one without halo staging (threads 0..NHALO-1) and other than the top
    // row's warp (which solves the top boundary y faces), so that no warp
    // solves more than one extra face per plane.
    static constexpr int kRightWarp = NT == 256 ? 3 : 2;
    static_assert(kRightWarp * 32 >= NHALO && kRightWarp < NT / 32 - 1 && TY <= 32 && 32 % TX == 0, "right boundary warp");
};

// The fields the engine stages: the state's cons, or the operator's prim.
template <int COMP>
__device__ __forceinline__ CBundle<float> const& staged(FluxParams<float> const& p)
{
    return COMP == kCompOperator ? p.prim : p.cons_in;
}

struct Prim7 {
    float d, p, u[3], c, e; // e: e + p, as the HLLC takes it
};

struct Raw5 {
    float d, e, m[3];
};

__device__ __forceinline__ Side<float> side_of(Prim7 const& q, int dir)
{
    Side<float> s;
    s.d = q.d;
    s.p = q.p;
    s.un = q.u[dir];
    s.ut1 = q.u[(dir + 1) % 3];
    s.ut2 = q.u[(dir + 2) % 3];
    s.c = q.c;
    s.e = q.e;
    return s;
}

// The flux of a face in global components (d, e, m0, m1, m2).
__device__ __forceinline__ void to_global(Flux<float> const& f, int dir, float* g)
{
    g[0] = f.d;
    g[1] = f.e;
    g[2 + dir] = f.n;
    g[2 + (dir + 1) % 3] = f.t1;
    g[2 + (dir + 2) % 3] = f.t2;
}

// Pressure (gamma-1) (e - m.u / 2) of an FP32 conservative cell from its
// velocities u = m / rho: the kinetic energy as m.u instead of |m|^2 / rho
// saves the product by 1/(2 rho).  (Sums of products are written as the fma
// they become here and below, so that every kernel of the engine gives the
// same bits whatever the compiler contracts.)  Compensated states redo the subtraction
// in FP64 where it lost more than 8 bits (pressure_f64_rescue).
template <int COMP>
__device__ __forceinline__ float col_pressure(Raw5 const& r, float u0, float u1, float u2, float ir, float gm1,
                                              const float* lo = nullptr)
{
    float const eint = fmaf(-0.5f, fmaf(r.m[2], u2, fmaf(r.m[1], u1, __fmul_rn(r.m[0], u0))), r.e);
    if (COMP == kCompNone || eint > kLowPressure * r.e) {
        return gm1 * eint;
    }
    return pressure_f64_rescue(r.d, r.e, r.m[0], r.m[1], r.m[2], ir, gm1, COMP == kCompHiLo ? lo : nullptr);
}

// sqrt(x / d) of the per-operator godunov's cells, x = gamma p: x / sqrt(x d)
// from the hardware reciprocal square root and one Newton step, within 1.5
// ulps of the correctly rounded value, where x d is a normal number.  Elsewhere
// that is NaN, and a root and a division answer, out of line so that they cost
// the others only the test (256^3: the operator 2 %):
// x d leaves FP32's range though x / d does not in a dilute gas in CGS units
// (rho 1e-27, p 1e-12), and p = 0 has c = 0.
static __device__ __noinline__ float sound_speed_rare(float x, float d) { return sqrtf(x * (1.0f / d)); }
__device__ __forceinline__ float operator_sound_speed(float x, float d)
{
    float const z = x * d;
    float const y = rsqrt_approx(z);
    float const c = x * fmaf(0.5f * y, fmaf(-z * y, y, 1.0f), y);
    return c == c ? c : sound_speed_rare(x, d);
}

// Primitive state, sound speed and e + p of an FP32 conservative cell.  1/rho
// is the hardware reciprocal (one MUFU.RCP), not the correctly rounded
// sequence: the FP32 step's error budget is set by the state's own rounding,
// and the 1000-step implosion error is the same either way.
template <int COMP>
__device__ __forceinline__ Prim7 prim_of(Raw5 const& r, FluxParams<float> const& p)
{
    Prim7 q;
    if constexpr (COMP == kCompOperator) {
        // r holds prim (d, p, u)
        q.d = r.d;
        q.p = r.e;
        q.u[0] = r.m[0];
        q.u[1] = r.m[1];
        q.u[2] = r.m[2];
        q.c = operator_sound_speed(p.gamma * r.e, r.d);
        float const uu = fmaf(r.m[2], r.m[2], fmaf(r.m[1], r.m[1], __fmul_rn(r.m[0], r.m[0])));
        q.e = __fadd_rn(fmaf(r.e, p.inv_gm1, __fmul_rn(0.5f * r.d, uu)), r.e);
        return q;
    }
    // The double-float state keeps the correctly rounded 1/rho (one FMA pair
    // more): its low words make the conversion's own rounding visible.
    float const ir = COMP == kCompHiLo ? rcp_rn(r.d) : rcp_approx(r.d);
    q.d = r.d;
    q.u[0] = r.m[0] * ir;
    q.u[1] = r.m[1] * ir;
    q.u[2] = r.m[2] * ir;
    q.p = col_pressure<COMP>(r, q.u[0], q.u[1], q.u[2], ir, p.gm1);
    q.c = fast_sound_speed(p.gamma * q.p * ir);
    q.e = __fadd_rn(r.e, q.p);
    return q;
}

// Keeps the compiler from turning field pointer + running offset into a
// running 64-bit pointer per field, which would hold up to 20 registers.
__device__ __forceinline__ void opaque(unsigned& o) { asm("" : "+r"(o)); }
__device__ __forceinline__ void opaque(long long& o) { asm("" : "+l"(o)); }

// Element offset of cell (i, j, k) in the type Off: unsigned (32-bit
// arithmetic, one instruction fewer per address) when the grid has fewer
// than 2^32 cells, long long otherwise.
template <class Off>
__device__ __forceinline__ Off cell_offset(Geom const& g, int i, int j, int k)
{
    return static_cast<Off>(i) + static_cast<Off>(g.s1) * static_cast<Off>(j) +
           static_cast<Off>(g.s2) * static_cast<Off>(k);
}

// A cell past the array's last ghost layer (a tile overhanging the grid)
// takes the state of the nearest ghost cell: physical values, read without a
// branch, and no face that touches such a cell is used.
template <class Off>
__device__ __forceinline__ Off clamped_offset(Geom const& g, int i, int j, int k)
{
    return cell_offset<Off>(g, min(i, g.n0 - 1), min(j, g.n1 - 1), k);
}

template <class Off>
__device__ __forceinline__ Raw5 load_raw(CBundle<float> const& src, Off o)
{
    return Raw5{__ldg(src.f[0] + o), __ldg(src.f[1] + o), {__ldg(src.f[2] + o), __ldg(src.f[3] + o), __ldg(src.f[4] + o)}};
}

// Asynchronous 4-byte global->shared copies (cp.async): the prefetched cons
// of the next planes wait in shared memory instead of registers.
__device__ __forceinline__ void cp_async4(float* dst, const float* src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// All of this thread's copy groups but the last committed one have landed.
__device__ __forceinline__ void cp_async_wait_all_but_last() { asm volatile("cp.async.wait_group 1;" ::: "memory"); }

// Starts copying the fields src of the cell at offset o to dst[f * stride].
template <class Off>
__device__ __forceinline__ void prefetch_raw(float* dst, int stride, CBundle<float> const& src, Off o)
{
#pragma unroll
    for (int f = 0; f < 5; ++f) {
        cp_async4(dst + f * stride, src.f[f] + o);
    }
}

__device__ __forceinline__ void write_raw(float* dst, int stride, Raw5 const& r)
{
    dst[0] = r.d;
    dst[stride] = r.e;
    dst[2 * stride] = r.m[0];
    dst[3 * stride] = r.m[1];
    dst[4 * stride] = r.m[2];
}

__device__ __forceinline__ Raw5 read_raw(float const* src, int stride)
{
    return Raw5{src[0], src[stride], {src[2 * stride], src[3 * stride], src[4 * stride]}};
}

template <class W>
__device__ __forceinline__ void halo_cell(int h, int& hx, int& hy)
{
    constexpr int TX = W::TX, TY = W::TY, HX = W::HX, HY = W::HY;
    if (h < TY) {
        hx = 0;
        hy = 1 + h;
    } else if (h < 2 * TY) {
        hx = HX - 1;
        hy = 1 + h - TY;
    } else if (h < 2 * TY + TX) {
        hx = 1 + h - 2 * TY;
        hy = 0;
    } else {
        hx = 1 + h - 2 * TY - TX;
        hy = HY - 1;
    }
}

// One plane slot: a staged cell is two 16-byte words, (d, p, u0, u1) and
// (u2, c, e + p, -), written and read with two vector accesses (STS.128 and
// LDS.128) instead of seven scalar ones.  Consecutive lanes touch
// consecutive words, so the accesses are free of bank conflicts.
template <class W>
struct SlotPlane {
    float4 a[W::PLANE];
    float4 b[W::PLANE];
};

template <class W>
__device__ __forceinline__ void put(SlotPlane<W>& q, int idx, Prim7 const& v)
{
    q.a[idx] = make_float4(v.d, v.p, v.u[0], v.u[1]);
    q.b[idx] = make_float4(v.u[2], v.c, v.e, v.e);
}

template <class W>
__device__ __forceinline__ Prim7 get(SlotPlane<W> const& q, int idx)
{
    float4 const a = q.a[idx];
    float4 const b = q.b[idx];
    Prim7 v;
    v.d = a.x;
    v.p = a.y;
    v.u[0] = a.z;
    v.u[1] = a.w;
    v.u[2] = b.x;
    v.c = b.y;
    v.e = b.z;
    return v;
}

// Five flux components through shared memory as one 16-byte word and one
// 4-byte word.
__device__ __forceinline__ void put_flux(float4* a, float* b, int idx, float const* f)
{
    a[idx] = make_float4(f[0], f[1], f[2], f[3]);
    b[idx] = f[4];
}

__device__ __forceinline__ void get_flux(float4 const* a, float const* b, int idx, float* f)
{
    float4 const v = a[idx];
    f[0] = v.x;
    f[1] = v.y;
    f[2] = v.z;
    f[3] = v.w;
    f[4] = b[idx];
}

// ---- paired FP32 arithmetic: on sm_100 and later, FADD2/FMUL2/FFMA2
// carry two FP32 operations per issued instruction, each rounded once.  The
// step is bound by instruction issue, so the compensated update of fields
// (d, e) and (m0, m1) runs in pairs (the same operations, the same bits).

// a - b, rounded once (b * -1 is exact)
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }

// The compensated update of two fields of a cubic cell: u + k (flux balance)
// with one rounding at the state's scale, operation for operation the scalar
// form below.  nk = -k gives the product's rounding error negated,
// P - k S, which the last step subtracts.
__device__ __forceinline__ float2 comp_update2(float2 u, float2 xl, float2 xr, float2 yb, float2 yt, float2 zl, float2 zh,
                                               float2 k, float2 nk)
{
    float2 const S = __fadd2_rn(__fadd2_rn(sub2(xl, xr), sub2(yb, yt)), sub2(zl, zh));
    float2 const P = __fmul2_rn(k, S);
    float2 const nP = __ffma2_rn(nk, S, P);
    float2 const s = __fadd2_rn(u, P);
    float2 const bb = sub2(s, u);
    float2 const err = __fadd2_rn(sub2(u, sub2(s, bb)), sub2(P, bb));
    return __fadd2_rn(s, sub2(err, nP));
}

// The double-float update of two fields: u + lo plus the six signed face
// terms, accumulated without rounding error in any product (TwoProduct) or
// running sum (TwoSum), the errors collected in lo; then one rounding of each
// word.  compensated_add's operations on two fields at once.
__device__ __forceinline__ void comp_add2(float2& sum, float2& err, float2 k, float2 nk, float2 f)
{
    float2 const prod = __fmul2_rn(k, f);
    float2 const nprod_err = __ffma2_rn(nk, f, prod); // -(k f - prod)
    float2 const s = __fadd2_rn(sum, prod);
    float2 const bb = sub2(s, sum);
    float2 const sum_err = __fadd2_rn(sub2(sum, sub2(s, bb)), sub2(prod, bb));
    sum = s;
    err = __fadd2_rn(err, sub2(sum_err, nprod_err));
}

__device__ __forceinline__ void hilo_update2(float2& u, float2& lo, float2 xl, float2 xr, float2 yb, float2 yt, float2 zl,
                                             float2 zh, float k0, float k1, float k2)
{
    float2 const p0 = make_float2(k0, k0), n0 = make_float2(-k0, -k0);
    float2 const p1 = make_float2(k1, k1), n1 = make_float2(-k1, -k1);
    float2 const p2 = make_float2(k2, k2), n2 = make_float2(-k2, -k2);
    float2 sum = u;
    float2 err = lo;
    comp_add2(sum, err, n0, p0, xr);
    comp_add2(sum, err, p0, n0, xl);
    comp_add2(sum, err, n1, p1, yt);
    comp_add2(sum, err, p1, n1, yb);
    comp_add2(sum, err, n2, p2, zh);
    comp_add2(sum, err, p2, n2, zl);
    u = __fadd2_rn(sum, err);
    lo = sub2(err, sub2(u, sum));
}

template <int COMP, class W>
struct ColShared {
    static constexpr int NT = W::NT, TY = W::TY, NHALO = W::NHALO;
    SlotPlane<W> slot[2];
    float4 yflux_a[NT]; // the y face below each cell
    float yflux_b[NT];
    float4 xflux_ra[TY]; // the tile's right boundary x faces
    float xflux_rb[TY];
    float raw_own[3][5 * NT];  // own column's staged fields: planes k, k+1, k+2 in turn
    float raw_halo[5 * NHALO]; // halo ring, one plane ahead
    float raw_lo[COMP == kCompHiLo ? 5 * NT : 1]; // own column's low words of the current plane
    long long warp_best[NT / 32];
    int any_bad;
};

// One work item: interior planes [kb, ke) of the column tile (tx, ty), with
// update coefficients k0..k2 (UNIFORM: cubic cells, k0..k2 all equal and
// 1/dx_d too).  BRANCHED: the cell update sits inside the
// interior test (the batch) rather than beside it (the single grid).
// Accumulates this thread's max wavespeed and non-physical flag.
template <int COMP, class W, bool UNIFORM, class Off, bool BRANCHED>
__device__ __forceinline__ void col_item(FluxParams<float> const& p, float k0, float k1, float k2, int tx, int ty,
                                         int kb, int ke, ColShared<COMP, W>& sh, float& wmaxf, bool& bad)
{
    constexpr int NT = W::NT, TX = W::TX, TY = W::TY, HX = W::HX, NHALO = W::NHALO;
    constexpr int kRightWarp = W::kRightWarp;
    CBundle<float> const& src = staged<COMP>(p);
    int const tid = threadIdx.x;
    int const ti = tid % TX;
    int const tj = tid / TX;
    int const own_idx = (tj + 1) * HX + ti + 1;
    int const i0 = 1 + tx * TX;
    int const j0 = 1 + ty * TY;
    bool const own = (i0 + ti < p.g.n0 - 1) && (j0 + tj < p.g.n1 - 1);
    // offsets of the thread's own cell and of its halo cell, kept running
    // from plane to plane
    Off const s2 = static_cast<Off>(p.g.s2);
    Off o = clamped_offset<Off>(p.g, i0 + ti, j0 + tj, kb);
    Off ho = 0;
    int halo_idx = 0;
    if (tid < NHALO) {
        int hx, hy;
        halo_cell<W>(tid, hx, hy);
        halo_idx = hy * HX + hx;
        ho = clamped_offset<Off>(p.g, i0 - 1 + hx, j0 - 1 + hy, kb);
    }

    // prologue: plane kb of the halo ring staged, kb+1 on its way; planes
    // kb-1 (z face below), kb, kb+1 of the own column
    if (tid < NHALO) {
        prefetch_raw(sh.raw_halo + tid, NHALO, src, ho);
        cp_async_wait_all();
        put(sh.slot[0], halo_idx, prim_of<COMP>(read_raw(sh.raw_halo + tid, NHALO), p));
        ho += s2;
        if (kb + 1 < ke) {
            prefetch_raw(sh.raw_halo + tid, NHALO, src, ho);
        }
    }
    cp_async_commit();
    Raw5 const rb = load_raw(src, o - s2);
    Raw5 const r0 = load_raw(src, o);
    Raw5 const r1 = load_raw(src, o + s2); // kb + 1 <= ke <= n2 - 1
    if constexpr (COMP != kCompOperator) {
        write_raw(sh.raw_own[0] + tid, NT, r0);
        write_raw(sh.raw_own[1] + tid, NT, r1);
    }
    Prim7 q0 = prim_of<COMP>(r0, p);
    Prim7 q1 = prim_of<COMP>(r1, p);
    float* raw_k = sh.raw_own[0] + tid; // this thread's words of plane k, and of plane k+2
    float* raw_n = sh.raw_own[2] + tid;
    float zlo[5];
    to_global(hllc_flux(side_of(prim_of<COMP>(rb, p), 2), side_of(q0, 2)), 2, zlo);

    // Unrolled twice: the plane-to-plane register rotation (q0 <- q1,
    // zlo <- fzh) becomes renaming instead of moves, and the slot of each
    // copy is a constant.
#pragma unroll 2
    for (int k = kb; k < ke; ++k) {
        SlotPlane<W>& q = sh.slot[(k - kb) & 1];
        // stage plane k: the own cell (its halo ring was staged a plane ahead)
        put(q, own_idx, q0);
        // own column plane k+2, consumed at the end of this plane
        if (k + 2 <= ke) {
            prefetch_raw(raw_n, NT, src, o + 2 * s2);
        }
        if constexpr (COMP == kCompHiLo) { // and the low words of plane k, consumed by this plane's update
            prefetch_raw(sh.raw_lo + tid, NT, p.lo_in, o);
        }
        float cons[5]; // the operator's cons, in flight while the faces are solved
        if (COMP == kCompOperator && own) {
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                cons[f] = p.cons_in.f[f][o];
            }
        }
        cp_async_commit();
        __syncthreads(); // plane k staged
        // the halo ring of plane k+1 into the other slot, off the path to the
        // barrier above (the slot's last reader finished before the previous
        // plane's second barrier)
        if (tid < NHALO && k + 1 < ke) {
            cp_async_wait_all_but_last(); // the halo copies of plane k+1 landed (own k+2 may be in flight)
            put(sh.slot[(k + 1 - kb) & 1], halo_idx, prim_of<COMP>(read_raw(sh.raw_halo + tid, NHALO), p));
            ho += s2;
            opaque(ho);
            if (k + 2 < ke) {
                prefetch_raw(sh.raw_halo + tid, NHALO, src, ho);
            }
        }
        cp_async_commit();

        // ---- faces
        float fxl[5], fyb[5], fzh[5], fxr[5], fyt[5];
        {
            float t[5];
            to_global(hllc_flux(side_of(get(q, own_idx - HX), 1), side_of(q0, 1)), 1, t);
            put_flux(sh.yflux_a, sh.yflux_b, tid, t); // read back after the barrier (registers are scarce here)
        }
        to_global(hllc_flux(side_of(get(q, own_idx - 1), 0), side_of(q0, 0)), 0, fxl);
        to_global(hllc_flux(side_of(q0, 2), side_of(q1, 2)), 2, fzh);
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            fxr[f] = __shfl_down_sync(0xffffffffu, fxl[f], 1);
        }
        int const lane = tid % 32;
        if (tid / 32 == kRightWarp && lane < TY) { // the tile's right boundary faces, one per row
            int const c = (lane + 1) * HX + TX;
            float t[5];
            to_global(hllc_flux(side_of(get(q, c), 0), side_of(get(q, c + 1), 0)), 0, t);
            put_flux(sh.xflux_ra, sh.xflux_rb, lane, t);
        }
        if (tj == TY - 1) { // the tile's top boundary faces
            to_global(hllc_flux(side_of(q0, 1), side_of(get(q, own_idx + HX), 1)), 1, fyt);
        }
        __syncthreads(); // y fluxes and right boundary fluxes written
        get_flux(sh.yflux_a, sh.yflux_b, tid, fyb);
        if (tj < TY - 1) {
            get_flux(sh.yflux_a, sh.yflux_b, tid + TX, fyt);
        }
        {
            float xr[5];
            get_flux(sh.xflux_ra, sh.xflux_rb, tj, xr); // one broadcast read per row
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                fxr[f] = ti == TX - 1 ? xr[f] : fxr[f];
            }
        }

        // ---- update of the own cell.  In the single-grid step every lane
        // computes it (a lane off the interior holds physical values of
        // clamped cells) and only the stores and the wavespeed are the
        // interior's, so no branch encloses the arithmetic (+1 %); the batch,
        // whose tiles overhang its small grids more often, keeps the branch
        // (measured 4 % faster there).
        if (!BRANCHED || own) {
            float u[5];
            float lo[COMP == kCompHiLo ? 5 : 1];
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                u[f] = COMP == kCompOperator ? cons[f] : raw_k[f * NT];
            }
            if constexpr (COMP == kCompHiLo) {
                cp_async_wait_all_but_last(); // the low words of plane k landed (and own k+2)
                Raw5 const rl = read_raw(sh.raw_lo + tid, NT);
                lo[0] = rl.d;
                lo[1] = rl.e;
                lo[2] = rl.m[0];
                lo[3] = rl.m[1];
                lo[4] = rl.m[2];
#pragma unroll
                for (int f = 0; f < 5; f += 2) { // (d, e), (m0, m1), (m2, -)
                    int const h = f + 1 < 5 ? f + 1 : f;
                    float2 uu = make_float2(u[f], u[h]), ll = make_float2(lo[f], lo[h]);
                    hilo_update2(uu, ll, make_float2(fxl[f], fxl[h]), make_float2(fxr[f], fxr[h]),
                                 make_float2(fyb[f], fyb[h]), make_float2(fyt[f], fyt[h]), make_float2(zlo[f], zlo[h]),
                                 make_float2(fzh[f], fzh[h]), k0, k1, k2);
                    u[f] = uu.x;
                    lo[f] = ll.x;
                    if (h != f) {
                        u[h] = uu.y;
                        lo[h] = ll.y;
                    }
                }
            }
            constexpr bool kPaired = COMP == kCompSum && UNIFORM;
            if (kPaired) { // fields (d, e) and (m0, m1) in pairs, m2 below
                float2 const kk = make_float2(k0, k0), nk = make_float2(-k0, -k0);
#pragma unroll
                for (int f = 0; f < 4; f += 2) {
                    float2 const r = comp_update2(make_float2(u[f], u[f + 1]), make_float2(fxl[f], fxl[f + 1]),
                                                  make_float2(fxr[f], fxr[f + 1]), make_float2(fyb[f], fyb[f + 1]),
                                                  make_float2(fyt[f], fyt[f + 1]), make_float2(zlo[f], zlo[f + 1]),
                                                  make_float2(fzh[f], fzh[f + 1]), kk, nk);
                    u[f] = r.x;
                    u[f + 1] = r.y;
                }
            }
#pragma unroll
            for (int f = COMP == kCompHiLo ? 5 : (kPaired ? 4 : 0); f < 5; ++f) {
                if (COMP == kCompNone || COMP == kCompOperator) {
                    u[f] = fmaf(-k2, __fsub_rn(fzh[f], zlo[f]),
                                fmaf(-k1, __fsub_rn(fyt[f], fyb[f]), fmaf(-k0, __fsub_rn(fxr[f], fxl[f]), u[f])));
                } else if (UNIFORM) {
                    // _rn intrinsics: no product may be fused into the sums
                    // the TwoSum and TwoProduct take apart
                    float const S = __fadd_rn(__fadd_rn(__fsub_rn(fxl[f], fxr[f]), __fsub_rn(fyb[f], fyt[f])),
                                              __fsub_rn(zlo[f], fzh[f]));
                    float const P = __fmul_rn(k0, S);
                    float const eP = fmaf(k0, S, -P);
                    float const s = __fadd_rn(u[f], P);
                    float const bb = __fsub_rn(s, u[f]);
                    float const err = __fadd_rn(__fsub_rn(u[f], __fsub_rn(s, bb)), __fsub_rn(P, bb));
                    u[f] = __fadd_rn(s, __fadd_rn(err, eP));
                } else {
                    float const d0 = __fsub_rn(fxl[f], fxr[f]);
                    float const d1 = __fsub_rn(fyb[f], fyt[f]);
                    float const d2 = __fsub_rn(zlo[f], fzh[f]);
                    float const P0 = __fmul_rn(k0, d0), P1 = __fmul_rn(k1, d1), P2 = __fmul_rn(k2, d2);
                    float const eP = __fadd_rn(__fadd_rn(fmaf(k0, d0, -P0), fmaf(k1, d1, -P1)), fmaf(k2, d2, -P2));
                    float const P = __fadd_rn(__fadd_rn(P0, P1), P2);
                    float const s = __fadd_rn(u[f], P);
                    float const bb = __fsub_rn(s, u[f]);
                    float const err = __fadd_rn(__fsub_rn(u[f], __fsub_rn(s, bb)), __fsub_rn(P, bb));
                    u[f] = __fadd_rn(s, __fadd_rn(err, eP));
                }
            }
            if (own) {
#pragma unroll
                for (int f = 0; f < 5; ++f) {
                    p.cons_out.f[f][o] = u[f];
                    if (COMP == kCompHiLo) {
                        p.lo_out.f[f][o] = lo[f];
                    }
                }
            }
            if constexpr (COMP != kCompOperator) {
            // next step's CFL wavespeed of the new state (time_step.hpp:28-33);
            // on cubic cells (3 cs + |v0| + |v1| + |v2|) / dx, one product
            Raw5 const nr{u[0], u[1], {u[2], u[3], u[4]}};
            float const r = COMP == kCompHiLo ? rcp_rn(u[0]) : rcp_approx(u[0]);
            float const v0 = u[2] * r, v1 = u[3] * r, v2 = u[4] * r;
            float const pr = col_pressure<COMP>(nr, v0, v1, v2, r, p.gm1, lo);
            float const cs = fast_sound_speed((p.gamma * r) * pr);
            float const invdt =
                    UNIFORM ? __fmul_rn(__fadd_rn(__fadd_rn(fmaf(3.0f, cs, fabsf(v0)), fabsf(v1)), fabsf(v2)), p.invdx0)
                            : fmaf(__fadd_rn(cs, fabsf(v2)), p.invdx2,
                                   fmaf(__fadd_rn(cs, fabsf(v1)), p.invdx1, __fmul_rn(__fadd_rn(cs, fabsf(v0)), p.invdx0)));
            wmaxf = own ? fmaxf(wmaxf, invdt) : wmaxf; // NaN never wins
            bad |= own && !cell_ok(u[0], pr, invdt);
            }
        }
        // march: plane k+1 becomes the current plane
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            zlo[f] = fzh[f];
        }
        q0 = q1;
        if (k + 2 <= ke) {
            cp_async_wait_all_but_last(); // the own copies of plane k+2 landed
            q1 = prim_of<COMP>(read_raw(raw_n, NT), p);
        }
        // the slots in turn: k <- k+1, k+1 <- k+2, and plane k's is free
        float* const end = sh.raw_own[2] + tid;
        raw_n = raw_k;
        raw_k = raw_k == end ? sh.raw_own[0] + tid : raw_k + 5 * NT;
        o += s2;
        opaque(o);
    }
    __syncthreads(); // the slots are restaged by the next item
}

// Block max of the threads' wavespeeds into *wmax (ordered bits, one
// atomicMax per CTA) and the non-physical flag into *status; clears both.
template <int COMP, class W>
__device__ __forceinline__ void col_flush(ColShared<COMP, W>& sh, float& wmaxf, bool& bad, unsigned long long* wmax,
                                          int* status)
{
    constexpr int NT = W::NT;
    int const tid = threadIdx.x;
    long long wk = wave_key(wmaxf);
#pragma unroll
    for (int s = 16; s > 0; s >>= 1) {
        long long const v = __shfl_xor_sync(0xffffffffu, wk, s);
        wk = v > wk ? v : wk;
    }
    __syncthreads();
    if (tid == 0) {
        sh.any_bad = 0;
    }
    __syncthreads();
    if (tid % 32 == 0) {
        sh.warp_best[tid / 32] = wk;
    }
    if (bad) {
        sh.any_bad = 1;
    }
    __syncthreads();
    if (tid == 0) {
        long long b = sh.warp_best[0];
#pragma unroll
        for (int v = 1; v < NT / 32; ++v) {
            b = sh.warp_best[v] > b ? sh.warp_best[v] : b;
        }
        atomicMax(wmax, static_cast<unsigned long long>(b));
        if (sh.any_bad) {
            atomicOr(status, 1);
        }
    }
    wmaxf = 0.0f;
    bad = false;
}

// CTAs per SM the registers are cut for.
template <int COMP, class W>
constexpr int kColPerSM = (COMP == kCompHiLo ? 512 : 768) / W::NT;

// One launch over a single grid: the fused step, or the operator.
template <int COMP, class W, bool UNIFORM, class Off>
__global__ void __launch_bounds__(W::NT, kColPerSM<COMP, W>) f32_step_kernel(const __grid_constant__ FluxParams<float> p)
{
    __shared__ __align__(16) ColShared<COMP, W> sh;
    float const dtodv = dt_over_dv(p);
    float const k0 = dtodv * p.ds0, k1 = dtodv * p.ds1, k2 = dtodv * p.ds2; // UNIFORM: all equal
    float wmaxf = 0.0f;
    bool bad = false;
    // (chunk, tile) items, tiles fastest: the CTAs at work at one time hold
    // neighbouring tiles of one chunk, whose halos they share in L2.  The
    // chunks (p.kchunk of them) are even to a plane.
    int const iz = p.g.n2 - 2;
    int const tiles = p.tiles_x * p.tiles_y;
    for (int w = blockIdx.x; w < p.nwork; w += gridDim.x) {
        int const chunk = w / tiles;
        int const tile = w - chunk * tiles;
        int const kb = 1 + static_cast<int>(static_cast<long long>(chunk) * iz / p.kchunk);
        int const ke = 1 + static_cast<int>(static_cast<long long>(chunk + 1) * iz / p.kchunk);
        col_item<COMP, W, UNIFORM, Off, false>(p, k0, k1, k2, tile % p.tiles_x, tile / p.tiles_x, kb, ke, sh, wmaxf, bad);
    }
    if constexpr (COMP != kCompOperator) {
        col_flush(sh, wmaxf, bad, p.wmax, p.status);
        step_done(p);
    }
}

// The column engine over a batch: CTAs pop (grid, tile x, tile y, chunk)
// items from the queue, as flux_batch_kernel does; each item's wavespeed goes
// to its own grid.  Grids of cubic cells take the cubic update and wavespeed.
template <int COMP, class W, class Off>
__global__ void __launch_bounds__(W::NT, kColPerSM<COMP, W>) f32_batch_kernel(const __grid_constant__ BatchParams<float> b)
{
    static_assert(sizeof(FluxParams<float>) % 4 == 0, "parameter copy in 4-byte words");
    __shared__ __align__(16) ColShared<COMP, W> sh;
    __shared__ __align__(16) FluxParams<float> gp;
    __shared__ int s_item;
    int const tid = threadIdx.x;
    float wmaxf = 0.0f;
    bool bad = false;
    for (;;) {
        __syncthreads(); // everyone is done with the previous item's parameters
        if (tid == 0) {
            s_item = static_cast<int>(atomicAdd(b.head, 1u));
        }
        __syncthreads();
        int const item = s_item;
        if (item >= b.nitems) {
            break;
        }
        int4 const it = b.items[item];
        for (int w = tid; w < static_cast<int>(sizeof(FluxParams<float>) / 4); w += W::NT) {
            reinterpret_cast<int*>(&gp)[w] = reinterpret_cast<const int*>(&b.grids[it.x])[w];
        }
        __syncthreads();
        float const dtodv = dt_over_dv(gp);
        float const k0 = dtodv * gp.ds0, k1 = dtodv * gp.ds1, k2 = dtodv * gp.ds2;
        int const kb = 1 + it.w * gp.kchunk;
        int const ke = min(kb + gp.kchunk, gp.g.n2 - 1);
        if (gp.ds0 == gp.ds1 && gp.ds1 == gp.ds2 && gp.invdx0 == gp.invdx1 && gp.invdx1 == gp.invdx2) {
            col_item<COMP, W, true, Off, true>(gp, k0, k1, k2, it.y, it.z, kb, ke, sh, wmaxf, bad);
        } else {
            col_item<COMP, W, false, Off, true>(gp, k0, k1, k2, it.y, it.z, kb, ke, sh, wmaxf, bad);
        }
        col_flush(sh, wmaxf, bad, gp.wmax, gp.status);
        item_done(gp);
    }
    batch_cta_done(b);
}

} // namespace f32col

// Grids up to this many cells index their fields with 32-bit offsets.
constexpr long long kNarrowCells = 0xffffffffLL;

template <int COMP>
cudaError_t configure_f32col(int* per_sm)
{
    return resident_ctas<f32col::f32_step_kernel<COMP, f32col::Tile<32>, false, long long>>(256, 0, per_sm);
}

// Tile width and chunks of planes of a single-grid launch.
// Width: the fewest tiles, a 16-column tile counted 2 % and an 8-column one
// 12 % dearer than a 32-column one (measured at 512^3: -2 to 8 % and 10 to
// 15 %), and 32-column tiles 6 % dearer where they leave a remainder (200^3,
// compensated state: 166 us a step in 32-wide tiles, 142 in 16-wide).
// Chunks: the least time of the busiest SM.  n items over its CTA slots are
// q full rounds and a rest of k items an SM.  A full round costs as many items'
// time as the SM has slots.  The rest costs what kRest says: less than a full
// round, but more than in proportion, as fewer CTAs hide less of each other's
// waits; after two full rounds the CTAs are out of step and most of a single
// item is hidden.  An item costs a plane besides its own (the z face and the
// two planes below it), and 2 % more per 64 planes beyond 64: neighbouring CTAs
// drift apart and lose the halos they share in L2.  Fitted to 10 to 30 counts
// of chunks on each of 43 grids of 38^3 to 512^3 and three states, where it is
// on average 1.6 % (plain and compensated) and 3.4 % (double-float) above the
// best count; the items of the busiest SM alone, each as dear, gave 4.9 and
// 6.9 %.  Plain state: 224^3 186 -> 169 us a step, 320^3 508 -> 470,
// 1024 x 32^2 25.7 -> 24.5.
struct ColPlan {
    int width, chunks;
};

ColPlan choose_columns(int ix, int iy, int iz, int sms, int per_sm)
{
    ColPlan best{32, 1};
    double least = 1e300;
    long long tiles = 1;
    for (int tx : {32, 16, 8}) {
        int const ty = 256 / tx;
        long long const n = static_cast<long long>((ix + tx - 1) / tx) * ((iy + ty - 1) / ty);
        double const cost = n * (tx == 32 ? (ix % 32 == 0 ? 1.0 : 1.06) : (tx == 16 ? 1.02 : 1.12));
        if (cost < least) {
            least = cost;
            best.width = tx;
            tiles = n;
        }
    }
    // time of a rest of k items an SM after 0, 1 and more full rounds, in 0.01 items
    constexpr int kRest2[3][3] = {{0, 110, 200}, {0, 120, 200}, {0, 90, 200}};
    constexpr int kRest3[3][4] = {{0, 130, 215, 300}, {0, 150, 250, 300}, {0, 90, 220, 300}};
    long long const slots = static_cast<long long>(sms) * per_sm;
    long long least_time = 0x7fffffffffffffffLL;
    for (int planes = iz < 128 ? iz : 128; planes >= 1; --planes) {
        int const c = (iz + planes - 1) / planes;
        long long const q = tiles * c / slots;
        int const k = static_cast<int>((tiles * c - q * slots + sms - 1) / sms);
        int const after = q < 2 ? static_cast<int>(q) : 2;
        int const rest = per_sm == 2 ? kRest2[after][k] : (per_sm == 3 ? kRest3[after][k] : 100 * k);
        int const longest = (iz + c - 1) / c;
        long long const time =
                (100 * per_sm * q + rest) * (longest + 1) * (3200 + (longest > 64 ? longest - 64 : 0));
        if (time < least_time) {
            least_time = time;
            best.chunks = c;
        }
    }
    return best;
}

template <int COMP, class W, class Off>
cudaError_t launch_f32col_as(FluxParams<float> p, int chunks, int sms, cudaStream_t s)
{
    int const per_sm = p.per_sm > 0 ? p.per_sm : 1;
    int const ix = p.g.n0 - 2;
    int const iy = p.g.n1 - 2;
    p.tiles_x = (ix + W::TX - 1) / W::TX;
    p.tiles_y = (iy + W::TY - 1) / W::TY;
    long long const slots = static_cast<long long>(sms) * per_sm;
    p.kchunk = chunks;
    p.nwork = p.tiles_x * p.tiles_y * chunks;
    int const grid = static_cast<int>(slots < p.nwork ? slots : p.nwork);
    // cubic cells: equal face areas give equal update coefficients dt/dv * ds_d,
    // and equal 1/dx_d the one-product wavespeed
    if (p.ds0 == p.ds1 && p.ds1 == p.ds2 && p.invdx0 == p.invdx1 && p.invdx1 == p.invdx2) {
        f32col::f32_step_kernel<COMP, W, true, Off><<<grid, W::NT, 0, s>>>(p);
    } else {
        f32col::f32_step_kernel<COMP, W, false, Off><<<grid, W::NT, 0, s>>>(p);
    }
    return cudaGetLastError();
}

template <int COMP>
cudaError_t launch_f32col(FluxParams<float> const& p, int sms, cudaStream_t s)
{
    if (p.g.n0 <= 2 || p.g.n1 <= 2 || p.g.n2 <= 2) {
        return cudaSuccess; // no interior cell
    }
    ColPlan const plan = choose_columns(p.g.n0 - 2, p.g.n1 - 2, p.g.n2 - 2, sms, p.per_sm > 0 ? p.per_sm : 1);
    if (p.g.ncell() > kNarrowCells) { // 64-bit offsets are built for one width
        return launch_f32col_as<COMP, f32col::Tile<32>, long long>(p, plan.chunks, sms, s);
    }
    switch (plan.width) {
    case 8: return launch_f32col_as<COMP, f32col::Tile<8>, unsigned>(p, plan.chunks, sms, s);
    case 16: return launch_f32col_as<COMP, f32col::Tile<16>, unsigned>(p, plan.chunks, sms, s);
    default: return launch_f32col_as<COMP, f32col::Tile<32>, unsigned>(p, plan.chunks, sms, s);
    }
}

// The column engine as the shapes of the FP32 batch.
template <int COMP, class W>
struct ColBatchKernel {
    static cudaError_t run(BatchParams<float> const* b, int grid, int* per_sm, cudaStream_t s)
    {
        if (b == nullptr) {
            int n = 0;
            cudaError_t const e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                    &n, f32col::f32_batch_kernel<COMP, W, long long>, W::NT, 0);
            *per_sm = n < 1 ? 1 : n;
            return e;
        }
        if (b->max_cells <= kNarrowCells) {
            f32col::f32_batch_kernel<COMP, W, unsigned><<<grid, W::NT, 0, s>>>(*b);
        } else {
            f32col::f32_batch_kernel<COMP, W, long long><<<grid, W::NT, 0, s>>>(*b);
        }
        return cudaGetLastError();
    }
};

} // namespace

cudaError_t configure_step_f32col(int comp, int* per_sm)
{
    switch (comp) {
    case kCompSum: return configure_f32col<kCompSum>(per_sm);
    case kCompHiLo: return configure_f32col<kCompHiLo>(per_sm);
    default: return configure_f32col<kCompNone>(per_sm);
    }
}

cudaError_t launch_step_f32col(FluxParams<float> const& p, int comp, int sms, cudaStream_t s)
{
    switch (comp) {
    case kCompSum: return launch_f32col<kCompSum>(p, sms, s);
    case kCompHiLo: return launch_f32col<kCompHiLo>(p, sms, s);
    default: return launch_f32col<kCompNone>(p, sms, s);
    }
}

cudaError_t launch_godunov_f32(FluxParams<float> const& p, int sms, cudaStream_t s)
{
    FluxParams<float> q = p;
    cudaError_t const e = configure_f32col<f32col::kCompOperator>(&q.per_sm);
    return e != cudaSuccess ? e : launch_f32col<f32col::kCompOperator>(q, sms, s);
}

template <int COMP>
static cudaError_t run_batch_f32col(int tx, int ty, BatchParams<float> const* b, int grid, int* per_sm, cudaStream_t s)
{
    if (tx * ty == 128) {
        return ColBatchKernel<COMP, f32col::Tile<16, 128>>::run(b, grid, per_sm, s);
    }
    return tx == 32 ? ColBatchKernel<COMP, f32col::Tile<32>>::run(b, grid, per_sm, s)
                    : ColBatchKernel<COMP, f32col::Tile<16>>::run(b, grid, per_sm, s);
}

cudaError_t launch_batch_f32col(int comp, int tx, int ty, BatchParams<float> const* b, int grid, int* per_sm, cudaStream_t s)
{
    switch (comp) {
    case kCompSum: return run_batch_f32col<kCompSum>(tx, ty, b, grid, per_sm, s);
    case kCompHiLo: return run_batch_f32col<kCompHiLo>(tx, ty, b, grid, per_sm, s);
    default: return run_batch_f32col<kCompNone>(tx, ty, b, grid, per_sm, s);
    }
}

} // namespace eulr
