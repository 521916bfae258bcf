// FP64 Godunov/HLLC flux kernels (sm_103a): the per-operator godunov and the
// fused simulation step share one z-marching tile engine.  (The FP32 ones run
// on the column engine of flux_f32.cu.)
//
// Work decomposition: the interior [1,n0-1) x [1,n1-1) x [1,n2-1) is cut into
// tiles of at most TX x TY columns, of even size.  Single grid: their extent
// is chosen for the grid (choose_tiles), and all tiles' planes are divided
// evenly among a resident grid of CTAs, a run of planes each.  Batch: chunks
// of planes popped from a queue.  A CTA marches up its run one plane at a
// time through a ring of plane slots in shared memory, each slot holding ten
// values (d, p, u0, u1, u2, c, e + p, m0, m1, m2) of a (TX+2) x (TY+2) plane
// with its one-cell halo.  Per plane:
//   1. face phase -- every x face and y face of plane k and every z face
//      between planes k and k+1 is solved ONCE (the reference solves each
//      interior face twice, once from each side, godunov.hpp:48-82).  The
//      FP64 pipe is the bound: the x, y and z faces share one index space
//      of exactly the tile's faces, and each face's family, cells and axis
//      are chosen by selects, so a warp whose lanes straddle two families
//      still runs the HLLC once -- the 800 faces of a 16x16 tile take exactly
//      25 warp-passes.  Three numbers a face go to shared memory
//      (hllc_upwind), b scaled by the ratio of the face's area to an x
//      face's where the areas differ;
//   2. cell phase -- each thread owns one column cell and forms div F of its
//      six faces, each term b times d, m or h of the face's upwind side, read
//      from the slots; then cons -= dt/dv ds_0 div F (godunov.hpp:84-90), one
//      rounding at the state's scale.  What the z face below the cell carries
//      stays in registers from the previous plane.
// Forming all five fluxes at the face took 27 FP64 operations a face and 30 a
// cell's update; this takes 22 and 32, with m staged besides u (loading 512^3
// and 4 steps: 141.0 -> 133.7 ms; the rounding error of a step 0.6 of the
// other form's against quadruple precision, 1.0 where pressure outweighs
// momentum).  That filled the FP64 pipe (553 G instructions/s of about 560)
// with 85 % of the issue slots idle, so products, reciprocals, square roots
// and the sum of the densities run on the integer pipes (mul_alu, rcp_alu,
// sqrt_alu, add_alu): 11 FP64 instructions stay of a face's 22 and seed, 34 of
// a cell's 51 and two seeds.  With three CTAs on an SM (two plane slots, 80
// registers) and kernels that know their mesh, a step of 512^3 takes 19.2 ms
// where it took 31.0, the operator godunov 21.1 where it took 31.6.
// The fused step then finishes the cell on chip: cons_to_prim, sound speed
// and the next step's CFL max-wavespeed, reduced warp -> block -> one
// atomicMax per CTA, so dt never leaves the device.
//
// Staging: the ten fields of a plane slot are fetched into a ring of two
// slots by TMA (cp.async.bulk.tensor, one 18x18x1 box per field, each slot
// completing on its own mbarrier) where the row pitch is a multiple of 16
// bytes, else and in the batch by 8-byte cp.async (20 steps of a
// 99 x 128 x 75 grid, odd pitch: 7.0 -> 5.9 ms against synchronous loads and
// whole tiles).  A slot is refilled once its plane's cell phase is over, and
// waited for before the next plane's first pass with z faces; the SM's other
// CTAs cover what is left of the wait.  (Three slots leave room for two CTAs:
// the same time a 512^3 step, 3.5 % more for 24 batched grids.)  The
// per-operator godunov, and the first step of a state whose cons the caller
// gave besides prim (its momenta need not be d u), copy what is stored the
// same way and compute the rest in place.  Every mbarrier wait is bounded: a
// wait that runs out sets bit 1 of the status word, waits (bounded) for the
// copies still in flight and ends the CTA.
#include "euler_device.cuh"
#include "kernels.h"
#include "step_common.cuh"

#include <algorithm>
#include <cfloat>

namespace eulr {

namespace {

constexpr int kWaitTries = 1 << 20; // mbarrier.try_wait attempts before giving up

// How a plane slot is filled.
enum Staging {
    kStageTma,   // fused FP64 step, row pitch a multiple of 16 bytes: TMA boxes
    kStageAsync, // fused FP64 step, any pitch, and the batch: 8-byte cp.async
    kStageDerive, // only prim is stored (per-operator godunov, FluxParams::own_momenta): cp.async, the rest computed
};
constexpr int kSlots = 2; // plane slots of the ring

// What a kernel knows of its mesh.  Code for the other kind of mesh is short
// and FP64: kept beside a run-time test it is predicated, and takes its slots
// of the FP64 pipe unused: a step of 512^3 20.6 -> 19.2 ms, of 64^3 63.0 -> 58.1
// us, of 24 batched grids 7.40 -> 7.22 ms with kernels of their own.
enum Mesh {
    kMeshAny,   // tested at run time: a batch with grids of both kinds, and the first step of FluxParams::own_momenta
    kMeshCubic, // equal spacings and face areas
    kMeshOther,
};

template <int TX, int TY, int NSLOT>
struct TileLayout {
    static constexpr int HX = TX + 2;
    static constexpr int HY = TY + 2;
    static constexpr int PLANE = HX * HY;
    static constexpr int PLANE_PAD = (PLANE + 15) / 16 * 16; // 128-byte aligned field tiles
    static constexpr int NFX = (TX + 1) * TY;
    static constexpr int NFY = TX * (TY + 1);
    static constexpr int NFZ = TX * TY;
    static_assert(NFX < 4096 && NFY < 4096 && NFZ < 4096, "face index range of div_runtime");
    static constexpr int NT = TX * TY;
    // shared memory, in double elements after a 128-byte mbarrier block
    static constexpr int Q_ELEMS = NSLOT * kFields * PLANE_PAD;
    static constexpr int FX_OFF = Q_ELEMS;
    static constexpr int FY_OFF = FX_OFF + 3 * NFX;
    static constexpr int FZ_OFF = FY_OFF + 3 * NFY;
    static constexpr int ELEMS = FZ_OFF + 3 * NFZ;
    static constexpr int MBAR_BYTES = 128;
    // + 128 bytes of slack to align the dynamic region to 128 bytes at run time
    static constexpr size_t BYTES = 128 + MBAR_BYTES + sizeof(double) * static_cast<size_t>(ELEMS);
    static constexpr unsigned TX_BYTES = kFields * PLANE * sizeof(double); // bytes one slot's TMA delivers
};

__device__ __forceinline__ void mbar_init(unsigned long long* bar, unsigned count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(unsigned long long* bar, unsigned bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}

// Bounded wait for the phase with the given parity; false if it never came.
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity)
{
    unsigned const a = smem_u32(bar);
    for (int it = 0; it < kWaitTries; ++it) {
        unsigned done;
        asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(a), "r"(parity)
                : "memory");
        if (done) {
            return true;
        }
    }
    return false;
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z,
                                            unsigned long long* bar)
{
    asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
            "l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
            : "memory");
}

template <int TX, int TY, int NSLOT>
__device__ __forceinline__ double* slot_field(double* smem, int slot, int field)
{
    using L = TileLayout<TX, TY, NSLOT>;
    return smem + (slot * kFields + field) * L::PLANE_PAD;
}

// Issue the TMA loads of plane k (x origin i0-1, y origin j0-1) into `slot`.
template <int TX, int TY, int NSLOT>
__device__ __forceinline__ void issue_plane(double* smem, unsigned long long* bars, int slot, TmaMaps const& maps, int i0,
                                            int j0, int k)
{
    using L = TileLayout<TX, TY, NSLOT>;
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    mbar_expect_tx(&bars[slot], L::TX_BYTES);
#pragma unroll
    for (int f = 0; f < kFields; ++f) {
        tma_load_3d(slot_field<TX, TY, NSLOT>(smem, slot, f), &maps.m[f], i0 - 1, j0 - 1, k, &bars[slot]);
    }
}

// The tile of one work item: its cells and the magic divisors of its face
// and cell indexes (div_runtime).
struct TileDims {
    int w, h;            // interior cells along x and y
    unsigned mw, mw1, mw2; // magics of w, w + 1 and w + 2
};

__device__ __forceinline__ TileDims tile_dims(int w, int h)
{
    return TileDims{w, h, div_magic20(w), div_magic20(w + 1), div_magic20(w + 2)};
}

// The halo cells a thread stages of every plane (a tile and its halo hold at
// most two cells per thread): their offset within a plane of the grid and
// their place in a slot's field (-1: none).  Found once per work item.
template <int N>
struct StageCells {
    long long src[N];
    int dst[N];
};

template <int TX, int TY>
constexpr int kStagePerThread = ((TX + 2) * (TY + 2) + TX * TY - 1) / (TX * TY);

template <int TX, int TY>
__device__ __forceinline__ StageCells<kStagePerThread<TX, TY>> stage_cells(FluxParams<double> const& p, TileDims const& t,
                                                                         int i0, int j0)
{
    StageCells<kStagePerThread<TX, TY>> s;
#pragma unroll
    for (int r = 0; r < kStagePerThread<TX, TY>; ++r) {
        int const c = threadIdx.x + r * TX * TY;
        int const hy = div_runtime(c, t.mw2);
        int const hx = c - hy * (t.w + 2);
        s.dst[r] = hy < t.h + 2 ? hy * (TX + 2) + hx : -1;
        s.src[r] = p.g.at(i0 - 1 + hx, j0 - 1 + hy, 0);
    }
    return s;
}

// Start copying plane k of the tile and its halo into `slot`: all ten values,
// or those that derive_plane does not compute.
template <int TX, int TY, int NSLOT, int MODE, int STAGE>
__device__ __forceinline__ void issue_plane_async(double* smem, int slot, FluxParams<double> const& p,
                                                  StageCells<kStagePerThread<TX, TY>> const& s, int k)
{
    using L = TileLayout<TX, TY, NSLOT>;
    constexpr int NF = STAGE == kStageAsync ? kFields : (MODE == kModeStep ? 7 : 5);
    unsigned const base = smem_u32(slot_field<TX, TY, NSLOT>(smem, slot, 0));
    long long const plane = p.g.s2 * k;
#pragma unroll
    for (int r = 0; r < kStagePerThread<TX, TY>; ++r) {
        if (s.dst[r] >= 0) {
            long long const o = s.src[r] + plane;
#pragma unroll
            for (int f = 0; f < NF; ++f) {
                const double* const src = (f < 5 ? p.prim.f[f] : (f == 5 ? p.cs : (f == 6 ? p.h : p.cons_in.f[f - 5]))) + o;
                asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                                     base + static_cast<unsigned>((f * L::PLANE_PAD + s.dst[r]) * sizeof(double))),
                             "l"(src)
                             : "memory");
            }
        }
    }
}

// The rest of a plane whose prim this thread has copied: the momenta d u and,
// for the per-operator godunov, the sound speed and e + p.
template <int TX, int TY, int NSLOT, int MODE>
__device__ __forceinline__ void derive_plane(double* smem, int slot, FluxParams<double> const& p,
                                             StageCells<kStagePerThread<TX, TY>> const& s)
{
    using L = TileLayout<TX, TY, NSLOT>;
#pragma unroll
    for (int r = 0; r < kStagePerThread<TX, TY>; ++r) {
        if (s.dst[r] >= 0) {
            double* const q = slot_field<TX, TY, NSLOT>(smem, slot, 0) + s.dst[r];
            double const d = q[0 * L::PLANE_PAD];
            double const u0 = q[2 * L::PLANE_PAD];
            double const u1 = q[3 * L::PLANE_PAD];
            double const u2 = q[4 * L::PLANE_PAD];
            double const m0 = mul_alu(d, u0);
            double const m1 = mul_alu(d, u1);
            double const m2 = mul_alu(d, u2);
            q[7 * L::PLANE_PAD] = m0;
            q[8 * L::PLANE_PAD] = m1;
            q[9 * L::PLANE_PAD] = m2;
            if (MODE != kModeStep) {
                // sqrt(gamma p / rho) from one reciprocal square root, and
                // e + p = p gamma/(gamma-1) + m.u / 2 with the halving on the
                // integer pipe
                double const pr = q[1 * L::PLANE_PAD];
                q[5 * L::PLANE_PAD] = sqrt_alu(mul_alu(mul_alu(p.gamma, pr), rcp_alu(d)));
                q[6 * L::PLANE_PAD] =
                        fma_rn(pr, p.h_over_p, half_exact(fma_rn(m2, u2, fma_rn(m1, u1, mul_alu(m0, u0)))));
            }
        }
    }
}

template <int PLANE_PAD>
__device__ __forceinline__ StagedSide load_side(double const* q, int c, int dir)
{
    StagedSide s;
    s.d = q[0 * PLANE_PAD + c];
    s.p = q[1 * PLANE_PAD + c];
    s.un = q[(2 + dir) * PLANE_PAD + c];
    s.mn = q[(7 + dir) * PLANE_PAD + c];
    s.c = q[5 * PLANE_PAD + c];
    s.h = q[6 * PLANE_PAD + c];
    return s;
}

// What a face carries into the cells beside it: its flux (b scaled by the
// ratio of its area to an x face's) and d and the momenta of its upwind side.
struct FaceTerms {
    double b, h, fn, d, m0, m1, m2;
};

template <int PLANE_PAD>
__device__ __forceinline__ FaceTerms face_terms(double const* f, int stride, int idx, double const* q, int left, int right)
{
    FaceTerms t;
    t.b = f[idx];
    t.h = f[stride + idx];
    t.fn = f[2 * stride + idx];
    double const* const u = q + (dbits(t.b) > 0 ? left : right);
    t.d = u[0 * PLANE_PAD];
    t.m0 = u[7 * PLANE_PAD];
    t.m1 = u[8 * PLANE_PAD];
    t.m2 = u[9 * PLANE_PAD];
    return t;
}

// Per-CTA state of the tile engine that lives across work items.
struct TileCtx {
    unsigned long long* bars; // one mbarrier per slot (TMA ring)
    double* smem;                  // plane slots
    double* fx;                    // x faces' b, h and fn (UpwindFlux)
    double* fy;                    // y faces'
    double* fz;                    // z faces'
    unsigned phase;           // bit s: parity of slot s's next completion (TMA ring)
    unsigned inflight;        // bit s: a TMA into slot s has not been waited for
    bool timed_out;           // a bounded mbarrier wait ran out
    long long wkey;           // ordered bits of this thread's max wavespeed
    unsigned wrun;            // fused step: the warp's running max of wavespeed estimates (WaveScreen)
    bool bad;                 // this thread saw a non-physical cell
};

template <int NSLOT>
__device__ __forceinline__ bool wait_slot(TileCtx& c, int s)
{
    bool const ok = mbar_wait(&c.bars[s], (c.phase >> s) & 1u);
    c.phase ^= 1u << s;
    c.inflight &= ~(1u << s);
    return ok;
}

// One work item: interior planes [kb, ke) of tile (tx, ty), with the update
// coefficient k0 (dt/dv times an x face's area).  Tiles are at most
// TX x TY cells, cut evenly out of the grid (p.sx, p.sy), so a warp solves no
// face and updates no cell that is not the grid's.  Returns false when a staged plane never arrived.
template <int TX, int TY, int MODE, int STAGE, int MESH>
__device__ __forceinline__ bool tile_item(TileCtx& c, FluxParams<double> const& p, TmaMaps const& maps, double k0, int tx,
                                          int ty, int kb, int ke)
{
    constexpr int NSLOT = kSlots;
    using L = TileLayout<TX, TY, NSLOT>;
    int const tid = threadIdx.x;
    bool const cubic = MESH == kMeshAny ? cubic_mesh(p) : MESH == kMeshCubic;
    double* const smem = c.smem;
    double* const fx = c.fx;
    double* const fy = c.fy;
    double* const fz = c.fz;

    int const i0 = 1 + p.sx.start(tx);
    int const j0 = 1 + p.sy.start(ty);
    TileDims const t = tile_dims(1 + p.sx.start(tx + 1) - i0, 1 + p.sy.start(ty + 1) - j0);
    int const tj = div_runtime(tid, t.mw);
    int const ti = tid - tj * t.w;
    int const center = (tj + 1) * L::HX + ti + 1;
    int const i = i0 + ti;
    int const j = j0 + tj;
    bool const own = tj < t.h;

    StageCells<kStagePerThread<TX, TY>> cells;
    if (STAGE != kStageTma) {
        cells = stage_cells<TX, TY>(p, t, i0, j0);
    }

    __syncthreads(); // the previous item's readers of slots and fluxes are done
    if (STAGE == kStageTma) {
        // planes kb-1 and kb -> slots 0 and 1
        if (tid == 0) {
            for (int s = 0; s < NSLOT; ++s) {
                issue_plane<TX, TY, NSLOT>(smem, c.bars, s, maps, i0, j0, kb - 1 + s);
            }
        }
        c.inflight |= (1u << NSLOT) - 1u;
        c.timed_out |= !wait_slot<NSLOT>(c, 0);
        c.timed_out |= !wait_slot<NSLOT>(c, 1);
    } else {
        for (int s = 0; s < NSLOT; ++s) {
            issue_plane_async<TX, TY, NSLOT, MODE, STAGE>(smem, s, p, cells, kb - 1 + s);
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        if (STAGE == kStageDerive) {
            for (int s = 0; s < NSLOT; ++s) {
                derive_plane<TX, TY, NSLOT, MODE>(smem, s, p, cells);
            }
        }
        __syncthreads();
    }
    // z face below the run's first plane, kept in registers
    FaceTerms zlo{};
    if (own) {
        double const* const q0 = slot_field<TX, TY, NSLOT>(smem, 0, 0);
        double const* const q1 = slot_field<TX, TY, NSLOT>(smem, 1, 0);
        UpwindFlux const f0 = hllc_upwind(load_side<L::PLANE_PAD>(q0, center, 2), load_side<L::PLANE_PAD>(q1, center, 2));
        double const* const u = (dbits(f0.b) > 0 ? q0 : q1) + center;
        zlo = FaceTerms{cubic ? f0.b : mul_rn(f0.b, p.rs2), f0.h, f0.fn, u[0], u[7 * L::PLANE_PAD], u[8 * L::PLANE_PAD],
                        u[9 * L::PLANE_PAD]};
    }
    if (__syncthreads_or(c.timed_out)) { // slot 0 is refilled next
        return false;
    }
    if (STAGE == kStageTma) { // plane kb + 1 <= ke
        if (tid == 0) {
            issue_plane<TX, TY, NSLOT>(smem, c.bars, 0, maps, i0, j0, kb + 1);
        }
        c.inflight |= 1u;
    } else {
        issue_plane_async<TX, TY, NSLOT, MODE, STAGE>(smem, 0, p, cells, kb + 1);
    }
    int const nfx = (t.w + 1) * t.h; // the faces of each family
    int const nfy = t.w * (t.h + 1);
    int const nface = nfx + nfy + t.w * t.h;

    // fused step: the next step's CFL wavespeed is screened (WaveScreen); the
    // running max carries over from the CTA's previous item of the same grid
    constexpr bool kScreen = MODE == kModeStep;
    WaveScreen screen(p.gamma, p.invdx0, p.invdx1, p.invdx2);
    screen.run = c.wrun;

    for (int k = kb; k < ke; ++k) {
        int const cur = (k - kb + 1) % NSLOT;
        int const nxt = (k - kb + 2) % NSLOT;
        // this cell's conservative state, fetched while the faces are solved
        // (where density and momenta are staged from cons, only the energy)
        double u[5];
        long long const o = p.g.at(i, j, k);
        if (own) {
            u[1] = p.cons_in.f[1][o];
            if (STAGE == kStageDerive) {
                u[0] = p.cons_in.f[0][o];
                u[2] = p.cons_in.f[2][o];
                u[3] = p.cons_in.f[3][o];
                u[4] = p.cons_in.f[4][o];
            }
        }
        // ---- face phase
        double const* qc = slot_field<TX, TY, NSLOT>(smem, cur, 0);
        double const* qn = slot_field<TX, TY, NSLOT>(smem, nxt, 0);
        // one index space over the three families; each face's family, left
        // cell and right cell are chosen by selects, so a warp that straddles
        // two families still runs the HLLC once
        // The z faces come last: plane k + 1, copied since the previous plane's
        // end, is waited for before the first pass that holds one.
        bool staged = false;
        for (int f = tid; f - tid < nface; f += L::NT) {
            if (!staged && f - tid + L::NT > nfx + nfy) {
                staged = true;
                if (STAGE == kStageTma) {
                    c.timed_out |= !wait_slot<NSLOT>(c, nxt);
                } else {
                    asm volatile("cp.async.wait_all;" ::: "memory");
                    if (STAGE == kStageDerive) {
                        derive_plane<TX, TY, NSLOT, MODE>(smem, nxt, p, cells);
                    }
                    __syncthreads();
                }
            }
            if (f >= nface) {
                break;
            }
            bool const is_x = f < nfx;
            bool const is_y = !is_x && f < nfx + nfy;
            int const g = is_x ? f : (is_y ? f - nfx : f - nfx - nfy);
            int const gj = div_runtime(g, is_x ? t.mw1 : t.mw);
            int const gi = g - gj * (is_x ? t.w + 1 : t.w);
            int const a = (is_y ? gj : gj + 1) * L::HX + (is_x ? gi : gi + 1);
            int const dir = is_x ? 0 : (is_y ? 1 : 2);
            double const* const qr = is_x || is_y ? qc : qn;
            int const ar = a + (is_x ? 1 : (is_y ? L::HX : 0));
            UpwindFlux u = hllc_upwind(load_side<L::PLANE_PAD>(qc, a, dir), load_side<L::PLANE_PAD>(qr, ar, dir));
            if (!cubic) {
                u.b = mul_rn(u.b, is_x ? 1.0 : (is_y ? p.rs1 : p.rs2));
            }
            double* const out = (is_x ? fx : (is_y ? fy : fz)) + g;
            int const stride = is_x ? L::NFX : (is_y ? L::NFY : L::NFZ);
            out[0] = u.b;
            out[stride] = u.h;
            out[2 * stride] = u.fn;
        }
        if (__syncthreads_or(c.timed_out)) {
            return false;
        }

        // ---- cell phase
        FaceTerms zhi{};
        double wv[4] = {0.0, 0.0, 0.0, 0.0}; // fused step: the new cs, v0, v1, v2, for the screened wavespeed
        if (own) {
            zhi = face_terms<L::PLANE_PAD>(fz, L::NFZ, tid, qc + center, 0, static_cast<int>(qn - qc));
            int const xl = tj * (t.w + 1) + ti;
            int const yb = tj * t.w + ti;
            FaceTerms const xlo = face_terms<L::PLANE_PAD>(fx, L::NFX, xl, qc + center, -1, 0);
            FaceTerms const xhi = face_terms<L::PLANE_PAD>(fx, L::NFX, xl + 1, qc + center, 0, 1);
            // div F in units of an x face's area: every term but the normal
            // momenta's is b times a value of the face's upwind side
            double rd = fma_rn(-xlo.b, xlo.d, mul_alu(xhi.b, xhi.d));
            double re = fma_rn(-xlo.b, xlo.h, mul_alu(xhi.b, xhi.h));
            double r0 = sub_rn(xhi.fn, xlo.fn);
            FaceTerms const ylo = face_terms<L::PLANE_PAD>(fy, L::NFY, yb, qc + center, -L::HX, 0);
            FaceTerms const yhi = face_terms<L::PLANE_PAD>(fy, L::NFY, yb + t.w, qc + center, 0, L::HX);
            double r1 = sub_rn(yhi.fn, ylo.fn);
            double r2 = sub_rn(zhi.fn, zlo.fn);
            if (!cubic) {
                r1 = mul_rn(r1, p.rs1);
                r2 = mul_rn(r2, p.rs2);
            }
            r1 = fma_rn(-xlo.b, xlo.m1, fma_rn(xhi.b, xhi.m1, r1));
            r2 = fma_rn(-xlo.b, xlo.m2, fma_rn(xhi.b, xhi.m2, r2));
            rd = fma_rn(-ylo.b, ylo.d, fma_rn(yhi.b, yhi.d, rd));
            re = fma_rn(-ylo.b, ylo.h, fma_rn(yhi.b, yhi.h, re));
            r0 = fma_rn(-ylo.b, ylo.m0, fma_rn(yhi.b, yhi.m0, r0));
            r2 = fma_rn(-ylo.b, ylo.m2, fma_rn(yhi.b, yhi.m2, r2));
            rd = fma_rn(-zlo.b, zlo.d, fma_rn(zhi.b, zhi.d, rd));
            re = fma_rn(-zlo.b, zlo.h, fma_rn(zhi.b, zhi.h, re));
            r0 = fma_rn(-zlo.b, zlo.m0, fma_rn(zhi.b, zhi.m0, r0));
            r1 = fma_rn(-zlo.b, zlo.m1, fma_rn(zhi.b, zhi.m1, r1));
            if (STAGE != kStageDerive) {
                u[0] = qc[center];
                u[2] = qc[7 * L::PLANE_PAD + center];
                u[3] = qc[8 * L::PLANE_PAD + center];
                u[4] = qc[9 * L::PLANE_PAD + center];
            }
            u[0] = fma_rn(-k0, rd, u[0]);
            u[1] = fma_rn(-k0, re, u[1]);
            u[2] = fma_rn(-k0, r0, u[2]);
            u[3] = fma_rn(-k0, r1, u[3]);
            u[4] = fma_rn(-k0, r2, u[4]);
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                p.cons_out.f[f][o] = u[f];
            }
            if constexpr (MODE == kModeStep) {
                // cons_to_prim of the new state (cons_to_prim.hpp:26-31)
                double const r = rcp_alu(u[0]);
                double const v0 = mul_alu(u[2], r);
                double const v1 = mul_alu(u[3], r);
                double const v2 = mul_alu(u[4], r);
                double const mv = fma_rn(u[4], v2, fma_rn(u[3], v1, mul_alu(u[2], v0))); // |m|^2 / rho
                double const pr = fma_rn(-p.half_gm1, mv, mul_alu(p.gm1, u[1])); // (gamma-1)(e - |m|^2/(2 rho))
                double const cs = sqrt_alu(mul_alu(mul_alu(p.gamma, r), pr));
                p.h_out[o] = u[1] + pr; // staged as e + p at the next step
                p.prim_out.f[0][o] = u[0];
                p.prim_out.f[1][o] = pr;
                p.prim_out.f[2][o] = v0;
                p.prim_out.f[3][o] = v1;
                p.prim_out.f[4][o] = v2;
                if (p.prim_rec.f[0] != nullptr) { // a second copy, for a recording caller
                    p.prim_rec.f[0][o] = u[0];
                    p.prim_rec.f[1][o] = pr;
                    p.prim_rec.f[2][o] = v0;
                    p.prim_rec.f[3][o] = v1;
                    p.prim_rec.f[4][o] = v2;
                }
                p.cs_out[o] = cs;
                wv[0] = cs;
                wv[1] = v0;
                wv[2] = v1;
                wv[3] = v2;
                c.bad |= !(finite_positive(u[0]) && finite_positive(pr)); // the wavespeed is checked below
            }
        }
        if constexpr (kScreen) {
            // next step's CFL wavespeed (time_step.hpp:28-33), in FP64 only
            // for the cells that can hold the max; the same expression as
            // the unscreened step, so the max and the dt are unchanged.
            // Every lane of the warp is here (the screen is warp-collective);
            // a non-finite wavespeed always takes the FP64 branch.
            if (screen.step_exact_needed(own, wv[0], wv[1], wv[2], wv[3], cubic)) {
                double const invdt = cubic ? (3.0 * wv[0] + abs_(wv[1]) + abs_(wv[2]) + abs_(wv[3])) * p.invdx0
                                      : (wv[0] + abs_(wv[1])) * p.invdx0 + (wv[0] + abs_(wv[2])) * p.invdx1 +
                                                (wv[0] + abs_(wv[3])) * p.invdx2;
                long long const key = wave_key(invdt);
                c.wkey = key > c.wkey ? key : c.wkey;
                c.bad |= dbits(invdt) >= kInfBits;
            }
        }
        zlo = zhi; // the z face above becomes the next plane's z face below
        __syncthreads(); // the next face phase rewrites the fluxes, and plane k is no longer read:
        if (k + 2 <= ke) { // refill its slot
            if (STAGE == kStageTma) {
                if (tid == 0) {
                    issue_plane<TX, TY, NSLOT>(smem, c.bars, cur, maps, i0, j0, k + 2);
                }
                c.inflight |= 1u << cur;
            } else {
                issue_plane_async<TX, TY, NSLOT, MODE, STAGE>(smem, cur, p, cells, k + 2);
            }
        }
    }
    c.wrun = screen.run;
    return !__syncthreads_or(c.timed_out);
}

// Block-wide max of the threads' wavespeed keys into *wmax, and the
// non-physical flag into *status; clears the per-thread values.
template <int NT>
__device__ __forceinline__ void flush_wavespeed(TileCtx& c, unsigned long long* wmax, int* status)
{
    __shared__ long long warp_best[NT / 32];
    __shared__ int any_bad;
    int const tid = threadIdx.x;
    long long w = c.wkey;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        long long const v = __shfl_xor_sync(0xffffffffu, w, o);
        w = v > w ? v : w;
    }
    __syncthreads();
    if (tid == 0) {
        any_bad = 0;
    }
    __syncthreads();
    if ((tid & 31) == 0) {
        warp_best[tid >> 5] = w;
    }
    if (c.bad) {
        any_bad = 1;
    }
    __syncthreads();
    if (tid == 0) {
        long long b = warp_best[0];
#pragma unroll
        for (int wv = 1; wv < NT / 32; ++wv) {
            b = warp_best[wv] > b ? warp_best[wv] : b;
        }
        atomicMax(wmax, static_cast<unsigned long long>(b));
        if (any_bad) {
            atomicOr(status, 1);
        }
    }
    c.wkey = 0;
    c.wrun = 0u; // the next item may be another grid's
    c.bad = false;
}

template <int TX, int TY, int NSLOT>
__device__ __forceinline__ TileCtx make_ctx(unsigned char* smem_dyn)
{
    using L = TileLayout<TX, TY, NSLOT>;
    // TMA destinations must sit on 128-byte boundaries of the shared window
    unsigned char* raw = smem_dyn + ((128u - (smem_u32(smem_dyn) & 127u)) & 127u);
    TileCtx c;
    c.bars = reinterpret_cast<unsigned long long*>(raw);
    c.smem = reinterpret_cast<double*>(raw + L::MBAR_BYTES);
    c.fx = c.smem + L::FX_OFF;
    c.fy = c.smem + L::FY_OFF;
    c.fz = c.smem + L::FZ_OFF;
    c.phase = 0;
    c.inflight = 0;
    c.timed_out = false;
    c.wkey = 0;
    c.wrun = 0u;
    c.bad = false;
    return c;
}

template <int TX, int TY, int MODE, int STAGE, int MESH>
__global__ void __launch_bounds__(TX* TY, 3) flux_tile_kernel(const __grid_constant__ FluxParams<double> p,
                                                           const __grid_constant__ TmaMaps maps)
{
    constexpr int NSLOT = kSlots;
    extern __shared__ __align__(128) unsigned char smem_dyn[];
    TileCtx c = make_ctx<TX, TY, NSLOT>(smem_dyn);
    double const dtodv = dt_over_dv(p);
    double const k0 = dtodv * p.ds0;

    if (STAGE == kStageTma) {
        if (threadIdx.x == 0) {
            for (int s = 0; s < NSLOT; ++s) {
                mbar_init(&c.bars[s], 1);
            }
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncthreads();
    }

    // CTA b's share of all tiles' planes, counted tile by tile: a run of
    // planes up one tile, and on into the next
    int const iz = p.g.n2 - 2;
    int w = static_cast<int>(static_cast<long long>(p.nwork) * blockIdx.x / gridDim.x);
    int const end = static_cast<int>(static_cast<long long>(p.nwork) * (blockIdx.x + 1) / gridDim.x);
    while (w < end) {
        int const tile = w / iz;
        int const k = w - tile * iz;
        int const run = min(end - w, iz - k);
        if (!tile_item<TX, TY, MODE, STAGE, MESH>(c, p, maps, k0, tile % p.tiles_x, tile / p.tiles_x, 1 + k, 1 + k + run)) {
            break;
        }
        w += run;
    }

    if (STAGE == kStageTma && __syncthreads_or(c.timed_out)) {
        // a staged plane never arrived: report, wait (bounded) for the copies
        // still in flight so none lands after the CTA is gone, and stop
        if (threadIdx.x == 0) {
            atomicOr(p.status, 2);
        }
        for (int s = 0; s < NSLOT; ++s) {
            if (c.inflight & (1u << s)) {
                wait_slot<NSLOT>(c, s);
            }
        }
        step_done(p); // the launch still counts this CTA, so the next launch starts from zero
        return;
    }
    if (MODE == kModeStep) {
        flush_wavespeed<TX * TY>(c, p.wmax, p.status);
        step_done(p);
    }
}

// Many independent grids in one launch: a persistent grid of CTAs pops
// (grid, tile, chunk) items from a global queue (largest grids first),
// copies the item's grid parameters to shared memory and runs the same tile
// engine; each item's wavespeed goes to its own grid's accumulator, so every
// grid keeps its own dt.  Staging by cp.async (grids of any shape).
template <int TX, int TY, int MESH>
__global__ void __launch_bounds__(TX* TY, TX* TY == 256 ? 3 : 6) flux_batch_kernel(const __grid_constant__ BatchParams<double> b)
{
    constexpr int NSLOT = kSlots;
    constexpr int NT = TX * TY;
    static_assert(sizeof(FluxParams<double>) % 4 == 0, "parameter copy in 4-byte words");
    extern __shared__ __align__(128) unsigned char smem_dyn[];
    __shared__ __align__(16) FluxParams<double> gp;
    __shared__ int s_item;
    TileCtx c = make_ctx<TX, TY, NSLOT>(smem_dyn);
    int const tid = threadIdx.x;
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
        for (int w = tid; w < static_cast<int>(sizeof(FluxParams<double>) / 4); w += NT) {
            reinterpret_cast<int*>(&gp)[w] = reinterpret_cast<const int*>(&b.grids[it.x])[w];
        }
        __syncthreads();
        double const dtodv = dt_over_dv(gp);
        int const kb = 1 + it.w * gp.kchunk;
        tile_item<TX, TY, kModeStep, kStageAsync, MESH>(c, gp, TmaMaps{}, dtodv * gp.ds0, it.y, it.z, kb,
                                                     min(kb + gp.kchunk, gp.g.n2 - 1));
        flush_wavespeed<NT>(c, gp.wmax, gp.status);
        item_done(gp);
    }
    batch_cta_done(b);
}

// Cells of the ghost layer (all cells of a grid without interior), and the
// offset of the c-th of them.
__host__ __device__ inline long long ghost_cells(Geom const& g)
{
    if (g.n0 < 3 || g.n1 < 3 || g.n2 < 3) {
        return g.ncell();
    }
    return 2 * g.s2 + (2LL * g.n0 + 2LL * (g.n1 - 2)) * (g.n2 - 2);
}

__device__ __forceinline__ long long ghost_offset(Geom const& g, long long c)
{
    long long const plane = g.s2;
    if (g.n0 < 3 || g.n1 < 3 || g.n2 < 3) {
        return c;
    }
    if (c < 2 * plane) {
        return (c < plane) ? c : c - plane + plane * (g.n2 - 1);
    }
    // grids hold < 2^31 cells: the ring index fits 32-bit division
    long long const ring = 2LL * g.n0 + 2LL * (g.n1 - 2);
    unsigned const r0 = static_cast<unsigned>(c - 2 * plane);
    unsigned const q = r0 / static_cast<unsigned>(ring);
    int const k = 1 + static_cast<int>(q);
    int const r = static_cast<int>(r0 - q * static_cast<unsigned>(ring));
    int i, j;
    if (r < g.n0) {
        i = r;
        j = 0;
    } else if (r < 2 * g.n0) {
        i = r - g.n0;
        j = g.n1 - 1;
    } else {
        int const r2 = r - 2 * g.n0;
        j = 1 + r2 / 2;
        i = (r2 & 1) ? g.n0 - 1 : 0;
    }
    return g.at(i, j, k);
}

// Ghost shell of the step's output: cons copied, prim = cons_to_prim(cons)
// (bit-identical to the reference's cons_to_prim over ghosts,
// cons_to_prim.hpp:26-27), sound speed and CFL contribution.
template <class T>
__device__ __forceinline__ void ghost_shell_body(GhostParams<T> const& p)
{
    Geom const g = p.g;
    long long const total = ghost_cells(g);
    T wmax = T(0);
    for (long long c = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; c < total;
         c += static_cast<long long>(gridDim.x) * blockDim.x) {
        long long const o = ghost_offset(g, c);
        T const d = p.cons_in.f[0][o];
        T const e = p.cons_in.f[1][o];
        T const m0 = p.cons_in.f[2][o];
        T const m1 = p.cons_in.f[3][o];
        T const m2 = p.cons_in.f[4][o];
        T pr, u0, u1, u2;
        if (p.prim_out.f[0] == nullptr) {
            // cons-only FP32 state: only the cons words and the wavespeed
            T const r = rcp_rn(d); // = 1/d correctly rounded
            u0 = m0 * r;
            u1 = m1 * r;
            u2 = m2 * r;
            pr = p.comp != kCompNone ? cons_pressure<kCompSum>(d, e, m0, m1, m2, r, p.gm1, nullptr)
                                     : cons_pressure<kCompNone>(d, e, m0, m1, m2, r, p.gm1, nullptr);
        } else {
            cons_to_prim_exact(d, e, m0, m1, m2, p.gm1, pr, u0, u1, u2);
        }
        p.cons_out.f[0][o] = d;
        p.cons_out.f[1][o] = e;
        p.cons_out.f[2][o] = m0;
        p.cons_out.f[3][o] = m1;
        p.cons_out.f[4][o] = m2;
        if (p.lo_in.f[0] != nullptr) {
#pragma unroll
            for (int f = 0; f < 5; ++f) {
                p.lo_out.f[f][o] = p.lo_in.f[f][o];
            }
        }
        if (p.h_out != nullptr) {
            p.h_out[o] = e + pr;
        }
        if (p.prim_out.f[0] != nullptr) {
            p.prim_out.f[0][o] = d;
            p.prim_out.f[1][o] = pr;
            p.prim_out.f[2][o] = u0;
            p.prim_out.f[3][o] = u1;
            p.prim_out.f[4][o] = u2;
            p.cs_out[o] = sqrt_rn(div_rn(mul_rn(p.gamma, pr), d));
        }
        T v;
        if (p.prim_out.f[0] == nullptr) {
            // FP32 states: the sound speed as their step kernel forms it
            T const cs = fast_sound_speed((p.gamma * rcp_rn(d)) * pr);
            v = (cs + abs_(u0)) * p.invdx0 + (cs + abs_(u1)) * p.invdx1 + (cs + abs_(u2)) * p.invdx2;
        } else {
            v = cell_invdt_exact(d, pr, u0, u1, u2, p.gamma, p.invdx0, p.invdx1, p.invdx2);
        }
        wmax = (v > wmax) ? v : wmax;
    }
    __shared__ T warp_best[8];
    wmax = warp_max(wmax);
    if ((threadIdx.x & 31) == 0) {
        warp_best[threadIdx.x >> 5] = wmax;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        T b = warp_best[0];
        for (int w = 1; w < static_cast<int>(blockDim.x >> 5); ++w) {
            b = (warp_best[w] > b) ? warp_best[w] : b;
        }
        atomicMax(p.wmax, order_bits(b));
    }
}

template <class T>
__global__ void __launch_bounds__(256) ghost_shell_kernel(GhostParams<T> p)
{
    ghost_shell_body(p);
}

__global__ void __launch_bounds__(256) ghost_prim_kernel(CBundle<double> prim, Geom g, double* base, size_t field,
                                                         int count)
{
    long long const total = ghost_cells(g);
    for (long long c = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; c < total;
         c += static_cast<long long>(gridDim.x) * blockDim.x) {
        long long const o = ghost_offset(g, c);
#pragma unroll
        for (int f = 0; f < 5; ++f) {
            double const v = prim.f[f][o];
            for (int b = 0; b < count; ++b) {
                base[(static_cast<size_t>(b) * 5 + f) * field + o] = v;
            }
        }
    }
}

template <class T>
__global__ void finalize_dt_kernel(SimScalars* s, T cfl, int add_time, const double* dt_seq, double* dt_log)
{
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        finalize_one(s, cfl, add_time, dt_seq, dt_log);
    }
}

// The single-grid tile, at most: 16x16 columns, whose 800 faces per plane
// fill exactly 25 warp-passes (a 32x8 tile's 808 need 26) with the same 256
// threads, 18x18 TMA boxes and three resident CTAs per SM.
constexpr int kStepTX = 16, kStepTY = 16;

} // namespace

// Picks the tiles by the time of the busiest SM.  The kernel divides all tiles'
// planes evenly among its CTAs, so with U planes in all on G CTAs, r of them
// on an SM, each solves m = ceil(U/G) planes of cost c and the z faces below
// its first plane, z: the SM's FP64 pipe is busy r (m c + z), and every plane
// adds a wait that its neighbours do not cover (its barriers and its last,
// partly filled pass of faces).  c and z count FP64 warp instructions, each
// holding its SM for 9.0 ns; the wait measured
// 1.1 us a plane with two CTAs on the SM and 1.6 us with one.  Both were
// measured on the kernel with two CTAs and all its work on the FP64 pipe; for
// today's, with three and half of its arithmetic on the integer pipes, they
// rank the tiles but do not give the time (512^3: 25.6 ms for 19.2, 64^3: 60
// us for 58), and count whole tiles too dear against small ones.  Whole
// 16 x 16 tiles are the best for large grids, smaller ones where their number
// leaves SMs idle.  Against whole 16 x 16 tiles in chunks of at least 8
// planes, all work on the FP64 pipe: 16^3 97 -> 12.5 us a step, 48^3 97 -> 46,
// 64^3 97 -> 86, 99 x 128 x 75 311 -> 270 (now 13.5, 34, 58 and 211).
TilePlan choose_tiles(int ix, int iy, int iz, int sms, int per_sm, int face, int cell, int stage, int q)
{
    constexpr double kInstr = 9.0e-3, kWait2 = 1.1, kWait1 = 1.6; // us
    // the last answer of this thread: a loop over one grid asks the same
    // again, and the search takes a few microseconds
    struct Asked {
        int key[9];
        TilePlan plan;
    };
    thread_local Asked last{};
    int const key[9] = {ix, iy, iz, sms, per_sm, face, cell, stage, q};
    if (std::equal(key, key + 9, last.key)) {
        return last.plan;
    }
    int const units = (ix + q - 1) / q;
    TilePlan best{};
    double best_us = 1e300;
    int last_nx = 0;
    for (int w = kStepTX / q; w >= 1; --w) {
        int const nx = (units + w - 1) / w;
        int const tw = (units + nx - 1) / nx * q;
        if (nx == last_nx) {
            continue; // the same tiles as the previous extent's
        }
        last_nx = nx;
        int last_ny = 0;
        for (int h = kStepTY; h >= 1; --h) {
            int const ny = (iy + h - 1) / h;
            int const th = (iy + ny - 1) / ny;
            if (ny == last_ny) {
                continue;
            }
            last_ny = ny;
            int const faces = (tw + 1) * th + tw * (th + 1) + tw * th;
            int const rows = (tw * th + 31) / 32;
            int const c = face * ((faces + 31) / 32) + cell * rows + stage * (((tw + 2) * (th + 2) + 31) / 32);
            long long const u = static_cast<long long>(nx) * ny * iz;
            long long const ctas = u < static_cast<long long>(sms) * per_sm ? u : static_cast<long long>(sms) * per_sm;
            long long const r = (ctas + sms - 1) / sms;
            long long const m = (u + ctas - 1) / ctas;
            double const us = m * (r * c * kInstr + (r > 1 ? kWait2 : kWait1)) + r * face * rows * kInstr;
            if (us < best_us * (1.0 - 1e-9)) {
                best_us = us;
                best = TilePlan{nx, ny};
            }
        }
    }
    std::copy(key, key + 9, last.key);
    last.plan = best;
    return best;
}

namespace {

template <int MODE, int STAGE, int MESH>
struct FluxKernel {
    using L = TileLayout<kStepTX, kStepTY, kSlots>;
    static auto fn() { return flux_tile_kernel<kStepTX, kStepTY, MODE, STAGE, MESH>; }

    // Resident CTAs per SM.  Called outside any stream capture (by the entry
    // points before they enqueue work).
    static cudaError_t configure(int* per_sm)
    {
        return resident_ctas<flux_tile_kernel<kStepTX, kStepTY, MODE, STAGE, MESH>>(L::NT, static_cast<int>(L::BYTES), per_sm);
    }

    static cudaError_t launch(FluxParams<double> p, TmaMaps const& maps, int sms, cudaStream_t s)
    {
        int const per_sm = p.per_sm > 0 ? p.per_sm : 1;
        int const ix = p.g.n0 - 2;
        int const iy = p.g.n1 - 2;
        int const iz = p.g.n2 - 2;
        if (ix <= 0 || iy <= 0 || iz <= 0) {
            return cudaSuccess; // no interior cell
        }
        int const q = STAGE == kStageTma ? 2 : 1;
        // in FP64 instructions, the integer work beside them included: 16 a
        // face; the step's 48 a cell, or the operator's 30 a cell and 17 a
        // staged one
        TilePlan const plan = MODE == kModeStep ? choose_tiles(ix, iy, iz, sms, per_sm, 16, 48, 0, q)
                                                : choose_tiles(ix, iy, iz, sms, per_sm, 16, 30, 17, q);
        p.h_over_p = p.inv_gm1 + 1.0;
        p.sx = split_tiles(ix, plan.nx, q);
        p.sy = split_tiles(iy, plan.ny, 1);
        p.tiles_x = plan.nx;
        p.tiles_y = plan.ny;
        p.nwork = plan.nx * plan.ny * iz;
        long long const slots = static_cast<long long>(sms) * per_sm;
        int const grid = static_cast<int>(slots < p.nwork ? slots : p.nwork);
        fn()<<<grid, L::NT, L::BYTES, s>>>(p, maps);
        return cudaGetLastError();
    }
};

// Tile shapes of the batch (the autotuner picks one).
constexpr int kBatchShapes[][2] = {{32, 8}, {16, 8}, {16, 16}};
constexpr int kNumBatchShapes = 3;

template <int TX, int TY, int MESH>
struct BatchKernel {
    using L = TileLayout<TX, TY, kSlots>;
    static cudaError_t configure(int* per_sm)
    {
        return resident_ctas<flux_batch_kernel<TX, TY, MESH>>(L::NT, static_cast<int>(L::BYTES), per_sm);
    }
    static cudaError_t launch(BatchParams<double> const& b, int grid, cudaStream_t s)
    {
        flux_batch_kernel<TX, TY, MESH><<<grid, L::NT, L::BYTES, s>>>(b);
        return cudaGetLastError();
    }
};

// b == nullptr: configure for every kind of mesh (the fewest resident CTAs).
template <int TX, int TY>
cudaError_t run_batch(BatchParams<double> const* b, int grid, int* per_sm, cudaStream_t s)
{
    if (b != nullptr) {
        return b->cubic == b->ngrids ? BatchKernel<TX, TY, kMeshCubic>::launch(*b, grid, s)
               : b->cubic == 0       ? BatchKernel<TX, TY, kMeshOther>::launch(*b, grid, s)
                                     : BatchKernel<TX, TY, kMeshAny>::launch(*b, grid, s);
    }
    int n[3] = {};
    cudaError_t e = BatchKernel<TX, TY, kMeshAny>::configure(&n[0]);
    e = e != cudaSuccess ? e : BatchKernel<TX, TY, kMeshCubic>::configure(&n[1]);
    e = e != cudaSuccess ? e : BatchKernel<TX, TY, kMeshOther>::configure(&n[2]);
    *per_sm = std::min(n[0], std::min(n[1], n[2]));
    return e;
}

} // namespace

int batch_shape_count() { return kNumBatchShapes; }
void batch_shape(int shape, int* tx, int* ty)
{
    *tx = kBatchShapes[shape][0];
    *ty = kBatchShapes[shape][1];
}

// b == nullptr: configure (dynamic shared memory opt-in) and report the
// resident CTAs per SM; otherwise launch `grid` persistent CTAs.
template <class T>
cudaError_t launch_flux_batch(int shape, int comp, BatchParams<T> const* b, int grid, int* per_sm, cudaStream_t s)
{
    if constexpr (sizeof(T) == sizeof(double)) {
        switch (shape) {
        case 0: return run_batch<32, 8>(b, grid, per_sm, s);
        case 1: return run_batch<16, 8>(b, grid, per_sm, s);
        default: return run_batch<16, 16>(b, grid, per_sm, s);
        }
    } else {
        return launch_batch_f32col(comp, kBatchShapes[shape][0], kBatchShapes[shape][1], b, grid, per_sm, s);
    }
}

template cudaError_t launch_flux_batch<double>(int, int, BatchParams<double> const*, int, int*, cudaStream_t);
template cudaError_t launch_flux_batch<float>(int, int, BatchParams<float> const*, int, int*, cudaStream_t);

template <class T>
struct FluxDispatch;

template <>
struct FluxDispatch<double> {
    // Both kinds of mesh, as the mesh is not known here; their kernels take
    // the same shared memory and no more than the registers of three CTAs.
    template <int MODE, int STAGE>
    static cudaError_t configure_meshes(int* per_sm)
    {
        cudaError_t const e = FluxKernel<MODE, STAGE, kMeshOther>::configure(per_sm);
        return e != cudaSuccess ? e : FluxKernel<MODE, STAGE, kMeshCubic>::configure(per_sm);
    }
    template <int MODE, int STAGE>
    static cudaError_t launch_mesh(FluxParams<double> const& p, TmaMaps const& maps, int sms, cudaStream_t s)
    {
        return cubic_mesh(p) ? FluxKernel<MODE, STAGE, kMeshCubic>::launch(p, maps, sms, s)
                             : FluxKernel<MODE, STAGE, kMeshOther>::launch(p, maps, sms, s);
    }

    static cudaError_t configure(int mode, bool tma, int /*comp*/, int* per_sm)
    {
        if (mode == kModeStep) {
            cudaError_t const e = FluxKernel<kModeStep, kStageDerive, kMeshAny>::configure(per_sm);
            if (e != cudaSuccess) {
                return e;
            }
            return tma ? configure_meshes<kModeStep, kStageTma>(per_sm) : configure_meshes<kModeStep, kStageAsync>(per_sm);
        }
        return configure_meshes<kModeGodunov, kStageDerive>(per_sm);
    }
    static cudaError_t launch(FluxParams<double> p, TmaMaps const* maps, int mode, int /*comp*/, int sms, cudaStream_t s)
    {
        p.rs1 = p.ds1 / p.ds0;
        p.rs2 = p.ds2 / p.ds0;
        if (mode == kModeStep) {
            if (p.own_momenta) {
                return FluxKernel<kModeStep, kStageDerive, kMeshAny>::launch(p, TmaMaps{}, sms, s);
            }
            return maps != nullptr ? launch_mesh<kModeStep, kStageTma>(p, *maps, sms, s)
                                   : launch_mesh<kModeStep, kStageAsync>(p, TmaMaps{}, sms, s);
        }
        return launch_mesh<kModeGodunov, kStageDerive>(p, TmaMaps{}, sms, s);
    }
};

template <>
struct FluxDispatch<float> {
    static cudaError_t configure(int mode, bool /*tma*/, int comp, int* per_sm)
    {
        return mode == kModeStep ? configure_step_f32col(comp, per_sm) : cudaSuccess;
    }
    static cudaError_t launch(FluxParams<float> const& p, TmaMaps const* /*maps*/, int mode, int comp, int sms,
                              cudaStream_t s)
    {
        return mode == kModeStep ? launch_step_f32col(p, comp, sms, s) : launch_godunov_f32(p, sms, s);
    }
};

template <class T>
cudaError_t configure_flux(int mode, bool tma, int comp, int* per_sm)
{
    return FluxDispatch<T>::configure(mode, tma, comp, per_sm);
}

template <class T>
cudaError_t launch_flux(FluxParams<T> p, TmaMaps const* maps, int mode, int comp, int sms, cudaStream_t s)
{
    return FluxDispatch<T>::launch(p, maps, mode, comp, sms, s);
}

static int ghost_blocks(Geom const& g, int sms)
{
    long long const blocks = (ghost_cells(g) + 255) / 256;
    long long const cap = static_cast<long long>(sms) * 8;
    return static_cast<int>(blocks < 1 ? 1 : (blocks < cap ? blocks : cap));
}

cudaError_t launch_ghost_prim(CBundle<double> prim, Geom g, double* base, size_t field, int count, int sms,
                              cudaStream_t s)
{
    ghost_prim_kernel<<<ghost_blocks(g, sms), 256, 0, s>>>(prim, g, base, field, count);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_ghost_shell(GhostParams<T> p, int sms, cudaStream_t s)
{
    ghost_shell_kernel<T><<<ghost_blocks(p.g, sms), 256, 0, s>>>(p);
    return cudaGetLastError();
}

template <class T>
cudaError_t launch_finalize_dt(SimScalars* sc, T cfl, int add_time, cudaStream_t s, const double* dt_seq, double* dt_log)
{
    finalize_dt_kernel<T><<<1, 32, 0, s>>>(sc, cfl, add_time, dt_seq, dt_log);
    return cudaGetLastError();
}

int flux_tile_x() { return kStepTX; } // the FP64 step's TMA boxes
int flux_tile_y() { return kStepTY; }

template cudaError_t configure_flux<double>(int, bool, int, int*);
template cudaError_t configure_flux<float>(int, bool, int, int*);
template cudaError_t launch_flux<double>(FluxParams<double>, TmaMaps const*, int, int, int, cudaStream_t);
template cudaError_t launch_flux<float>(FluxParams<float>, TmaMaps const*, int, int, int, cudaStream_t);
template cudaError_t launch_ghost_shell<double>(GhostParams<double>, int, cudaStream_t);
template cudaError_t launch_ghost_shell<float>(GhostParams<float>, int, cudaStream_t);
template cudaError_t launch_finalize_dt<double>(SimScalars*, double, int, cudaStream_t, const double*, double*);
template cudaError_t launch_finalize_dt<float>(SimScalars*, float, int, cudaStream_t, const double*, double*);

} // namespace eulr
