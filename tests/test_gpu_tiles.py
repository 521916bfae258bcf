"""The FP64 tile engine's work split at the sizes where it can go wrong: tiles
cut evenly out of the interior (one cell, one tile, a tile and a cell, thin
slabs), runs of planes that cross from one tile into the next, and both ways
of staging (even row pitch: TMA; odd: cp.async)."""
import numpy as np
import pytest

from conftest import rel_linf

pytestmark = pytest.mark.gpu

SHAPES = [(3, 3, 3), (4, 3, 5), (18, 18, 18), (19, 19, 5), (20, 35, 3), (3, 50, 41), (50, 3, 41), (35, 21, 66),
          (52, 37, 23), (131, 34, 19)]


@pytest.mark.parametrize("shape", SHAPES)
def test_step_and_godunov_match_oracle(cuda, euler, oracle_lib, shape):
    """Tolerances: the bars of the fused step and the operator after one call, 1e-12 of each field's scale;
    4e-12 after four steps."""
    O = oracle_lib
    n0, n1, n2 = shape
    dx = (0.11, 0.07, 0.13)
    prim0 = O.random_prim(n0, n1, n2, seed=n0 + 100 * n1 + 10000 * n2)
    for steps, tol in ((1, 1e-12), (4, 4e-12)):
        pref, cref = prim0.copy(), O.prim_to_cons(prim0, 1.4)
        tref = O.simulate(pref, cref, 1.4, dx, 0.4, steps)
        with euler.Simulation(n0, n1, n2, 1.4, dx, 0.4) as s:
            s.set_prim(prim0)
            s.advance(steps)
            assert s.status() == 0
            prim, cons = s.state_numpy()
            t = s.time()[0]
        assert abs(t - tref) <= 1e-12 * tref
        assert max(rel_linf(cons, cref) + rel_linf(prim, pref)) <= tol
    pg = cuda.from_numpy(prim0).cuda()
    cg = euler.prim_to_cons(pg, 1.4)
    euler.godunov(pg, cg, 1.4, dx, 0.01)
    cref = O.godunov(prim0, O.prim_to_cons(prim0, 1.4), 1.4, dx, 0.01)
    assert max(rel_linf(cg.cpu().numpy(), cref)) <= 1e-12


def test_batch_tiles_equal_single_grid(cuda, euler, oracle_lib):
    """Every shape as one grid of a batch (queue items, chunks): the bits of the same grid stepped alone."""
    grids = [(*s, 1.4, 0.11, 0.07, 0.13) for s in SHAPES]
    prims = [oracle_lib.random_prim(*s, seed=7 + i) for i, s in enumerate(SHAPES)]
    with euler.Batch(grids, cfl=0.4) as b:
        for g, p in enumerate(prims):
            b.set_prim(g, p)
        b.advance(4)
        got = [b.state_numpy(g) for g in range(len(grids))]
    for shape, p0, (pb, cb) in zip(SHAPES, prims, got):
        with euler.Simulation(*shape, 1.4, (0.11, 0.07, 0.13), 0.4) as s:
            s.set_prim(p0)
            s.advance(4)
            ps, cs = s.state_numpy()
        assert np.array_equal(pb, ps) and np.array_equal(cb, cs), shape


@pytest.mark.parametrize("shape", [(4, 3, 5), (19, 35, 5), (34, 21, 23)])
def test_first_step_of_a_state_loaded_with_its_own_cons(cuda, euler, oracle_lib, shape):
    """set_state with momenta that are not d u: the first step's faces take the velocities from prim, the update
    starts from cons, as the operator does.  1e-12 of each field's scale, the bar of one step."""
    O = oracle_lib
    dx = (0.11, 0.07, 0.13)
    prim0 = O.random_prim(*shape, seed=sum(shape))
    cons0 = O.prim_to_cons(prim0, 1.4)
    cons0[2:] += 0.2 * np.random.default_rng(5).standard_normal(cons0[2:].shape)
    with euler.Simulation(*shape, 1.4, dx, 0.3) as s:
        s.set_state(prim0, cons0)
        s.advance(1)
        dt = s.time()[0]
        cons = s.state_numpy()[1]
    assert max(rel_linf(cons, O.godunov(prim0, cons0.copy(), 1.4, dx, dt))) <= 1e-12


@pytest.mark.parametrize("k", [-300, -129, 130, 254, 300])
def test_step_and_godunov_scale_with_density_and_pressure(cuda, euler, oracle_lib, k):
    """Density and pressure times 2^k scale the conserved state by 2^k and leave dt: within, across and outside the
    magnitudes the integer products, reciprocals and roots take.  Each differs by at most an ulp from the FP64 unit's:
    1e-13 of each field's scale after four steps."""
    shape = (19, 12, 9)
    prim = oracle_lib.random_prim(*shape, seed=11)
    scaled = prim.copy()
    scaled[:2] = np.ldexp(scaled[:2], k)
    out = []
    for p in (prim, scaled):
        with euler.Simulation(*shape, 1.4, (0.11, 0.07, 0.13), 0.3) as s:
            s.set_prim(p)
            s.advance(4)
            assert s.status() == 0
            cons = s.state_numpy()[1]
        pg = cuda.from_numpy(p).cuda()
        cg = euler.prim_to_cons(pg, 1.4)
        euler.godunov(pg, cg, 1.4, (0.11, 0.07, 0.13), 0.01)
        out.append((cons, cg.cpu().numpy()))
    for a, b in zip(out[1], out[0]):
        assert max(rel_linf(np.ldexp(a, -k), b)) <= 1e-13


@pytest.mark.parametrize("kinds", ["cubic", "both"])
def test_batch_of_cubic_and_other_meshes_equals_single_grids(cuda, euler, oracle_lib, kinds):
    """A batch whose grids are all of cubic cells, and one with both kinds: the bits of each grid stepped alone."""
    shapes = [(19, 19, 5), (20, 35, 3), (35, 21, 26), (18, 18, 18)]
    meshes = [(0.1, 0.1, 0.1) if kinds == "cubic" or i % 2 else (0.11, 0.07, 0.13) for i in range(len(shapes))]
    prims = [oracle_lib.random_prim(*s, seed=50 + i) for i, s in enumerate(shapes)]
    with euler.Batch([(*s, 1.4, *dx) for s, dx in zip(shapes, meshes)], cfl=0.4) as b:
        for g, p in enumerate(prims):
            b.set_prim(g, p)
        b.advance(4)
        got = [b.state_numpy(g) for g in range(len(shapes))]
    for shape, dx, p0, (pb, cb) in zip(shapes, meshes, prims, got):
        with euler.Simulation(*shape, 1.4, dx, 0.4) as s:
            s.set_prim(p0)
            s.advance(4)
            ps, cs = s.state_numpy()
        assert np.array_equal(pb, ps) and np.array_equal(cb, cs), shape


@pytest.mark.parametrize("precision", ["f32", "f32c", "f32c_hilo"])
def test_fp32_columns_match_oracle_and_batch(cuda, euler, oracle_lib, precision):
    """The FP32 column engine at its tile widths and chunk edges.  Against the FP64 oracle after four steps: 4 steps
    of at most about 20 roundings (2^-24) each at a field's scale, 5e-6 of it; the batch's bits equal the single
    grid's."""
    O = oracle_lib
    dx = (0.11, 0.07, 0.13)
    grids = [(*s, 1.4, *dx) for s in SHAPES]
    prims = [O.random_prim(*s, seed=31 + i) for i, s in enumerate(SHAPES)]
    with euler.Batch(grids, cfl=0.4, precision=precision) as b:
        for g, p in enumerate(prims):
            b.set_prim(g, p)
        b.advance(4)
        batch = [b.state_numpy(g)[1] for g in range(len(grids))]
    for shape, p0, cb in zip(SHAPES, prims, batch):
        pref, cref = p0.copy(), O.prim_to_cons(p0, 1.4)
        O.simulate(pref, cref, 1.4, dx, 0.4, 4)
        with euler.Simulation(*shape, 1.4, dx, 0.4, precision=precision) as s:
            s.set_prim(p0)
            s.advance(4)
            assert s.status() == 0
            cons = s.state_numpy()[1]
        assert max(rel_linf(cons, cref)) <= 5e-6, shape
        assert np.array_equal(cb, cons), shape


@pytest.mark.parametrize("shape", SHAPES)
def test_fp32_godunov_matches_oracle(cuda, euler, oracle_lib, shape):
    """The per-operator FP32 godunov against the FP64 oracle on the same FP32 inputs, cubic and uneven cells: the
    operator's bar, 2e-5 of each field's scale."""
    O = oracle_lib
    p32 = O.random_prim(*shape, seed=sum(shape)).astype(np.float32)
    for dx in ((0.11, 0.07, 0.13), (0.1, 0.1, 0.1)):
        pg = cuda.from_numpy(p32).cuda()
        cg = euler.prim_to_cons(pg, 1.4)
        c0 = cg.cpu().numpy().astype(np.float64)
        euler.godunov(pg, cg, 1.4, dx, 0.01)
        ref = O.godunov(p32.astype(np.float64), c0, 1.4, dx, 0.01)
        assert max(rel_linf(cg.cpu().numpy(), ref)) <= 2e-5


def _bits(a):
    return a.view(np.uint64 if a.dtype == np.float64 else np.uint32)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("shape", SHAPES + [(258, 162, 130)])
def test_exact_godunov_tiles_bit_identical(cuda, euler, oracle_lib, dtype, shape):
    """The bit-identical godunov at tile edges, on random states with patches of gas at rest (zero numerators of the
    shared-reciprocal quotients), signed zeros, and cells out of the quotients' mid range; the last shape is large
    enough for FP32's whole-tile kernel.  Every bit, the signs of zeros included."""
    O = oracle_lib
    n0, n1, n2 = shape
    prim = O.random_prim(n0, n1, n2, seed=n0 + n1 + n2).astype(dtype)
    prim[1, : n2 // 2 + 1] = 1.0
    prim[2:, : n2 // 2 + 1] = 0.0
    prim[2:, : n2 // 4 + 1] = -0.0
    prim[2:, -1] *= dtype(1e25 if dtype == np.float32 else 1e150) ** dtype(0.5)  # out of the mid range, squares finite
    cons = O.prim_to_cons(prim, 1.4)
    dx, dt = (0.11, 0.07, 0.13), 1e-3
    ref = O.godunov(prim, cons, 1.4, dx, dt)
    cg = cuda.from_numpy(cons.copy()).cuda()
    euler.godunov(cuda.from_numpy(prim).cuda(), cg, 1.4, dx, dt, exact=True)
    got = cg.cpu().numpy()
    same = (_bits(got) == _bits(ref)) | (np.isnan(got) & np.isnan(ref))
    assert same.all(), (int((~same).sum()), got[~same][:4], ref[~same][:4])
