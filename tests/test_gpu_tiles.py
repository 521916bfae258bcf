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
