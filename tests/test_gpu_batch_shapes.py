"""FP32 batches in each of the column engine's tile shapes: batches whose grids
make 16 x 8, 16 x 16 and (plain state) 32 x 8 tiles the default, at tile edges
and remainders, cubic and other cells, as picked and after the autotuner.  The
bits of every grid equal the grid's stepped alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

BATCHES = {
    "tiny": [(3, 3, 3), (6, 7, 8), (10, 10, 40), (18, 9, 20), (5, 34, 11)],
    "narrow": [(3, 43, 17), (10, 41, 40), (17, 10, 5), (4, 130, 6)],
    "24s": [(26, 26, 26), (26, 26, 9), (58, 26, 14)],
    "square": [(18, 18, 18), (34, 18, 26), (50, 50, 21), (19, 35, 14)],
}


@pytest.mark.parametrize("precision", ["f32", "f32c", "f32c_hilo"])
@pytest.mark.parametrize("name", list(BATCHES))
def test_batch_equals_single_grids(euler, cuda, oracle_lib, precision, name):
    shapes = BATCHES[name]
    meshes = [(0.1, 0.1, 0.1) if i % 2 else (0.11, 0.07, 0.13) for i in range(len(shapes))]
    prims = [oracle_lib.random_prim(*s, seed=70 + i) for i, s in enumerate(shapes)]
    got = []
    with euler.Batch([(*s, 1.4, *dx) for s, dx in zip(shapes, meshes)], cfl=0.4, precision=precision) as b:
        for tuned in (False, True):
            for g, p in enumerate(prims):
                b.set_prim(g, p)
            if tuned:
                b.autotune(trial_steps=1)
            b.advance(4)
            got.append([b.state_numpy(g)[1] for g in range(len(shapes))])
    for i, (shape, dx, p0) in enumerate(zip(shapes, meshes, prims)):
        with euler.Simulation(*shape, 1.4, dx, 0.4, precision=precision) as s:
            s.set_prim(p0)
            s.advance(4)
            alone = s.state_numpy()[1]
        assert np.array_equal(got[0][i], alone) and np.array_equal(got[1][i], alone), shape
