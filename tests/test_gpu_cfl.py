"""time_step's screened max at the sizes and states where the screen could
miss the cell that holds it: partial blocks and threads with one cell or
several, states whose wavespeeds tie or differ by ulps everywhere, values past
the FP32 estimate's range.  dt equals the oracle's bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SHAPES = [(1, 1, 1), (5, 17, 3), (257, 1, 2), (64, 16, 2), (130, 67, 71)]


def states(O, shape, dtype):
    rng = np.random.default_rng(sum(shape))
    base = O.random_prim(*shape, seed=sum(shape)).astype(dtype)
    yield base
    tied = base.copy()
    tied[:] = base.reshape(5, -1)[:, 0][:, None, None, None]
    yield tied
    near = tied.copy()
    near *= (1 + np.finfo(dtype).eps * rng.integers(-40, 41, size=near.shape)).astype(dtype)
    yield near
    wide = base.copy()
    span = 12 if dtype == np.float32 else 45  # FP32: squares and quotients stay finite
    wide[:2] *= (10.0 ** rng.uniform(-span, span, size=wide[:2].shape)).astype(dtype)
    yield wide
    rest = tied.copy()
    rest[2:] = 0.0
    rest[1] *= dtype(1e-35) if dtype == np.float32 else dtype(1e-200)  # estimates at and below FP32's normal range
    yield rest


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("shape", SHAPES)
def test_time_step_bit_identical(cuda, euler, oracle_lib, dtype, shape):
    for prim in states(oracle_lib, shape, dtype):
        ref = oracle_lib.time_step(prim, 1.4, (0.11, 0.07, 0.13))
        got = euler.time_step(cuda.from_numpy(prim).cuda(), 1.4, (0.11, 0.07, 0.13)).cpu().numpy()
        assert got.dtype == dtype and got == dtype(ref)


@pytest.mark.parametrize("shape", SHAPES)
def test_loaded_dt_is_time_steps(cuda, euler, oracle_lib, shape):
    """The load's own max: the first dt of a simulation is cfl * time_step of the loaded state."""
    dx = (0.11, 0.07, 0.13)
    for prim in states(oracle_lib, shape, np.float64):
        with euler.Simulation(*shape, 1.4, dx, 0.4) as s:
            s.set_prim(prim)
            assert s.time()[1] == 0.4 * oracle_lib.time_step(prim, 1.4, dx)
