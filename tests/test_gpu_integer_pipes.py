"""The bit-identical FP64 operators, whose products and reciprocals run on the
integer pipes: within, across and outside the magnitudes [2^-255, 2^257) that
those take, with zeros, powers of two and values of few bits (exact products
and ties) among the inputs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("k", [-300, -130, 0, 129, 254, 300])
def test_bit_identical_operators(cuda, euler, oracle_lib, k):
    """Bit for bit the oracle's prim_to_cons, cons_to_prim and godunov."""
    O = oracle_lib
    prim = O.random_prim(21, 18, 9, seed=3)
    rng = np.random.default_rng(4)
    few = rng.random(prim.shape) < 0.2
    prim[few] = np.round(prim[few] * 1024) / 1024
    prim[2:][rng.random(prim[2:].shape) < 0.2] = 0.0
    prim[0][rng.random(prim[0].shape) < 0.1] = 2.0 - 2.0**-52
    prim[:2] = np.ldexp(np.maximum(prim[:2], 2.0**-10), k)
    cons = O.prim_to_cons(prim, 1.4)
    pg = cuda.from_numpy(prim).cuda()
    cg = euler.prim_to_cons(pg, 1.4)
    assert np.array_equal(cg.cpu().numpy(), cons)
    assert np.array_equal(euler.cons_to_prim(cg, 1.4).cpu().numpy(), O.cons_to_prim(cons, 1.4))
    dx = (0.11, 0.07, 0.13)
    euler.godunov(pg, cg, 1.4, dx, 0.01, exact=True)
    assert np.array_equal(cg.cpu().numpy(), O.godunov(prim, cons.copy(), 1.4, dx, 0.01))
