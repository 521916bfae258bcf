"""The per-operator FP32 godunov over FP32's range: density and pressure scaled
by powers of two, together and apart, so that their product leaves the normal
range while their quotient, the fluxes and the HLLC's own products stay inside
it; and cells without pressure."""
import numpy as np
import pytest

from conftest import rel_linf

pytestmark = pytest.mark.gpu

DX = (0.11, 0.07, 0.13)


def _godunov_f32(cuda, euler, prim, dt):
    pg = cuda.from_numpy(prim).cuda()
    cg = euler.prim_to_cons(pg, 1.4)
    cons = cg.cpu().numpy().astype(np.float64)
    euler.godunov(pg, cg, 1.4, DX, dt)
    return cons, cg.cpu().numpy()


@pytest.mark.parametrize("kd,kp", [(-110, -20), (110, 20), (-50, 50), (50, -50), (50, 50), (-50, -50), (0, 0)])
def test_scaled_density_and_pressure(cuda, euler, oracle_lib, kd, kp):
    """rho 2^kd, p 2^kp and velocities (time steps) scaled by the sound speed's 2^((kp - kd)/2) (its inverse) are the
    same flow, every field times a power of two.  Against the FP64 oracle: the operator's bar, 2e-5 of each field's
    scale."""
    ku = (kp - kd) // 2
    prim = oracle_lib.random_prim(19, 12, 9, seed=21, dtype=np.float32)
    scaled = np.ldexp(prim, np.array([kd, kp, ku, ku, ku]).reshape(5, 1, 1, 1))
    assert scaled.dtype == np.float32
    _, got = _godunov_f32(cuda, euler, scaled, float(np.ldexp(0.01, -ku)))
    cons = oracle_lib.prim_to_cons(prim, 1.4).astype(np.float64)
    ref = oracle_lib.godunov(prim.astype(np.float64), cons, 1.4, DX, 0.01)
    back = np.ldexp(got.astype(np.float64), -np.array([kd, kp, kd + ku, kd + ku, kd + ku]).reshape(5, 1, 1, 1))
    assert np.isfinite(back).all()
    assert max(rel_linf(back, ref)) <= 2e-5


def test_cells_without_pressure(cuda, euler, oracle_lib):
    """Pairs of cells with p = 0 (sound speed 0) that collide along x, amid warm gas: finite, and the FP64 oracle's
    update within the operator's bar."""
    prim = oracle_lib.random_prim(14, 11, 10, seed=22, dtype=np.float32)
    for k in (2, 5, 7):
        for j in (2, 5, 8):
            prim[1, k, j, 4:6] = 0.0
            prim[2, k, j, 4:6] = 0.7, -0.7
    cons, got = _godunov_f32(cuda, euler, prim, 0.005)
    ref = oracle_lib.godunov(prim.astype(np.float64), cons, 1.4, DX, 0.005)
    assert np.isfinite(got).all()
    assert max(rel_linf(got, ref)) <= 2e-5
