"""Loading and reading a state through device arrays (read and written in
place) and through host arrays (copied): the same bits, for every precision,
single grid and batch, whole bundles and single fields."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

PRECISIONS = ["f64", "f32c", "f32", "f32c_hilo"]


@pytest.mark.parametrize("precision", PRECISIONS)
@pytest.mark.parametrize("shape", [(3, 2, 4), (19, 33, 7), (70, 41, 29)])
def test_device_and_host_arrays_agree(cuda, euler, oracle_lib, precision, shape):
    torch = cuda
    n0, n1, n2 = shape
    prim = oracle_lib.random_prim(n0, n1, n2, seed=n0)
    cons = oracle_lib.prim_to_cons(prim, 1.4)
    on_device = torch.from_numpy(prim).cuda()
    cons_device = torch.from_numpy(cons).cuda()
    torch.cuda.synchronize()

    def read(sim):
        host = sim.state_numpy()
        dev = [torch.zeros((5, n2, n1, n0), dtype=torch.float64, device="cuda") for _ in range(4)]
        torch.cuda.synchronize()
        sim.get_state(dev[0], dev[1])
        sim.get_state(cons=dev[2])  # cons alone
        one = euler.null_bundle()
        one.f3 = dev[3][3].data_ptr()  # a single prim field
        euler.check(euler.load().eulr_sim_get_state_f64(sim._h, one, euler.null_bundle()))
        got = [d.cpu().numpy() for d in dev]
        assert np.array_equal(got[0], host[0]) and np.array_equal(got[1], host[1])
        assert np.array_equal(got[2], host[1])
        assert np.array_equal(got[3][3], host[0][3]) and not got[3][:3].any() and not got[3][4].any()
        return host + (sim.time()[0],)

    for with_cons in (False, True):
        res = []
        for p, c in ((prim, cons), (on_device, cons_device)):
            with euler.Simulation(n0, n1, n2, dx=(0.1, 0.07, 0.12), precision=precision) as s:
                s.set_state(p, c) if with_cons else s.set_prim(p)
                first = read(s)
                s.advance(3)
                res.append(first + read(s))
        for a, b in zip(*res):
            assert np.array_equal(a, b)


@pytest.mark.parametrize("precision", PRECISIONS)
def test_batch_device_and_host_arrays_agree(cuda, euler, oracle_lib, precision):
    torch = cuda
    shapes = [(9, 12, 7), (34, 18, 21), (2, 5, 4)]
    grids = [(*s, 1.4, 0.1, 0.07, 0.12) for s in shapes]
    prims = [oracle_lib.random_prim(*s, seed=3 + i) for i, s in enumerate(shapes)]
    device = [torch.from_numpy(p).cuda() for p in prims]
    torch.cuda.synchronize()
    res = []
    for src in (prims, device):
        with euler.Batch(grids, precision=precision) as b:
            for g, p in enumerate(src):
                b.set_prim(g, p)
            b.autotune(trial_steps=1)
            b.advance(4)
            host = [b.state_numpy(g) for g in range(len(grids))]
            out = [torch.empty((2, 5, s[2], s[1], s[0]), dtype=torch.float64, device="cuda") for s in shapes]
            torch.cuda.synchronize()
            for g, o in enumerate(out):
                euler.check(euler.load().eulr_batch_get_state_f64(b._h, g, euler.bundle(o[0]), euler.bundle(o[1])))
                assert np.array_equal(o[0].cpu().numpy(), host[g][0])
                assert np.array_equal(o[1].cpu().numpy(), host[g][1])
            res.append(host)
    for (pa, ca), (pb, cb) in zip(*res):
        assert np.array_equal(pa, pb) and np.array_equal(ca, cb)
