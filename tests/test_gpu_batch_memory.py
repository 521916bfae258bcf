"""Device memory of an FP64 batch: 11 fields a copy, two copies.  The density
is a field of prim and of cons, equal in both in a batch, and is held once."""
import pytest

pytestmark = pytest.mark.gpu


def test_fp64_batch_holds_22_fields(cuda, euler):
    torch = cuda
    shape = (130, 126, 128)
    with euler.Batch([(8, 8, 8, 1.4, 0.1, 0.1, 0.1)]):
        pass  # kernels and streams of a first batch
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    with euler.Batch([(*shape, 1.4, 0.1, 0.1, 0.1)]):
        used = before - torch.cuda.mem_get_info()[0]
    field = shape[0] * shape[1] * shape[2] * 8
    assert used <= 22 * field + (8 << 20)  # parameters, items and the allocator's granularity
