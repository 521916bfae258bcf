"""Scalars that are no C floating-point numbers are refused by the Python
operators with the error of the conversion itself, before anything is launched."""
import pytest
import torch


class NoStream:
    cuda_stream = 0


@pytest.mark.parametrize("dtype", [torch.float64, torch.float32])
@pytest.mark.parametrize("bad, error", [("1.4", TypeError), (None, TypeError), ([1.4], TypeError),
                                        (10**400, OverflowError)])
def test_scalars_of_the_wrong_kind_are_refused(euler, dtype, bad, error):
    a = torch.ones((5, 3, 4, 5), dtype=dtype)
    b = torch.ones_like(a)
    dx, s = (0.1, 0.1, 0.1), NoStream()
    calls = [
        lambda: euler.prim_to_cons(a, bad, out=b, stream=s),
        lambda: euler.cons_to_prim(a, bad, out=b, stream=s),
        lambda: euler.time_step(a, 1.4, (0.1, bad, 0.1), stream=s),
        lambda: euler.godunov(a, b, 1.4, dx, bad, stream=s),
        lambda: euler.godunov(a, b, bad, dx, 0.01, stream=s, exact=True),
        lambda: euler.init_implode(5, 4, 3, (0.1, 0.1, bad), dtype=dtype, device="cpu", stream=s),
    ]
    if dtype == torch.float64:
        calls.append(lambda: euler.godunov(a, b, 1.4, dx, (torch.ones((), dtype=dtype), bad), stream=s))
    for call in calls:
        with pytest.raises(error):
            call()
