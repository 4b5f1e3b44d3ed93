"""A reduction asks for the scratch that its kernel uses, and no more."""

import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def abi():
    if not torch.cuda.is_available():
        pytest.fail("the gpu tests need a CUDA device")
    from tessiq_b200 import _lib

    return _lib


# one cluster takes each tile of columns whole: no partials and no tickets, where the form with tickets would need more than the
# built-in scratch (3072 x 4096), some (1000 x 1000), or is only an estimate for another alignment (700 x 1003: rows between vectors)
SHAPES = [(1, 3072, 4096), (1, 1000, 1000), (1, 700, 1003), (3, 2000, 640)]


@pytest.mark.parametrize("outer, reduce, inner", SHAPES)
@pytest.mark.parametrize("op", ["ARGMAX", "SUM"])
def test_no_scratch_is_asked_for_where_none_is_used(abi, op, outer, reduce, inner):
    # small whole numbers: sums are exact in any order, and columns have ties
    x = torch.randint(-8, 9, (outer, reduce, inner), generator=torch.Generator(device="cuda").manual_seed(1), device="cuda").float()
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    make = lambda: torch.full((outer, inner), -7, dtype=torch.int64 if op == "ARGMAX" else torch.float32, device="cuda")  # noqa: E731
    bare, static = make(), make()
    abi.check(abi.lib.tq_reduce_launch(getattr(abi, op), abi.F32, x.data_ptr(), bare.data_ptr(), outer, reduce, inner, None, 0, 0, stream))
    abi.check(abi.lib.tq_reduce_launch_static(getattr(abi, op), abi.F32, x.data_ptr(), static.data_ptr(), outer, reduce, inner, 0, stream))
    torch.cuda.synchronize()
    if op == "SUM":
        expected = x.sum(1)
    else:      # the first of the largest
        expected = (x == x.amax(1, keepdim=True)).to(torch.int8).argmax(1)
    assert torch.equal(bare, expected) and torch.equal(static, expected)


def test_scratch_that_is_used_is_still_asked_for(abi):
    x, out = torch.randn(131072, 128, device="cuda"), torch.full((128,), -7.0, device="cuda")
    need = ctypes.c_size_t()
    abi.check(abi.lib.tq_reduce_workspace_bytes(abi.SUM, abi.F32, 1, 131072, 128, 0, ctypes.byref(need)))
    assert need.value > 0
    assert abi.lib.tq_reduce_launch(abi.SUM, abi.F32, x.data_ptr(), out.data_ptr(), 1, 131072, 128, None, 0, 0, None) == abi.TQ_INVALID_ARGUMENT
    torch.cuda.synchronize()
    assert (out == -7).all()
