"""What a plan of the native launcher (csrc/launcher.cpp) does not stand for, and what it leaves behind."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tq():
    if not torch.cuda.is_available():
        pytest.fail("the gpu tests need a CUDA device")
    from tessiq_b200 import ops

    return ops


def drawn(shape, seed, dtype=torch.float32):
    return torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").to(dtype)


def on_device(value):
    return torch.tensor(value, device="cuda")


# ---- numbers that come as tensors: their values are no part of a signature ----------------------


@pytest.mark.parametrize("name", ["layer_norm", "layer_norm of a view", "native_layer_norm", "batch_norm", "attention", "softmax", "argmax", "sum"])
def test_a_number_given_as_a_tensor_is_read_on_every_call(tq, name):
    x, w = drawn((48, 64), 1), drawn((64,), 2)
    q = drawn((1, 2, 32, 64), 3, torch.bfloat16)
    call, values = {
        "layer_norm": (lambda eps: tq.layer_norm(x, [64], w, w, eps), (1e-5, 3.0)),
        "layer_norm of a view": (lambda eps: tq.layer_norm(x.t(), [48], None, None, eps), (1e-5, 3.0)),
        "native_layer_norm": (lambda eps: tq.native_layer_norm(x, [64], w, w, eps)[0], (1e-5, 3.0)),
        "batch_norm": (lambda eps: tq.batch_norm_eval(x, w, w, w, w.abs(), eps), (1e-5, 3.0)),
        "attention": (lambda scale: tq.attention(q, q, q, scale, False), (0.125, 1.0)),
        "softmax": (lambda half_to_float: tq.softmax(x.bfloat16(), -1, half_to_float), (False, True)),
        "argmax": (lambda dim: tq.argmax(x, dim), (0, 1)),
        "sum": (lambda keepdim: tq.sum(x, 0, keepdim), (False, True)),
    }[name]
    expected = [call(value) for value in values]
    for _ in range(2):
        for value, right in zip(values, expected):
            got = call(on_device(value))
            assert got.dtype == right.dtype and torch.equal(got, right)

# ---- results of later calls -----------------------------------------------------------------------


def test_strides_of_later_results_are_those_of_the_first(tq):
    wide = drawn((8, 16), 5)
    for x in (wide[:1, :8], wide[:, :1], wide[3:4, 2:3], drawn((6, 4, 5), 6)[:, 2:3], drawn((6, 5), 7).t()):
        first = tq.elementwise("mul", x, 2.0)
        for _ in range(2):
            again = tq.elementwise("mul", x, 2.0)
            assert again.stride() == first.stride() and torch.equal(again, first)


# ---- scratch ---------------------------------------------------------------------------------------


def test_a_failed_allocation_leaves_no_reference_to_the_scratch(tq):
    """The result does not fit: torch's error, the scratch block as it was, and the next call works."""
    import sys

    from tessiq_b200 import kernel as K

    x = drawn((2048, 4096), 8)
    expected = tq.softmax(x.t(), -1)
    assert torch.equal(tq.softmax(x.t(), -1), expected)
    block = K.workspace(0, torch.cuda.current_stream().cuda_stream, 1)
    before = sys.getrefcount(block)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    torch.cuda.set_per_process_memory_fraction(torch.cuda.memory_reserved() / torch.cuda.get_device_properties(0).total_memory)
    try:
        for _ in range(3):
            with pytest.raises(torch.OutOfMemoryError):
                held = [tq.softmax(x.t(), -1) for _ in range(64)]      # (what the allocator has left over may serve the first ones)
                del held
    finally:
        torch.cuda.set_per_process_memory_fraction(1.0)
    assert sys.getrefcount(block) == before
    assert torch.equal(tq.softmax(x.t(), -1), expected)


# ---- the table ------------------------------------------------------------------------------------


def test_a_plan_in_use_outlasts_others(tq):
    from tessiq_b200 import _launcher

    x, hot = torch.arange(5000, device="cuda", dtype=torch.float32), drawn((3, 7), 9)
    tq.clone(hot)
    for n in range(1, 4800):
        tq.clone(x[:n])
        if n % 100 == 0:
            assert torch.equal(_launcher.call(tq._CODES["pack"], hot), hot), n
    assert _launcher.size() <= 2048
