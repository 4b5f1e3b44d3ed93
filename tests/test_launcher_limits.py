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


# ---- what takes the long way ------------------------------------------------------------------------


class Tagged(torch.Tensor):
    pass


def planned(tq, x):
    from tessiq_b200 import _launcher

    return _launcher.call(tq._CODES["softmax"], x, -1, False)


def test_only_plain_tensors_have_plans(tq):
    from torch.utils._python_dispatch import TorchDispatchMode

    class Watching(TorchDispatchMode):
        def __torch_dispatch__(self, function, types, args=(), kwargs=None):
            return function(*args, **(kwargs or {}))

    x = drawn((9, 33), 10)
    expected = tq.softmax(x, -1)
    assert torch.equal(planned(tq, x), expected)
    assert torch.equal(planned(tq, torch.nn.Parameter(x)), expected)
    assert planned(tq, x.as_subclass(Tagged)) is None and torch.equal(tq.softmax(x.as_subclass(Tagged), -1).as_subclass(torch.Tensor), expected)
    assert planned(tq, x.cpu()) is None and planned(tq, x.to("meta")) is None
    with Watching():
        assert planned(tq, x) is None and torch.equal(tq.softmax(x, -1), expected)
    seen = []

    def inside(row):
        seen.append(planned(tq, row))
        return row.sum()

    torch.func.vmap(inside)(x.expand(2, 9, 33).contiguous())
    torch.func.grad(inside)(x)
    torch.func.functionalize(inside)(x)
    assert seen == [None, None, None]


def test_inference_mode_and_gradients(tq):
    x = drawn((9, 35), 11)
    with torch.inference_mode():
        results = [tq.softmax(x, -1) for _ in range(3)]
        assert all(r.is_inference() for r in results)
    leaf = x.clone().requires_grad_()
    for _ in range(3):
        plain, of_leaf = tq.softmax(x, -1), tq.softmax(leaf, -1)
        assert not plain.is_inference() and torch.equal(plain, results[0])
        assert not of_leaf.requires_grad and torch.equal(of_leaf, plain)


def test_another_alignment_of_a_shape_is_another_signature(tq):
    for dtype in (torch.float32, torch.bfloat16):
        data = drawn((40 * 64 + 8,), 12, dtype)
        for _ in range(2):
            for start in (0, 1, 2, 4, 0, 3):
                x = data[start : start + 40 * 64].view(40, 64)
                exact = x.double()
                assert torch.equal(tq.clone(x), x) and torch.equal(tq.elementwise("mul", x, 2.0), x * 2)
                rel = 2.0**-8 if dtype == torch.bfloat16 else 1e-6
                for dim in (0, 1):
                    assert ((tq.sum(x, dim).double() - exact.sum(dim)).abs() <= rel * exact.abs().sum(dim)).all()
                    assert torch.equal(tq.amax(x, dim), x.amax(dim))
