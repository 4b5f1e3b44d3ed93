"""Reductions over columns and over transposed views, around the forms one cluster of CTAs takes whole: one CTA and clusters
of two to eight, row pieces of 32 to 1024 bytes, rows that divide nothing, one row a thread, special values in each part."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def tq():
    if not torch.cuda.is_available():
        pytest.fail("the gpu tests need a CUDA device")
    from tessiq_b200 import ops

    return ops


SHAPES = [  # outer, reduce, inner
    (1, 1, 64), (1, 2, 8), (1, 31, 2048), (1, 64, 2048), (1, 257, 40), (1, 512, 768), (1, 700, 32), (1, 1000, 1000), (1, 1003, 1003), (3, 300, 520),
    (1, 2049, 333), (1, 5003, 1250), (1, 4096, 768), (1, 20000, 64), (1, 300, 9999), (5, 1111, 96), (1, 3072, 4096), (2, 40, 24), (1, 9000, 8), (1, 40000, 301),
]
DTYPES = [torch.float32, torch.bfloat16, torch.float16, torch.float64, torch.int32]


def drawn(shape, dtype, seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    if dtype == torch.int32:
        return torch.randint(-1000, 1000, shape, generator=g, device="cuda", dtype=torch.int32)
    return torch.randn(shape, generator=g, device="cuda", dtype=torch.float64).to(dtype)


@pytest.mark.parametrize("dtype", DTYPES, ids=lambda d: str(d)[6:])
@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
def test_columns(tq, shape, dtype):
    """Sums within the rounding of a tree with chains of up to 60 additions (2^-24 each, 2^-53 for f64) and of the result; the others exact."""
    outer, reduce, inner = shape
    for off in (0, 1):       # and a base between vectors
        x = drawn((outer * reduce * inner + off,), dtype, reduce + inner)[off:].view(shape)
        wide = x.double()
        unit = {torch.float32: 2.0**-24, torch.bfloat16: 2.0**-8, torch.float16: 2.0**-11, torch.float64: 2.0**-53, torch.int32: 0.0}[dtype]
        bound = 60 * (2.0**-53 if dtype == torch.float64 else 2.0**-24) * wide.abs().sum(1) * (dtype != torch.int32)
        total = wide.sum(1)
        assert ((tq.sum(x, 1).double() - total).abs() <= bound + unit * total.abs()).all()
        if dtype != torch.int32:
            assert ((tq.mean(x, 1).double() - total / reduce).abs() <= bound / reduce + 2 * unit * total.abs() / reduce + 2.0**-24).all()
        assert torch.equal(tq.amax(x, 1), x.amax(1)) and torch.equal(tq.amin(x, 1), x.amin(1))
        best = x.max(1, keepdim=True).values
        first = torch.where(x == best, torch.arange(reduce, device="cuda").view(1, -1, 1), reduce).amin(1)      # the lowest index of the largest value
        assert torch.equal(tq.argmax(x, 1), first)


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("shape", [(64, 2048), (512, 768), (700, 32), (1000, 1000), (5184, 1000), (3072, 4096), (16384, 1024), (20000, 64)], ids=str)
def test_rows_of_a_transposed_view(tq, shape, dtype):
    x = drawn(shape, dtype, 7)
    w, b = drawn(shape[:1], dtype, 8), drawn(shape[:1], dtype, 9)
    wide = x.t().double()
    exact = torch.softmax(wide, -1)
    got = tq.softmax(x.t(), -1).double()
    rel = 2e-6 if dtype == torch.float32 else 2.0**-8 + 2e-6      # f32: ex2, the sum and a product, a few 2^-24 each
    assert ((got - exact).abs() <= rel * exact).all()
    exact = torch.nn.functional.layer_norm(wide, [shape[0]], w.double(), b.double(), 1e-5)
    got = tq.layer_norm(x.t(), [shape[0]], w, b, 1e-5).double()
    assert ((got - exact).abs() <= rel * exact.abs() + 4e-6 * (1 + exact.abs().max())).all()


def test_large_f32_views_of_short_columns_take_three_passes(tq):
    from tessiq_b200 import kernel as K

    forms = {(1, 4096, 16384): "three-pass", (1, 8192, 8192): "three-pass", (1, 16384, 4096): "three-pass",
             (2, 16384, 2048): "panels", (1, 24576, 4096): "panels", (1, 32768, 4096): "panels", (1, 32768, 1024): "three-pass"}
    for (batch, rows, cols), form in forms.items():
        assert K.transposed_form("softmax", torch.float32, batch, rows, cols) == form
    x = drawn((4096, 16384), torch.float32, 13)
    w, b = drawn((4096,), torch.float32, 14), drawn((4096,), torch.float32, 15)
    exact = torch.softmax(x.t().double(), -1)
    assert ((tq.softmax(x.t(), -1).double() - exact).abs() <= 2e-6 * exact).all()
    exact = torch.nn.functional.layer_norm(x.t().double(), [4096], w.double(), b.double(), 1e-5)
    assert ((tq.layer_norm(x.t(), [4096], w, b, 1e-5).double() - exact).abs() <= 2e-6 * exact.abs() + 4e-6 * (1 + exact.abs().max())).all()


@pytest.mark.parametrize("shape", [(64, 2048), (512, 768), (3072, 4096), (700, 32)], ids=str)
def test_special_values_in_columns(tq, shape):
    rows, cols = shape
    x = drawn(shape, torch.float32, 11)
    x[rows - 1, 0] = float("nan")
    x[rows // 2, 1] = float("inf")
    x[:, 2] = float("-inf")
    x[0, 3] = float("-inf")
    x[:, 4] = torch.finfo(torch.float32).min
    assert torch.equal(tq.amax(x, 0).isnan(), x.amax(0).isnan()) and torch.equal(tq.amax(x, 0)[1:], x.amax(0)[1:])
    arg = tq.argmax(x, 0)
    assert arg[0] == rows - 1 and arg[1] == rows // 2 and arg[2] == 0 and arg[4] == 0
    sums = tq.sum(x, 0)
    assert sums[0].isnan() and sums[1] == float("inf") and sums[2] == float("-inf") and sums[3] == float("-inf")
    soft, exact = tq.softmax(x.t(), -1), torch.softmax(x.t().double(), -1)
    assert torch.equal(soft.isnan(), exact.isnan())
    keep = ~exact.isnan().any(1)
    assert ((soft.double() - exact).abs()[keep] <= 2e-6 * exact[keep]).all()


def test_f64_columns_move_at_the_pace_of_memory(tq):
    """A sum down f64 columns reads what a copy reads and writes next to nothing: it takes less time than the copy. (With a register too few for
    its rows in flight it took 1.1 to 1.3 times as long.)"""
    for shape in ((60632, 2208), (6749, 5879), (3102, 11648)):
        x = torch.randn(shape, dtype=torch.float64, device="cuda")
        times = {}
        for name, call in (("sum", lambda: tq.sum(x, 0)), ("copy", lambda: x.clone())):
            call()
            for _ in range(5):
                start, end = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
                start.record()
                call()
                end.record()
                end.synchronize()
                times[name] = min(times.get(name, 1e9), start.elapsed_time(end))
        assert times["sum"] < 0.95 * times["copy"], (shape, times)
        assert (tq.sum(x, 0) - x.sum(0)).abs().max() <= 2.0**-52 * 40 * x.abs().sum(0).max()


def test_f32_column_sums_lose_no_digits_to_long_chains(tq):
    """Sums of values in [1, 2) round at every addition. Brought together in pairs, chains and trees the error of 16384 of them is that of the
    last few additions, 0.58 to 0.64 units of 2^-24 (root of the mean square, simulated for 32 to 256 threads a column); one chain
    a thread is at 0.77 and more with the 64 threads a column that the kernel has here. The bound lies between."""
    x = torch.rand(16384, 8192, generator=torch.Generator(device="cuda").manual_seed(16), device="cuda") + 1
    x.clamp_(max=2.0 - 2.0**-23)
    exact = x.double().sum(0)
    units = lambda got: (((got.double() - exact) / exact) ** 2).mean().sqrt().item() * 2.0**24  # noqa: E731
    rows = torch.zeros(64, 8192, device="cuda")
    for step in x.view(256, 64, 8192):
        rows += step
    while rows.shape[0] > 1:
        rows = rows[0::2] + rows[1::2]
    assert units(rows[0]) > 0.7      # one chain a thread, and a tree
    assert units(tq.sum(x, 0)) <= 0.7


@pytest.mark.parametrize("dtype, rows, cols", [(torch.float64, 79, 48000), (torch.float64, 80, 48000), (torch.float64, 80, 46800), (torch.float64, 2000, 77),
                                               (torch.float32, 300, 100000), (torch.float32, 300, 99968), (torch.int32, 300, 100004)], ids=str)
def test_both_sides_of_where_the_form_changes(tq, dtype, rows, cols):
    """f64 of 80 rows and 30 MB or less, 120 MB of four-byte elements: whole numbers, whose sums are exact in any order, with ties."""
    x = torch.randint(-9, 10, (rows, cols), generator=torch.Generator(device="cuda").manual_seed(rows), device="cuda").to(dtype)
    assert torch.equal(tq.sum(x, 0), x.sum(0)) and torch.equal(tq.amax(x, 0), x.amax(0)) and torch.equal(tq.amin(x, 0), x.amin(0))
