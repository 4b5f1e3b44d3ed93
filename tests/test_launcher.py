"""Repeated calls of one signature go through the native launcher (csrc/launcher.cpp), and chains of view operators through
one step (executor._Views): both give what the first call, the long way, gave."""

import operator
import threading

import pytest
import torch
import torch.nn.functional as F
from torch import fx


# ---- views, on the CPU -------------------------------------------------------------------------


def view_recipe(functions, keep=()):
    """x -> functions[0] -> functions[1] -> ... as view steps, then a step that copies the last value."""
    from tessiq_b200.executor import Recipe, Step

    graph = fx.Graph()
    nodes = [graph.placeholder("x")] + [graph.call_function(operator.pos, (None,), name=f"v{i}") for i in range(len(functions))]
    copied = graph.call_function(operator.pos, (None,), name="copied")
    recipe = Recipe(inputs=["x"])
    for i, function in enumerate(functions):
        source = nodes[i].name
        recipe.steps.append(Step("view", nodes[i + 1].name, lambda env, f=function, s=source: f(env[s]), [source], view=function))
    recipe.steps.append(Step("pack", "copied", lambda env: env[nodes[-1].name].clone(), [nodes[-1].name]))
    recipe.outputs = tuple([copied] + [nodes[1 + i] for i in keep])
    recipe.finish()
    return recipe


CHAINS = {
    "split of a projection": [lambda t: t.view(2, 6, 24), lambda t: t.split([8, 8, 8], -1), lambda t: t[1], lambda t: t.view(2, 6, 2, 4), lambda t: t.permute(0, 2, 1, 3)],
    "identity": [lambda t: t.view(12, 24), lambda t: t.view(12, 24)],
    "expanded": [lambda t: t[:1], lambda t: t.expand(5, 24), lambda t: t.unsqueeze(0)],
    "a slice, then a copy": [lambda t: t[:, 3:9], lambda t: t.t(), lambda t: t.reshape(-1)],
    "nothing left": [lambda t: t[:0], lambda t: t.t()],
}


@pytest.mark.parametrize("name", CHAINS)
def test_a_chain_of_views_is_one_step_with_the_same_result(name):
    functions = CHAINS[name]
    inner = len(functions) - 1
    recipe = view_recipe(functions, keep=(inner,))
    assert len(recipe._schedule) == 2 and len(recipe.steps) == len(functions) + 1
    base = torch.arange(4 * 12 * 24).reshape(48, 24)
    # twice the same layout, another offset, another layout (where the views allow it)
    inputs = [base[:12], base[12:24].clone(), base[24:36], torch.nn.Parameter(base[:12].float(), requires_grad=False)]
    if name in ("expanded", "a slice, then a copy", "nothing left"):
        inputs.append(base.t()[:12, :24].t().contiguous().t()[:12])
    for x in inputs:
        expected = x
        for function in functions:
            expected = function(expected)
        copied, last = recipe.run(x)
        assert torch.equal(copied, expected) and torch.equal(last, expected)
        assert last.stride() == expected.stride() and last is not x
        assert (last.untyped_storage().data_ptr() == x.untyped_storage().data_ptr()) == (expected.untyped_storage().data_ptr() == x.untyped_storage().data_ptr())


def test_an_inner_view_that_is_also_read_by_itself():
    functions = [lambda t: t.view(4, 6), lambda t: t.t(), lambda t: t[1:3]]
    recipe = view_recipe(functions, keep=(0, 2))
    x = torch.arange(24)
    copied, first, last = recipe.run(x)
    assert torch.equal(first, x.view(4, 6)) and torch.equal(last, x.view(4, 6).t()[1:3]) and torch.equal(copied, last)
    assert len(recipe._schedule) == 3


# ---- the launcher, on the GPU -------------------------------------------------------------------


@pytest.fixture(scope="module")
def tq():
    if not torch.cuda.is_available():
        pytest.fail("the gpu tests need a CUDA device")
    from tessiq_b200 import ops

    return ops


def shaped(kind, rows, width, dtype, seed):
    """[rows, width] in one of the layouts a signature tells apart."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*shape):
        return torch.randn(shape, generator=g, device="cuda").to(dtype)

    if kind == "packed":
        return normal(rows, width)
    if kind == "transposed":
        return normal(width, rows).t()
    if kind == "columns":
        return normal(rows, 2 * width)[:, ::2]
    if kind == "off its boundary":
        return normal(rows * width + 1)[1:].view(rows, width)
    return normal(1, width).expand(rows, width)


def calls(tq, x, w, eps):
    rows, width = x.shape
    yield "add", tq.elementwise("add", x, w), x + w
    yield "scaled", tq.elementwise("mul", x, 0.5), x * 0.5
    yield "above", tq.elementwise("gt", x, 1), x > 1
    yield "sum", tq.sum(x, -1), x.float().sum(-1)
    yield "mean", tq.mean(x, [0], True), x.float().mean(0, keepdim=True)
    yield "amax", tq.amax(x), x.amax()
    yield "argmax", tq.argmax(x, 0), x.argmax(0)
    yield "pack", tq.clone(x), x
    yield "softmax", tq.softmax(x, -1), torch.softmax(x.float(), -1)
    yield "softmax 0", tq.softmax(x, 0), torch.softmax(x.float(), 0)
    yield "layer_norm", tq.layer_norm(x, [width], w, None, eps), F.layer_norm(x.float(), [width], w.float(), None, eps)
    y, mean, rstd = tq.native_layer_norm(x, (width,), w, w, eps)
    yield "native_layer_norm", y, F.layer_norm(x.float(), [width], w.float(), w.float(), eps)
    yield "its mean", mean, x.float().mean(-1, keepdim=True)
    if x.is_contiguous():
        yield "batch_norm", tq.batch_norm_eval(x, w, w, w, w.abs() + 1, eps), F.batch_norm(x.float(), w.float(), w.float().abs() + 1, w.float(), w.float(), False, 0.0, eps)


@pytest.mark.gpu
@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
@pytest.mark.parametrize("kind", ["packed", "transposed", "columns", "off its boundary", "expanded"])
@pytest.mark.parametrize("rows, width", [(64, 128), (17, 33), (1, 8)], ids=str)
def test_every_call_of_a_signature_gives_what_the_first_gives(tq, dtype, kind, rows, width):
    """First, second and third call of a signature, with other values and an epsilon of their own: 16-bit results within a rounding of the result and of
    the inputs' statistics, 32-bit ones within sums in another order."""
    rel = 1e-5 if dtype == torch.float32 else 2.0**-7
    for seed, eps in ((1, 1e-5), (2, 1e-5), (3, 1e-3), (4, 1e-3)):
        x = shaped(kind, rows, width, dtype, seed)
        w = torch.nn.Parameter(shaped("packed", 1, width, dtype, 10 + seed)[0], requires_grad=False)
        for name, got, expected in calls(tq, x, w, eps):
            assert got.shape == expected.shape, name
            if expected.dtype in (torch.bool, torch.int64):
                assert torch.equal(got, expected), name
            else:
                bound = rel * expected.float().abs() + rel * max(expected.float().abs().max().item(), 1e-3)
                assert ((got.float() - expected.float()).abs() <= bound).all(), name


@pytest.mark.gpu
def test_products_and_attention_again(tq):
    for seed in range(3):
        a, b = shaped("packed", 40, 64, torch.bfloat16, seed), shaped("packed", 72, 64, torch.bfloat16, 5 + seed)
        odd = shaped("off its boundary", 40, 64, torch.bfloat16, 9 + seed)      # copied first by the long way, every time
        bias = shaped("packed", 1, 72, torch.bfloat16, 20 + seed)[0]
        for left in (a, odd):
            expected = F.linear(left.float(), b.float(), bias.float())
            assert (tq.addmm(bias, left, b.t()).float() - expected).abs().max() <= 2.0**-7 * expected.abs().max()
        q = torch.randn(2, 3, 40, 64, device="cuda").bfloat16()
        for causal in (False, True):
            got = tq.attention(q, q, q, None, causal)
            expected = F.scaled_dot_product_attention(q.float(), q.float(), q.float(), is_causal=causal)
            assert (got.float() - expected).abs().max() <= 2.0**-6 * expected.abs().max() and got.transpose(1, 2).is_contiguous()


@pytest.mark.gpu
def test_what_is_refused_is_refused_again(tq):
    from tessiq_b200._lib import Declined

    x = torch.randn(4, 8, device="cuda")
    for _ in range(3):
        with pytest.raises(Declined):
            tq.sum(torch.empty(0, 4, device="cuda"), 0)
        with pytest.raises(ValueError):
            tq.elementwise("add", x, x.cpu())
        with pytest.raises(Declined):
            tq.elementwise("add", x, x.half())
        with pytest.raises(ValueError):
            tq.softmax(torch.randn(4, 8), -1)


@pytest.mark.gpu
def test_more_signatures_than_the_table_holds_and_several_threads(tq):
    from tessiq_b200 import _launcher

    x = torch.arange(3000, device="cuda", dtype=torch.float32)
    assert torch.equal(tq.clone(x[::2]), x[::2])
    for n in range(1, 2200):
        tq.clone(x[:n])
    assert _launcher.size() <= 2048
    assert torch.equal(tq.clone(x[::2]), x[::2])
    wrong = []

    def work(seed):
        with torch.cuda.stream(torch.cuda.Stream()):
            y = torch.full((257, 129), float(seed), device="cuda")
            for i in range(200):
                if not torch.equal(tq.sum(tq.elementwise("add", y, i), -1), (y + i).sum(-1)):
                    wrong.append((seed, i))

    threads = [threading.Thread(target=work, args=(seed,)) for seed in range(4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong


@pytest.mark.gpu
def test_planned_calls_under_capture(tq):
    x = torch.randn(300, 129, device="cuda")
    for _ in range(2):
        tq.softmax(tq.elementwise("mul", x, 2.0), -1)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        out = tq.softmax(tq.elementwise("mul", x, 2.0), -1)
    x.copy_(torch.randn(300, 129, device="cuda"))
    graph.replay()
    torch.cuda.synchronize()
    torch.testing.assert_close(out, torch.softmax(x * 2, -1), rtol=1e-5, atol=1e-6)
