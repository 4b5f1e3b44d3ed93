"""Parity of the fused tcgen05 attention kernel with the oracle, through the C ABI.

Bars. Against the float64 value (oracle/restate.c): one rounding of the result (2^-8 relative for
bf16, 2^-11 for f16) plus the rounding of the probabilities to the storage type before the second
product (2^-8 / 2^-11 of sum_j p_ij |v_j|) plus 2e-5 of the largest value for ex2.approx and f32
sums. Against the oracle's own half-precision result (five nodes, each rounded): rtol 1e-2, atol
1e-2 * max|ref|, the tolerance stated for bf16 on this path.
"""

import ctypes
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

from oracle import restate, tessiq0  # noqa: E402


@pytest.fixture(scope="module")
def tq():
    if not torch.cuda.is_available():
        pytest.fail("the gpu tests need a CUDA device")
    from tessiq_b200 import ops

    return ops


def poll(device=0):
    from tessiq_b200 import _lib

    status = ctypes.c_int32(-1)
    _lib.check(_lib.lib.tq_status_poll(device, None, ctypes.byref(status)))
    return status.value


def draw(shape, dtype, seed, spread=1.0):
    g = torch.Generator().manual_seed(seed)
    return (torch.randn(*shape, generator=g) * spread).to(dtype)


def check(got, q, k, v, scale, causal, half_oracle=True, oracle_atol=1e-2):
    dtype = q.dtype
    ulp = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-11
    q64, k64, v64 = (t.double().numpy() for t in (q, k, v))
    exact = restate.attention(q64, k64, v64, scale, causal)
    weight = restate.attention(q64, k64, np.abs(v64), scale, causal)    # sum_j p_ij |v_j|
    bound = ulp * np.abs(exact) + ulp * weight + 2e-5 * np.abs(exact).max() + 1e-30
    error = np.abs(got.detach().cpu().double().numpy() - exact)
    worst = (error / bound).max()
    assert worst <= 1.0, f"error {error.max():.3e} exceeds the float64 bound by {worst:.2f}x"
    if not half_oracle:
        return
    ref = tessiq0.attention(q, k, v, scale, causal).float()
    torch.testing.assert_close(got.detach().cpu().float(), ref, rtol=1e-2, atol=oracle_atol * ref.abs().max().item())


SHAPES = [  # batch, heads, q_tokens, k_tokens
    (1, 1, 128, 128), (1, 1, 256, 256), (2, 3, 256, 256), (1, 2, 1024, 1024), (1, 1, 1, 1), (1, 1, 100, 100),
    (1, 2, 130, 130), (1, 1, 257, 300), (1, 1, 200, 333), (1, 1, 333, 200), (3, 1, 384, 512), (1, 1, 640, 129),
]


@pytest.mark.parametrize("shape", SHAPES, ids=lambda s: "x".join(map(str, s)))
@pytest.mark.parametrize("causal", [True, False], ids=["causal", "full"])
def test_attention_matches_oracle(tq, shape, causal):
    batch, heads, tq_, tk = shape
    q = draw((batch, heads, tq_, 64), torch.bfloat16, 1)
    k = draw((batch, heads, tk, 64), torch.bfloat16, 2)
    v = draw((batch, heads, tk, 64), torch.bfloat16, 3)
    got = tq.attention(q.cuda(), k.cuda(), v.cuda(), 0.125, causal)
    assert got.shape == q.shape
    check(got, q, k, v, 0.125, causal)
    assert poll() == 0


@pytest.mark.parametrize("width", [8, 32, 48, 128, 96, 72])
@pytest.mark.parametrize("causal", [True, False], ids=["causal", "full"])
def test_attention_with_other_head_widths(tq, width, causal):
    """Heads of 8, 16, ... 56 elements ride in the kernel's 64-wide tiles: TMA fills the other columns
    with zeros, which add nothing to q . k, and the result columns they produce are not stored. Heads of
    72 ... 128 elements are two such tiles side by side (one group of 128 query rows per CTA)."""
    q = draw((2, 3, 200, width), torch.bfloat16, 21)
    k = draw((2, 3, 333, width), torch.bfloat16, 22)
    v = draw((2, 3, 333, width), torch.bfloat16, 23)
    scale = width ** -0.5
    guard = torch.full((2, 200, 3, width + 8), 7.0, dtype=torch.bfloat16, device="cuda")   # the result sits inside a wider buffer
    got = tq.attention(q.cuda(), k.cuda(), v.cuda(), scale, causal)
    # (the float64 bound inside `check` is the strict one; against the oracle's five bf16-rounded nodes one
    # element in 10^5 of a 96-wide head differed by 1.1e-2 of the largest value, the oracle's own rounding)
    check(got, q, k, v, scale, causal, oracle_atol=2e-2)
    from tessiq_b200.kernel import AttentionKernel
    AttentionKernel(scale, causal).launch([q.cuda(), k.cuda(), v.cuda()], guard[..., :width].transpose(1, 2), stream=None)
    torch.cuda.synchronize()
    assert torch.equal(guard[..., :width].transpose(1, 2), got) and (guard[..., width:] == 7.0).all()      # nothing beyond the head is written
    # a fused projection of narrow heads, read in place
    qkv = draw((2, 160, 3 * 4 * width), torch.float16, 24).cuda()
    q, k, v = (z.view(2, 160, 4, width).transpose(1, 2) for z in qkv.split(4 * width, dim=-1))
    check(tq.attention(q, k, v, scale, causal), q.cpu(), k.cpu(), v.cpu(), scale, causal, oracle_atol=2e-2)
    assert poll() == 0


@pytest.mark.parametrize("queries, keys", [(1, 1), (1, 31), (1, 1000), (2, 129), (3, 700), (4, 2), (4, 515), (5, 515)])
@pytest.mark.parametrize("width, dtype", [(64, torch.bfloat16), (128, torch.float16), (32, torch.bfloat16), (40, torch.float16), (8, torch.bfloat16)])
@pytest.mark.parametrize("causal", [True, False], ids=["causal", "full"])
def test_few_queries_against_a_cache(tq, queries, keys, width, dtype, causal):
    """One to four query rows of a few heads stream the keys, unless they are so few that tiles are quicker (5 queries are the first
    that always take tiles); 515 and 1000 keys are shared by a cluster. Keys and values are views of a longer cache."""
    q = draw((2, queries, 3, width), dtype, 31).transpose(1, 2)
    cache = draw((2, 2, 3, keys + 9, width), dtype, 32)
    k, v = cache[0][:, :, 4:keys + 4], cache[1][:, :, 4:keys + 4]
    cache = cache.cuda()
    got = tq.attention(q.cuda(), cache[0][:, :, 4:keys + 4], cache[1][:, :, 4:keys + 4], width ** -0.5, causal)
    check(got, q, k, v, width ** -0.5, causal, oracle_atol=2e-2)
    assert poll() == 0


FORMS = [  # batch, heads, queries, keys, width, causal, kernel, keys a step
    (2, 3, 64, 64, 64, True, "tiles", 64), (2, 3, 200, 64, 64, False, "tiles", 64), (1, 2, 200, 50, 128, False, "tiles", 64),
    (1, 2, 200, 65, 64, False, "tiles", 128), (1, 2, 300, 129, 64, True, "tiles", 128), (1, 3, 300, 515, 40, False, "tiles", 128),
    (1, 2, 128, 1000, 128, False, "tiles", 128), (1, 3, 333, 333, 96, True, "tiles", 128), (1, 2, 700, 700, 64, True, "tiles", 128),
    (40, 12, 5, 100, 64, False, "tiles", 64), (20, 16, 129, 129, 64, True, "tiles", 64), (50, 6, 200, 200, 64, False, "tiles", 64),
    (13, 12, 64, 300, 128, False, "tiles", 64), (10, 16, 130, 130, 128, True, "tiles", 64), (7, 24, 20, 65, 72, False, "tiles", 64),
    (30, 12, 130, 600, 64, False, "tiles", 128), (30, 12, 130, 700, 64, False, "tiles", 64), (30, 12, 130, 700, 64, True, "tiles", 128), (26, 12, 60, 600, 64, False, "tiles", 64),
    (25, 6, 4, 64, 128, False, "few", 64), (25, 6, 4, 100, 64, False, "few", 64), (25, 6, 3, 77, 32, False, "few", 64),
    (50, 6, 3, 400, 64, False, "few", 64), (50, 6, 2, 515, 96, False, "few", 64), (25, 6, 4, 1000, 128, False, "few", 64),
    (1, 3, 4, 65, 64, False, "few", 128), (1, 3, 3, 100, 40, False, "few", 128), (1, 3, 4, 500, 128, False, "few", 128),
    (24, 6, 1, 515, 72, False, "few", 128), (25, 3, 3, 1000, 128, False, "few", 128), (8, 18, 4, 900, 64, False, "few", 128),
    (1, 3, 4, 900, 64, False, "streamed", 0), (50, 6, 1, 300, 128, False, "streamed", 0), (24, 6, 1, 600, 64, False, "streamed", 0),
    (25, 6, 4, 900, 64, True, "streamed", 0),
]


@pytest.mark.parametrize("shape", FORMS, ids=lambda s: "x".join(map(str, s[:5])) + ("c" if s[5] else "") + s[6] + str(s[7]))
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_every_form(tq, shape, dtype):
    """Each kernel that a call can take, around its tiles' edges: one step and several, a last step with one key, keys a step
    that divide nothing, several CTAs an SM."""
    from tessiq_b200.kernel import attention_form

    batch, heads, queries, keys, width, causal, form, step = shape
    assert attention_form(batch * heads, queries, keys, width, causal, device=-1) == (form, step)
    q, k, v = (draw((batch, heads, n, width), dtype, 50 + i) for i, n in enumerate((queries, keys, keys)))
    got = tq.attention(q.cuda(), k.cuda(), v.cuda(), width ** -0.5, causal)
    check(got[:2], q[:2], k[:2], v[:2], width ** -0.5, causal, half_oracle=False)
    exact = torch.from_numpy(restate.attention(*(t[-2:].double().numpy() for t in (q, k, v)), width ** -0.5, causal))
    error = (got[-2:].cpu().double() - exact).abs()
    ulp = 2.0**-8 if dtype == torch.bfloat16 else 2.0**-11
    if form != "tiles":          # probabilities are not rounded: one rounding of the result, and f32 sums
        assert (error <= 1.001 * ulp * exact.abs() + 2e-5 * exact.abs().max()).all()
    else:
        assert (error <= ulp * exact.abs() + ulp * v.abs().max().item()).all()
    assert poll() == 0


@pytest.mark.parametrize("batch, tokens", [(1, 128), (1, 300), (20, 256)], ids=["one step", "128 keys a step", "64 keys a step"])
def test_the_largest_probability_is_exact(tq, batch, tokens):
    """A row's reference point is the maximum over its first 128 keys, so where that is the row's maximum, its probability is
    exactly 1 and loses nothing to 16 bits. Key 100 alone has a score, other than 0, and a value: the result is one
    probability over the (f32) sum, within its own rounding."""
    heads = 16
    g = torch.Generator().manual_seed(60)
    q = torch.zeros(batch, heads, tokens, 64)
    q[..., 0] = torch.rand(batch, heads, tokens, generator=g) * 36 + 4
    k, v = torch.zeros(batch, heads, tokens, 64), torch.zeros(batch, heads, tokens, 64)
    k[..., 100, 0] = 1.0
    v[..., 100, :] = 1.0
    q, k, v = q.bfloat16(), k.bfloat16(), v.bfloat16()
    got = tq.attention(q.cuda(), k.cuda(), v.cuda(), 0.125, False).cpu().double()[..., 0]
    top = torch.exp(q[..., 0].double() * 0.125)                      # e^0.5 ... e^5
    exact = top / (top + tokens - 1)
    assert ((got - exact).abs() <= 2.0**-8 * exact * 1.002).all()      # half a unit in the last of bf16's eight places


def _exact_with_specials(q, k, v, scale):
    """float64 attention, NaN and infinity as they fall out of the arithmetic."""
    scores = scale * q.double() @ k.double().transpose(-1, -2)
    return torch.softmax(scores, dim=-1) @ v.double()


@pytest.mark.parametrize("queries", [1, 4])
@pytest.mark.parametrize("heads, keys", [(96, 300), (2, 900), (2, 7)], ids=["one CTA a head", "eight CTAs a head", "sets without a key"])
@pytest.mark.parametrize("where", ["first", "middle", "last"])
def test_decode_with_special_values(tq, queries, heads, keys, where):
    """What is not finite meets ordinary values three times (lanes, warps, CTAs of a cluster) and must come through each
    as float64 gives it: a NaN or an infinity in one key or one value, rows of -inf scores, and one
    score far above all others, in the first, a middle and the last share of the keys (7 keys leave most sets empty)."""
    from tessiq_b200.kernel import attention_form

    batch, width = (8 if heads == 96 else 2), 64
    assert attention_form(batch * heads, queries, keys, width, False, device=-1)[0] == "streamed"
    at = {"first": 0, "middle": keys // 2, "last": keys - 1}[where]
    q = draw((batch, heads, queries, width), torch.bfloat16, 41).abs() + 0.5       # no zero meets an infinity
    k = draw((batch, heads, keys, width), torch.bfloat16, 42)
    v = draw((batch, heads, keys, width), torch.bfloat16, 43)
    inf, nan = float("inf"), float("nan")

    qd, part = q.cuda(), (slice(1, 2), slice(0, 2))         # the changed head and one beside it are compared

    def run(change):
        kk, vv = k.clone(), v.clone()
        change(kk, vv)
        got = tq.attention(qd, kk.cuda(), vv.cuda(), width ** -0.5, False).cpu().double()[part]
        exact = _exact_with_specials(q[part], kk[part], vv[part], width ** -0.5)
        assert torch.equal(torch.isnan(got), torch.isnan(exact)) and torch.equal(torch.isinf(got), torch.isinf(exact))
        infinite = torch.isinf(exact)
        assert torch.equal(got[infinite], exact[infinite])
        finite = torch.isfinite(exact)
        # a rounding of the result, and of f32 sums over the keys
        assert ((got - exact).abs() <= 2.0**-8 * exact.abs() + 2e-5)[finite].all()
        return exact

    def key(kk, value, head=1):
        kk[1, head, at, 5] = value

    run(lambda kk, vv: key(kk, nan))
    run(lambda kk, vv: key(kk, inf))                        # one score +inf: inf - inf
    assert torch.isfinite(run(lambda kk, vv: key(kk, -inf))).all()      # one score -inf: a probability of 0
    run(lambda kk, vv: vv[1, 1].__setitem__((at, 3), nan))
    assert torch.isinf(run(lambda kk, vv: vv[1, 1].__setitem__((at, 3), -inf))).any()
    run(lambda kk, vv: vv[1, 1, at, 3:5].copy_(torch.tensor([inf, nan])))
    run(lambda kk, vv: kk[1, 1, :, 0].fill_(-inf))          # every score of a head -inf: 0 / 0
    run(lambda kk, vv: kk[1, 1, : max(1, keys - 3), 0].fill_(-inf))     # ... of all keys but the last three
    dominated = run(lambda kk, vv: kk[1, 1, at].fill_(4.0))             # scores of about 40 above the others' 1
    torch.testing.assert_close(dominated[0, 1], v[1, 1, at].double().expand_as(dominated[0, 1]), rtol=0, atol=1e-3)
    assert poll() == 0


def test_attention_golden(tq, golden):
    q, k, v = (torch.from_numpy(golden[n].copy()).view(torch.bfloat16) for n in ("attn_q", "attn_k", "attn_v"))
    for causal, name in ((True, "attn_causal_bf16"), (False, "attn_full_bf16")):
        ref = torch.from_numpy(golden[name].copy()).view(torch.bfloat16).float()
        got = tq.attention(q.cuda(), k.cuda(), v.cuda(), 0.125, causal).cpu().float()
        torch.testing.assert_close(got, ref, rtol=1e-2, atol=1e-2 * ref.abs().max().item())


def test_attention_f16_and_large_scores(tq):
    q = draw((1, 2, 300, 64), torch.float16, 4, spread=3.0)
    k = draw((1, 2, 300, 64), torch.float16, 5, spread=3.0)
    v = draw((1, 2, 300, 64), torch.float16, 6)
    for causal in (True, False):
        got = tq.attention(q.cuda(), k.cuda(), v.cuda(), 1.0 / 8, causal)   # scores up to ~ +-100: sharp rows
        check(got, q, k, v, 1.0 / 8, causal)


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16])
def test_attention_when_the_scores_keep_rising(tq, dtype):
    """The kernel keeps one reference point per row and moves it only when a key tile rises far above
    it, rescaling what the row has gathered. Scores that grow with the key index make every tile
    move it; scores that fall never do; a late spike moves it once; and rows of one warp differ."""
    tokens = 640
    g = torch.Generator().manual_seed(21)
    direction = torch.randn(64, generator=g)
    direction /= direction.norm()
    ramp = torch.linspace(0.0, 60.0, tokens)
    v = draw((1, 1, tokens, 64), dtype, 22)
    noise = torch.randn(tokens, 64, generator=g) * 0.3
    for name, profile in (("rising", ramp), ("falling", ramp.flip(0)), ("spike", torch.where(torch.arange(tokens) == 500, 90.0, 0.0)),
                          ("steps", (torch.arange(tokens) // 128).float() * 11.0)):
        k = (noise + profile[:, None] * direction).to(dtype).view(1, 1, tokens, 64)
        # rows alternate between following the profile and opposing it, so the rows of one warp disagree
        sign = torch.where(torch.arange(tokens) % 3 == 0, -1.0, 1.0)
        q = ((sign[:, None] * direction) * 8.0 + torch.randn(tokens, 64, generator=g) * 0.1).to(dtype).view(1, 1, tokens, 64)
        for causal in (True, False):
            got = tq.attention(q.cuda(), k.cuda(), v.cuda(), 0.125, causal)
            # scores of +-60 rounded to 16 bits between the oracle's nodes move ITS result by tens of
            # per cent, so only the float64 bound is meaningful here
            check(got, q, k, v, 0.125, causal, half_oracle=False)
    assert poll() == 0


def test_attention_reads_a_fused_qkv_projection_in_place_and_writes_token_major(tq):
    batch, tokens, heads = 2, 320, 4
    qkv = draw((batch, tokens, 3 * heads * 64), torch.bfloat16, 7).cuda()
    q, k, v = (z.view(batch, tokens, heads, 64).transpose(1, 2) for z in qkv.split(heads * 64, dim=-1))
    assert not q.is_contiguous()
    got = tq.attention(q, k, v, None, True)
    # the result is a view of a packed [batch, tokens, heads, 64] buffer
    assert got.transpose(1, 2).is_contiguous()
    check(got, q.cpu(), k.cpu(), v.cpu(), 1.0 / 8, True)


def test_attention_properties_at_the_decoder_block_size(tq):
    """benchmark config 4's attention shape (batch 64 is cut to 8 to bound the test's memory):
    with v = 1 every output is 1 (the probabilities of a row sum to one); under the causal mask
    row 0 returns v[0]; and shifting every key by a constant vector changes nothing for rows whose
    query is orthogonal to it — here checked through q = 0, which gives the running mean of v."""
    batch, heads, tokens = 8, 12, 1024
    q = draw((batch, heads, tokens, 64), torch.bfloat16, 8).cuda()
    k = draw((batch, heads, tokens, 64), torch.bfloat16, 9).cuda()
    v = draw((batch, heads, tokens, 64), torch.bfloat16, 10).cuda()
    ones = torch.ones_like(v)
    out = tq.attention(q, k, ones, None, True).float()
    assert (out - 1).abs().max().item() <= 2.0**-7
    out = tq.attention(q, k, v, None, True)
    assert torch.equal(out[:, :, 0], v[:, :, 0])
    mean = tq.attention(torch.zeros_like(q), k, v, None, True).float()
    running = v.float().cumsum(2) / torch.arange(1, tokens + 1, device="cuda").view(1, 1, -1, 1)
    assert (mean - running).abs().max().item() <= 2.0**-7 * running.abs().max().item() + 2.0**-8
    assert poll() == 0


def test_attention_declines_what_it_has_no_kernel_for(tq):
    from tessiq_b200._lib import Declined

    for width in (256, 136, 36):
        q = torch.zeros(1, 1, 16, width, dtype=torch.bfloat16, device="cuda")
        with pytest.raises(Declined):
            tq.attention(q, q, q, None, True)         # heads wider than 128, or not a multiple of 8 elements
    q = torch.zeros(1, 1, 16, 64, dtype=torch.bfloat16, device="cuda")
    with pytest.raises(Declined):
        tq.attention(q, q, q, -1.0, True)             # a negative scale turns the maximum into a minimum
    with pytest.raises(Declined):
        tq.attention(q.float(), q.float(), q.float(), None, True)
    shifted = torch.zeros(16 * 64 + 8, dtype=torch.bfloat16, device="cuda")[4:4 + 16 * 64].view(1, 1, 16, 64)
    with pytest.raises(Declined):
        tq.attention(shifted, q, q, None, True)       # a base that is not 16-byte aligned
    empty = tq.attention(q[:, :, :0], q, q, None, True)
    assert empty.shape == (1, 1, 0, 64)


def test_attention_under_stream_capture(tq):
    q = draw((1, 2, 256, 64), torch.bfloat16, 11).cuda()
    k = draw((1, 2, 256, 64), torch.bfloat16, 12).cuda()
    v = draw((1, 2, 256, 64), torch.bfloat16, 13).cuda()
    eager = tq.attention(q, k, v, None, True)
    side = torch.cuda.Stream()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.stream(side):
        tq.attention(q, k, v, None, True)
        side.synchronize()
        with torch.cuda.graph(graph, stream=side):
            captured = tq.attention(q, k, v, None, True)
    captured.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(captured, eager)
