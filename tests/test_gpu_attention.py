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
    """One to four query rows stream the keys (5 is the first size the tensor-core kernel takes); 515 and 1000
    keys are shared by a cluster. Keys and values are views of a longer cache."""
    q = draw((2, queries, 3, width), dtype, 31).transpose(1, 2)
    cache = draw((2, 2, 3, keys + 9, width), dtype, 32)
    k, v = cache[0][:, :, 4:keys + 4], cache[1][:, :, 4:keys + 4]
    cache = cache.cuda()
    got = tq.attention(q.cuda(), cache[0][:, :, 4:keys + 4], cache[1][:, :, 4:keys + 4], width ** -0.5, causal)
    check(got, q, k, v, width ** -0.5, causal, oracle_atol=2e-2)
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
