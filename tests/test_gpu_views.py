"""View operators of a compiled graph over values whose strides are not the traced ones."""

import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dtype", [torch.float32, torch.bfloat16], ids=["f32", "bf16"])
def test_a_view_of_a_result_that_torch_would_lay_out_otherwise(dtype):
    """torch lays the result of `x * 2 + 1` out like a transposed x, and traces a view that joins its axes; the fused kernel's is packed."""
    from tessiq_b200.backend import compile_graph

    def joined(x):
        y = x * 2 + 1
        return (y.t().reshape(-1) - 1).view(4, -1).sum(0)

    torch._dynamo.reset()
    compiled = torch.compile(joined, backend=compile_graph, dynamic=False)
    for seed in range(3):
        x = torch.randint(-8, 9, (8, 6), generator=torch.Generator(device="cuda").manual_seed(seed), device="cuda").to(dtype).t()
        assert torch.equal(compiled(x), joined(x))
    packed = torch.ones(6, 8, device="cuda", dtype=dtype)
    assert torch.equal(compiled(packed), joined(packed))
