"""Which kernel a shape gets, against recorded kernel times (B200, bf16, microseconds; graphs of launches over rotating
operands): a changed constant or rule that sends a shape to a form recorded as slower fails here, without a GPU."""

import pytest

from tessiq_b200.kernel import attention_form

# (batch * heads, queries, keys, head, causal): {(kernel, keys a step): time}
ATTENTION_TIMES = {
    (768, 1024, 1024, 64, True): {("tiles", 64): 228.7, ("tiles", 128): 228.7},
    (96, 1024, 1024, 64, True): {("tiles", 64): 41.9, ("tiles", 128): 38.4},
    (8, 4096, 4096, 64, True): {("tiles", 64): 69.0, ("tiles", 128): 54.4},
    (12, 4096, 4096, 64, False): {("tiles", 64): 90.6, ("tiles", 128): 92.8},
    (768, 64, 64, 64, True): {("tiles", 64): 11.4, ("tiles", 128): 15.5},
    (384, 1024, 1024, 128, True): {("tiles", 64): 174.7, ("tiles", 128): 225.0},
    (16, 1024, 1024, 128, True): {("tiles", 64): 21.1, ("tiles", 128): 15.7},
    (8, 100, 8000, 64, False): {("tiles", 64): 107.9, ("tiles", 128): 77.6},
    (96, 16, 1000, 64, False): {("tiles", 64): 18.5, ("tiles", 128): 14.4},
    (96, 128, 2000, 128, False): {("tiles", 64): 40.9, ("tiles", 128): 30.0},
    (320, 200, 200, 64, False): {("tiles", 64): 19.0, ("tiles", 128): 19.4},
    (768, 8, 1000, 128, False): {("tiles", 64): 75.2, ("tiles", 128): 87.9},
    (3072, 16, 16, 64, False): {("tiles", 64): 30.8, ("tiles", 128): 47.4},
    (768, 4, 1000, 64, False): {("streamed", 0): 72.9, ("few", 64): 52.8, ("few", 128): 78.6},
    (768, 4, 1000, 128, False): {("streamed", 0): 143.3, ("few", 64): 73.9, ("few", 128): 90.7},
    (768, 2, 1000, 128, False): {("streamed", 0): 84.9, ("few", 64): 74.3, ("few", 128): 90.8},
    (768, 2, 1000, 64, False): {("streamed", 0): 49.2, ("few", 64): 53.1, ("few", 128): 78.4},
    (768, 4, 100, 64, False): {("streamed", 0): 13.9, ("few", 64): 17.2, ("few", 128): 28.1},
    (96, 4, 4000, 128, False): {("streamed", 0): 79.7, ("few", 64): 71.3, ("few", 128): 50.1},
    (96, 4, 4000, 64, False): {("streamed", 0): 41.0, ("few", 64): 53.7, ("few", 128): 43.4},
    (8, 4, 4000, 128, False): {("streamed", 0): 36.1, ("few", 64): 66.0, ("few", 128): 44.0},
    (8, 4, 100, 64, False): {("streamed", 0): 5.7, ("few", 64): 5.5, ("few", 128): 5.1},
    (1024, 3, 4000, 64, False): {("streamed", 0): 289.9, ("few", 64): 212.1, ("few", 128): 288.7},
    (768, 2, 4000, 96, False): {("streamed", 0): 307.9, ("few", 64): 229.6, ("few", 128): 280.6},
    (8, 2, 4000, 64, False): {("streamed", 0): 11.8, ("few", 64): 51.6, ("few", 128): 40.9},
    (288, 4, 1000, 64, False): {("streamed", 0): 27.2, ("few", 64): 20.5, ("few", 128): 28.7},
}


def slower(chosen, times):
    """How much longer the chosen form took than the best, beyond what two runs differ by (3 %, 0.3 us)."""
    return times[chosen] - 1.03 * min(times.values()) - 0.3


@pytest.mark.parametrize("shape", ATTENTION_TIMES, ids=str)
def test_attention_takes_the_form_recorded_as_fastest(shape):
    assert slower(attention_form(*shape, device=-1), ATTENTION_TIMES[shape]) <= 0


def test_forms_of_impossible_shapes_are_refused():
    with pytest.raises(ValueError):
        attention_form(0, 1, 1, 64, False, device=-1)
    with pytest.raises(TypeError):
        attention_form(1, 1, 1, 36, False, device=-1)
