"""A kernel may touch the shared memory of another CTA of its cluster only once that CTA runs, so every path to
such an access leads through a cluster barrier first. Nothing on a GPU shows a missing one (CTAs of a cluster
begin within a few cycles of each other, almost always), so the sources are read."""

import re
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "tessiq_b200" / "csrc"

TOUCH = re.compile(r"map_shared_rank\(|peer_address\(|shared::cluster\.(?:v4\.)?b32 \[")
BARRIER = re.compile(r"cluster_started\(\)|cluster_sync_all\(\)|\b(?:cluster|group)\.sync\(\)")
# A function's head up to the brace of its body.
FUNCTION = re.compile(r"__(?:global|device)__\b[^;{}]*?\b(?!__launch_bounds__)(\w+)\s*\((?:[^;{}]|\{\})*?\)\s*\{", re.S)


def functions(text):
    """[(is a kernel, name, body)] of the device code in `text`, comments taken out."""
    text = re.sub(r"//[^\n]*", "", text)
    found = []
    for match in FUNCTION.finditer(text):
        depth, at = 1, match.end()
        while depth:
            depth += {"{": 1, "}": -1}.get(text[at], 0)
            at += 1
        head = re.sub(r"__launch_bounds__\s*\([^()]*(?:\([^()]*\)[^()]*)*\)", "", match.group(0))
        name = re.search(r"(\w+)\s*\(", head).group(1)
        found.append(("__global__" in head, name, text[match.end():at]))
    return found


def unguarded(text):
    """The kernels in `text` that may touch a peer's shared memory before they have passed a cluster barrier."""
    found = functions(text)
    exposed = set()         # device functions that touch before any barrier of their own
    while True:
        def touches_first(body):
            touch = TOUCH.search(body)
            calls = [m for name in exposed for m in re.finditer(rf"\b{name}\s*(?:<[^;(){{}}]*>)?\(", body)]
            first = min([m.start() for m in ([touch] if touch else []) + calls], default=None)
            if first is None:
                return False
            barrier = BARRIER.search(body)
            return barrier is None or barrier.start() > first

        grown = {name for kernel, name, body in found if not kernel and touches_first(body)}
        if grown == exposed:
            return sorted({name for kernel, name, body in found if kernel and touches_first(body)})
        exposed = grown


@pytest.mark.parametrize("source", ["rownorm.cu", "reduce.cu", "slabnorm.cu", "decode.cu", "gemm.cu"])
def test_no_peer_is_touched_before_it_runs(source):
    text = (CSRC / source).read_text()
    assert any(TOUCH.search(body) for _, _, body in functions(text)), "the file no longer uses a peer's shared memory"
    assert unguarded(text) == []


def test_the_reader_finds_what_it_looks_for():
    helper = "__device__ void push(float v) { float* p = group.map_shared_rank(slots, 0); *p = v; group.sync(); }"
    assert unguarded(helper + "__global__ void __launch_bounds__(256) k(int n) { if (n) { push(1.f); } }") == ["k"]
    assert unguarded(helper + "__global__ void k(int n) { cluster_start(); load(); cluster_started(); push(1.f); }") == []
    assert unguarded("__global__ void k() { slots[0] = 1; cluster.sync(); v = *cluster.map_shared_rank(slots, 1); }") == []
