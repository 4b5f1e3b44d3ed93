"""Host threads that share a stream, its scratch, or a kernel."""

import threading
import time

import pytest
import torch


def run_threads(work, count):
    failures, start = [], threading.Barrier(count)

    def body(index):
        try:
            start.wait()
            work(index)
        except Exception as reason:  # noqa: BLE001
            failures.append(repr(reason))

    threads = [threading.Thread(target=body, args=(i,)) for i in range(count)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures


def test_threads_that_find_no_scratch_make_one_block(monkeypatch):
    from tessiq_b200 import kernel as K

    made = []

    def slow_empty(size, dtype, device):
        time.sleep(0.05)
        made.append(torch.zeros(size, dtype=dtype))
        return made[-1]

    monkeypatch.setattr(K, "torch", type("Slow", (), {"empty": staticmethod(slow_empty), "uint8": torch.uint8}))
    monkeypatch.setattr(K, "_workspaces", {})
    monkeypatch.setattr(K, "_outgrown", {})
    for nbytes in (64, 3 << 20):
        got = []
        run_threads(lambda i: got.append(K.workspace(0, 77, nbytes)), 4)
        assert len({id(block) for block in got}) == 1 and got[0].numel() >= nbytes
    assert len(made) == 2 and K._outgrown == {(0, 77): [made[0]]} and K._workspaces[(0, 77)] is made[1]


@pytest.mark.gpu
@pytest.mark.parametrize("own_stream", [False, True], ids=["the default stream", "a stream of their own"])
def test_threads_on_one_stream(own_stream):
    """Reductions that meet over tickets in scratch and normalisations that leave their statistics there: every thread's calls, one among
    the others', give what they give alone."""
    from tessiq_b200 import ops

    count, rounds = 6, 60
    g = torch.Generator(device="cuda").manual_seed(5)
    tall = [torch.randn(65536, 64, generator=g, device="cuda") for _ in range(count)]
    long = [torch.randn(1 << 21, generator=g, device="cuda") for _ in range(count)]
    view = [torch.randn(1024, 2048, generator=g, device="cuda").t() for _ in range(count)]

    def results(i):
        return ops.sum(tall[i], 0), ops.argmax(tall[i], 0), ops.sum(long[i]), ops.softmax(view[i], -1), ops.layer_norm(view[i], [1024], None, None, 1e-5)

    stream = torch.cuda.Stream() if own_stream else torch.cuda.default_stream()
    stream.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(stream):
        expected = [results(i) for i in range(count)]
    stream.synchronize()

    def work(i):
        with torch.cuda.stream(stream):
            for _ in range(rounds):
                for got, right in zip(results(i), expected[i]):
                    assert torch.equal(got, right)

    run_threads(work, count)


@pytest.mark.gpu
def test_threads_with_tiles_of_different_widths():
    """One kernel, launched by threads on streams of their own with other amounts of shared memory: no launch is refused for another's."""
    from tessiq_b200 import kernel as K
    from tessiq_b200 import ops

    shapes = {"argmax": [(1000, 8192), (3000, 64), (700, 512), (2000, 2048)], "sum": [(1000, 8192), (3000, 64), (700, 512), (2000, 2048)]}
    data = {shape: torch.randn(shape, generator=torch.Generator(device="cuda").manual_seed(6), device="cuda").bfloat16() for shape in shapes["sum"]}
    columns = [torch.randn(rows, 16, device="cuda").t() for rows in (8192, 12288, 32768, 49152)]      # slabs of other lengths
    assert all(K.transposed_form("softmax", torch.float32, 1, c.shape[1], 16) == "slab" for c in columns)
    expected = {(op, shape): getattr(ops, op)(data[shape], 0) for op in shapes for shape in data}
    rows = [ops.softmax(c, -1) for c in columns]
    torch.cuda.synchronize()

    def work(i):
        shape = shapes["sum"][i]
        with torch.cuda.stream(torch.cuda.Stream()):
            for _ in range(300):
                for op in shapes:
                    assert torch.equal(getattr(ops, op)(data[shape], 0), expected[op, shape])
                assert torch.equal(ops.softmax(columns[i], -1), rows[i])

    run_threads(work, 4)
