"""Kernels that are launched while the one before them ends read what it wrote, and write nothing that it still reads."""

import numpy as np
import pytest
import torch

from tests.gpu_util import graph_ms, random_blocks, to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize(("batch", "columns"), (
    (1, 640),           # row kernel
    (5, 640),           # group sums, few rows
    (70, 1408),         # group sums on tcgen05
    (8, 1024)))         # mma.sync out of registers
def test_a_chain_of_calls_equals_one_call_at_a_time(batch, columns):
    """gather -> product -> rows for the next gather, buffers reused: without a synchronisation between the calls the results
    are those of a run that waits after every call."""
    from ternel_b200.ops import tq1_get_rows, tq1_matmul
    rows = 20000
    table, weight = (to_dev(random_blocks(n, columns, seed=n)[0]) for n in (rows, 4096))
    first = torch.arange(batch, device="cuda") * 7

    def run(wait):
        ids, seen = first.clone(), []
        for _ in range(40):
            x = tq1_get_rows(table, ids)
            if wait:
                torch.cuda.synchronize()
            y = tq1_matmul(weight, x, out_dtype=torch.float32)
            if wait:
                torch.cuda.synchronize()
            # the next rows come from the bits of this result
            torch.remainder(y[:, :3].contiguous().view(torch.int32).to(torch.int64).sum(dim=1), rows, out=ids)
            seen.append(ids.clone())
        return torch.stack(seen).cpu()

    want = run(True)
    assert len(torch.unique(want)) > 1
    for _ in range(5):
        assert torch.equal(run(False), want)


def test_a_captured_call_depends_fully_on_another_library_s_kernel():
    """In a graph a programmatic edge pays behind a kernel that lets the next one in. Behind any other kernel it costs time: a
    call there is an ordinary node, whichever stream and capture came before."""
    import ctypes
    from ternel_b200.ops import tq1_get_rows, tq1_matmul
    table, weight, ragged = (to_dev(random_blocks(n, k, seed=n)[0]) for n, k in ((500, 1024), (1024, 1024), (500, 640)))
    ids, x, other = torch.arange(16, device="cuda"), torch.ones((8, 1024), device="cuda").half(), torch.zeros(32, device="cuda")
    short = x[:, :640].contiguous()
    # gather, slice kernel, group sums of few rows, row kernel
    calls = (lambda: tq1_get_rows(table, ids), lambda: tq1_matmul(weight, x), lambda: tq1_matmul(ragged, short),
             lambda: tq1_matmul(ragged, short[:1]))
    cudart = ctypes.CDLL("libcudart.so.12")

    def edges(run):
        """Programmatic edges and all edges of the graph that `run` is captured as."""
        run()
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(graph):
            run()
        raw, count = ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
        assert cudart.cudaGraphGetEdges_v2(raw, None, None, None, ctypes.byref(count)) == 0
        nodes, data = (ctypes.c_void_p * (2 * count.value))(), (ctypes.c_uint8 * (8 * count.value))()
        assert cudart.cudaGraphGetEdges_v2(raw, nodes, ctypes.byref(nodes, 8 * count.value), data, ctypes.byref(count)) == 0
        return sum(data[8 * i + 2] != 0 for i in range(count.value)), count.value       # .type: 0 is a full dependency

    for call in calls:
        def apart():
            for _ in range(4):
                other.add_(1)
                call()

        def in_a_row():
            other.add_(1)
            for _ in range(4):
                call()

        assert edges(apart)[0] == 0
        assert edges(in_a_row) == (3, 4)
        assert edges(apart)[0] == 0


@pytest.mark.parametrize("tokens", (1, 3, 2049))
def test_gathers_of_both_forms_are_the_same(tokens):
    """The first gather of a graph is an ordinary launch, the ones behind it are dependent ones."""
    from ternel_b200.ops import tq1_get_rows
    table = to_dev(random_blocks(3000, 640, seed=8)[0])
    ids = torch.randint(-5, 3005, (tokens,), device="cuda")
    for dtype in (torch.float16, torch.float32):
        want = tq1_get_rows(table, ids, dtype=dtype)
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            got = [tq1_get_rows(table, ids, dtype=dtype) for _ in range(3)]
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(g, want) for g in got)


@pytest.mark.parametrize(("batch", "rows", "columns"), ((1, 300, 640), (5, 4099, 640), (16, 2400, 1408), (32, 4800, 640), (64, 9600, 640)))
def test_products_of_both_forms_are_the_same(batch, rows, columns):
    from ternel_b200.ops import tq1_matmul
    blocks, rng = random_blocks(rows, columns, seed=batch)
    w, x = to_dev(blocks), to_dev(rng.standard_normal((batch, columns)).astype(np.float16))
    want = tq1_matmul(w, x, out_dtype=torch.float32)
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        got = [tq1_matmul(w, x, out_dtype=torch.float32) for _ in range(3)]
    graph.replay()
    torch.cuda.synchronize()
    assert all(torch.equal(g, want) for g in got)


@pytest.mark.parametrize(("batch", "rows", "columns"), (
    (1, 1000, 1408), (1, 2048, 2176), (1, 4400, 9856), (1, 3300, 13184), (1, 5120, 17280), (1, 4400, 5248), (1, 512, 9856),
    (16, 4400, 9856), (16, 10000, 2176)))               # group sums of few rows
def test_calls_in_a_row_are_no_slower_than_calls_apart(batch, rows, columns):
    """Calls that come in while the one before them ends must not crowd on some SMs: in a row they take no longer than with a
    small kernel between them (1.9 times as long where they did)."""
    from ternel_b200.ops import tq1_matmul
    blocks, rng = random_blocks(rows, columns, seed=3)
    weight, x = to_dev(blocks), to_dev(rng.standard_normal((batch, columns)).astype(np.float16))
    other = torch.zeros(32, device="cuda")

    def apart(_):
        other.add_(1)
        tq1_matmul(weight, x)

    assert graph_ms(lambda _: tq1_matmul(weight, x)) <= 1.1 * graph_ms(apart)


@pytest.mark.parametrize(("batch", "rows", "columns", "form"), (
    (1, 4096, 640, "rows"), (5, 4096, 640, "groups_few"), (100, 9000, 640, "groups_many"), (48, 4099, 2176, "groups_tcgen05"),
    (8, 4096, 1024, "slices"), (64, 1024, 1024, "tcgen05"), (1, 1024, 1024, "stream_gemv")))
def test_no_kernel_writes_what_an_earlier_one_reads(batch, rows, columns, form):
    """Nothing but this library's kernels on a stream: a gather overwrites the activations that the product before it reads, two
    products in a row read them, and the second one's results are overwritten each time. As with a synchronisation after every
    call, eagerly and as a graph."""
    import ctypes
    from ternel_b200 import _native
    from ternel_b200.dispatch import plan
    assert plan(batch, rows, columns).form == form
    lib, turns = _native.lib(), 12
    table, weight = (to_dev(random_blocks(n, columns, seed=n)[0]) for n in (500, rows))
    ids = torch.randint(0, 500, (turns, batch), device="cuda")
    x = torch.zeros((batch, columns), dtype=torch.float16, device="cuda")
    last, kept = torch.zeros((batch, rows), device="cuda"), torch.zeros((turns, batch, rows), device="cuda")
    need = lib.tq1_linear_workspace_bytes(batch, rows, columns)
    scratch = torch.zeros(max(need, 256), dtype=torch.uint8, device="cuda")

    def run(wait):
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)

        def done(status):
            assert status == 0
            if wait:
                torch.cuda.synchronize()

        def product(y):
            done(lib.tq1_linear_f16(weight.data_ptr(), x.data_ptr(), y.data_ptr(), 1, batch, rows, columns, scratch.data_ptr(),
                                    need, stream))

        for i in range(turns):
            done(lib.tq1_embedding_f16(table.data_ptr(), ids[i].data_ptr(), x.data_ptr(), 0, batch, 500, columns, stream))
            product(kept[i])
            product(last)

    run(True)
    want, want_last = kept.clone(), last.clone()
    assert torch.equal(want[-1], want_last) and not torch.equal(want[0], want[1])

    def check(go):
        kept.zero_()
        last.zero_()
        go()
        torch.cuda.synchronize()
        assert torch.equal(kept, want) and torch.equal(last, want_last)

    for _ in range(10):
        check(lambda: run(False))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        run(False)
    for _ in range(10):
        check(graph.replay)
    assert int(scratch[:4].view(torch.int32).item()) == 0
