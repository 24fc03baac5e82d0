"""One and two activation rows by the tile kernel: bit for bit what the chain kernel gives for one link. Needs a B200."""

import numpy as np
import pytest
import torch

from oracle import tq1_oracle as o
from tests.gpu_util import random_blocks, to_dev

pytestmark = pytest.mark.gpu

# (rows, columns): one row, tile remainders, twenty sets of one chunk and fewer; the widest K range of one CTA (18 chunks), and
# clusters of four (19 and 34 chunks: parts of unequal length) and eight (80 chunks, the most for two activation rows, and 128,
# where two rows are links of the chain kernel); several tiles per set
SHAPES = ((1, 512), (15, 512), (2375, 512), (50002, 512), (33, 1536), (4100, 4096), (12018, 5120), (2400, 9216), (2390, 9728),
          (1202, 17408), (49, 40960), (49, 65536))


def single_links(blocks, x, swiglu):
    from ternel_b200.chain import ChainPlan, Link
    rows = blocks.shape[0] // 2 if swiglu else blocks.shape[0]
    y = torch.empty((x.shape[0], rows), dtype=torch.float32, device="cuda")
    for m in range(x.shape[0]):
        ChainPlan([Link(blocks=blocks, x=x[m], y=y[m], swiglu=swiglu)]).run()
    torch.cuda.synchronize()
    return y


@pytest.mark.parametrize(("rows", "columns"), SHAPES)
def test_equals_the_chain_kernel(rows, columns):
    from ternel_b200.dispatch import ring_layout
    from ternel_b200.ops import tq1_matmul, tq1_swiglu
    for batch in (1, 2):
        layout = ring_layout("stream_gemv", batch, rows, columns)
        assert layout is None if (batch, columns) == (2, 65536) else layout.preferred
    host, rng = random_blocks(rows, columns, seed=rows + columns, dist="tests")
    blocks = to_dev(host)
    x = to_dev(rng.standard_normal((2, columns)).astype(np.float16))
    x[1, ::3] *= 2.0 ** -9                      # groups of a wide range
    want = single_links(blocks, x, False)
    if rows * columns < 6_000_000:
        exact = o.float64_matmul(host, x.cpu().numpy(), rows=rows, columns=columns)
        assert o.normalised_error(want.cpu().numpy(), exact) < 1e-5
    for batch in (1, 2):
        assert torch.equal(tq1_matmul(blocks, x[:batch], out_dtype=torch.float32), want[:batch])
        assert torch.equal(tq1_matmul(blocks, x[:batch]), want[:batch].half())
    if rows % 2 == 0:
        gated = single_links(blocks, x, True)
        for batch in (1, 2):
            assert torch.equal(tq1_swiglu(blocks, x[:batch], out_dtype=torch.float32), gated[:batch])


# Rings that are gone round: two sets of warps on eight stages, three on twelve, five and two on twenty, twenty on sixty, and two
# and one on six in a cluster of two
ROUND = ((40961, 5120, 1), (34816, 3072, 1), (50001, 2048, 1), (50001, 2048, 2), (151934, 512, 1), (34815, 10240, 1), (34815, 10240, 2))


@pytest.mark.parametrize(("rows", "columns", "batch"), ROUND)
def test_stages_that_are_filled_again(rows, columns, batch):
    from ternel_b200.dispatch import ring_layout
    from ternel_b200.ops import tq1_matmul
    from ternel_b200.stack import random_blocks_device
    layout = ring_layout("stream_gemv", batch, rows, columns)
    assert layout.tiles > layout.stages
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows + columns)
    blocks = random_blocks_device(rows, columns, gen, "cuda")
    x = torch.randn((batch, columns), generator=gen, device="cuda").to(torch.float16)
    want = single_links(blocks, x, False)
    for _ in range(3):
        assert torch.equal(tq1_matmul(blocks, x, out_dtype=torch.float32), want)


@pytest.mark.parametrize(("rows", "columns"), ((151936, 5120), (60000, 10240)))
def test_two_rows_of_more_than_two_links_have_slots_for(rows, columns):
    from ternel_b200.dispatch import plan
    from ternel_b200.ops import tq1_matmul, tq1_swiglu
    from ternel_b200.stack import random_blocks_device
    assert plan(2, rows, columns).kernel == "stream_gemv"
    gen = torch.Generator(device="cuda")
    gen.manual_seed(rows)
    blocks = random_blocks_device(rows, columns, gen, "cuda")
    x = torch.randn((2, columns), generator=gen, device="cuda").to(torch.float16)
    for call in (tq1_matmul, tq1_swiglu):
        both = call(blocks, x, out_dtype=torch.float32)
        for m in range(2):
            assert torch.equal(both[m:m + 1], call(blocks, x[m:m + 1], out_dtype=torch.float32))


@pytest.mark.parametrize("value", (np.inf, -np.inf, np.nan))
@pytest.mark.parametrize(("rows", "columns"), ((70, 1024), (40, 10240)))
def test_non_finite_groups(rows, columns, value):
    """In the first, in the middle and in the last group, of either activation row."""
    from ternel_b200.ops import tq1_matmul
    host, rng = random_blocks(rows, columns, seed=3)
    blocks = to_dev(host)
    x = rng.standard_normal((2, columns)).astype(np.float16)
    x[0, 5] = x[0, columns // 2 + 130] = x[1, columns - 1] = value
    x = to_dev(x)
    want = single_links(blocks, x, False)
    assert not torch.isfinite(want).all()
    got = tq1_matmul(blocks, x, out_dtype=torch.float32)
    torch.testing.assert_close(got, want, rtol=0, atol=0, equal_nan=True)
    torch.testing.assert_close(tq1_matmul(blocks, x[:1], out_dtype=torch.float32), want[:1], rtol=0, atol=0, equal_nan=True)


def test_calls_that_follow_one_another_and_replays():
    """Back to back on a stream and in a graph, each call reading what the one before wrote."""
    from ternel_b200.ops import tq1_matmul
    host, rng = random_blocks(2560, 2560, seed=9)
    blocks = to_dev(host)
    x = to_dev((rng.standard_normal((1, 2560)) * 0.05).astype(np.float16))

    def chain():
        y = x
        for _ in range(12):
            y = tq1_matmul(blocks, y)
        return y

    want = x
    for _ in range(12):
        want = tq1_matmul(blocks, want)
        torch.cuda.synchronize()
    assert torch.equal(chain(), want)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        y = chain()
    for _ in range(3):
        y.zero_()
        graph.replay()
        assert torch.equal(y, want)
