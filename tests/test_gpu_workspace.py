"""Scratch buffers of the packed ops on the GPU: what graphs, growth and several streams do to them."""

import subprocess
import sys
from pathlib import Path

import pytest
import torch

pytestmark = pytest.mark.gpu

GRAPH_SCRIPT = """
import torch
from ternel_b200 import ops
from ternel_b200.graphs import GraphedStep
from ternel_b200.stack import random_blocks_device
gen = torch.Generator(device="cuda")
gen.manual_seed(5)
small, large = (random_blocks_device(n, 5120, gen, "cuda") for n in (1024, 17408))
x, other, long = (torch.randn((m, 5120), generator=gen, device="cuda").half() for m in (17, 17, 2048))
step = GraphedStep(lambda v: ops.tq1_matmul(small, v), [x])             # five K parts: partial tiles and counters in use
want = step(other).clone()
first = ops._workspaces[0]
before = first.data_ptr()
del first
ops.tq1_matmul(large, long)                                             # needs more: a larger buffer takes over
assert ops._workspaces[0].data_ptr() != before
junk = [torch.full((1 << 20,), 255, dtype=torch.uint8, device="cuda") for _ in range(96)]    # over anything given back
for _ in range(3):
    assert torch.equal(step(other), want) and torch.equal(step(x), ops.tq1_matmul(small, x))
assert all(bool((j == 255).all()) for j in junk)
ops.check_status()
print("fine")
"""


def test_a_graph_outlives_the_growth_of_the_workspace():
    """A process of its own, because the buffer has to start small."""
    run = subprocess.run([sys.executable, "-c", GRAPH_SCRIPT], capture_output=True, text=True, timeout=300,
                         cwd=Path(__file__).resolve().parents[1])
    assert run.returncode == 0 and "fine" in run.stdout, run.stdout + run.stderr


def test_streams_may_overlap():
    """Products that share tiles between different numbers of K parts, on three streams at once and over and over: every one
    as on the default stream alone, and afterwards the default stream's too."""
    from ternel_b200 import ops
    from ternel_b200.stack import random_blocks_device
    gen = torch.Generator(device="cuda")
    gen.manual_seed(11)
    shapes = ((8, 5120, 17408), (64, 5120, 17408), (3, 1024, 5120), (1, 5120, 5120), (300, 1024, 5120),
              (17, 1024, 5120), (48, 1024, 5120))
    cases = [(random_blocks_device(n, k, gen, "cuda"), torch.randn((m, k), generator=gen, device="cuda").half())
             for m, n, k in shapes]
    want = [ops.tq1_matmul(b, x) for b, x in cases]
    streams = [torch.cuda.Stream() for _ in range(3)]
    torch.cuda.synchronize()
    got = []
    for turn in range(30):
        for s, stream in enumerate(streams):
            with torch.cuda.stream(stream):
                which = (turn + 2 * s) % len(cases)
                got.append((which, ops.tq1_matmul(*cases[which])))
    torch.cuda.synchronize()
    assert all(torch.equal(y, want[which]) for which, y in got)
    for (b, x), y in zip(cases, want):
        assert torch.equal(ops.tq1_matmul(b, x), y)
    ops.check_status()
    assert len(ops._stream_workspaces) <= ops.MAX_STREAM_WORKSPACES
    for _ in range(2 * ops.MAX_STREAM_WORKSPACES):                      # more streams than keep a buffer
        with torch.cuda.stream(torch.cuda.Stream()):
            got = ops.tq1_matmul(*cases[0])
        torch.cuda.synchronize()
        assert torch.equal(got, want[0])
    assert len(ops._stream_workspaces) <= ops.MAX_STREAM_WORKSPACES


def test_counters_that_are_not_zero_are_reported():
    """The counters of shared tiles have to be zero when a call begins. One that is beyond its tile's number of parts (here as
    a stale workspace would leave it) cannot complete the tile: status 8, and good results again after a zero-fill."""
    import ctypes
    from ternel_b200 import _native
    from ternel_b200.dispatch import plan
    from ternel_b200.ops import tq1_matmul
    from ternel_b200.stack import random_blocks_device
    m, n, k = 17, 1024, 5120
    assert plan(m, n, k).kernel == "tensor_core" and plan(m, n, k).parts > 1
    gen = torch.Generator(device="cuda")
    gen.manual_seed(2)
    blocks, x = random_blocks_device(n, k, gen, "cuda"), torch.randn((m, k), generator=gen, device="cuda").half()
    lib = _native.lib()
    need = lib.tq1_linear_workspace_bytes(m, n, k)
    ws = torch.zeros(need, dtype=torch.uint8, device="cuda")
    slots_end = 256 + (16 << 20)
    ws[slots_end - 4096:slots_end + 4096].view(torch.int32).fill_(99)       # the counters, and slots and scratch beside them
    y = torch.zeros((m, n), dtype=torch.float16, device="cuda")

    def call():
        stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
        assert lib.tq1_linear_f16(blocks.data_ptr(), x.data_ptr(), y.data_ptr(), 0, m, n, k, ws.data_ptr(), need, stream) == 0
        return int(ws[:4].view(torch.int32).item())

    assert call() == 8
    ws.zero_()
    assert call() == 0 and torch.equal(y, tq1_matmul(blocks, x))
    assert call() == 0 and torch.equal(y, tq1_matmul(blocks, x))
