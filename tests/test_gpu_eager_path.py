"""The eager call path (csrc/torch_binding.cpp) against the dispatcher's: same bytes out, and everything that is
not the plain case declined. Needs a B200."""

import numpy as np
import pytest
import torch

from tests.gpu_util import random_blocks

pytestmark = pytest.mark.gpu


def _setup(rows=48, columns=640, batch=3):
    packed, rng = random_blocks(rows, columns, rows + columns)
    blocks = torch.from_numpy(packed).cuda()
    return blocks, torch.from_numpy(rng.standard_normal((batch, columns)).astype(np.float16)).cuda()


@pytest.mark.parametrize("rows,columns", [(1, 512), (48, 640), (1000, 1536)])
@pytest.mark.parametrize("lead", [(), (1,), (3,), (2, 17)])
@pytest.mark.parametrize("dtype", [torch.float16, torch.float32])
def test_same_bytes_as_the_dispatcher(rows, columns, lead, dtype):
    from ternel_b200.layout import PackedTensorLayout
    from ternel_b200.modules import packed_matmul
    from ternel_b200.ops import eager_embedding, eager_linear, tq1_get_rows
    blocks, _ = _setup(rows, columns)
    x = torch.randn((*lead, columns), device="cuda").half()
    got = packed_matmul(blocks, x, layout=PackedTensorLayout.for_tensor(rows, columns), out_dtype=dtype)
    want = torch.ops.ternel.tq1_linear(blocks, x.reshape(-1, columns), dtype == torch.float32)
    assert got.shape == (*lead, rows) and got.dtype == dtype
    assert torch.equal(got.reshape(-1, rows), want)
    assert torch.equal(eager_linear(blocks, x, dtype, False, False), got)         # the workspace has grown: taken here
    if rows % 2 == 0 and columns % 512 == 0:
        want = torch.ops.ternel.tq1_linear_swiglu(blocks, x.reshape(-1, columns), dtype == torch.float32)
        assert torch.equal(eager_linear(blocks, x, dtype, True, False).reshape(-1, rows // 2), want)
    ids = torch.randint(-1, rows + 1, (*lead, 5), device="cuda")
    assert torch.equal(eager_embedding(blocks, ids, dtype, False).reshape(-1, columns),
                       torch.ops.ternel.tq1_embedding(blocks, ids.reshape(-1), dtype == torch.float32))
    assert tq1_get_rows(blocks, ids.reshape(-1).int(), dtype=dtype).shape == (ids.numel(), columns)


def test_declines_what_is_not_the_plain_case():
    from torch._subclasses.fake_tensor import FakeTensorMode
    from ternel_b200.ops import eager_embedding, eager_linear, tq1_matmul
    blocks, x = _setup()
    tq1_matmul(blocks, x)
    ids = torch.zeros(3, dtype=torch.int64, device="cuda")
    assert eager_linear(blocks, x, None, False, False) is not None
    for b, v, dtype, swiglu, flat in (
            (blocks, x.float(), None, False, False), (blocks, x.cpu(), None, False, False),
            (blocks.cpu(), x, None, False, False), (blocks[:, :, :27], x, None, False, False),
            (blocks[:, 1:], x, None, False, False), (blocks, x[:, 128:], None, False, False),
            (blocks, x[:, ::2], None, False, False), (blocks, x[0], None, False, True), (blocks, x[:0], None, False, False),
            (blocks, x, torch.bfloat16, False, False), (blocks, x, "f16", False, False), (None, x, None, False, False),
            (blocks, x.clone().requires_grad_(), None, False, False), (blocks[:47].contiguous(), x, None, True, False)):
        assert eager_linear(b, v, dtype, swiglu, flat) is None
    for i, flat in ((ids.int(), True), (ids.cpu(), True), (ids[:0], True), (ids[None], True), (ids.float(), True)):
        assert eager_embedding(blocks, i, torch.float16, flat) is None
    assert eager_embedding(blocks, ids, torch.bfloat16, True) is None
    with FakeTensorMode() as mode:
        fake = mode.from_tensor(x)
        assert eager_linear(mode.from_tensor(blocks), fake, None, False, False) is None
        assert tq1_matmul(mode.from_tensor(blocks), fake).shape == (3, 48)


def test_what_a_thread_has_switched_on_is_seen():
    """A trace records the operations and follows its input (a result made outside the dispatcher would be a constant in
    it), a negative view counts as its values, and functionalization goes through."""
    from ternel_b200.ops import eager_embedding, eager_linear, tq1_get_rows, tq1_matmul, tq1_swiglu
    blocks, x = _setup(48, 1024)
    ids = torch.tensor([3, 0, 47], device="cuda")
    other, other_ids = torch.randn_like(x), ids.flip(0) - 1
    tq1_matmul(blocks, x)
    for op, call, first, second in (("tq1_linear", lambda v: tq1_matmul(blocks, v), x, other),
                                    ("tq1_linear_swiglu", lambda v: tq1_swiglu(blocks, v), x, other),
                                    ("tq1_embedding", lambda v: tq1_get_rows(blocks, v), ids, other_ids)):
        traced = torch.jit.trace(call, (first,))
        assert f"ternel::{op}" in str(traced.graph)
        assert torch.equal(traced(second), call(second))
    assert torch.equal(tq1_matmul(blocks, torch._neg_view(x)), tq1_matmul(blocks, -x))
    assert eager_linear(blocks, torch._neg_view(x), None, False, True) is None
    assert torch.equal(torch.func.functionalize(lambda v: tq1_matmul(blocks, v))(x), tq1_matmul(blocks, x))
    assert eager_linear(blocks, x, None, False, True) is not None               # nothing stays switched on
    assert eager_embedding(blocks, ids, torch.float16, True) is not None


def test_torch_functions_are_called():
    """A TorchFunctionMode sees the operation and a subclass gets its own type back, as from any operator; the mode that a
    default device puts up changes nothing."""
    from torch.overrides import TorchFunctionMode
    from ternel_b200.ops import eager_embedding, eager_linear, tq1_get_rows, tq1_matmul
    blocks, x = _setup()
    ids = torch.zeros(3, dtype=torch.int64, device="cuda")
    want = tq1_matmul(blocks, x)

    class Watch(TorchFunctionMode):
        def __init__(self):
            super().__init__()
            self.seen = []

        def __torch_function__(self, func, types, args=(), kwargs=None):
            self.seen.append(str(func))
            return func(*args, **(kwargs or {}))

    class Named(torch.Tensor):
        pass

    with Watch() as watch:
        assert torch.equal(tq1_matmul(blocks, x), want)
        tq1_get_rows(blocks, ids)
    assert any("tq1_linear" in f for f in watch.seen) and any("tq1_embedding" in f for f in watch.seen)
    named = tq1_matmul(blocks, x.as_subclass(Named))
    assert type(named) is Named and torch.equal(named.as_subclass(torch.Tensor), want)
    assert type(tq1_get_rows(blocks.as_subclass(Named), ids)) is Named
    with torch.device("cuda"):
        assert torch.equal(eager_linear(blocks, x, None, False, True), want)
        assert eager_embedding(blocks, ids, torch.float16, True) is not None
        with Watch():
            assert eager_linear(blocks, x, None, False, True) is None
    parameter = torch.nn.Parameter(blocks, requires_grad=False)
    assert torch.equal(eager_linear(parameter, x, None, False, True), want)


def test_a_profiler_sees_the_operations():
    from torch.profiler import ProfilerActivity, profile
    from ternel_b200.ops import eager_linear, tq1_get_rows, tq1_matmul
    blocks, x = _setup()
    tq1_matmul(blocks, x)
    with profile(activities=[ProfilerActivity.CPU]) as record:
        tq1_matmul(blocks, x)
        tq1_get_rows(blocks, torch.zeros(3, dtype=torch.int64, device="cuda"))
    names = {event.key for event in record.key_averages()}
    assert {"ternel::tq1_linear", "ternel::tq1_embedding"} <= names
    assert eager_linear(blocks, x, None, False, True) is not None               # and afterwards the short path again


def test_other_threads_run_while_a_launch_waits():
    """More launches than a stream's queue holds, behind a kernel that keeps the GPU busy for about a second: the launching
    thread waits, and another Python thread has to go on meanwhile (the kernel might wait for what it does)."""
    import threading
    import time
    from ternel_b200.ops import tq1_matmul
    blocks, x = _setup()
    tq1_matmul(blocks, x)
    torch.cuda.synchronize()
    gaps, stop = [], threading.Event()

    def tick():
        last = time.perf_counter()
        while not stop.is_set():
            time.sleep(0.001)
            now = time.perf_counter()
            gaps.append(now - last)
            last = now

    thread = threading.Thread(target=tick)
    thread.start()
    try:
        torch.cuda._sleep(2_000_000_000)                    # about a second
        begin = time.perf_counter()
        for _ in range(3000):
            tq1_matmul(blocks, x)
        waited = time.perf_counter() - begin
    finally:
        stop.set()
        thread.join()
    torch.cuda.synchronize()
    assert waited > 0.5                                     # the queue did fill up
    assert max(gaps) < 0.3, max(gaps)


FIRST_CALLS = """
import threading
import torch
from ternel_b200.ops import tq1_get_rows, tq1_matmul
from ternel_b200.stack import random_blocks_device
gen = torch.Generator(device="cuda")
gen.manual_seed(1)
blocks = random_blocks_device(1024, 1024, gen, "cuda")
xs = [torch.randn((m, 1024), generator=gen, device="cuda").half() for m in (1, 5, 40, 1, 5, 40, 300, 2)]
torch.cuda.synchronize()
start, got = threading.Barrier(len(xs)), [None] * len(xs)

def first(i):
    start.wait()
    got[i] = tq1_matmul(blocks, xs[i])

threads = [threading.Thread(target=first, args=(i,)) for i in range(len(xs))]
for t in threads: t.start()
for t in threads: t.join()
torch.cuda.synchronize()
for x, y in zip(xs, got):
    assert y is not None and torch.equal(y, tq1_matmul(blocks, x))
print("fine")
"""


def test_the_first_calls_may_come_from_several_threads():
    """In a process of its own: whatever is looked up or made once is complete for every thread that finds it there."""
    import subprocess
    import sys
    from pathlib import Path
    for _ in range(3):
        run = subprocess.run([sys.executable, "-c", FIRST_CALLS], capture_output=True, text=True, timeout=300,
                             cwd=Path(__file__).resolve().parents[1])
        assert run.returncode == 0 and "fine" in run.stdout, run.stdout + run.stderr
