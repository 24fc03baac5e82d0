"""Three to sixteen activation rows where the slice kernel takes them, against the oracle."""

import ctypes

import numpy as np
import pytest
import torch

from oracle import tq1_oracle as o
from tests.gpu_util import graph_ms, random_blocks, run_linear, to_dev

pytestmark = pytest.mark.gpu

# Relative error (2-norm): an accumulator of 64 columns truncates four times, on average half of an ulp of 0.72 * 2^-23 of a
# value that grows from zero (1.92 * 2^-24 in all), and up to eight FP32 additions in a row, twice (a slice's accumulators,
# the slices), round by 0.58 * 2^-24 of a sum that grows from zero: 2 * 0.58 * sqrt(8 / 2) * 2^-24.
BOUND = (1.92 + 2 * 0.58 * 2.0) * 2.0 ** -24


@pytest.mark.parametrize("batch", (3, 8, 9, 16))
@pytest.mark.parametrize(("rows", "columns"), (
    (1, 512), (15, 1024), (16, 512), (17, 1536),        # a tile and its edges, one to three slices, eleven sets of warps
    (100, 2560), (4099, 1024), (2400, 5632),            # sets of warps that take turns, eleven slices, rows off the 4-row grid
    (2369, 5120),                                       # a CTA's second tile, the last one of one row
    (48, 6144), (264, 17408), (640, 8704)))             # two and more CTAs in a cluster, K parts that begin inside a chunk
def test_slices_against_float64(rows, columns, batch):
    from ternel_b200.dispatch import plan
    assert plan(batch, rows, columns).form == "slices"
    blocks, rng = random_blocks(rows, columns, seed=rows + columns + batch)
    x = rng.standard_normal((batch, columns)).astype(np.float16)
    want = o.float64_matmul(blocks, x, rows=rows, columns=columns)
    got = run_linear(blocks, x)
    assert np.linalg.norm(got - want) <= BOUND * np.linalg.norm(want)
    assert np.array_equal(run_linear(blocks, x), got)
    half = run_linear(blocks, x, out_dtype=torch.float16)
    assert np.array_equal(half, got.astype(np.float16).astype(np.float32))


@pytest.mark.parametrize(("rows", "columns", "batch"), ((70001, 512, 4), (34810, 2560, 8), (50001, 2048, 3), (70001, 512, 12)))
def test_stages_that_are_filled_again(rows, columns, batch):
    """Several sets of warps whose ring is gone round, by the C ABI's name for this kernel. Whole numbers, so every sum is exact."""
    from ternel_b200 import _native
    from ternel_b200.dispatch import ring_layout
    layout = ring_layout("slices", batch, rows, columns)
    assert layout.sets > 1 and layout.tiles > layout.stages
    rng = np.random.default_rng(rows)
    groups = rows * columns // 128
    trits = rng.integers(0, 3, size=(groups, 128), dtype=np.uint8)
    scales = np.ones(groups, np.float16).view(np.uint8).reshape(-1, 2)
    blocks = to_dev(o.encode_blocks(scales, trits).reshape(rows, columns // 128, 28))
    x = torch.randint(-1, 2, (batch, columns), device="cuda").to(torch.float16)
    want = x.float() @ (to_dev(trits.reshape(rows, columns)).float() - 1).T
    y, ws = torch.empty((batch, rows), dtype=torch.float32, device="cuda"), torch.zeros(1 << 16, dtype=torch.uint8, device="cuda")
    run = _native.lib().tq1_debug_linear_as
    run.restype = ctypes.c_int
    run.argtypes = [ctypes.c_int, *_native.SIGNATURES["tq1_linear_f16"][1][:8], ctypes.c_void_p]
    for _ in range(3):
        assert run(3, blocks.data_ptr(), x.data_ptr(), y.data_ptr(), 1, batch, rows, columns, ws.data_ptr(),
                   torch.cuda.current_stream().cuda_stream) == 0
        assert torch.equal(y, want) and int(ws[:4].view(torch.int32)) == 0


@pytest.mark.parametrize("batch", (3, 16))
@pytest.mark.parametrize("offset", (1, 2, 4))
def test_results_off_the_wide_grid(batch, offset):
    """Results that do not begin on an 8- or 16-byte boundary are stored one by one; the elements around them stay."""
    from ternel_b200 import _native
    from ternel_b200.ops import _workspace
    rows, columns = 100, 1024
    blocks, rng = random_blocks(rows, columns, seed=offset)
    x = rng.standard_normal((batch, columns)).astype(np.float16)
    bd, xd = to_dev(blocks), to_dev(x)
    lib = _native.lib()
    need = lib.tq1_linear_workspace_bytes(batch, rows, columns)
    ws = _workspace(xd.device, need)
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    for dtype in (torch.float16, torch.float32):
        y = torch.full((batch * rows + 2 * offset,), 7.0, dtype=dtype, device="cuda")
        assert lib.tq1_linear_f16(bd.data_ptr(), xd.data_ptr(), y[offset:].data_ptr(), int(dtype == torch.float32), batch, rows,
                                  columns, ws.data_ptr(), need, stream) == 0
        got = y[offset:-offset].float().cpu().numpy().reshape(batch, rows)
        assert np.array_equal(got, run_linear(blocks, x, out_dtype=dtype))
        assert bool((y[:offset] == 7).all()) and bool((y[-offset:] == 7).all())


@pytest.mark.parametrize("batch", (3, 8, 16))
@pytest.mark.parametrize(("half_rows", "columns"), ((9, 512), (1001, 5120), (40, 17408)))
def test_gated_activation(half_rows, columns, batch):
    """silu(gate) * up of row pairs equals the activation applied to the plain products, which add in the same order."""
    from ternel_b200.ops import tq1_matmul, tq1_swiglu
    blocks, rng = random_blocks(2 * half_rows, columns, seed=half_rows)
    both, x = to_dev(blocks), to_dev(rng.standard_normal((batch, columns)).astype(np.float16))
    plain = tq1_matmul(both, x, out_dtype=torch.float32).double()
    want = torch.nn.functional.silu(plain[:, 0::2]) * plain[:, 1::2]
    got = tq1_swiglu(both, x, out_dtype=torch.float32)
    # expf, a division and two products in FP32: a few units in the last place of each value
    assert bool(((got - want).abs() <= 2e-6 * want.abs()).all())


@pytest.mark.parametrize("batch", (8, 16))
def test_counters_of_other_kernels_do_not_matter(batch):
    """The slice kernel adds nothing up in the workspace: counters that another kernel is using, or has left behind, are no
    fault of its results."""
    from ternel_b200 import _native
    rows, columns = 1024, 5120
    blocks, rng = random_blocks(rows, columns, seed=4)
    x = rng.standard_normal((batch, columns)).astype(np.float16)
    bd, xd = to_dev(blocks), to_dev(x)
    lib = _native.lib()
    ws = torch.full((lib.tq1_linear_workspace_bytes(batch, rows, columns),), 99, dtype=torch.uint8, device="cuda")
    ws[:256].zero_()
    y = torch.zeros((batch, rows), dtype=torch.float32, device="cuda")
    assert lib.tq1_linear_f16(bd.data_ptr(), xd.data_ptr(), y.data_ptr(), 1, batch, rows, columns, ws.data_ptr(), ws.numel(),
                              ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)) == 0
    assert int(ws[:4].view(torch.int32).item()) == 0 and bool((ws[256:] == 99).all())
    assert np.array_equal(y.cpu().numpy(), run_linear(blocks, x))


@pytest.mark.parametrize(("batch", "rows", "columns"), (
    (8, 2048, 512), (8, 34816, 512), (16, 17408, 1536), (16, 4096, 4096), (8, 12000, 6144), (8, 1024, 5120)))
def test_the_choice_is_not_the_slower_kernel(batch, rows, columns):
    """In a row of calls and behind another kernel, weights out of HBM: the kernel that is chosen against the tcgen05 kernel."""
    from ternel_b200 import _native
    from ternel_b200.ops import tq1_matmul
    from ternel_b200.stack import random_blocks_device
    gen = torch.Generator(device="cuda")
    gen.manual_seed(3)
    first = random_blocks_device(rows, columns, gen, "cuda")
    weights = [first.clone() for _ in range(min(40, 260_000_000 // first.numel() + 1))]
    x, other = torch.randn((batch, columns), generator=gen, device="cuda").half(), torch.zeros(32, device="cuda")

    def in_a_row(i):
        tq1_matmul(weights[i % len(weights)], x)

    def apart(i):
        other.add_(1)
        tq1_matmul(weights[i % len(weights)], x)

    lib = _native.lib()
    lib.tq1_debug_force_token_tile.argtypes = [ctypes.c_int]
    chosen = [graph_ms(in_a_row), graph_ms(apart)]
    try:
        assert lib.tq1_debug_force_token_tile(16) == 0
        tcgen05 = [graph_ms(in_a_row), graph_ms(apart)]
    finally:
        assert lib.tq1_debug_force_token_tile(0) == 0
    assert all(a <= 1.07 * b for a, b in zip(chosen, tcgen05)), (chosen, tcgen05)


@pytest.mark.parametrize("batch", (3, 16, 17))          # slice kernel, and the tcgen05 kernel, which has the same rule
def test_nonfinite_scales_are_folded_into_the_weights(batch):
    """A weight is -s, 0 or s: an infinite or NaN scale makes infinities and NaN of the products with trits other than zero, and
    with activations of zero; the products with zero trits stay zero."""
    rows, columns = 300, 1024
    blocks, rng = random_blocks(rows, columns, seed=12)
    scales, trits = o.decode_blocks(blocks.reshape(-1, 28))
    values = scales.copy().view(np.float16)[:, 0]
    hit = rng.random(values.shape) < 0.02
    values[hit] = rng.choice(np.array([np.inf, -np.inf, np.nan], dtype=np.float16), hit.sum())
    trits = trits.copy()
    trits[hit] = np.where(rng.random((int(hit.sum()), 128)) < 0.985, 1, trits[hit])       # few products decide: infinities remain
    blocks = o.encode_blocks(values.view(np.uint8).reshape(-1, 2), trits).reshape(rows, columns // 128, 28)
    x = rng.integers(-3, 4, (batch, columns)).astype(np.float16)
    with np.errstate(invalid="ignore", over="ignore"):
        weights = np.where(trits == 1, 0.0, (trits.astype(np.float64) - 1.0) * values.astype(np.float64)[:, None])
        want = x.astype(np.float64) @ weights.reshape(rows, columns).T
    classes = o.nonfinite_classes(want)
    assert len(np.unique(classes)) == 4                 # finite, NaN, and infinities of both signs
    assert np.array_equal(o.nonfinite_classes(run_linear(blocks, x)), classes)
